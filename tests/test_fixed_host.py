"""The twiddle product of the integer-pipe transforms (melt_ibm_gb300/csrc/fixed.cuh) and the guarded sum of six
(fpconv.cuh), built for the host by g++ from the source the kernels use and checked against exact arithmetic."""
from __future__ import annotations

import ctypes as C
import math
import random
import shutil
import subprocess
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    out = tmp_path_factory.mktemp("fixed") / "libfixed_host.so"
    subprocess.run([gxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-I", str(ROOT / "melt_ibm_gb300" / "csrc"),
                    str(ROOT / "tests" / "fixed_host.cpp"), "-o", str(out)], check=True)
    return C.CDLL(str(out))


def _values():
    """Components below 2^60.5 in magnitude whose low word is one of the edges of a signed half, or any."""
    rnd = random.Random(5)
    low = [0x80000000, 0x80000001, 0x7fffffff, 0, 1, 0xffffffff]
    comp = lambda: (rnd.randrange(-(1 << 28), 1 << 28) << 32) | (rnd.choice(low) if rnd.random() < 0.7 else rnd.getrandbits(32))
    v = [(comp(), comp()) for _ in range(4000)]
    v += [(-(1 << 31), 1 << 31), (1 << 31, -(1 << 31)), (0, 1 << 31), (0, -(1 << 31)), (1 << 31, 0)]
    return v


@pytest.mark.parametrize("shift", [1, 2])
@pytest.mark.parametrize("inverse", [0, 1])
def test_product_is_within_its_bound(lib, shift, inverse):
    """Half a unit of rounding, and two products of low halves left out per component: each below 2^62 / 2^(62 + shift)."""
    v = _values()
    rnd = random.Random(6)
    w = []
    for _ in v:
        a = 2 * math.pi * rnd.random()
        c, s = (int(Fraction(f(a)) * (1 << 62)) for f in (math.cos, lambda x: -math.sin(x)))
        if rnd.random() < 0.3:                          # a factor whose low half is the most negative one
            c, s = (c >> 32 << 32) + (1 << 31), (s >> 32 << 32) + (1 << 31)
        w.append((c, s))
    halves = lambda x: ((x - ((x + (1 << 31)) % (1 << 32) - (1 << 31))) >> 32, (x + (1 << 31)) % (1 << 32) - (1 << 31))
    vin = np.array(v, dtype=np.int64)
    win = np.array([halves(c) + halves(s) for c, s in w], dtype=np.int32)
    out = np.empty_like(vin)
    lib.fixed_twiddle(shift, inverse, C.c_longlong(len(v)), C.c_void_p(vin.ctypes.data), C.c_void_p(win.ctypes.data),
                      C.c_void_p(out.ctypes.data))
    bound = Fraction(1, 2) + 2 * Fraction(1, 1 << shift)
    for (x, y), (c, s), got in zip(v, w, out.tolist()):
        s = -s if inverse else s
        for g, exact in zip(got, (x * c - y * s, y * c + x * s)):
            assert abs(g - Fraction(exact, 1 << (62 + shift))) <= bound, (x, y, c, s)


def test_guarded_sum_is_taken_only_where_it_is_good(lib):
    """Six cuts of less than a unit of a sum of 2^57 units at least (0.4 of 2^-53) and one rounding: within 1.5 times 2^-53 of
    the sum wherever one is given; given wherever the sum is a quarter of the largest."""
    rnd = random.Random(8)
    rows = []
    for _ in range(6000):
        spread = rnd.choice([0, 1, 8, 40, 200])
        row = [rnd.gauss(0, 1) * 2.0 ** rnd.uniform(-spread, 0) for _ in range(6)]
        if rnd.random() < 0.3:
            row[1] = -row[0] * (1 + rnd.choice([0.0, 2.0 ** -52, 1e-3, 0.3]))
        scale = rnd.choice([1.0, 2.0 ** 900, 2.0 ** -900])
        rows.append([v * scale for v in row])
    rows += [[math.inf, 1, 1, 1, 1, 1], [math.nan, 1, 1, 1, 1, 1], [1e308] * 6, [0.0] * 6, [-0.0] * 6, [5e-324] * 6,
             [2.0 ** -1000] * 6, [1, -1, 1e-12, 2e-12, 0, 0], [-1.0, 0, 0, 0, 0, 0], [1.0] * 6]
    x = np.array(rows)
    out, ok = np.empty(len(rows)), np.empty(len(rows), dtype=np.int32)
    lib.guarded_sum6(C.c_longlong(len(rows)), C.c_void_p(x.ctypes.data), C.c_void_p(out.ctypes.data),
                     C.c_void_p(ok.ctypes.data))
    taken = 0
    for row, got, given in zip(rows, out.tolist(), ok.tolist()):
        if not all(map(math.isfinite, row)):
            assert not given
            continue
        exact, top = sum(map(Fraction, row)), max(abs(Fraction(v)) for v in row)
        if given:
            taken += 1
            if math.isinf(got):
                assert abs(exact) >= Fraction(2) ** 1024 - Fraction(2) ** 970
            else:
                assert abs(Fraction(got) - exact) <= Fraction(3, 2) * abs(exact) / (1 << 53), row
        else:
            assert abs(exact) < top / 4 or top < Fraction(2) ** -950, row
    assert taken > 3000
