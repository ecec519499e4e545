"""The FP64 Poisson solve with its x and y transforms on the integer pipe.

Line lengths at the edges of the radix plans (a single stage of every radix,
odd numbers of radix-3 stages, the shortest and longest lines), and inputs at
the edges of the block exponent: a single spike, fields near the ends of the
FP64 range, zeros, infinities and NaN.
"""
from __future__ import annotations

import numpy as np
import pytest

from melt_ibm_gb300 import abi as A
from melt_ibm_gb300.case import Case
from tests.helpers import pair, rel_l2, small_config

pytestmark = pytest.mark.gpu


def _solve(case, oracle_lib, gpu_lib):
    co, cg = pair(case, oracle_lib, gpu_lib, initial_tag=False)
    for c, lib in ((co, oracle_lib), (cg, gpu_lib)):
        c.bind(lib)
        lib.phcalc_()
        lib.check("phcalc")
    cg.sync_to_host(gpu_lib, 1 << A.MIBM_F_DPH)
    return cg.interior(A.MIBM_F_DPH), co.interior(A.MIBM_F_DPH)


def _case(n, n3, x):
    case = Case(small_config(n=n, n3=n3, velocity="rest", imlsfor=0))
    case.interior(A.MIBM_F_DPH)[...] = x
    return case


@pytest.mark.parametrize("n, n3", [(8, 16), (12, 8), (18, 24), (36, 8), (54, 16), (108, 8), (162, 8), (486, 8), (512, 8)])
@pytest.mark.parametrize("kind", ["noise", "spike"])
def test_poisson_solve_matches_oracle(oracle_lib, gpu_lib, n, n3, kind):
    """Against the oracle's transforms.  The solution is dominated by the lowest modes, which the z lines (or the
    oracle's z transform) carry with an error of about (n/pi)^2 units of 2^-53; 16 times that is allowed."""
    rng = np.random.default_rng(n + n3)
    x = rng.standard_normal((n, n, n3))
    if kind == "spike":
        x *= 1e-3
        x[n // 2, n // 3, n3 // 2] = 1e3
    got, ref = _solve(_case(n, n3, x), oracle_lib, gpu_lib)
    m = max(n, n3)
    assert rel_l2(got, ref) <= 16 * 2.0 ** -53 * max((m / np.pi) ** 2, 8.0)


@pytest.mark.parametrize("scale", [2.0 ** -960, 2.0 ** 960])
def test_scaled_by_a_power_of_two(oracle_lib, gpu_lib, scale):
    """The block exponent carries the scale: the solution scales exactly."""
    x = np.random.default_rng(1).standard_normal((24, 24, 16))
    a, _ = _solve(_case(24, 16, x), oracle_lib, gpu_lib)
    a = a.copy()
    b, _ = _solve(_case(24, 16, x * scale), oracle_lib, gpu_lib)
    assert np.array_equal(a * scale, b)


def test_zeros_and_non_finite(oracle_lib, gpu_lib):
    x = np.zeros((16, 16, 16))
    got, _ = _solve(_case(16, 16, x), oracle_lib, gpu_lib)
    assert np.all(got == 0.0)
    for bad in (np.nan, np.inf):
        y = np.random.default_rng(2).standard_normal((16, 16, 16))
        y[3, 4, 5] = bad
        got, _ = _solve(_case(16, 16, y), oracle_lib, gpu_lib)
        assert not np.isfinite(got).any()
