"""The FP64 Poisson solve against extended precision, on inputs whose low words have a structure."""
from __future__ import annotations

import numpy as np
import pytest

from melt_ibm_gb300 import abi as A
from melt_ibm_gb300.case import Case
from tests.helpers import rel_l2, small_config

pytestmark = pytest.mark.gpu


def _solve(gpu_lib, n, n3, x, stretch=1.0):
    case = Case(small_config(n=n, n3=n3, velocity="rest", imlsfor=0))
    case.zlen *= stretch
    case.dx3 = n3 / case.zlen
    case.interior(A.MIBM_F_DPH)[...] = x
    case.attach(gpu_lib, initial_tag=False)
    gpu_lib.phcalc_()
    gpu_lib.check("phcalc")
    case.sync_to_host(gpu_lib, 1 << A.MIBM_F_DPH)
    out = case.interior(A.MIBM_F_DPH).copy()
    case.detach(gpu_lib)
    return out


def _exact(n, n3, x, stretch=1.0):
    """phcalc.f90:11-97 in extended precision: the eigenvalues by the half-angle formula, the mean set to zero."""
    L = np.longdouble
    length = L(np.float64(2.0 * np.pi))

    def wave(m, size):
        s = np.sin(np.arange(m).astype(L) * (np.arctan(L(1)) * 4 / m))
        d = L(np.float64(m / np.float64(size)))
        return 4 * s * s * (d * d)

    zlen = np.float64(length) * stretch
    lam = (wave(n, length)[:, None, None] + wave(n, length)[None, :, None] + wave(n3, zlen)[None, None, :])
    lam[0, 0, 0] = 1
    spec = np.fft.fftn(x.astype(L))
    assert spec.dtype == np.clongdouble
    spec /= -lam
    spec[0, 0, 0] = 0
    return np.fft.ifftn(spec).real


@pytest.mark.parametrize("n, n3", [(8, 16), (36, 24), (48, 8), (54, 16), (64, 32), (108, 8)])
@pytest.mark.parametrize("kind", ["noise", "single", "integers", "planes", "spike"])
def test_solve_against_extended_precision(gpu_lib, n, n3, kind):
    """Five passes, each rounding its results to FP64 and holding its lines to a few units of 2^-53 of their norm; the
    gradient (what the projection takes from phi) and phi itself carry no more than that: 24 units of 2^-53 in all.
    single: FP32 values; integers and planes: values whose sums have many zero bits at the end."""
    rng = np.random.default_rng(n + n3)
    x = rng.standard_normal((n, n, n3))
    if kind == "single":
        x = x.astype(np.float32).astype(np.float64)
    elif kind == "integers":
        x = np.rint(8 * x)
    elif kind == "planes":
        x = np.broadcast_to(x[:, :1, :1].astype(np.float32).astype(np.float64), x.shape).copy()
    elif kind == "spike":
        x *= 1e-3
        x[n // 2, n // 3, n3 // 2] = 1e3
    got, ref = _solve(gpu_lib, n, n3, x), _exact(n, n3, x)
    assert rel_l2(got, ref) <= 24 * 2.0 ** -53
    for axis in range(3):
        a, b = np.roll(got, 1, axis) - got, np.roll(ref, 1, axis) - ref
        assert np.sqrt(np.sum((a - b) ** 2)) <= 24 * 2.0 ** -53 * np.sqrt(
            sum(np.sum((np.roll(ref, 1, q) - ref) ** 2) for q in range(3)))
