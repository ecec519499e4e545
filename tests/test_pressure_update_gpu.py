"""The drop-in pressure update where the largest neighbours of a cell cancel."""
from __future__ import annotations

import numpy as np
import pytest

from melt_ibm_gb300 import abi as A
from melt_ibm_gb300.case import Case
from tests.helpers import set_substep, small_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("small", [1e-12, 1e-6, 1.0])
def test_small_terms_beside_cancelling_ones(gpu_lib, axis, small):
    """phi = 0, 1, 0, -1 along an axis plus small values: at the zeros the two large neighbours cancel and the others
    are left.  Pair sums, products and their sum in FP64: 8 units of 2^-53 of the pair sums and the centre."""
    n = 16
    case = Case(small_config(n=n, velocity="rest", imlsfor=0))
    set_substep(case, 0)
    rng = np.random.default_rng(axis)
    wave = np.array([0.0, 1.0, 0.0, -1.0] * (n // 4)).reshape([n if d == axis else 1 for d in range(3)])
    phi = small * rng.standard_normal((n, n, n)) + wave
    case.interior(A.MIBM_F_DPH)[...] = phi
    case.attach(gpu_lib, initial_tag=False)
    gpu_lib.prcalc_()
    gpu_lib.check("prcalc")
    case.sync_to_host(gpu_lib, 1 << A.MIBM_F_PR)
    got = case.interior(A.MIBM_F_PR).copy()
    case.detach(gpu_lib)
    x = phi.astype(np.longdouble)
    b = np.longdouble(case.S(A.MIBM_S_AL)) * np.longdouble(case.S(A.MIBM_S_BETA)) * np.longdouble(case.dx1) ** 2
    pairs = [np.roll(x, 1, d) + np.roll(x, -1, d) for d in range(3)]
    want = (1 + 6 * b) * x - b * sum(pairs)
    size = (1 + 6 * b) * abs(x) + b * sum(abs(p) for p in pairs)
    assert np.all(abs(got - want) <= 8 * 2.0 ** -53 * size)
