"""Mean force removal and forcing updates: dense, sparse and empty forces, rows off the warp width, more rows than blocks."""
from __future__ import annotations

import numpy as np
import pytest

from melt_ibm_gb300 import abi as A
from melt_ibm_gb300.case import Case
from tests.helpers import small_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, n3", [(8, 8), (18, 24), (36, 8), (64, 32)])
@pytest.mark.parametrize("share", [0.0, 0.01, 1.0])
def test_forces_are_added_and_their_mean_removed(gpu_lib, n, n3, share):
    """Against extended precision: a few roundings of the operands per cell, and 64 units of 2^-53 of the mean
    magnitude for the sum (at most 13 additions per lane and 23 levels of trees)."""
    case = Case(small_config(n=n, n3=n3, mesh_level=1, velocity="rest"))
    rng = np.random.default_rng(n)
    vel, force = (A.MIBM_F_VX, A.MIBM_F_VY, A.MIBM_F_VZ), (A.MIBM_F_FORXC, A.MIBM_F_FORYC, A.MIBM_F_FORZC)
    for f in vel + force + (A.MIBM_F_TEMP, A.MIBM_F_FORTEMP):
        case.interior(f)[...] = rng.standard_normal((n, n, n3)) * (1.0 if f in vel else rng.random((n, n, n3)) < share)
    before = {f: case.interior(f).astype(np.longdouble) for f in vel + force + (A.MIBM_F_TEMP, A.MIBM_F_FORTEMP)}
    case.attach(gpu_lib, initial_tag=False)
    case.bind(gpu_lib)
    gpu_lib.velforce_()
    gpu_lib.tempforce_()
    gpu_lib.check("forcing")
    case.sync_to_host(gpu_lib, sum(1 << f for f in vel + (A.MIBM_F_TEMP,)))
    eps = 2.0 ** -53
    for v, f in zip(vel, force):
        mean, size = before[f].mean(), np.abs(before[f]).mean()
        want = before[v] + before[f] - mean
        bound = 4 * eps * (np.abs(before[v]) + np.abs(before[f]) + abs(mean)) + 64 * eps * size
        assert np.all(np.abs(case.interior(v) - want) <= bound)
    assert np.array_equal(case.interior(A.MIBM_F_TEMP),
                          (before[A.MIBM_F_TEMP] + before[A.MIBM_F_FORTEMP]).astype(np.float64))
    case.detach(gpu_lib)
