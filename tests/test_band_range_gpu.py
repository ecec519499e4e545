"""The narrow band in boxes of every size: culling must not lose a nearest face where FP32 coordinates are coarse."""
from __future__ import annotations

import numpy as np
import pytest

from melt_ibm_gb300 import abi as A
from melt_ibm_gb300.case import Case
from tests.helpers import pair, small_config

pytestmark = pytest.mark.gpu
FIELDS = (A.MIBM_F_VOFP, A.MIBM_F_VOFX, A.MIBM_F_VOFY, A.MIBM_F_VOFZ)


@pytest.mark.parametrize("length, rad", [(1e-3, 1e-5), (2 * np.pi, 0.3), (100.0, 1.0), (400.0, 1.0), (1e3, 1.0), (1e4, 3.0)])
@pytest.mark.parametrize("seed", range(6))
def test_band_matches_the_oracle_in_any_box(oracle_lib, gpu_lib, length, rad, seed):
    """A body within 1e-7 of the box's size of a cell's centre, whose faces are then almost equally far away: the
    distances come from the same operations on both sides, so they agree to rounding."""
    n, h = 16, length / 16
    rng = np.random.default_rng(seed)
    case = Case(small_config(n=n, mesh_level=3, velocity="rest", length=length, rad_p=rad))
    x = case.mesh_arrays[A.MIBM_M_XYZV]
    x += (0.5 * h + 3e-8 * length * rng.standard_normal(3))[:, None]
    case._geometry_refresh()
    co, cg = pair(case, oracle_lib, gpu_lib, initial_tag=False)
    for c, lib in ((co, oracle_lib), (cg, gpu_lib)):
        c.bind(lib)
        lib.tagcells_()
        lib.check("tagcells")
    cg.sync_to_host(gpu_lib, sum(1 << f for f in FIELDS + (A.MIBM_F_SDF,)))
    a, b = cg.interior(A.MIBM_F_SDF), co.interior(A.MIBM_F_SDF)
    assert np.array_equal(a == 999.0, b == 999.0)
    assert np.max(np.abs(a - b)) <= 1e-13 * length
    for f in FIELDS:
        assert np.max(np.abs(cg.interior(f) - co.interior(f))) <= 1e-9, f
    cg.detach(gpu_lib)
    co.detach(oracle_lib)
