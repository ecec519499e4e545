"""The literal heat flux in its two splits of the work (up to 4096 faces, and more) against the oracle, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from melt_ibm_gb300 import abi as A
from melt_ibm_gb300.case import Case
from tests.helpers import pair, small_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level, ghosts", [(1, 0), (2, 7), (3, 0), (4, 0)])
def test_heat_flux_has_the_oracles_bits(oracle_lib, gpu_lib, level, ghosts):
    """80 to 5120 faces (40 probes to 10240, the last block part empty for 80), some of them ghosts; the same
    operations in the same order on both sides, so equal bits."""
    case = Case(small_config(n=32, mesh_level=level, velocity="rest"))
    rng = np.random.default_rng(level)
    case.interior(A.MIBM_F_TEMP)[...] += 0.1 * rng.standard_normal((32, 32, 32))
    case.fill_ghosts(A.MIBM_F_TEMP)
    if ghosts:
        case.mesh_arrays[A.MIBM_M_GHOST_FACE][::ghosts] = 1
    co, cg = pair(case, oracle_lib, gpu_lib, initial_tag=False)
    for c, lib in ((co, oracle_lib), (cg, gpu_lib)):
        c.bind(lib)
        lib.findprobeindices_()
        lib.mls_heatflux_()
        lib.check("heat flux")
    cg.sync_to_host(gpu_lib, -1)
    for m in (A.MIBM_M_QW_O, A.MIBM_M_QW_I):
        assert np.array_equal(cg.mesh_arrays[m], co.mesh_arrays[m])
