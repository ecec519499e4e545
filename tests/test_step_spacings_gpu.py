"""Whole FP64 steps on boxes with one, two and three spacings and on grids that do not fill the kernels' tiles."""
from __future__ import annotations

import numpy as np
import pytest

from melt_ibm_gb300 import abi as A
from melt_ibm_gb300.case import Case
from tests.helpers import FIELDS_OUT, pair, rel_l2, small_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, n3", [(24, 16), (36, 54)])
@pytest.mark.parametrize("stretch", [(1.0, None), (1.0, 0.8), (1.25, 0.8)])
@pytest.mark.parametrize("body", ["none", "melt"])
def test_steps_match_the_oracle(oracle_lib, gpu_lib, n, n3, stretch, body):
    """Three steps with buoyancy and ABC forcing from a random flow; stretch None: as many cells per length as in x.  The
    bound of the whole-step tests, 1e-10."""
    case = Case(small_config(n=n, n3=n3, mesh_level=2, velocity="rest", imlsfor=int(body != "none"),
                             imelt=int(body != "none"), betagz=0.3, forcing=1, which_hit=2, dt=1e-3, dtmax=1e-3))
    case.ylen *= stretch[0]
    case.zlen *= n3 / n if stretch[1] is None else stretch[1]
    case._grid()
    case._params()
    case._geometry()
    case._initial_condition()
    rng = np.random.default_rng(n)
    for f in (A.MIBM_F_VX, A.MIBM_F_VY, A.MIBM_F_VZ):
        case.interior(f)[...] = rng.standard_normal((n, n, n3))
        case.fill_ghosts(f)
    co, cg = pair(case, oracle_lib, gpu_lib)
    for c, lib in ((co, oracle_lib), (cg, gpu_lib)):
        c.run(lib, 3)
    cg.sync_to_host(gpu_lib, -1)
    for name, f in FIELDS_OUT.items():
        assert rel_l2(cg.interior(f), co.interior(f)) <= 1e-10, name
    cg.detach(gpu_lib)
    co.detach(oracle_lib)
