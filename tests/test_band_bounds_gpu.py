"""The narrow band's culling bounds where they are weakest: slivers, degenerate faces, centroids off their faces, coarse grids."""
from __future__ import annotations

import numpy as np
import pytest

from melt_ibm_gb300 import abi as A
from melt_ibm_gb300.case import Case
from tests.helpers import pair, small_config

pytestmark = pytest.mark.gpu
FIELDS = (A.MIBM_F_VOFP, A.MIBM_F_VOFX, A.MIBM_F_VOFY, A.MIBM_F_VOFZ, A.MIBM_F_SDF)


@pytest.mark.parametrize("n, level", [(8, 1), (32, 3), (48, 2)])
@pytest.mark.parametrize("kind", ["plain", "sliver", "point", "shifted"])
def test_band_matches_the_oracle(oracle_lib, gpu_lib, n, level, kind):
    """Culling leaves the minimum distance and the first face at it: the distances come from the same operations."""
    case = Case(small_config(n=n, mesh_level=level, velocity="rest"))
    x, bar = case.mesh_arrays[A.MIBM_M_XYZV], case.mesh_arrays[A.MIBM_M_TRI_BAR]
    tri = case.mesh_arrays[A.MIBM_M_VERT_OF_FACE] - 1
    for f in range(0, tri.shape[1], 9):
        a, b, c = tri[:, f]
        if kind == "sliver":                         # the vertex almost on the opposite edge
            x[:, a] = 0.3 * x[:, b] + 0.7 * x[:, c] + 1e-7 * (x[:, a] - x[:, b])
        elif kind == "point":
            x[:, a] = x[:, b]
    bar[...] = (x[:, tri[0]] + x[:, tri[1]] + x[:, tri[2]]) / 3.0
    if kind == "shifted":
        bar += 0.02 * np.random.default_rng(n).standard_normal(bar.shape)
    co, cg = pair(case, oracle_lib, gpu_lib, initial_tag=False)
    for c, lib in ((co, oracle_lib), (cg, gpu_lib)):
        c.bind(lib)
        lib.tagcells_()
        lib.check("tagcells")
    cg.sync_to_host(gpu_lib, sum(1 << f for f in FIELDS))
    for f in FIELDS:
        assert np.max(np.abs(cg.interior(f) - co.interior(f))) <= 1e-12, f
