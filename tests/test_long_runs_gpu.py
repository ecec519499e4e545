"""The scatter plan where many faces share a cell: fine meshes on coarse grids, bodies melted to a few cells."""
from __future__ import annotations

import numpy as np
import pytest

from melt_ibm_gb300 import abi as A
from melt_ibm_gb300.case import Case
from tests.helpers import pair, small_config

pytestmark = pytest.mark.gpu
FORCES = (A.MIBM_F_FORXC, A.MIBM_F_FORYC, A.MIBM_F_FORZC, A.MIBM_F_FORTEMP)


@pytest.mark.parametrize("n, level, rad", [(16, 3, 1.0), (16, 4, 0.3), (8, 4, 0.01), (8, 5, 0.4), (8, 5, 1e-3)])
def test_forces_of_many_faces_per_cell(oracle_lib, gpu_lib, n, level, rad):
    """Runs from a dozen to 20480 entries.  Each force is a sum of its run's terms, on the device by lanes and a tree, by
    the oracle in triangle order: at most (len + 5) units of 2^-53 of the sum of the magnitudes apart, of which the
    terms' own roundings (MLS weights of the same bits) take two."""
    case = Case(small_config(n=n, mesh_level=level, rad_p=rad))
    co, cg = pair(case, oracle_lib, gpu_lib, initial_tag=False)
    for c, lib in ((co, oracle_lib), (cg, gpu_lib)):
        c.bind(lib)
        lib.findcentroidindices_()
        lib.mlsweight_()
        lib.mlsforce_()
        lib.check("mlsforce")
    cg.sync_to_host(gpu_lib, sum(1 << f for f in FORCES))
    again = case.clone()                          # slots are given out by atomics: the order must not depend on them
    again.attach(gpu_lib, initial_tag=False)
    for routine in ("findcentroidindices_", "mlsweight_", "mlsforce_"):
        getattr(gpu_lib, routine)()
    again.sync_to_host(gpu_lib, sum(1 << f for f in FORCES))
    faces = case.maxnf
    for f in FORCES:
        a, b = cg.interior(f), co.interior(f)
        assert np.array_equal(a, again.interior(f))
        assert np.array_equal(a == 0.0, b == 0.0)
        assert np.max(np.abs(a - b)) <= (faces + 8) * 2.0 ** -53 * 27 * np.max(np.abs(b)), f
    for c, lib in ((cg, gpu_lib), (again, gpu_lib), (co, oracle_lib)):
        c.detach(lib)
