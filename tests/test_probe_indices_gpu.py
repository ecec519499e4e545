"""The registered cage indices after a step that does not run ahead into the next substep's geometry work."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from melt_ibm_gb300 import abi as A
from melt_ibm_gb300.case import Case
from tests.helpers import CoarseningRemesher, pair, small_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("why", ["profiled", "remesher"])
@pytest.mark.parametrize("precision", [0, 1])
def test_step_leaves_the_probes(oracle_lib, gpu_lib, why, precision):
    """particle.f90 leaves the probes' cells in pind; so does a step whose kernels are timed one by one, or one that may stop
    for the host's remesher (here never: no edge is below a threshold of zero)."""
    case = Case(small_config(n=24, mesh_level=2, seed=1, iremesh=int(why == "remesher"), perc_ethresh=0.0))
    co, cg = pair(case, oracle_lib, gpu_lib)
    remeshers = []
    for c, lib in ((co, oracle_lib), (cg, gpu_lib)):
        c.bind(lib)
        if why == "remesher":
            remeshers.append(CoarseningRemesher(c, 1))
            remeshers[-1].install(lib)
    gpu_lib.mibm_set_precision_(C.byref(C.c_int(precision)), C.byref(C.c_int(2)))
    if why == "profiled":
        gpu_lib.mibm_profile_(C.byref(C.c_int(1)))
    for c, lib in ((co, oracle_lib), (cg, gpu_lib)):
        c.step(lib, 1)
    if why == "profiled":
        gpu_lib.mibm_profile_(C.byref(C.c_int(0)))
    assert all(r.calls == 0 for r in remeshers)
    cg.sync_to_host(gpu_lib, -1)
    assert np.array_equal(cg.mesh_arrays[A.MIBM_M_PIND], co.mesh_arrays[A.MIBM_M_PIND])
    cg.detach(gpu_lib)
    co.detach(oracle_lib)
