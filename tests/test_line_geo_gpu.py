"""Edges of the FP64 line solves on the factored circulant form.

Lines of one chunk (8 cells), of odd numbers of chunks (18, 54), the longest
line (512) and a length without a chunk (486: tile kernels); a negative
off-diagonal weight, weights whose powers die out within a chunk, and ones
for which every chunk of the line contributes to an entry value.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from melt_ibm_gb300 import abi as A
from melt_ibm_gb300.case import Case
from tests.helpers import pair, rel_l2, small_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, n3", [(8, 512), (18, 54), (54, 8), (24, 486), (48, 36)])
@pytest.mark.parametrize("betadx", [-0.1, 1e-6, 0.03, 2.0, 3e3])
def test_line_solves_match_oracle(oracle_lib, gpu_lib, n, n3, betadx):
    """solxi_, solxj_, solxk_ against the oracle's Thomas sweep.  Both sides are backward stable to a few units of
    2^-53, so they agree to the condition number of the system, (1 + 4 beta) / min(1, 1 + 4 beta), times that:
    64 units allowed for three directions of up to 512 cells."""
    case = Case(small_config(n=n, n3=n3, velocity="rest", imlsfor=0))
    rng = np.random.default_rng(n * n3)
    case.fields[A.MIBM_F_RHS][...] = rng.standard_normal(case.fields[A.MIBM_F_RHS].shape)
    case.fields[A.MIBM_F_VX][...] = rng.standard_normal(case.fields[A.MIBM_F_VX].shape)
    co, cg = pair(case, oracle_lib, gpu_lib, initial_tag=False)
    for c, lib in ((co, oracle_lib), (cg, gpu_lib)):
        c.bind(lib)
        bd = C.byref(C.c_double(betadx))
        vx = c.fields[A.MIBM_F_VX]
        lib.solxi_(bd)
        lib.solxj_(bd)
        lib.solxk_(C.c_void_p(vx.ctypes.data + vx.shape[0] * vx.shape[1] * 8), bd)
        lib.check("line solves")
    cg.sync_to_host(gpu_lib, -1)
    tol = 64 * 2.0 ** -53 * max(1 + 4 * betadx, 1 / (1 + 4 * betadx), 1.0)
    for fid in (A.MIBM_F_RHS, A.MIBM_F_VX):
        assert rel_l2(cg.interior(fid), co.interior(fid)) <= tol
