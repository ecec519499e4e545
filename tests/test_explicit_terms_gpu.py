"""The FP64 step's explicit terms, read back from the RK history after a step of vanishing length."""
from __future__ import annotations

import numpy as np
import pytest

from melt_ibm_gb300 import abi as A
from melt_ibm_gb300.case import Case
from tests.helpers import small_config

pytestmark = pytest.mark.gpu
VEL = (A.MIBM_F_VX, A.MIBM_F_VY, A.MIBM_F_VZ)
HIST = (A.MIBM_F_RU1, A.MIBM_F_RU2, A.MIBM_F_RU3, A.MIBM_F_RUT)


def _case(n, n3, scale, stretch, seed=0):
    """u(y, z), v(x, z), w(x, y): divergence-free to the last bit, so that a step of length 1e-30 leaves the
    velocity as it is and its history holds the explicit terms of exactly this flow."""
    case = Case(small_config(n=n, n3=n3, velocity="rest", imlsfor=0))
    case.ylen *= stretch[0]
    case.zlen *= stretch[1]
    case.dx2, case.dx3 = n / case.ylen, n3 / case.zlen
    rng = np.random.default_rng(seed)
    case.interior(VEL[0])[...] = scale[0] * (0.3 + rng.standard_normal((1, n, n3)))
    case.interior(VEL[1])[...] = scale[1] * rng.standard_normal((n, 1, n3))
    case.interior(VEL[2])[...] = scale[2] * rng.standard_normal((n, n, 1))
    case.interior(A.MIBM_F_TEMP)[...] = rng.standard_normal((n, n, n3))
    for f in VEL + (A.MIBM_F_TEMP,):
        case.fill_ghosts(f)
    case.set_S(A.MIBM_S_DT, 1e-30)
    return case


def _step(case, lib):
    case.attach(lib, initial_tag=False)
    lib.tschem_()
    lib.check("tschem")
    case.sync_to_host(lib, sum(1 << f for f in VEL + HIST + (A.MIBM_F_TEMP, A.MIBM_F_PR)))
    case.detach(lib)


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_bad_temperature_leaves_the_velocity(gpu_lib, bad):
    """Without buoyancy nothing of T reaches u, v, w or p: they have the bits of the step with a finite T."""
    good, spoilt = _case(24, 16, (1.0, 1.0, 1.0), (1.0, 1.0), 3), _case(24, 16, (1.0, 1.0, 1.0), (1.0, 1.0), 3)
    for c in (good, spoilt):
        c.set_S(A.MIBM_S_DT, 1e-3)
    spoilt.interior(A.MIBM_F_TEMP)[5, 7, 9] = bad
    for c in (good, spoilt):
        _step(c, gpu_lib)
    for f in VEL + HIST[:3] + (A.MIBM_F_PR,):
        assert np.array_equal(spoilt.interior(f), good.interior(f)), f
    assert not np.isfinite(spoilt.interior(A.MIBM_F_TEMP)).any()
