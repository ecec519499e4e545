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
EPS = 2.0 ** -53


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


def _terms(case):
    """hdnl1-3 and hdnlte (hdnl1.f90, hdnl2.f90, hdnl3.f90, hdnlte.f90) in extended precision, and for each the sum of
    the magnitudes of its products."""
    q = [case.interior(f).astype(np.longdouble) for f in VEL]
    T = case.interior(A.MIBM_F_TEMP).astype(np.longdouble)
    dx = [np.longdouble(case.dx1), np.longdouble(case.dx2), np.longdouble(case.dx3)]
    up, dn = lambda a, d: np.roll(a, -1, d), lambda a, d: np.roll(a, 1, d)
    out = []
    for c in range(3):
        h, m = 0, 0
        for d in range(3):
            if d == c:
                hi, lo = (up(q[c], d) + q[c]) ** 2, (q[c] + dn(q[c], d)) ** 2
            else:
                f = q[d] + dn(q[d], c)                       # the advecting component at this face
                hi, lo = up(f, d) * (up(q[c], d) + q[c]), f * (q[c] + dn(q[c], d))
            h = h - dx[d] / 4 * (hi - lo)
            m = m + dx[d] / 4 * (abs(hi) + abs(lo))
        out.append((h, m))
    h, m = 0, 0
    for d in range(3):
        hi, lo = up(q[d], d) * (up(T, d) + T), q[d] * (T + dn(T, d))
        h, m = h - dx[d] / 2 * (hi - lo), m + dx[d] / 2 * (abs(hi) + abs(lo))
    out.append((h, m))
    return out


@pytest.mark.parametrize("n, n3", [(8, 8), (36, 18), (48, 32), (54, 12)])
@pytest.mark.parametrize("scale", [(1.0, 1.0, 1.0), (1.0, 1e-4, 1e-8), (1e-7, 1.0, 1e-3), (1e-3, 1e-9, 1.0)])
@pytest.mark.parametrize("stretch", [(1.0, 1.0), (1.0, 0.75), (1.25, 0.75)])
def test_terms_to_the_scale_of_their_component(gpu_lib, n, n3, scale, stretch):
    """Blocks in part beyond the grid's end, one, two and three spacings, components of very different size.  FP64
    products and sums of this cell, 8 units of 2^-53 of their magnitudes, and the fixed point's last place: 2^-55 of the
    largest value of the component that is carried times the largest velocity, per spacing."""
    case = _case(n, n3, scale, stretch)
    want = _terms(case)
    before = [case.interior(f).copy() for f in VEL]
    _step(case, gpu_lib)
    for f, b in zip(VEL, before):
        assert np.array_equal(case.interior(f), b)
    top = [np.abs(b).max() for b in before] + [np.abs(case.interior(A.MIBM_F_TEMP)).max()]
    for c, (f, (h, m)) in enumerate(zip(HIST, want)):
        bound = 8 * EPS * m + 2.0 ** -55 * top[c] * max(top[:3]) * (case.dx1 + case.dx2 + case.dx3)
        assert np.all(np.abs(case.interior(f) - h) <= bound), c


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
