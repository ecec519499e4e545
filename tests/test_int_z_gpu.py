"""The z lines of the FP64 Poisson solve on the integer pipe: every chunk length, few and many chunks, flat and tall boxes."""
from __future__ import annotations

import numpy as np
import pytest

from melt_ibm_gb300 import abi as A
from melt_ibm_gb300.case import Case
from tests.helpers import pair, rel_l2, small_config

pytestmark = pytest.mark.gpu


def _solve(n, n3, stretch, x, oracle_lib, gpu_lib):
    case = Case(small_config(n=n, n3=n3, velocity="rest", imlsfor=0))
    case.zlen *= stretch
    case.dx3 = n3 / case.zlen
    case.interior(A.MIBM_F_DPH)[...] = x
    co, cg = pair(case, oracle_lib, gpu_lib, initial_tag=False)
    for c, lib in ((co, oracle_lib), (cg, gpu_lib)):
        c.bind(lib)
        lib.phcalc_()
        lib.check("phcalc")
    cg.sync_to_host(gpu_lib, 1 << A.MIBM_F_DPH)
    return cg.interior(A.MIBM_F_DPH), co.interior(A.MIBM_F_DPH)


@pytest.mark.parametrize("n, n3, stretch", [
    (8, 8, 1.0), (8, 12, 1.0), (8, 18, 1.0), (8, 36, 1.0), (16, 54, 1.0), (8, 162, 1.0), (8, 256, 1.0),
    (12, 432, 1.0), (8, 486, 1.0), (8, 512, 1.0), (18, 16, 4.0), (16, 48, 0.25), (16, 48, 0.1)])
@pytest.mark.parametrize("kind", ["noise", "spike", "constant"])
def test_z_lines_match_the_oracle(oracle_lib, gpu_lib, n, n3, stretch, kind):
    """Against the oracle's transforms.  The lowest modes dominate: the oracle carries them with an error of about (n/pi)^2
    units of 2^-53, the lines with the square of their growth, G = (n3 / (2 pi stretch))^2; 16 times the larger is
    allowed.  stretch 0.1: a box too flat for the fixed point, solved by the tables."""
    rng = np.random.default_rng(n + n3)
    x = rng.standard_normal((n, n, n3))
    if kind == "spike":
        x *= 1e-3
        x[n // 2, n // 3, n3 // 2] = 1e3
    if kind == "constant":                       # only the zero line: phi depends on z alone
        x[...] = x[:1, :1, :]
    got, ref = _solve(n, n3, stretch, x, oracle_lib, gpu_lib)
    m = max(n, n3)
    assert rel_l2(got, ref) <= 16 * 2.0 ** -53 * max((m / np.pi) ** 2, (n3 / (2 * np.pi * stretch)) ** 2, 8.0)


def test_a_constant_has_no_solution_but_zero(oracle_lib, gpu_lib):
    got, _ = _solve(8, 24, 1.0, np.full((8, 8, 24), 0.1), oracle_lib, gpu_lib)
    assert np.all(got == 0.0)
