"""A batch graph follows its cases' step graphs when a host changes a constant of a case between steps."""
from __future__ import annotations

import numpy as np
import pytest

from melt_ibm_gb300 import abi
from melt_ibm_gb300.batch import BatchRunner
from melt_ibm_gb300.case import Case
from tests.helpers import FIELDS_OUT, small_config

pytestmark = pytest.mark.gpu


def _case(lib, seed, precision):
    c = Case(small_config(n=16, level=2, seed=seed))
    c.attach(lib)
    c.bind(lib)
    lib.mibm_set_precision_(abi.ref_int(precision), abi.ref_int(2))
    lib.check("precision")
    return c


def _change(c, step):
    """Scalars that a step reads by value: each change makes the next step capture its graph again."""
    c.set_S(abi.MIBM_S_LATHEAT, 1.0 + 0.25 * (step % 4))
    c.set_S(abi.MIBM_S_REN, 100.0 + 20.0 * (step % 3))
    c.set_S(abi.MIBM_S_PEC, 100.0 + 20.0 * (step % 3))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("members", [1, 3])
def test_changed_constants_reach_the_batch(gpu_lib, precision, members):
    steps = 14
    want = []
    for q in range(members):
        c = _case(gpu_lib, q + 1, precision)
        for s in range(steps):
            _change(c, s)
            c.step(gpu_lib, s + 1)
        c.sync_to_host(gpu_lib, -1)
        want.append([c.interior(f).copy() for f in FIELDS_OUT.values()] + [c.mesh_arrays[abi.MIBM_M_XYZV].copy()])
        c.detach(gpu_lib)
    cs = [_case(gpu_lib, q + 1, precision) for q in range(members)]
    with BatchRunner(gpu_lib, cs) as b:
        for s in range(steps):
            for c in cs:
                _change(c, s)
            b.step()
    for c, ref in zip(cs, want):
        c.sync_to_host(gpu_lib, -1)
        got = [c.interior(f) for f in FIELDS_OUT.values()] + [c.mesh_arrays[abi.MIBM_M_XYZV]]
        for a, r in zip(got, ref):
            assert np.array_equal(a, r)
        c.detach(gpu_lib)
