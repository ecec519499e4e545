"""A batch whose members change at every step: a case's steps keep their bits and their launches."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from melt_ibm_gb300 import abi
from melt_ibm_gb300.case import Case
from tests.helpers import FIELDS_OUT, small_config

pytestmark = pytest.mark.gpu
SIZES = [16, 16, 24, 16, 16, 16, 16, 16, 16, 48]


def _attached(lib, precision):
    out = []
    for q, n in enumerate(SIZES):
        c = Case(small_config(n=n, level=2, seed=q + 1))
        c.attach(lib)
        c.bind(lib)
        lib.mibm_set_precision_(abi.ref_int(precision), abi.ref_int(2))
        lib.check("precision")
        out.append(c)
    return out


def _state(c, lib):
    c.sync_to_host(lib, -1)
    return [c.interior(f).copy() for f in FIELDS_OUT.values()] + [c.mesh_arrays[abi.MIBM_M_XYZV].copy(), c.S(abi.MIBM_S_DT)]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("launch", [0, 1])
def test_membership_changes_neither_bits_nor_launches(gpu_lib, precision, launch):
    """Few members, many, and a large one among them, in turn, with tschem_ between: the step graph's form follows the
    company, and each form is captured once.  A form that dropped the other's graph or the geometry work done ahead would
    launch that work again."""
    alone = _attached(gpu_lib, precision)
    for c in alone:
        c.run(gpu_lib, 13)
    want = [_state(c, gpu_lib) for c in alone]
    for c in alone:
        c.detach(gpu_lib)
    cs = _attached(gpu_lib, precision)
    ids = np.array([c.ctx[gpu_lib.path] for c in cs], dtype=np.int32)
    few, many, all_ = list(range(3)), list(range(9)), list(range(10))
    plan = [many, many, many, few, many, few, all_, few, few, many, "alone", many]
    done, per_step = [0] * len(cs), []
    handle = int(gpu_lib.mibm_batch_create_(ids.ctypes.data, abi.ref_int(len(ids))))
    assert gpu_lib.mibm_batch_set_launch_(abi.ref_int(handle), abi.ref_int(launch)) == 0
    members = set(all_)
    for step, who in enumerate(plan):
        cs[0].bind(gpu_lib)
        before = gpu_lib.mibm_launch_count_()
        if who == "alone":
            cs[0].step(gpu_lib, done[0] + 1)
            done[0] += 1
        else:
            for q in members - set(who):
                gpu_lib.mibm_batch_remove_(abi.ref_int(handle), abi.ref_int(int(ids[q])))
            for q in set(who) - members:
                assert gpu_lib.mibm_batch_add_(abi.ref_int(handle), abi.ref_int(int(ids[q]))) == 0
            members = set(who)
            assert gpu_lib.mibm_batch_step_(abi.ref_int(handle), abi.ref_int(0)) == 0
            for q in who:
                done[q] += 1
        cs[0].bind(gpu_lib)
        per_step.append(gpu_lib.mibm_launch_count_() - before)
    gpu_lib.mibm_batch_destroy_(abi.ref_int(handle))
    # from the third step on the geometry work of a step's start is always already there (no change of members before it)
    assert len(set(per_step[2:])) == 1, per_step
    for q, c in enumerate(cs):
        for nt in range(done[q] + 1, 14):
            c.step(gpu_lib, nt)
        for got, ref in zip(_state(c, gpu_lib), want[q]):
            assert np.array_equal(got, ref), q
        c.detach(gpu_lib)
