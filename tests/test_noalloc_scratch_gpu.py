"""Which lines mibm_solxi_noalloc solves without the shared factor table: a captured call is then one kernel."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from melt_ibm_gb300 import abi as A
from melt_ibm_gb300.case import Case
from tests.helpers import small_config

pytestmark = pytest.mark.gpu
LENGTHS = sorted(2 ** a * 3 ** b for a in range(1, 10) for b in range(6) if 2 ** a * 3 ** b <= 512)


def _kernels(gpu_lib, torch, n, pitch, beta):
    """Nodes of a captured call: the solve, and the table's kernel where there is one."""
    buf = torch.randn(3 * 2 * pitch, dtype=torch.float64, device="cuda")
    stream = torch.cuda.Stream()
    call = lambda: gpu_lib.mibm_solxi_noalloc(C.c_void_p(buf.data_ptr()), n, 3, 2, pitch, beta,
                                              C.c_void_p(stream.cuda_stream))
    assert call() == A.MIBM_OK
    torch.cuda.synchronize()
    graph, cuda = torch.cuda.CUDAGraph(keep_graph=True), C.CDLL("libcuda.so.1")
    with torch.cuda.graph(graph, stream=stream):
        assert call() == A.MIBM_OK
    count = C.c_size_t(0)
    assert cuda.cuGraphGetNodes(C.c_void_p(graph.raw_cuda_graph()), None, C.byref(count)) == 0
    return count.value


def test_even_lengths_need_no_table(gpu_lib):
    torch = pytest.importorskip("torch")
    assert 486 in LENGTHS and len(LENGTHS) > 25
    for n in LENGTHS:
        assert _kernels(gpu_lib, torch, n, n + n % 2, 0.05) == 1, n
    assert _kernels(gpu_lib, torch, 96, 97, 0.05) == 2           # rows off the 16-byte boundaries
    assert _kernels(gpu_lib, torch, 100, 100, 0.05) == 1         # 25 chunks of 4
    assert _kernels(gpu_lib, torch, 97, 98, 0.05) == 2


@pytest.mark.parametrize("betadx", [-0.1, 1e-3, 0.37, 40.0])
def test_longest_odd_power_of_three(gpu_lib, betadx):
    """solxi_ on 486 cells against the eigenvalues of the periodic system: backward stable, 64 units of 2^-53 times its
    condition number."""
    n, n3 = 486, 8
    case = Case(small_config(n=n, n3=n3, velocity="rest", imlsfor=0))
    r = np.random.default_rng(1).standard_normal((n, n, n3))
    case.interior(A.MIBM_F_RHS)[...] = r
    case.attach(gpu_lib, initial_tag=False)
    gpu_lib.solxi_(C.byref(C.c_double(betadx)))
    gpu_lib.check("solxi")
    case.sync_to_host(gpu_lib, 1 << A.MIBM_F_RHS)
    lam = 1.0 + 2.0 * betadx * (1.0 - np.cos(2.0 * np.pi * np.arange(n) / n))
    ref = np.fft.ifft(np.fft.fft(r, axis=0) / lam[:, None, None], axis=0).real
    err = np.linalg.norm(case.interior(A.MIBM_F_RHS) - ref)
    case.detach(gpu_lib)
    assert err <= 64 * 2.0 ** -53 * np.abs(lam).max() / np.abs(lam).min() * np.linalg.norm(ref)
