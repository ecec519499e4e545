"""mibm_solxi_noalloc on lines of two cells in rows of every pitch."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from melt_ibm_gb300 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pitch", [2, 3, 4, 6, 32])
@pytest.mark.parametrize("n2, n3", [(1, 1), (3, 2), (200, 3)])
def test_lines_of_two_cells(gpu_lib, pitch, n2, n3):
    """(1 + 2 b) x_i - 2 b x_{1-i} = r_i: mean and difference divided by 1 and 1 + 4 b; the padding keeps its values."""
    torch = pytest.importorskip("torch")
    beta = 0.37
    host = np.random.default_rng(pitch + n2).standard_normal((n2 * n3, pitch))
    mean, half = (host[:, 0] + host[:, 1]) / 2, (host[:, 0] - host[:, 1]) / 2 / (1 + 4 * beta)
    want = host.copy()
    want[:, 0], want[:, 1] = mean + half, mean - half
    buf = torch.from_numpy(host).cuda()
    st = gpu_lib.mibm_solxi_noalloc(C.c_void_p(buf.data_ptr()), 2, n2, n3, pitch, beta,
                                    C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == abi.MIBM_OK
    got = buf.cpu().numpy()
    assert np.array_equal(got[:, 2:], host[:, 2:])
    assert np.max(np.abs(got - want)) <= 16 * 2.0 ** -53 * np.abs(host[:, :2]).max()
