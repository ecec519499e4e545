"""mibm_solxi_noalloc on both of its routes: line lengths, row pitches and base addresses where the route changes."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from melt_ibm_gb300 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, n2, n3, pitch, offset", [
    (2, 3, 2, 2, 0), (2, 3, 2, 3, 0), (16, 1, 1, 16, 0), (27, 5, 3, 27, 0), (27, 5, 3, 28, 1), (48, 37, 2, 48, 0), (96, 7, 5, 96, 0),
    (96, 7, 5, 97, 0), (96, 7, 5, 98, 0), (96, 7, 5, 96, 1), (97, 7, 5, 98, 0), (256, 50, 130, 256, 0), (486, 3, 2, 488, 0),
    (512, 9, 3, 512, 0)])
@pytest.mark.parametrize("beta", [-0.1, 1e-3, 0.37, 40.0])
def test_both_routes_solve_the_periodic_system(gpu_lib, n, n2, n3, pitch, offset, beta):
    """(1 + 2 b) x_i - b (x_{i-1} + x_{i+1}) = r_i by its eigenvalues.  Both routes are stable
    eliminations: 64 units of 2^-53 times the condition number; the padding keeps its values."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + pitch)
    r = rng.standard_normal((n3 * n2, n))
    lam = 1.0 + 2.0 * beta * (1.0 - np.cos(2.0 * np.pi * np.arange(n) / n))
    cond = np.abs(lam).max() / np.abs(lam).min()
    ref = np.fft.ifft(np.fft.fft(r, axis=1) / lam, axis=1).real
    host = rng.standard_normal((n3 * n2, pitch))
    host[:, :n] = r
    flat = torch.zeros(host.size + offset, dtype=torch.float64, device="cuda")
    buf = flat[offset:]
    buf.copy_(torch.from_numpy(host.ravel()))
    st = gpu_lib.mibm_solxi_noalloc(C.c_void_p(buf.data_ptr()), n, n2, n3, pitch, beta,
                                    C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == abi.MIBM_OK
    out = buf.cpu().numpy().reshape(n3 * n2, pitch)
    assert np.linalg.norm(out[:, :n] - ref) <= 64 * 2.0 ** -53 * cond * np.linalg.norm(ref)
    assert np.array_equal(out[:, n:], host[:, n:])
