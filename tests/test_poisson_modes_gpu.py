"""The FP64 Poisson solve on single modes of z: lines that oscillate do not grow in the sweeps, and keep their digits."""
from __future__ import annotations

import numpy as np
import pytest

from tests.helpers import rel_l2
from tests.test_poisson_inputs_gpu import _exact, _solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, n3, stretch", [(16, 96, 1.0), (8, 216, 1.0), (16, 256, 1.0), (8, 512, 1.0), (16, 512, 1.0),
                                            (8, 256, 0.6), (8, 144, 0.4), (8, 256, 2.0)])
@pytest.mark.parametrize("mode", [0, 1, 2, 4, 8])
def test_a_single_mode_of_z(gpu_lib, n, n3, stretch, mode):
    """cos x times cos k z, k = n3/2, n3/2 - 1, n3/4, n3/8 (0: the alternating one, 8: the lowest).  A pass rounds each value
    to 2^-53 of it; where those roundings fall on the line's mean, the solution has them by the ratio of the two
    eigenvalues.  Half of that, a typical rounding, is allowed in all, and no less than 24 units of 2^-53."""
    k = {0: n3 // 2, 1: n3 // 2 - 1, 2: n3 // 4, 4: n3 // 8, 8: 1}[mode]
    wave = np.cos(2 * np.pi * np.arange(n) / n)[:, None, None] * np.ones((1, n, 1))
    x = wave * np.cos(2 * np.pi * k * np.arange(n3) / n3)[None, None, :]
    low = 4 * np.sin(np.pi / n) ** 2 * (n / (2 * np.pi)) ** 2
    ratio = (low + 4 * np.sin(np.pi * k / n3) ** 2 * (n3 / (2 * np.pi * stretch)) ** 2) / low
    got, ref = _solve(gpu_lib, n, n3, x, stretch), _exact(n, n3, x, stretch)
    assert rel_l2(got, ref) <= 2.0 ** -53 * max(0.5 * ratio, 24.0)
