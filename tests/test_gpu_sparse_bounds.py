"""Windows built against the error bound of the sparse path's distances, bit for bit against the CPU oracle.

Each set makes one share of the error as large as it gets; a bound without that share gives a wrong core distance
and no fallback.
"""

import numpy as np
import pytest

from tests.test_gpu_sparse import _check

pytestmark = pytest.mark.gpu


def tiny_window(n=3000, d=32):
    """A float64 cluster so small that the squares of its points' coordinates have no place in float32, in a window of ordinary
    range whose centre lies in that cluster."""
    rng = np.random.default_rng(11)
    x = rng.uniform(-4, 4, (8, d))[rng.integers(0, 8, n)] + rng.normal(0, 0.5, (n, d))
    samples = np.arange(16) * n // 16
    others = rng.choice(np.setdiff1d(np.arange(n), samples), 24, replace=False)
    x[np.concatenate([samples, others])] = rng.normal(0, 1, (40, d)) * 2e-22 / np.sqrt(d)
    return x


def test_squares_below_float32(cuda):
    _check([tiny_window()], 5, 5, 0.0, "float64")
