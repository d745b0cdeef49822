"""The LU's panels at the ends of the range: pivots that are subnormal, near the largest number or
infinite scale their column as getrf does (a quotient by a subnormal pivot, else a product with
the correctly rounded reciprocal), bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from tests.test_gpu_panel import _factor

pytestmark = pytest.mark.gpu
TINY = np.finfo(float).tiny


@pytest.mark.parametrize("pivot", [3.7, -1.1e-200, 1.3e200, TINY, -0.6 * TINY, 5e-324, 2.3e307, -1.79e308, np.inf])
@pytest.mark.parametrize("n", [64, 200, 300, 700])
def test_scaled_column(cuda, n, pivot):
    """One column of multipliers, in the first window and in the last: the rest is the unit matrix's."""
    import torch

    rng = np.random.default_rng(n)
    for j in (0, min(n, 64) - 5):
        a = np.eye(n)
        a[j, j] = pivot
        with np.errstate(over="ignore", under="ignore"):
            column = np.float64(abs(pivot) if np.isfinite(pivot) else 1e300) * rng.uniform(-0.9, 0.9, n - j - 1)
            a[j + 1:, j] = column
            want = column / pivot if abs(pivot) < TINY else column * (1.0 / np.float64(pivot))
        lu, piv, info = _factor(torch, a)
        assert info == 0 and np.array_equal(piv, np.arange(n))
        assert np.array_equal(lu[j + 1:, j], want)
