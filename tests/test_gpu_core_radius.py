"""The cutoff kernel without a core radius: whatever is off the filament's line counts, at the value of
the reference; exactly collinear targets, ends, a filament without length and NaN do not."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import uvlm_ref as R

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def test_off_the_line(cuda):
    import flapjax_b200 as fj

    rng = np.random.default_rng(6)
    n = 2048
    y0, e = rng.normal(size=(n, 3)), rng.normal(size=(n, 3))
    e /= np.linalg.norm(e, axis=1, keepdims=True)
    y1 = y0 + 0.3 * e
    p = np.cross(e, rng.normal(size=(n, 3)))
    p /= np.linalg.norm(p, axis=1, keepdims=True)
    away = 10.0 ** rng.uniform(-9, 1, n)  # from 1e6 roundings of the line on, between the ends
    x = y0 + rng.uniform(0.01, 0.29, (n, 1)) * e + away[:, None] * p
    got, want = fj.cutoff_kernel(0.0)(x, np.stack([y0, y1], 1)), R.bs_cutoff(x, y0, y1, 0.0)
    r1, r2, r0 = x - y0, x - y1, y1 - y0
    n1, n2, nr = (np.linalg.norm(a, axis=1) for a in (r1, r2, r0))
    c = np.linalg.norm(np.cross(r1, r2), axis=1)
    dot = np.abs((r0 * (r1 / n1[:, None] - r2 / n2[:, None])).sum(1))
    bound = np.linalg.norm(want, axis=1) * EPS * (20 + 20 * n1 * n2 / c + 20 * nr / dot)  # as in test_gpu_pairs
    assert np.all(np.any(got != 0, 1)) and np.all(np.any(want != 0, 1))
    assert np.all(np.linalg.norm(got - want, axis=1) <= bound)


def test_on_the_line(cuda):
    """Coordinates whose products and quotients are exact."""
    import flapjax_b200 as fj

    at = np.array([0.0, 0.5, 0.25, 2.0, -4.0, 0.125, 0.25])
    x, y0 = np.zeros((len(at), 3)), np.zeros((len(at), 3))
    x[:, 0] = at
    y1 = y0 + [0.5, 0.0, 0.0]
    x[5, 1], y1[5] = 1.0, y0[5]  # off the point of a filament without length
    x[6, 2] = np.nan
    with np.errstate(all="ignore"):
        assert np.all(R.bs_cutoff(x, y0, y1, 0.0) == 0.0)
    assert np.all(fj.cutoff_kernel(0.0)(x, np.stack([y0, y1], 1)) == 0.0)
