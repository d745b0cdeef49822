"""The Biot-Savart sum's adjoints where a pair must add nothing, or next to nothing: targets that are
not numbers under the cutoff kernel (within the core radius by the reference's test, as any pair
that is dropped, whatever the other factors are), filaments of no length, with an infinite end, and
targets so far away that the sixth power of their distance overflows."""
from __future__ import annotations

import numpy as np
import pytest

from flapjax_b200 import _lib
from tests.test_gpu_vjp import EPS, _adjoint, _device, _err, _filaments

pytestmark = pytest.mark.gpu
KERNELS = {"epsilon": _lib.FJ_KERNEL_EPSILON, "cutoff": _lib.FJ_KERNEL_CUTOFF}


def _case(rows=6, cols=11, n=300):
    rng = np.random.default_rng(8)
    k, l = np.meshgrid(np.linspace(0, 1, rows + 1), np.linspace(0, 2, cols + 1), indexing="ij")
    z, gamma = np.stack([k + 0.3 * l, l, -0.1 * k], -1), rng.normal(size=(rows, cols))
    x = rng.normal(size=(n, 3)) + [0.5, 1.0, 0.0]
    x[:, 2] = np.where(x[:, 2] < 0, -0.4, 0.3) + x[:, 2]
    return z, gamma, x, rng.normal(size=x.shape)


@pytest.mark.parametrize("bad", [np.nan, -np.nan, np.inf])
@pytest.mark.parametrize("r_cut", [0.0, 1e-3])
def test_targets_that_are_not_numbers(cuda, r_cut, bad):
    z, gamma, x, lam = _case()
    rows, none = [3, 200], lam.copy()
    none[rows] = 0.0  # adds exact zeros
    want = _device(x, z, gamma, none, _lib.FJ_KERNEL_CUTOFF, r_cut, False)
    x[3, 1], x[200] = bad, bad
    lam[rows] = bad
    got = _device(x, z, gamma, lam, _lib.FJ_KERNEL_CUTOFF, r_cut, False)
    want[0][rows] = 0.0
    for g, w in zip(got, want):
        assert np.array_equal(g, w)


@pytest.mark.parametrize("kernel", ["epsilon", "cutoff"])
def test_filaments_of_no_length(cuda, kernel):
    z, gamma, x, lam = _case()
    z[1] = z[2]
    f, g = _filaments(*gamma.shape, gamma)
    zf = z.reshape(-1, 3)
    some = np.linalg.norm(zf[f[:, 0]] - zf[f[:, 1]], axis=1) > 0
    want_t, want_z, *_ = _adjoint(x, zf, f[some], g[some], lam, KERNELS[kernel], 1e-3)
    tb, zb, gb = _device(x, z, gamma, lam, KERNELS[kernel], 1e-3, False)
    assert _err(tb, want_t) <= 12800 * EPS  # as off the surface in test_gpu_vjp
    assert _err(zb.reshape(-1, 3), want_z) <= 12800 * EPS
    assert np.all(np.isfinite(gb))


@pytest.mark.parametrize("r_cut", [0.0, 1e-3])
def test_infinite_ends(cuda, r_cut):
    z, gamma, x, lam = _case()
    f, g = _filaments(*gamma.shape, gamma)
    some = ~np.any(f == 2 * 12 + 3, axis=1)
    want_t, want_z, *_ = _adjoint(x, z.reshape(-1, 3), f[some], g[some], lam, _lib.FJ_KERNEL_CUTOFF, r_cut)
    z[2, 3, 0] = np.inf
    tb, zb, gb = _device(x, z, gamma, lam, _lib.FJ_KERNEL_CUTOFF, r_cut, False)
    assert _err(tb, want_t) <= 12800 * EPS and _err(zb.reshape(-1, 3), want_z) <= 12800 * EPS
    assert np.all(np.isfinite(gb))


@pytest.mark.parametrize("far", [1e52, 1e60, 1e80, 1e100])
@pytest.mark.parametrize("kernel", ["epsilon", "cutoff"])
def test_far_targets(cuda, kernel, far):
    z, gamma, x, lam = _case()
    none = lam.copy()
    none[[3, 200]] = 0.0
    want = _device(x, z, gamma, none, KERNELS[kernel], 1e-3, False)
    x[3], x[200] = [far, 2 * far, 3 * far], [-far, 0.0, 0.0]
    got = _device(x, z, gamma, lam, KERNELS[kernel], 1e-3, False)
    assert np.all(np.abs(got[0][[3, 200]]) <= 1e-30)
    got[0][[3, 200]], want[0][[3, 200]] = 0.0, 0.0
    for a, b in zip(got, want):  # what they add is far below the last place
        assert _err(a, b) <= 12800 * EPS
