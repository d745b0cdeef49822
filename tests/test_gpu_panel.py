"""The LU's panels at the edges of their forms (one CTA up to 384 rows, clusters of 128-row
CTAs above, narrow panels beyond 2048): getrf's factors within the backward error bound
|P A - L U| <= n eps |L||U| of elimination (Higham, Accuracy and Stability, 9.3), multipliers
of at most one, pivots that name rows below, and the first zero pivot."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from flapjax_b200 import _lib

pytestmark = pytest.mark.gpu


def _factor(torch, a):
    n = a.shape[0]
    lu = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    piv = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    nb = C.c_size_t()
    _lib.call("fj_lu_workspace_size", n, C.byref(nb))
    ws = torch.zeros(nb.value, dtype=torch.uint8, device="cuda")
    _lib.call("fj_lu_factor", lu.data_ptr(), n, piv.data_ptr(), ws.data_ptr(), ws.numel(),
              torch.cuda.current_stream().cuda_stream)
    return lu.cpu().numpy(), piv.cpu().numpy(), int(ws[:4].cpu().numpy().view(np.int32)[0])


def _matrix(kind, n):
    rng = np.random.default_rng(n)
    if kind == "random":
        return rng.normal(size=(n, n))
    if kind == "ties":  # equal magnitudes within and across warps and CTAs
        return rng.integers(-1, 2, size=(n, n)) + 3.0 * np.eye(n)[rng.permutation(n)]
    if kind == "permutation":
        return np.eye(n)[rng.permutation(n)]
    a = rng.normal(size=(n, n))  # a column that elimination finds empty
    a[:, n // 2] = 0.0
    return a


@pytest.mark.parametrize("kind", ["random", "ties", "permutation", "zero column"])
@pytest.mark.parametrize("n", [1, 2, 17, 64, 65, 128, 129, 200, 256, 257, 384, 385, 513, 1100, 2048, 2049])
def test_factors(cuda, n, kind):
    import torch

    a = _matrix(kind, n)
    lu, piv, info = _factor(torch, a)
    assert np.all((piv >= np.arange(n)) & (piv < n))
    assert info == (n // 2 + 1 if kind == "zero column" else 0)
    perm = np.arange(n)
    for i, p in enumerate(piv):
        perm[[i, p]] = perm[[p, i]]
    lo, up = np.tril(lu, -1) + np.eye(n), np.triu(lu)
    assert np.abs(lo).max() <= 1.0
    err = np.abs(a[perm] - lo @ up)
    assert np.all(err <= 2 * n * np.finfo(float).eps * (np.abs(lo) @ np.abs(up)) + 1e-300)
    if kind == "permutation":
        assert np.array_equal(lo, np.eye(n)) and np.array_equal(up, np.eye(n))
    if kind != "zero column":
        first = np.abs(a[:, 0])
        assert piv[0] == int(np.argmax(first))  # the first of equals
