"""getrs of orders whose row permutation needs a smaller scratch in shared memory (from 51 969), or
does not fit there (many right-hand sides), and those whose tiles have two buffers (from 17 400):
factors of the unit matrix with a few entries beside it, and pivots at random."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from flapjax_b200 import _lib

pytestmark = pytest.mark.gpu


def _case(torch, n):
    rng = np.random.default_rng(n)
    entries = [(n - 1, 0, 0.5), (n // 2 + 7, n // 2 - 70, -0.25), (3, n - 5, 0.75), (n // 3, n // 3 + 100, 1.5), (n - 1, n - 1, 4.0)]
    lu = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    lu.diagonal().fill_(1.0)
    for i, j, v in entries:
        lu[i, j] = v
    piv = (np.arange(n) + (rng.integers(0, 1 << 30, n) % (n - np.arange(n)))).astype(np.int32)
    perm = np.arange(n)
    for i, p in enumerate(piv):
        perm[i], perm[p] = perm[p], perm[i]
    return lu, torch.from_numpy(piv).cuda(), perm, rng.integers(-8, 9, n).astype(float), entries


def _solve(entries, perm, b, transposed):
    """The substitutions with the few entries, whose powers of two make them exact."""
    low, up = [e for e in entries if e[0] > e[1]], [e for e in entries if e[0] < e[1]]
    (d, _, dv), = [e for e in entries if e[0] == e[1]]
    x = b.copy() if transposed else b[perm]
    if transposed:
        for i, j, v in up:
            x[j] -= v * x[i]
        x[d] /= dv
        for i, j, v in low:
            x[j] -= v * x[i]
        out = np.empty_like(x)
        out[perm] = x
        return out
    for i, j, v in low:
        x[i] -= v * x[j]
    x[d] /= dv
    for i, j, v in up:
        x[i] -= v * x[j]
    return x


@pytest.mark.parametrize("n", [17500, 51969, 56320])
def test_one_right_hand_side(cuda, n):
    import torch

    lu, piv, perm, b, entries = _case(torch, n)
    nb = C.c_size_t()
    _lib.call("fj_lu_workspace_size", n, C.byref(nb))
    ws = torch.zeros(nb.value + 8 * n, dtype=torch.uint8, device="cuda")
    for transposed in (False, True):
        x = torch.from_numpy(b).cuda()
        _lib.call("fj_lu_solve_t" if transposed else "fj_lu_solve", lu.data_ptr(), n, piv.data_ptr(), x.data_ptr(),
                  ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
        assert np.array_equal(x.cpu().numpy(), _solve(entries, perm, b, transposed))


def test_many_right_hand_sides(cuda):
    import torch

    n = 51969
    lu, piv, perm, b, entries = _case(torch, n)
    x, nb = torch.from_numpy(np.stack([b, -2.0 * b], 1).copy()).cuda(), C.c_size_t()
    _lib.call("fj_lu_solve_many_workspace_size", n, 2, C.byref(nb))
    ws = torch.zeros(nb.value, dtype=torch.uint8, device="cuda")
    _lib.call("fj_lu_solve_many", lu.data_ptr(), n, piv.data_ptr(), x.data_ptr(), 2, 2, ws.data_ptr(), ws.numel(),
              torch.cuda.current_stream().cuda_stream)
    want = _solve(entries, perm, b, False)
    assert np.array_equal(x.cpu().numpy(), np.stack([want, -2.0 * want], 1))
