"""getrs for one right-hand side at the edges of its blocks of 64 rows and of its clusters
(one CTA below 512 rows, up to eight above; odd orders, whose rows begin unaligned), both
directions: |op(A) x - b| <= (3 n eps) |L||U||x|, the bound of elimination with the
substitutions' own rounding (Higham, Accuracy and Stability, theorem 9.4), doubled for the
residual's own evaluation."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from flapjax_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 128, 129, 255, 256, 257, 320, 511, 512, 513, 769, 1088, 2049])
def test_backward_error(cuda, n, transposed):
    import torch

    rng = np.random.default_rng(n)
    a, b = rng.normal(size=(n, n)), rng.normal(size=n)
    lu, x = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    piv = torch.empty(n, dtype=torch.int32, device="cuda")
    nb = C.c_size_t()
    _lib.call("fj_lu_workspace_size", n, C.byref(nb))
    ws = torch.zeros(nb.value + 8 * n, dtype=torch.uint8, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    _lib.call("fj_lu_factor", lu.data_ptr(), n, piv.data_ptr(), ws.data_ptr(), ws.numel(), s)
    _lib.call("fj_lu_solve_t" if transposed else "fj_lu_solve", lu.data_ptr(), n, piv.data_ptr(), x.data_ptr(),
              ws.data_ptr(), ws.numel(), s)
    f, x = lu.cpu().numpy(), x.cpu().numpy()
    lo, up = np.abs(np.tril(f, -1)) + np.eye(n), np.abs(np.triu(f))
    perm = np.arange(n)
    for i, p in enumerate(piv.cpu().numpy()):
        perm[[i, p]] = perm[[p, i]]
    size = np.empty((n, n))
    size[perm] = lo @ up  # of A's rows
    op = (lambda m: m.T) if transposed else (lambda m: m)
    assert np.all(np.abs(op(a) @ x - b) <= 6 * n * np.finfo(float).eps * (op(size) @ np.abs(x)))
