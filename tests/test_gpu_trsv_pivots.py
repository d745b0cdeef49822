"""getrs with pivots whose reciprocal is no normal number (subnormal ones, and above 2^1022), in the
first, a middle and the last, ragged block: a diagonal system's quotients, exactly."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from flapjax_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("pivot,value", [(3e-309, 6e-309), (-5e-324, 1e-300), (1.7e308, 1.1e308), (2.0**-1022, 1.0)])
@pytest.mark.parametrize("n", [5, 100, 600])
def test_quotients(cuda, n, pivot, value, transposed):
    import torch

    odd = np.isin(np.arange(n) % 64, [0, 3, 40, 63]) & (np.arange(n) // 64 % 2 == 0)
    odd[-1] = True
    d, b = np.where(odd, pivot, 1.0), np.where(odd, value, np.random.default_rng(n).normal(size=n))
    lu, x = torch.from_numpy(np.diag(d)).cuda(), torch.from_numpy(b).cuda()
    piv, nb = torch.arange(n, dtype=torch.int32, device="cuda"), C.c_size_t()
    _lib.call("fj_lu_workspace_size", n, C.byref(nb))
    ws = torch.zeros(nb.value + 8 * n, dtype=torch.uint8, device="cuda")
    _lib.call("fj_lu_solve_t" if transposed else "fj_lu_solve", lu.data_ptr(), n, piv.data_ptr(), x.data_ptr(),
              ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
    assert np.array_equal(x.cpu().numpy(), b / d)
