"""A cluster's waits that expire: a build of the kernels in which every wait gives up at once.  The
panel writes no row, names each row as its own pivot, reports the order + 1 and leaves a NaN pivot; the
substitutions' solution is NaN."""
from __future__ import annotations

import ctypes as C
import subprocess

import numpy as np
import pytest

from flapjax_b200 import build

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(cuda, tmp_path_factory):
    so = tmp_path_factory.mktemp("waits") / "waits.so"
    src = [build.ROOT / "tests" / "expired_waits.cu", build.CSRC / "fj_panel.cu", build.CSRC / "fj_trsv.cu"]
    subprocess.run([build.nvcc(), *build.ARCH, *build.NVCC_FLAGS, "-DFJ_WAIT_CYCLES=-1", "-I", str(build.INCLUDE), "-I",
                    str(build.CSRC), "-shared", "-o", str(so), *map(str, src), "-lcudart"], check=True)
    return C.CDLL(str(so))


@pytest.mark.parametrize("dtype,cols", [("float64", 64), ("float64", 40), ("float32", 128)])
@pytest.mark.parametrize("n", [385, 700, 2048])
def test_panel(lib, n, dtype, cols):
    import torch

    a = torch.randn((n, n), dtype=getattr(torch, dtype), device="cuda")
    before = a.clone()
    piv, info = torch.full((n,), -7, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    call = lib.panel64 if dtype == "float64" else lib.panel32
    p = lambda t: C.c_void_p(t.data_ptr())
    assert call(p(a), n, cols, p(piv), p(info), C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    assert int(info) == n + 1
    assert torch.isnan(a[0, 0])
    a[0, 0] = before[0, 0]
    assert torch.equal(a, before)
    want = np.full(n, -7)
    want[:cols] = np.arange(cols)
    assert np.array_equal(piv.cpu().numpy(), want)


@pytest.mark.parametrize("transposed", [0, 1])
@pytest.mark.parametrize("n", [64, 600, 2049])
def test_substitutions(lib, n, transposed):
    import torch

    lu, b, work = (torch.randn(s, dtype=torch.float64, device="cuda") for s in ((n, n), (n,), (n,)))
    piv = torch.arange(n, dtype=torch.int32, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())
    assert lib.solve(p(lu), n, p(piv), p(b), p(work), transposed, C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    assert torch.all(torch.isnan(b))
