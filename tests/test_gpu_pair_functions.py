"""The pair arithmetic's 1 / sqrt(x) and 1 / x against extended precision and CUDA's own functions.

With u = 2^-53 and e the seed's relative error, at most 2^-18.5 (its argument and result have 20 bits
of mantissa): the reciprocal's step leaves e^3 < 0.2 u and rounds once, 1.3 u; the square root's leaves
5/16 e^3 and half of the rounding of x y beside its own, 1.6 u.  CUDA's are known to half a unit and one
unit in the last place."""
from __future__ import annotations

import ctypes as C
import subprocess

import numpy as np
import pytest

from flapjax_b200 import build

pytestmark = pytest.mark.gpu
LD, U = np.longdouble, np.longdouble(2.0) ** -53


@pytest.fixture(scope="module")
def lib(cuda, tmp_path_factory):
    so = tmp_path_factory.mktemp("pairs") / "pairs.so"
    subprocess.run([build.nvcc(), *build.ARCH, *build.NVCC_FLAGS, "-I", str(build.INCLUDE), "-I", str(build.CSRC),
                    "-shared", "-o", str(so), str(build.ROOT / "tests" / "pair_functions.cu"), "-lcudart"], check=True)
    return C.CDLL(str(so))


def _evaluate(lib, x):
    import torch

    t = torch.from_numpy(x).cuda()
    out = torch.empty((4, len(x)), dtype=torch.float64, device="cuda")
    assert lib.pair_functions(C.c_void_p(t.data_ptr()), C.c_int64(len(x)), C.c_void_p(out.data_ptr()),
                              C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    return out.cpu().numpy()


@pytest.mark.parametrize("part", ["exponents", "mantissas", "ends"])
def test_against_extended_precision(lib, part):
    rng = np.random.default_rng(7)
    if part == "exponents":  # every exponent used: above the subnormals, below 2^1022
        x = np.ldexp(rng.uniform(1.0, 2.0, 2044 * 256), np.repeat(np.arange(-1022, 1022), 256))
    elif part == "mantissas":
        x = rng.uniform(0.25, 4.0, 1 << 20)
    else:  # beside the powers of two, and the two ends
        p = np.ldexp(1.0, np.arange(-1021, 1022))
        x = np.concatenate([p, np.nextafter(p, 0), np.nextafter(p, np.inf),
                            [2.0**-1022, np.array([0x7FCFFFFFFFFFFFFF], np.uint64).view(float)[0]]])
    root, root_cuda, rcp, rcp_cuda = _evaluate(lib, x)
    want_root, want_rcp = 1 / np.sqrt(x.astype(LD)), 1 / x.astype(LD)
    assert np.max(np.abs(root - want_root) / want_root) <= LD(1.6) * U
    assert np.max(np.abs(rcp - want_rcp) / want_rcp) <= LD(1.3) * U
    assert np.max(np.abs(root - root_cuda) / np.spacing(root_cuda)) <= 2
    assert np.max(np.abs(rcp - rcp_cuda) / np.spacing(rcp_cuda)) <= 1
