"""FP64 sums whose targets or vertices are not numbers, are infinite or far away: a NaN target
keeps no pair of the cutoff kernel (its radial distance is not above the radius) and has NaN
under the others; a filament one of whose ends is NaN is left out of the sums."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from flapjax_b200 import _lib
from oracle import uvlm_ref as R

pytestmark = pytest.mark.gpu
KERNELS = {"epsilon": _lib.FJ_KERNEL_EPSILON, "cutoff": _lib.FJ_KERNEL_CUTOFF, "plain": _lib.FJ_KERNEL_PLAIN}
NANS = [np.nan, np.array([0xFFF8000000000000], np.uint64).view(float)[0]]  # both signs
ROWS, COLS, R_CUT = 6, 11, 1e-3


def _lattice():
    rng = np.random.default_rng(4)
    k, l = np.meshgrid(np.linspace(0, 1, ROWS + 1), np.linspace(0, 2, COLS + 1), indexing="ij")
    z = np.stack([k + 0.3 * l, l, -0.1 * k], -1)
    return z, rng.normal(size=(ROWS, COLS)), rng.normal(size=(300, 3)) + [0.5, 1.0, 3.0]


def _vind(x, z, g, kernel):
    import torch

    t, zd, gd = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (x, z, g))
    rows, cols, v, nb = (C.c_int * 1)(g.shape[0]), (C.c_int * 1)(g.shape[1]), torch.empty_like(t), C.c_size_t()
    _lib.call("fj_vind_workspace_size", len(x), rows, cols, 1, 0, _lib.FJ_PREC_FP64, C.byref(nb))
    ws = torch.empty(nb.value, dtype=torch.uint8, device="cuda")
    p = lambda a: (C.c_void_p * 1)(a.data_ptr())
    _lib.call("fj_vind", t.data_ptr(), len(x), p(zd), p(gd), rows, cols, 1, None, None, kernel, R_CUT, _lib.FJ_PREC_FP64,
              v.data_ptr(), ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
    return v.cpu().numpy()


def _filaments(g):
    """(vertex, vertex, strength) of a ring lattice's filaments."""
    p = np.zeros((ROWS + 2, COLS + 2))
    p[1:-1, 1:-1] = g
    out = [((k, l), (k + 1, l), p[k + 1, l + 1] - p[k + 1, l]) for k in range(ROWS) for l in range(COLS + 1)]
    return out + [((k, l), (k, l + 1), p[k, l + 1] - p[k + 1, l + 1]) for k in range(ROWS + 1) for l in range(COLS)]


def _sum(x, z, filaments, kernel):
    pair = {"epsilon": R.bs_epsilon, "plain": R.bs_plain, "cutoff": lambda *a: R.bs_cutoff(*a, R_CUT)}[kernel]
    at = lambda v: np.broadcast_to(z[v], x.shape)
    return sum(g * pair(x, at(a), at(b)) for a, b, g in filaments)


@pytest.mark.parametrize("nan", NANS)
@pytest.mark.parametrize("kernel", ["epsilon", "cutoff", "plain"])
def test_targets(cuda, kernel, nan):
    z, g, x = _lattice()
    want = _vind(x, z, g, KERNELS[kernel])
    bad = x.copy()
    bad[3, 1], bad[200] = nan, nan
    got = _vind(bad, z, g, KERNELS[kernel])
    others = np.setdiff1d(np.arange(len(x)), [3, 200])
    assert np.array_equal(got[others], want[others])
    if kernel == "cutoff":
        assert np.all(got[[3, 200]] == 0.0)
    else:
        assert np.all(np.isnan(got[[3, 200]]))


@pytest.mark.parametrize("nan", NANS)
@pytest.mark.parametrize("whole", [False, True])
@pytest.mark.parametrize("kernel", ["epsilon", "cutoff", "plain"])
def test_vertices(cuda, kernel, whole, nan):
    z, g, x = _lattice()
    bad = z.copy()
    bad[2, 3, 0 if whole else 1:] = nan
    want = _sum(x, z, [f for f in _filaments(g) if (2, 3) not in f[:2]], kernel)
    got = _vind(x, bad, g, KERNELS[kernel])
    # 20 eps |r1||r2| / |c| a pair, of pairs up to 1e3 of the sum, distances of 2 to 5 to filaments of 0.2
    assert np.all(np.linalg.norm(got - want, axis=1) <= 1e-9 * np.linalg.norm(want, axis=1).max())


@pytest.mark.parametrize("kernel", ["epsilon", "cutoff"])
def test_far_targets(cuda, kernel):
    """|r1 x r2|^2 overflows: nothing to add, and nothing that is not a number."""
    z, g, x = _lattice()
    x[3], x[200] = [1e100, 2e100, 3e100], [-1e90, 1e90, 0.0]
    assert np.all(np.abs(_vind(x, z, g, KERNELS[kernel])[[3, 200]]) <= 1e-80)
