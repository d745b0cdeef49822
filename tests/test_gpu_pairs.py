"""The FP64 pair arithmetic and the cuts of the sums, against the oracle.

The pair takes its reciprocal square root and reciprocal from approximate seeds and one
cubic step: a few units in the last place.  With the cross product's own rounding (relative
to |r1||r2|) the velocity of a pair is known to about 20 eps |r1||r2| / |r1 x r2|, and the
difference of the two direction cosines to about 10 eps of its terms."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from flapjax_b200 import _lib
from oracle import uvlm_ref as R
from tests.helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("distance", [1e-3, 1.0, 1e3])
@pytest.mark.parametrize("kernel", ["epsilon", "cutoff"])
def test_pairs_over_distances(cuda, kernel, distance):
    import flapjax_b200 as fj

    rng = np.random.default_rng(3)
    y0 = rng.normal(size=(8192, 3))
    y1 = y0 + rng.normal(size=y0.shape)
    x = 0.5 * (y0 + y1) + distance * rng.normal(size=y0.shape)
    if kernel == "epsilon":
        got, want = fj.biot_savart_epsilon(x, np.stack([y0, y1], 1)), R.bs_epsilon(x, y0, y1)
    else:
        got, want = fj.cutoff_kernel(1e-5)(x, np.stack([y0, y1], 1)), R.bs_cutoff(x, y0, y1, 1e-5)
    r1, r2, r0 = x - y0, x - y1, y1 - y0
    n1, n2, nr = (np.linalg.norm(a, axis=1) for a in (r1, r2, r0))
    c = np.linalg.norm(np.cross(r1, r2), axis=1)
    eps = np.finfo(float).eps
    dot = np.abs((r0 * (r1 / n1[:, None] - r2 / n2[:, None])).sum(1))
    size = np.linalg.norm(want, axis=1)
    bound = size * eps * (20 + 20 * n1 * n2 / c + 20 * nr / np.maximum(dot, 1e-300))
    assert np.all(np.linalg.norm(got - want, axis=1) <= bound)


@pytest.mark.parametrize("r_cut", [0.0, 1e-4, 1e-2])
def test_core_radius_decides_as_the_reference(cuda, r_cut):
    """Targets from far inside to far outside the core radius, some within 1e-12 of it,
    collinear ones, ends, a filament without length and NaN: kept or dropped as the
    reference's radial distance says."""
    import flapjax_b200 as fj

    rng = np.random.default_rng(5)
    n = 2048
    y0 = rng.normal(size=(n, 3))
    e = rng.normal(size=(n, 3))
    e /= np.linalg.norm(e, axis=1, keepdims=True)
    y1 = y0 + 0.3 * e
    p = np.cross(e, rng.normal(size=(n, 3)))
    p /= np.linalg.norm(p, axis=1, keepdims=True)
    f = 1.0 + np.concatenate([10.0 ** rng.uniform(-12, 0, n // 2), -(10.0 ** rng.uniform(-12, -0.001, n // 2))])
    x = y0 + rng.uniform(-0.5, 0.8, (n, 1)) * e + (max(r_cut, 1e-6) * f)[:, None] * p
    x[0], x[1], x[2], y1[3], x[4] = y0[0], y1[1], y0[2] + 2.0 * (y1[2] - y0[2]), y0[3], np.nan
    with np.errstate(all="ignore"):
        want = R.bs_cutoff(x, y0, y1, r_cut)
        r0 = y1 - y0
        away = (x - y0) - ((x - y0) * r0).sum(1)[:, None] / (r0 * r0).sum(1)[:, None] * r0
        side = np.abs((away * away).sum(1) / max(r_cut, 1e-300) ** 2 - 1.0)
    got = fj.cutoff_kernel(r_cut)(x, np.stack([y0, y1], 1))
    # the radial distance itself is known to about 1e-15 / r_cut here
    clear = side > (1e-13 / r_cut if r_cut else np.inf)
    clear[:5] = r_cut > 0
    assert np.array_equal(np.any(got[clear] != 0, 1), np.any(want[clear] != 0, 1))
    assert np.all(np.isfinite(got[clear]))


def _vind(torch, targets, lats, kernel, precision, noalloc=False):
    n = len(lats)
    t = torch.from_numpy(np.ascontiguousarray(targets)).cuda()
    zs = [torch.from_numpy(z).cuda() for z, _ in lats]
    gs = [torch.from_numpy(g).cuda() for _, g in lats]
    zp, gp = (C.c_void_p * n)(*[z.data_ptr() for z in zs]), (C.c_void_p * n)(*[g.data_ptr() for g in gs])
    rows, cols = (C.c_int * n)(*[g.shape[0] for g in gs]), (C.c_int * n)(*[g.shape[1] for g in gs])
    v, s = torch.full_like(t, np.nan), torch.cuda.current_stream().cuda_stream
    args = (t.data_ptr(), t.shape[0], zp, gp, rows, cols, n, None, None, kernel, 1e-3, precision, v.data_ptr())
    if noalloc:
        _lib.call("fj_vind_noalloc", *args, s)
    else:
        nb = C.c_size_t()
        _lib.call("fj_vind_workspace_size", t.shape[0], rows, cols, n, 0, precision, C.byref(nb))
        ws = torch.full((nb.value,), 0xFF, dtype=torch.uint8, device="cuda")
        _lib.call("fj_vind", *args, ws.data_ptr(), ws.numel(), s)
    return v.cpu().numpy()


@pytest.mark.parametrize("n_targets,rows,cols", [(1, 1, 1), (3, 1, 130), (255, 7, 5), (257, 40, 9), (700, 33, 31),
                                                 (5000, 3, 2), (1, 120, 60)])
@pytest.mark.parametrize("precision,tol", [(_lib.FJ_PREC_FP64, 1e-12), (_lib.FJ_PREC_MIXED, 2e-6)])
def test_pieces_cover_the_stream(cuda, n_targets, rows, cols, precision, tol):
    """Sums at the edges of tiles, splits, pieces and chunks: every filament counted once,
    with a caller's workspace and with the library's fixed one."""
    import torch

    rng = np.random.default_rng(n_targets + rows)
    z = np.zeros((rows + 1, cols + 1, 3))
    z[..., 0] = np.linspace(0, 2, rows + 1)[:, None]
    z[..., 1] = np.linspace(0, 3, cols + 1)[None]
    z += 0.02 / max(rows, cols) * rng.normal(size=z.shape)
    g = rng.uniform(0.5, 1.5, (rows, cols))
    x = rng.uniform((-1, -1, 0.2), (3, 4, 1), (n_targets, 3))
    for ker, ref in ((_lib.FJ_KERNEL_EPSILON, R.KERNEL_EPSILON), (_lib.FJ_KERNEL_CUTOFF, R.KERNEL_CUTOFF)):
        want = R.compute_v_ind(x, [z], [g], ref, r_cut=1e-3)
        for noalloc in (False, True):
            assert rel_err(_vind(torch, x, [(z, g)], ker, precision, noalloc), want) < tol
