"""The Biot-Savart sum's adjoints against the derivative's formula in extended precision:
splits of one to many targets and links, both kernels, a call for the targets alone (the
linearisation's) and one for everything, targets off the surface and at the middles of its own
filaments (where the derivative is of 1 / (eps |r0|^3) and others lie on the target's line).

A pair is some 100 operations, a sum in the largest of its pairs' roundings: 64 eps of the
result's norm, doubled for the sums' own.  Off the surface the pairs are no larger than the
result by more than 100 (distances of 0.3 or more of a span of 2), which multiplies that.  A strength's adjoint at a
filament's own middle is s (lam.c) with a c of nothing but rounding, 4 eps |r1||r2|: its bound."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from flapjax_b200 import _lib

pytestmark = pytest.mark.gpu
LD = np.longdouble
EPS = np.finfo(float).eps


def _filaments(rows, cols, gamma):
    g = np.zeros((rows + 2, cols + 2))
    g[1:-1, 1:-1] = gamma
    v = np.arange((rows + 1) * (cols + 1)).reshape(rows + 1, cols + 1)
    out = [(v[k, l], v[k + 1, l], g[k + 1, l + 1] - g[k + 1, l]) for k in range(rows) for l in range(cols + 1)]
    out += [(v[k, l], v[k, l + 1], g[k, l + 1] - g[k + 1, l + 1]) for k in range(rows + 1) for l in range(cols)]
    return np.array([o[:2] for o in out]), np.array([o[2] for o in out]).astype(LD)


def _adjoint(x, z, f, g, lam, kernel, rc):
    """(targets_bar, vertices_bar, strengths_bar, sum of |s||lam||r1||r2|) in extended precision."""
    dot, n = (lambda a, b: (a * b).sum(-1)), (lambda a: a[..., None])
    x, z, lam, e = x.astype(LD), z.astype(LD), lam.astype(LD), LD(1e-7)
    r1, r2 = x[:, None] - z[f[:, 0]], x[:, None] - z[f[:, 1]]
    r0, c, lam = r1 - r2, np.cross(r1, r2), np.broadcast_to(lam[:, None], r1.shape)
    i1, i2 = 1 / np.sqrt(dot(r1, r1) + e * e), 1 / np.sqrt(dot(r2, r2) + e * e)
    u1, u2, sq = r1 * n(i1), r2 * n(i2), dot(r0, r0)
    d, keep = dot(c, c) + e * sq * sq, np.ones(sq.shape, bool)
    if kernel == _lib.FJ_KERNEL_CUTOFF:
        m = r1 - n(dot(r0, r1) / sq) * r0
        d, keep = dot(c, c), dot(m, m) > LD(rc) * LD(rc)
    inv = keep / np.where(keep, d, 1) / (16 * np.arctan(LD(1)))
    s, a = dot(r0, u1 - u2) * inv, dot(lam, c)
    p = LD(0) if kernel == _lib.FJ_KERNEL_CUTOFF else 4 * e * n(sq) * r0
    q = n(dot(r0, u1 - u2) / np.where(keep, d, 1))
    d1 = u1 - u2 + (r0 - n(dot(r0, u1)) * u1) * n(i1) - q * (2 * np.cross(r2, c) + p)
    d2 = u2 - u1 - (r0 - n(dot(r0, u2)) * u2) * n(i2) - q * (2 * np.cross(c, r1) - p)
    b1, b2 = n(s) * np.cross(r2, lam) + n(a * inv) * d1, n(s) * np.cross(lam, r1) + n(a * inv) * d2
    w = g[None, :, None]
    zb = np.zeros(z.shape, LD)
    np.add.at(zb, f[:, 0], -(w * b1).sum(0))
    np.add.at(zb, f[:, 1], -(w * b2).sum(0))
    size = np.abs(s) * np.sqrt(dot(lam, lam) * dot(r1, r1) * dot(r2, r2))
    return (w * (b1 + b2)).sum(1), zb, (s * a).sum(0), size.sum(0)


def _device(x, z, gamma, lam, kernel, rc, alone):
    import torch

    rows, cols = (C.c_int * 1)(gamma.shape[0]), (C.c_int * 1)(gamma.shape[1])
    t, zd, gd, ld = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (x, z, gamma, lam))
    tb, zb, gb = torch.zeros_like(t), torch.zeros_like(zd), torch.zeros_like(gd)
    nb = C.c_size_t()
    _lib.call("fj_vind_vjp_workspace_size", len(x), rows, cols, 1, 0, C.byref(nb))
    ws = torch.empty(nb.value, dtype=torch.uint8, device="cuda")
    p = lambda a: (C.c_void_p * 1)(a.data_ptr())
    _lib.call("fj_vind_vjp", t.data_ptr(), len(x), p(zd), p(gd), rows, cols, 1, None, None, kernel, rc, ld.data_ptr(),
              tb.data_ptr(), None if alone else p(zb), None if alone else p(gb), ws.data_ptr(), ws.numel(),
              torch.cuda.current_stream().cuda_stream)
    return tb.cpu().numpy(), zb.cpu().numpy(), gb.cpu().numpy()


def _err(got, want):
    return float(np.linalg.norm((got - want).astype(float)) / np.linalg.norm(want.astype(float)))


@pytest.mark.parametrize("alone", [False, True])
@pytest.mark.parametrize("kernel", [_lib.FJ_KERNEL_EPSILON, _lib.FJ_KERNEL_CUTOFF])
@pytest.mark.parametrize("n,rows,cols", [(1, 1, 1), (15, 2, 3), (127, 1, 64), (129, 7, 9), (700, 4, 16), (None, 6, 12),
                                         (None, 3, 20)])
def test_adjoints(cuda, n, rows, cols, kernel, alone):
    rng = np.random.default_rng(rows * 100 + cols)
    k, l = np.meshgrid(np.linspace(0, 1, rows + 1), np.linspace(0, 2, cols + 1), indexing="ij")
    z, gamma = np.stack([k + 0.3 * l, l, -0.1 * k], -1), rng.normal(size=(rows, cols))
    f, g = _filaments(rows, cols, gamma)
    zf = z.reshape(-1, 3)
    if n is None:
        x, tol = 0.5 * (zf[f[:, 0]] + zf[f[:, 1]]), 128 * EPS
    else:
        x, tol = rng.normal(size=(n, 3)) + [0.5, 1.0, 0.0], 12800 * EPS
        x[:, 2] = np.where(x[:, 2] < 0, -0.4, 0.3) + x[:, 2]
    lam = rng.normal(size=x.shape)
    want_t, want_z, *want_k = _adjoint(x, zf, f, g, lam, kernel, 1e-3)
    tb, zb, gb = _device(x, z, gamma, lam, kernel, 1e-3, alone)
    assert _err(tb, want_t) <= tol
    if alone:
        return
    assert _err(zb.reshape(-1, 3), want_z) <= tol
    n_chord = rows * (cols + 1)
    (mk, sk), (mc, sc) = ((w[:n_chord].reshape(rows, cols + 1), w[n_chord:].reshape(rows + 1, cols)) for w in want_k)
    want_g = mk[:, :-1] - mk[:, 1:] - sk[:-1] + sk[1:]
    if n is None:
        assert np.all(np.abs(gb - want_g) <= 4 * EPS * (mc[:, :-1] + mc[:, 1:] + sc[:-1] + sc[1:]))
    else:
        assert _err(gb, want_g) <= tol
