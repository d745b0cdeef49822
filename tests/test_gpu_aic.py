"""The influence matrix at the edges of its tiles: odd numbers of rows, one ring, strips wider
than a CTA, wakes of one row and of more rows than parts, images, all kernels, and surfaces whose
filaments leave room for one target only.  A ring is four filaments of some 20 roundings each
and a lumped strip a sum of W: 1e-13 (500 eps) of the largest entries' norm."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import uvlm_ref as R
from tests.helpers import rel_err
from tests.test_gpu_parity import _fj_aic

pytestmark = pytest.mark.gpu
MIRROR = (np.array([0.0, -0.5, 0.0]), np.array([0.0, 1.0, 0.0]))


@pytest.mark.parametrize("kernel", ["epsilon", "cutoff", "plain"])
@pytest.mark.parametrize("dims,wake,mirror", [([(1, 1)], None, False), ([(1, 1)], 1, True), ([(3, 5), (2, 7)], 9, False),
                                              ([(1, 261)], 3, False), ([(5, 43), (1, 2)], 40, True),
                                              ([(2, 700)], 2, True)])
def test_influence(cuda, dims, wake, mirror, kernel):
    from flapjax_b200 import _lib

    rng = np.random.default_rng(len(dims) + dims[0][1])
    zs, zw = [], []
    for q, (m, n) in enumerate(dims):
        k, l = np.meshgrid(np.arange(m + 1) * 0.3, np.arange(n + 1) * 0.25, indexing="ij")
        zs.append(np.stack([k + 2.0 * q, l, -0.05 * k], -1) + 0.02 * rng.normal(size=(m + 1, n + 1, 3)))
        if wake:
            zw.append(zs[q][-1] + np.arange(wake + 1)[:, None, None] * np.array([0.2, 0.01, 0.01]))
    cs, ns = [R.compute_surf_c(z) for z in zs], [R.compute_surf_nc(z) for z in zs]
    want = R.compute_aic_solve(cs, ns, zs, zw or None, kernel, MIRROR if mirror else None, 1e-3)
    ids = {"epsilon": _lib.FJ_KERNEL_EPSILON, "cutoff": _lib.FJ_KERNEL_CUTOFF, "plain": _lib.FJ_KERNEL_PLAIN}
    got = _fj_aic(cuda, zs, zw or None, ids[kernel], 1e-3, MIRROR if mirror else None)
    assert rel_err(got, want) < 1e-13
