"""A device case's outputs in one allocation: a slot written and read back as a whole, field by
field, in part and with fields that are empty (no wake), each value in its place."""
from __future__ import annotations

import numpy as np
import pytest

from flapjax_b200 import cases
from tests.helpers import device_uvlm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m_star", [0, 3])
@pytest.mark.parametrize("n_tstep", [1, 2, 5])
def test_slots(cuda, n_tstep, m_star):
    import torch

    from flapjax_b200.runtime import FIELDS

    c = cases.wing_heave(m=3, n=5, m_star=m_star, n_steps=2)
    uv, _ = device_uvlm(c, "fp64")
    dc = uv.make_device_case(n_tstep)
    rng = np.random.default_rng(n_tstep)
    want = {k: np.zeros(tuple(dc.arrays[k].shape)) for k in FIELDS}
    want.update(t=np.zeros(n_tstep), force_total=np.zeros((n_tstep, 3)))
    for slot in list(range(n_tstep)) + [0, -1]:
        vals = {k: rng.normal(size=want[k].shape[1]) for k in FIELDS}
        t, ft = rng.normal(), rng.normal(size=3)
        dc.load_slot(slot, vals, t, ft)
        for k in FIELDS:
            want[k][slot] = vals[k]
        want["t"][slot], want["force_total"][slot] = t, ft
    part = {"gamma_b": rng.normal(size=want["gamma_b"].shape[1])}  # one field: the others stay
    dc.load_slot(0, part, 2.0)
    want["gamma_b"][0], want["t"][0] = part["gamma_b"], 2.0
    for slots in (None, slice(0, 1), slice(n_tstep - 1, n_tstep), slice(None, None, 2), [0], slice(1, 1)):
        got = dc.host_arrays(slots)
        for k, a in want.items():
            assert np.array_equal(got[k], a[slice(None) if slots is None else slots]), (k, slots)
    for k, a in dc.arrays.items():
        assert a.is_contiguous() and (a.numel() == 0 or a.data_ptr() % 512 == 0)
    assert torch.equal(dc.t.cpu(), torch.from_numpy(want["t"]))
