"""One launch for several parts of a step: cases with a free and with a prescribed wake in one
batch (the shed wake and the force targets of all of them then come after the free wake's
velocities), against each alone.  And captured FP64 batches whose cases change, each with a
factorisation and a solve of its own cluster size.  FP64 1e-12, mixed 1e-6, as in
test_gpu_batch."""
from __future__ import annotations

from dataclasses import replace

import pytest

from flapjax_b200 import cases
from tests.helpers import device_uvlm, rel_err
from tests.test_gpu_batch import FIELDS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-6)])
def test_free_and_prescribed_wakes_in_one_batch(cuda, precision, tol):
    from flapjax_b200.serving import BatchStepper

    mix = [replace(cases.wing_free(m=4, n=10, m_star=12, n_steps=4, alpha_deg=3.0, seed=1), free_wake=False),
           cases.wing_free(m=3, n=8, m_star=6, n_steps=4, seed=4),
           replace(cases.wing_free(m=1, n=1, m_star=1, n_steps=4, seed=2), free_wake=False)]
    alone, uvs, dcs = [], [], []
    for c in mix:
        uv, _ = device_uvlm(c, precision)
        alone.append(uv.solve_prescribed_dynamic(uv.solve_static(), c.hg_t, c.hg_dot_t))
        uv, _ = device_uvlm(c, precision)
        dc = uv.make_device_case(c.n_tstep)
        uv.load_initial(dc, uv.solve_static())
        dc.set_hg(c.hg_t, c.hg_dot_t)
        uvs.append(uv)
        dcs.append(dc)
    st = BatchStepper(4, cuda)
    for i in range(1, mix[0].n_tstep):
        st.step(dcs, [i] * 3, [i > 1] * 3)
    for uv, dc, want in zip(uvs, dcs, alone):
        got = uv._to_case(dc)
        for f in FIELDS:
            for a, b in zip(getattr(got, f), getattr(want, f)):
                assert rel_err(a, b) < tol, (f, rel_err(a, b))


def test_captured_fp64_batches_of_changing_orders(cuda):
    from flapjax_b200.serving import BatchStepper

    sizes = [(4, 10), (8, 40), (6, 90), (3, 7), (9, 70)]
    mix = [cases.wing_heave(m=m, n=n, m_star=6, n_steps=4, alpha_deg=3.0, seed=k) for k, (m, n) in enumerate(sizes)]
    alone, uvs, dcs = [], [], []
    for c in mix:
        uv, _ = device_uvlm(c, "fp64")
        alone.append(uv.solve_prescribed_dynamic(uv.solve_static(), c.hg_t, c.hg_dot_t))
        uv, _ = device_uvlm(c, "fp64")
        dc = uv.make_device_case(c.n_tstep)
        uv.load_initial(dc, uv.solve_static())
        dc.set_hg(c.hg_t, c.hg_dot_t)
        uvs.append(uv)
        dcs.append(dc)
    st = BatchStepper(2, cuda)
    for i in range(1, mix[0].n_tstep):
        for pair in ((0, 1), (2, 3), (4,)):  # two cases, then two of other orders, then one
            st.step([dcs[q] for q in pair], [i] * len(pair), [i > 1] * len(pair))
    for uv, dc, want in zip(uvs, dcs, alone):
        got = uv._to_case(dc)
        for f in FIELDS:
            for a, b in zip(getattr(got, f), getattr(want, f)):
                assert rel_err(a, b) < 1e-12, (f, rel_err(a, b))
