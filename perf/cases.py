"""Workloads that users of the library run, through its public entry points.

A case is a dict of plain values; ``prepare`` builds what a user's program holds before the
call (wings, motions, flows, device cases) from the seed alone, ``run`` makes the call, and
``exact`` gives the same results from a plain FP64 PyTorch restatement of the method.

Wings have chord 1 and a span of 8 in a stream of speed 1; the angle of attack, twist,
camber, amplitudes and gusts are drawn from the seed.  The time step is one chordwise panel.
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.utils.checkpoint

CHORD, SPAN, RHO, RELAX = 1.0, 8.0, 1.225, 0.7
EPS = 1e-7
FIELDS = ("zeta_b", "zeta_b_dot", "zeta_w", "c", "n", "gamma_b", "gamma_b_dot", "gamma_w", "f_steady", "f_unsteady",
          "alpha")
SERVED = ("gamma_b", "gamma_b_dot", "f_steady", "f_unsteady")  # what the serving loop's clients read back
FIRST_SLOTS = {"stream": 2, "serve": 2}


# --------------------------------------------------------------------------------------
# The cases
# --------------------------------------------------------------------------------------
def listed():
    return [
        # One call of a fluid-structure iteration: the beam hands new node frames to
        # case_solve and reads the loads back.  Small wing, free wake, 1-cos gust: latency.
        dict(name="fsi_iterate_4x8", kind="fsi", m=4, n=8, w=20, kernel="cutoff", free=True, precision="fp64",
             motion="heave"),
        # The static solution of a wing and tail mirrored at the symmetry plane (ragged
        # sizes): the start of every study.
        dict(name="static_wing_tail_7x45", kind="static", m=7, n=45, w=83, m2=5, n2=19, kernel="epsilon",
             precision="fp64", mirror=True),
        # A heaving wing over 50 steps from the static solution, in both precisions: the
        # small prescribed-motion run of a parameter study, host arrays in and out.
        dict(name="heave_8x32_mixed", kind="run", m=8, n=32, w=64, steps=50, kernel="epsilon", free=False,
             precision="mixed", motion="heave"),
        dict(name="heave_8x32_fp64", kind="run", m=8, n=32, w=64, steps=50, kernel="epsilon", free=False,
             precision="fp64", motion="heave"),
        # A pitching, twisted wing of ordinary size, state kept on the device.
        dict(name="pitch_12x64_mixed", kind="device", m=12, n=64, w=100, steps=100, kernel="epsilon", free=False,
             precision="mixed", motion="pitch"),
        dict(name="pitch_12x64_fp64", kind="device", m=12, n=64, w=100, steps=40, kernel="epsilon", free=False,
             precision="fp64", motion="pitch"),
        # The benchmark's wing: 16 x 128 with a free wake of 200 rows.  Mixed: one chunk of a
        # streaming run of the wing in heave (the factors are kept from the first step);
        # FP64: the first steps of the wing at rest, the factorisation included.
        dict(name="free_16x128_mixed", kind="stream", m=16, n=128, w=200, steps=8, kernel="cutoff", free=True,
             precision="mixed", motion="heave"),
        dict(name="free_16x128_fp64", kind="device", m=16, n=128, w=200, steps=3, kernel="cutoff", free=True,
             precision="fp64", motion="none"),
        # Continuous batching: 16 heaving wings of uneven size, four batched steps.
        dict(name="serve_16_mixed", kind="serve", batch=16, sizes=1, steps=4, kernel="epsilon", free=False,
             precision="mixed", motion="heave"),
        # The gradient of a time-mean force with respect to the lattice (forward, recomputed
        # segments, reverse sweep).
        dict(name="gradient_12x64", kind="gradient", m=12, n=64, w=100, steps=6, kernel="epsilon", free=False,
             precision="fp64", motion="pitch"),
        # The linearised model about a static solution and a march of it.
        dict(name="linear_8x32", kind="linear", m=8, n=32, w=64, steps=200, kernel="epsilon", precision="fp64"),
        # The velocity induced by a wake at scattered points and its reverse mode, the seam
        # that other programs bind to.
        dict(name="induced_velocity_grad", kind="velocity", m=75, n=93, targets=2531, kernel="cutoff",
             precision="fp64"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("fsi", "static", "run", "run", "device", "device", "stream", "serve", "gradient", "linear",
                       "velocity"))
    precision = rng.choice(("fp64", "mixed"))
    m, n, w = rng.randint(4, 12), _log_int(rng, 12, 72), _log_int(rng, 16, 120)
    if kind == "fsi":
        return dict(kind=kind, m=rng.randint(3, 8), n=_log_int(rng, 6, 40), w=_log_int(rng, 8, 60), kernel="cutoff",
                    free=rng.random() < 0.7, precision=precision, motion="heave")
    if kind == "static":
        return dict(kind=kind, m=m, n=n, w=w, m2=rng.randint(2, 6), n2=rng.randint(6, 24),
                    kernel=rng.choice(("epsilon", "cutoff")), precision="fp64", mirror=rng.random() < 0.5)
    if kind in ("run", "device"):
        free = rng.random() < 0.4
        return dict(kind=kind, m=m, n=n, w=w, steps=rng.randint(3, 8) if free else rng.randint(6, 60),
                    kernel="cutoff" if free else "epsilon", free=free, precision=precision,
                    motion=rng.choice(("heave", "pitch")))
    if kind == "stream":
        return dict(kind=kind, m=rng.randint(8, 16), n=_log_int(rng, 40, 128), w=_log_int(rng, 60, 200),
                    steps=rng.randint(3, 8), kernel="cutoff", free=True, precision="mixed", motion="heave")
    if kind == "serve":
        return dict(kind=kind, batch=rng.randint(4, 16), sizes=rng.randint(2, 10**6), steps=rng.randint(2, 4),
                    kernel="epsilon", free=False, precision="mixed", motion="heave")
    if kind == "gradient":
        return dict(kind=kind, m=rng.randint(4, 12), n=_log_int(rng, 12, 64), w=_log_int(rng, 16, 100),
                    steps=rng.randint(3, 6), kernel="epsilon", free=False, precision="fp64", motion="pitch")
    if kind == "linear":
        return dict(kind=kind, m=rng.randint(4, 8), n=_log_int(rng, 10, 36), w=_log_int(rng, 16, 72),
                    steps=rng.randint(50, 200), kernel="epsilon", precision="fp64")
    return dict(kind=kind, m=_log_int(rng, 8, 120), n=_log_int(rng, 8, 120), targets=_log_int(rng, 200, 4000),
                kernel=rng.choice(("epsilon", "cutoff")), precision="fp64")


def _wings(case, seed):
    """The (m, n, w) of every wing of the case; a serving batch draws its own."""
    if case["kind"] != "serve":
        return [(case["m"], case["n"], case["w"])]
    rng = np.random.default_rng(case["sizes"])
    return [(int(rng.integers(4, 17)), int(rng.integers(16, 129)), int(rng.integers(20, 201)))
            for _ in range(case["batch"])]


# --------------------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------------------
def _frames(n_nodes, span):
    hg = np.zeros((n_nodes, 4, 4))
    hg[:, :3, :3] = np.eye(3)
    hg[:, 1, 3] = np.linspace(0.0, span, n_nodes)
    hg[:, 3, 3] = 1.0
    return hg


def _grid(m, n, chord, twist, camber):
    """Cambered section twisted per spanwise station about the quarter chord."""
    xc = np.linspace(0.0, 1.0, m + 1)
    x, z = (xc - 0.25) * chord, np.where(xc < 0.4, camber / 0.16 * (0.8 * xc - xc**2),
                                         camber / 0.36 * (0.2 + 0.8 * xc - xc**2)) * chord
    c, s = np.cos(twist), np.sin(twist)
    g = np.zeros((m + 1, n + 1, 3))
    g[..., 0] = x[:, None] * c + z[:, None] * s
    g[..., 2] = -x[:, None] * s + z[:, None] * c
    return g


def _motion(hg0, motion, steps, dt, rng):
    t = np.arange(steps + 1) * dt
    hg, hgd = np.repeat(hg0[None], steps + 1, axis=0), np.zeros((steps + 1,) + hg0.shape)
    if motion == "heave":
        a, om = rng.uniform(0.03, 0.08), rng.uniform(0.3, 0.6)
        hg[:, :, 2, 3] += (a * np.sin(om * t))[:, None]
        hgd[:, :, 2, 3] = (a * om * np.cos(om * t))[:, None]
    elif motion == "pitch":
        a, om = np.deg2rad(rng.uniform(1.0, 3.0)), rng.uniform(0.4, 0.8)
        th, thd = a * np.sin(om * t), a * om * np.cos(om * t)
        hg[:, :, 0, 0] = hg[:, :, 2, 2] = np.cos(th)[:, None]
        hg[:, :, 0, 2] = np.sin(th)[:, None]
        hg[:, :, 2, 0] = -np.sin(th)[:, None]
        hgd[:, :, 0, 2], hgd[:, :, 2, 0] = thd[:, None], -thd[:, None]
    return hg, hgd


def _setup(case, m, n, w, rng):
    """One wing (and tail): every number the solver is configured with."""
    alpha = np.deg2rad(rng.uniform(1.0, 7.0))
    twist = np.deg2rad(rng.uniform(-3.0, 3.0)) * np.linspace(0.0, 1.0, n + 1) + np.deg2rad(
        rng.normal(0.0, 0.3, n + 1))
    s = dict(dims=[(m, n, w)], zeta0=[_grid(m, n, CHORD, twist, rng.uniform(0.0, 0.04))], dof=[np.arange(n + 1)],
             hg0=_frames(n + 1, SPAN), dt=CHORD / m, u_inf=np.array((np.cos(alpha), 0.0, np.sin(alpha))), gust=None,
             mirror=bool(case.get("mirror")), kernel=case["kernel"], r_cut=1e-3, free=bool(case.get("free")),
             precision=case["precision"])
    if case.get("m2"):
        m2, n2 = case["m2"], case["n2"]
        tail = _frames(n2 + 1, 0.4 * SPAN)
        tail[:, 0, 3], tail[:, 2, 3] = 4.0, 0.5
        s["dims"].append((m2, n2, w))
        s["zeta0"].append(_grid(m2, n2, 0.6 * CHORD, np.deg2rad(rng.uniform(-2.0, 2.0)) * np.ones(n2 + 1), 0.0))
        s["dof"].append(n + 1 + np.arange(n2 + 1))
        s["hg0"] = np.concatenate([s["hg0"], tail])
    steps = {"fsi": 2, "static": 0, "linear": 0}.get(case["kind"], case.get("steps", 0) + FIRST_SLOTS.get(case["kind"], 1) - 1)
    s["hg"], s["hgd"] = _motion(s["hg0"], case.get("motion", "none"), steps, s["dt"], rng)
    if case["kind"] == "fsi":
        s["gust"] = dict(gust_length=5.0, gust_amplitude=rng.uniform(0.03, 0.08), gust_x0=np.array((-2.0, 0.0, 0.0)))
        s["hg"][2, :, 2, 3] += 1e-3 * rng.normal(size=s["hg0"].shape[0]).cumsum()  # the beam's deflection
    return s


def _setups(case, seed):
    rng = np.random.default_rng([seed, 17])
    return [_setup(case, m, n, w, rng) for m, n, w in _wings(case, seed)]


def _solver(s):
    import flapjax_b200 as fj

    kernel = fj.cutoff_kernel(s["r_cut"]) if s["kernel"] == "cutoff" else fj.biot_savart_epsilon
    more = dict(mirror_point=np.zeros(3), mirror_normal=np.array((0.0, 1.0, 0.0))) if s["mirror"] else {}
    uv = fj.UVLM([fj.GridDiscretisation(*d) for d in s["dims"]], s["dof"], kernel=kernel, free_wake=s["free"],
                 precision=s["precision"], gamma_dot_relaxation=RELAX, **more)
    flow = (fj.Constant(s["u_inf"], RHO, True) if s["gust"] is None
            else fj.OneMinusCosine(s["u_inf"], RHO, True, **s["gust"]))
    uv.set_design_variables(dt=s["dt"], flowfield=flow, zeta_b0=s["zeta0"], hg0=s["hg0"])
    return uv


def _device_case(uv, s, slots):
    dc = uv.make_device_case(slots)
    uv.load_initial(dc, uv.solve_static())
    dc.set_hg(s["hg"], s["hgd"])
    return dc


def _velocity_inputs(case, seed):
    """A rolled-up wake sheet of m x n panels and points around it."""
    rng = np.random.default_rng([seed, 29])
    m, n = case["m"], case["n"]
    x, y = np.meshgrid(np.linspace(0.0, 8.0, m + 1), np.linspace(0.0, SPAN, n + 1), indexing="ij")
    z = np.stack([x, y, 0.2 * np.sin(0.7 * x + rng.uniform(0, 6)) * (y / SPAN) ** 2], -1)
    z += 0.1 * SPAN / max(m, n) * rng.uniform(-1, 1, z.shape)
    g = (1.0 - (np.linspace(-1, 1, n)[None] * 0.95) ** 2) ** 0.5 * (1.0 + 0.2 * rng.normal(size=(m, n)))
    t = rng.uniform((-1.0, 0.0, -1.0), (9.0, SPAN, 1.0), (case["targets"], 3))
    return z, g, t, rng.normal(size=t.shape)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "velocity":
        z, g, t, vb = (torch.from_numpy(a).cuda() for a in _velocity_inputs(case, seed))
        return dict(kind=kind, x=t.requires_grad_(), z=z.requires_grad_(), g=g.requires_grad_(), v_bar=vb,
                    kernel=0 if case["kernel"] == "epsilon" else 1)
    ss = _setups(case, seed)
    s = ss[0]
    st = dict(kind=kind, steps=case.get("steps", 0))
    if kind == "serve":
        from flapjax_b200.serving import BatchStepper

        st["cases"] = [_device_case(_solver(q), q, q["hg"].shape[0]) for q in ss]
        for dc in st["cases"]:
            dc.solve_dynamic(1, 2)
        st["stepper"] = BatchStepper(len(ss))
        return st
    uv = st["uv"] = _solver(s)
    if kind in ("device", "stream"):
        st["dc"] = _device_case(uv, s, s["hg"].shape[0])
        if kind == "stream":
            st["dc"].solve_dynamic(1, 2)
    elif kind in ("run", "linear"):
        st["init"] = uv.solve_static()
        st["hg"], st["hgd"] = s["hg"], s["hgd"]
        if kind == "linear":
            rng = np.random.default_rng([seed, 31])
            from flapjax_b200.linear import LinearUVLM

            k = LinearUVLM(uv, st["init"], "frozen", skip_linearisation=True).n_inputs
            st["u"] = torch.from_numpy(1e-3 * rng.normal(size=(case["steps"] + 1, k))).cuda()
    elif kind == "fsi":
        st["case"] = uv.solve_prescribed_dynamic(uv.solve_static(), s["hg"], s["hgd"])
        st["frames"] = (s["hg"][2], s["hg"][1], s["hgd"][2])
    elif kind == "gradient":
        from flapjax_b200.adjoint import PrescribedAdjoint

        st["adjoint"] = PrescribedAdjoint(uv)
        st["hg"], st["hgd"], st["weights"] = s["hg"], s["hgd"], _weights(case, s)
    return st


def _weights(case, s):
    lift = np.array((-s["u_inf"][2], 0.0, s["u_inf"][0]))
    return np.repeat((lift / (0.5 * RHO * CHORD * SPAN * case["steps"]))[None], case["steps"] + 1, axis=0)


# --------------------------------------------------------------------------------------
# The calls
# --------------------------------------------------------------------------------------
def _case_outputs(c):
    out = {k: list(getattr(c, "nc" if k == "n" else k)) for k in FIELDS}
    out["force_total"] = c.force_total
    return out


def _device_outputs(dc, first):
    out = {k: dc.arrays["nc" if k == "n" else k][first:] for k in FIELDS}
    out["force_total"] = dc.force_total[first:]
    return out


def run(state):
    kind = state["kind"]
    if kind == "run":
        return _case_outputs(state["uv"].solve_prescribed_dynamic(state["init"], state["hg"], state["hgd"]))
    if kind == "device":
        dc = state["dc"]
        dc.solve_dynamic(1, 1 + state["steps"])
        return _device_outputs(dc, 1)
    if kind == "stream":
        dc = state["dc"]
        dc.solve_dynamic(2, 2 + state["steps"], reuse_factors=True)
        return _device_outputs(dc, 2)
    if kind == "serve":
        cs = state["cases"]
        for i in range(2, 2 + state["steps"]):
            state["stepper"].step(cs, [i] * len(cs), [True] * len(cs))
        return [{k: dc.arrays[k][2:] for k in SERVED} for dc in cs]
    if kind == "fsi":
        hg_n, hg_nm1, hgd_n = state["frames"]
        return _case_outputs(state["uv"].case_solve(state["case"], 2, hg_n, hg_nm1, hgd_n, static=False,
                                                    horseshoe=False))
    if kind == "static":
        return _case_outputs(state["uv"].solve_static())
    if kind == "gradient":
        j, g = state["adjoint"].gradient(state["hg"], state["hgd"], state["weights"])
        return {"j": j, "zeta_b0": g}
    if kind == "linear":
        sys = state["uv"].linearise(state["init"], "frozen").sys
        x, y = sys.run(state["u"])
        return {"a": sys.a, "b": sys.b, "c": sys.c, "d": sys.d, "x": x, "y": y}
    from flapjax_b200.autograd import induced_velocity

    x, z, g = state["x"], state["z"], state["g"]
    v = induced_velocity(x, z, g, state["kernel"], 1e-3)
    return {"v": v, "bars": torch.autograd.grad(v, (x, z, g), state["v_bar"])}


# --------------------------------------------------------------------------------------
# What a pass cannot do without
# --------------------------------------------------------------------------------------
PAIR, PAIR_VJP = 70, 150  # flop per (target, filament): the sum, and its reverse mode for targets and filaments


def _step_pairs(m, n, w, free):
    nb, sb, sw = m * n, m * (n + 1) + (m + 1) * n, w * (n + 1) + (w + 1) * n
    return nb * sw + sb * (sb + sw) + (w * (n + 1) * (sb + sw) if free else 0)


def _slot_doubles(m, n, w):
    return 14 * (m + 1) * (n + 1) + 6 * m * n + 3 * (w + 1) * (n + 1) + w * n


def work(case):
    kind, k = case["kind"], case.get("steps", 1) or 1
    if kind == "velocity":
        m, n, t = case["m"], case["n"], case["targets"]
        pairs, size = t * (m * (n + 1) + (m + 1) * n), 3 * (m + 1) * (n + 1) + m * n + 6 * t
        return {"bytes": 8.0 * 3 * size, "flops": float(pairs * (PAIR + PAIR_VJP))}
    if kind == "static":
        dims = [(case["m"], case["n"], case["w"]), (case["m2"], case["n2"], case["w"])]
        img = 2 if case["mirror"] else 1
        nb = sum(m * n for m, n, _ in dims)
        sb = sum(m * (n + 1) + (m + 1) * n for m, n, _ in dims)
        sw = sum(w * (n + 1) + (w + 1) * n for m, n, w in dims)
        return {"bytes": 8.0 * sum(_slot_doubles(*d) for d in dims),
                "flops": img * (nb + sb) * (sb + sw) * PAIR + 2 / 3 * nb**3}
    flops = bytes_ = 0.0
    for m, n, w in _wings(case, 0):
        nb, sb = m * n, m * (n + 1) + (m + 1) * n
        slot = 8.0 * (_slot_doubles(m, n, w) + 32 * (n + 1))
        factor = nb * sb * PAIR + 2 / 3 * nb**3
        if kind == "linear":
            rows, cols = 2 * nb + w * n + 6 * (m + 1) * (n + 1), 2 * nb + w * n + 9 * (m + 1) * (n + 1) + 3 * (w + 1) * (n + 1)
            bytes_ += 8.0 * rows * cols
            flops += factor + 2.0 * nb * nb * cols + 2.0 * rows * cols * k
        elif kind == "gradient":
            bytes_ += slot * k
            flops += 2 * (factor + k * _step_pairs(m, n, w, False) * PAIR) + k * _step_pairs(m, n, w, False) * PAIR_VJP
        else:
            bytes_ += slot * k
            flops += (0.0 if kind in ("stream", "serve") else factor) + k * _step_pairs(m, n, w, case.get("free")) * PAIR
    return {"bytes": bytes_, "flops": flops}


# --------------------------------------------------------------------------------------
# The same results in plain FP64 PyTorch
# --------------------------------------------------------------------------------------
def _t(a):
    return torch.as_tensor(np.asarray(a), dtype=torch.float64, device="cuda" if torch.cuda.is_available() else "cpu")


def _cross(a, b):
    return [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]]


def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _segment(x, y0, y1, kernel, r_cut):
    """Unit-strength velocities (three (T, F) tensors) of segments y0 -> y1 at points x."""
    r1 = [x[:, None, d] - y0[None, :, d] for d in range(3)]
    r2 = [x[:, None, d] - y1[None, :, d] for d in range(3)]
    r0 = [(y1 - y0)[None, :, d] for d in range(3)]
    n1, n2 = torch.sqrt(_dot(r1, r1) + EPS**2), torch.sqrt(_dot(r2, r2) + EPS**2)
    c = _cross(r1, r2)
    dot = _dot(r0, [a / n1 - b / n2 for a, b in zip(r1, r2)])
    c2, r0sq = _dot(c, c), _dot(r0, r0)
    if kernel == "epsilon":
        k = dot / (4 * math.pi * (c2 + EPS * r0sq * r0sq))
    else:
        s = _dot(r0, r1) / r0sq
        away = [a - s * b for a, b in zip(r1, r0)]
        far = _dot(away, away) > r_cut**2
        k = torch.where(far, dot / (4 * math.pi * torch.where(far, c2, torch.ones_like(c2))), torch.zeros_like(c2))
    return [a * k for a in c]


def _filaments(lats, mirror):
    y0, y1, gs = [], [], []
    for z, g in lats:
        gc = torch.nn.functional.pad(g, (0, 1)) - torch.nn.functional.pad(g, (1, 0))
        gs_ = torch.nn.functional.pad(g, (0, 0, 1, 0)) - torch.nn.functional.pad(g, (0, 0, 0, 1))
        strength = torch.cat([gc.reshape(-1), gs_.reshape(-1)])
        for sign in (1.0, -1.0) if mirror else (1.0,):
            zz = z if sign > 0 else z * _t((1.0, -1.0, 1.0))
            y0 += [zz[:-1].reshape(-1, 3), zz[:, :-1].reshape(-1, 3)]
            y1 += [zz[1:].reshape(-1, 3), zz[:, 1:].reshape(-1, 3)]
            gs.append(sign * strength)
    return torch.cat(y0), torch.cat(y1), torch.cat(gs)


def _velocity(x, lats, s):
    y0, y1, g = _filaments([q for q in lats if q[1].numel()], s["mirror"])

    def part(xp, y0, y1, g):
        return torch.stack([q @ g for q in _segment(xp, y0, y1, s["kernel"], s["r_cut"])], -1)

    step = max(1, 6_000_000 // max(1, y0.shape[0]))
    grad = torch.is_grad_enabled()
    return torch.cat([torch.utils.checkpoint.checkpoint(part, xp, y0, y1, g, use_reentrant=False) if grad
                      else part(xp, y0, y1, g) for xp in x.split(step)])


def _rings(x, nrm, z, s):
    """Normal velocity of unit rings of lattice z at points x: (T, R, C)."""
    out = 0.0
    for sign in (1.0, -1.0) if s["mirror"] else (1.0,):
        zz = z if sign > 0 else z * _t((1.0, -1.0, 1.0))
        fam = []
        for a, b in ((zz[:-1], zz[1:]), (zz[:, :-1], zz[:, 1:])):
            v = _segment(x, a.reshape(-1, 3), b.reshape(-1, 3), s["kernel"], s["r_cut"])
            fam.append(sum(q * nrm[:, None, d] for d, q in enumerate(v)).reshape((-1,) + a.shape[:2]))
        ch, sp = fam
        out = out + sign * (ch[:, :, :-1] - ch[:, :, 1:] + sp[:, 1:] - sp[:, :-1])
    return out


def _flow(s, x, t):
    u = _t(s["u_inf"])
    if s["gust"] is None:
        return u.expand_as(x)
    q = s["gust"]
    g = (x - _t(q["gust_x0"]) - u * t) @ u
    w = 0.5 * q["gust_amplitude"] * (1.0 - torch.cos(math.pi * g / q["gust_length"]))
    return u + torch.where((g > 0) & (g < 2 * q["gust_length"]), w, torch.zeros_like(w))[..., None] * _t((0.0, 0.0, 1.0))


def _cat(v):
    return torch.cat([a.reshape(-1, 3) if a.shape[-1:] == (3,) else a.reshape(-1) for a in v])


def _split(flat, like):
    out, o = [], 0
    for a in like:
        k = a.shape[0] * a.shape[1]
        out.append(flat[o:o + k].reshape(a.shape[:2] + flat.shape[1:]))
        o += k
    return out


def _mean4(z):
    return 0.25 * (z[:-1, :-1] + z[1:, :-1] + z[:-1, 1:] + z[1:, 1:])


def _place(s, zeta0, hg):
    return [torch.einsum("jkl,ijl->ijk", hg[d][:, :3, :3], z) + hg[d][None, :, :3, 3] for z, d in zip(zeta0, s["dof"])]


def _solve(s, q, prev, t):
    """Circulations, forces and strip incidence of one slot; ``q`` holds its lattices (and,
    for a dynamic step, its wake); ``prev`` is the slot before (None: static)."""
    q["c"] = [_mean4(z) for z in q["zeta_b"]]
    q["n"] = [torch.linalg.cross(z[1:, 1:] - z[:-1, :-1], z[1:, :-1] - z[:-1, 1:]) for z in q["zeta_b"]]
    c, nrm = _cat(q["c"]), _cat(q["n"])
    blocks = []
    for k, z in enumerate(q["zeta_b"]):
        a = _rings(c, nrm, z, s)
        if prev is None and q["zeta_w"][k].shape[0] > 1:
            a = torch.cat([a[:, :-1], a[:, -1:] + _wake_rows(c, nrm, q["zeta_w"][k], s)[:, None]], 1)
        blocks.append(a.reshape(c.shape[0], -1))
    u = _flow(s, c, t)
    if prev is not None:
        u = u - _cat([_mean4(z) for z in q["zeta_b_dot"]]) + _velocity(c, list(zip(q["zeta_w"], q["gamma_w"])), s)
    gb = torch.linalg.solve(torch.cat(blocks, 1), -(u * nrm).sum(-1))
    q["gamma_b"] = _split(gb, q["c"])
    if prev is None:
        q["gamma_w"] = [g[-1:].expand(d[2], -1) for g, d in zip(q["gamma_b"], s["dims"])]
    lats = list(zip(q["zeta_w"], q["gamma_w"])) + list(zip(q["zeta_b"], q["gamma_b"]))
    mids = [m for z in q["zeta_b"] for m in (0.5 * (z[:-1] + z[1:]), 0.5 * (z[:, :-1] + z[:, 1:]))]
    v = _split(_velocity(_cat(mids), lats, s), mids)
    pad = torch.nn.functional.pad
    q["f_steady"], q["f_unsteady"], q["alpha"], q["gamma_b_dot"] = [], [], [], []
    for k, (z, zd, g, gw) in enumerate(zip(q["zeta_b"], q["zeta_b_dot"], q["gamma_b"], q["gamma_w"])):
        gc = pad(g, (0, 1)) - pad(g, (1, 0))
        gs = pad(g, (0, 0, 1, 0)) - pad(g, (0, 0, 0, 1))
        if gw.shape[0]:
            gs = gs - pad(gw[:1], (0, 0, z.shape[0] - 1, 0))
        fc = RHO * gc[..., None] * torch.linalg.cross(_flow(s, mids[2 * k], t) + v[2 * k] - 0.5 * (zd[:-1] + zd[1:]),
                                                      z[1:] - z[:-1])
        fs = RHO * gs[..., None] * torch.linalg.cross(
            _flow(s, mids[2 * k + 1], t) + v[2 * k + 1] - 0.5 * (zd[:, :-1] + zd[:, 1:]), z[:, 1:] - z[:, :-1])
        steady = 0.5 * (pad(fc, (0, 0, 0, 0, 0, 1)) + pad(fc, (0, 0, 0, 0, 1, 0)) + pad(fs, (0, 0, 0, 1))
                        + pad(fs, (0, 0, 1, 0)))
        if prev is None:
            gd = torch.zeros_like(g)
        else:
            gd = RELAX * (g - prev["gamma_b"][k]) / s["dt"] + (1.0 - RELAX) * prev["gamma_b_dot"][k]
        fu = 0.25 * RHO * gd[..., None] * q["n"][k]
        unsteady = (pad(fu, (0, 0, 0, 1, 0, 1)) + pad(fu, (0, 0, 1, 0, 0, 1)) + pad(fu, (0, 0, 0, 1, 1, 0))
                    + pad(fu, (0, 0, 1, 0, 1, 0)))
        le, te = 0.5 * (z[0, :-1] + z[0, 1:]), 0.5 * (z[-1, :-1] + z[-1, 1:])
        sp = 0.5 * (z[0, 1:] + z[-1, 1:] - z[0, :-1] - z[-1, :-1])
        vr, b = _flow(s, 0.5 * (le + te), t), sp.norm(dim=-1)
        el = torch.linalg.cross(vr, sp / b[:, None])
        el = el / el.norm(dim=-1, keepdim=True)
        cl = ((0.5 * (steady[:, :-1] + steady[:, 1:])).sum(0) * el).sum(-1) / (
            0.5 * RHO * (vr * vr).sum(-1) * (te - le).norm(dim=-1) * b)
        q["f_steady"].append(steady)
        q["f_unsteady"].append(unsteady)
        q["alpha"].append(cl / (2 * math.pi))
        q["gamma_b_dot"].append(gd)
    q["force_total"] = sum((a + b).sum((0, 1)) for a, b in zip(q["f_steady"], q["f_unsteady"]))
    return q


def _wake_rows(c, nrm, zw, s):
    """The wake rings of each spanwise strip, summed over the wake rows: (T, C)."""
    rows = max(1, 20_000_000 // max(1, c.shape[0] * zw.shape[1]))
    return sum(_rings(c, nrm, zw[r:r + rows + 1], s).sum(1) for r in range(0, zw.shape[0] - 1, rows))


def _slots(s, steps, zeta0=None):
    """Slot 0 (static) and ``steps`` dynamic slots."""
    zeta0 = [_t(z) for z in s["zeta0"]] if zeta0 is None else zeta0
    hg, hgd, u, dt = _t(s["hg"]), _t(s["hgd"]), _t(s["u_inf"]), s["dt"]
    zb = _place(s, zeta0, _t(s["hg0"]))
    rows = [torch.arange(d[2] + 1, dtype=torch.float64, device=u.device)[:, None, None] * dt * u for d in s["dims"]]
    out = [_solve(s, dict(zeta_b=zb, zeta_b_dot=[torch.zeros_like(z) for z in zb],
                          zeta_w=[z[-1:] + r for z, r in zip(zb, rows)]), None, 0.0)]
    for i in range(1, steps + 1):
        p, t = out[-1], i * dt
        q = dict(zeta_b=_place(s, zeta0, hg[i]),
                 zeta_b_dot=[torch.einsum("jkl,ijl->ijk", hgd[i][d][:, :3, :3], z) + hgd[i][d][None, :, :3, 3]
                             for z, d in zip(zeta0, s["dof"])])
        move = [_flow(s, z[:-1], t) for z in p["zeta_w"]]
        if s["free"]:
            lats = list(zip(_place(s, zeta0, hg[i - 1]), p["gamma_b"])) + list(zip(p["zeta_w"], p["gamma_w"]))
            v = _split(_velocity(_cat([z[:-1] for z in p["zeta_w"]]), lats, s), move)
            move = [a + b for a, b in zip(move, v)]
        q["zeta_w"] = [torch.cat([z[-1:], zw[:-1] + dt * a]) for z, zw, a in zip(q["zeta_b"], p["zeta_w"], move)]
        q["gamma_w"] = [torch.cat([g[-1:], gw[:-1]]) for g, gw in zip(p["gamma_b"], p["gamma_w"])]
        out.append(_solve(s, q, p, t))
    return out


def _flat(slots, k):
    return torch.stack([torch.cat([a.reshape(-1) for a in q[k]]) for q in slots])


def exact(case, seed):
    kind = case["kind"]
    if kind == "linear":
        return None
    if kind == "velocity":
        z, g, x, vb = (_t(a) for a in _velocity_inputs(case, seed))
        for a in (x, z, g):
            a.requires_grad_()
        v = _velocity(x, [(z, g)], dict(mirror=False, kernel=case["kernel"], r_cut=1e-3))
        return {"v": v.detach(), "bars": torch.autograd.grad(v, (x, z, g), vb)}
    ss = _setups(case, seed)
    s = ss[0]
    if kind == "gradient":
        zeta0 = [_t(z).requires_grad_() for z in s["zeta0"]]
        w = _t(_weights(case, s))
        j = sum((w[i] * q["force_total"]).sum() for i, q in enumerate(_slots(s, case["steps"], zeta0)) if i)
        return {"j": float(j), "zeta_b0": torch.autograd.grad(j, zeta0)[0]}
    with torch.no_grad():
        if kind == "serve":
            out = [_slots(q, q["hg"].shape[0] - 1)[2:] for q in ss]
            return [{k: _flat(v, k) for k in SERVED} for v in out]
        slots = _slots(s, s["hg"].shape[0] - 1)
        if kind in ("device", "stream"):
            slots = slots[FIRST_SLOTS.get(kind, 1):]
            out = {k: _flat(slots, k) for k in FIELDS}
        elif kind == "static":
            return {**{k: [a for a in slots[0][k]] for k in FIELDS}, "force_total": slots[0]["force_total"]}
        else:
            out = {k: [torch.stack([q[k][i] for q in slots]) for i in range(len(s["dims"]))] for k in FIELDS}
        out["force_total"] = torch.stack([q["force_total"] for q in slots])
        return out
