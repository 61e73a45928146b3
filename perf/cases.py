"""What this framework is timed on: the calls that programs make of it, from one step of a small
box coupled to a host code up to the 513.9 M-node box of the benchmark.

A case is a dict of plain values; `prepare` makes what a user's program has in hand (mesh, model,
solver, network, inputs), `run` is one pass through the public entry points, `exact` the same
results in 64 bits in plain torch.  Axis convention as in the package: fields are [y][z][x], node
= ix + iz*nx + iy*nx*nz.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "proxy-geos-hc_gb300"))

import semgb  # noqa: E402

H = 10.0  # element size (m) of every box
N_IN, N_HID = 81, 64


# ---- the cases ----------------------------------------------------------------------------------

def listed():
    return [
        # A host code advances a small box one step per call, handing in that step's source sample
        # and reading that step's receivers: the smallest calls, all latency.
        dict(name="stream_q2_12", kind="stream", ex=12, ey=12, ez=12, order=2, steps=16, sponge=2, nrec=16),
        # One shot on the CPU-runnable configuration of the benchmark (40^3, order 2), with the
        # final wavefield read back: levels that stay in L2, launches that count.
        dict(name="shot_q2_40", kind="shot", ex=40, ey=40, ez=40, order=2, steps=300, sponge=10, nrec=64,
             variant="default", field=True),
        # An ordinary shot on a ragged box (sizes that divide no tile).
        dict(name="shot_q4_61x70x53", kind="shot", ex=61, ey=70, ez=53, order=4, steps=100, sponge=12, nrec=1024,
             variant="default", field=False),
        # The at-scale configuration of the benchmark: 200^3 order 4, 513.9 M nodes.
        dict(name="shot_q4_200", kind="shot", ex=200, ey=200, ez=200, order=4, steps=20, sponge=20, nrec=1024,
             variant="default", field=False),
        # The highest order the package has, on a ragged box of the size of its order-5 profile.
        dict(name="shot_q5_80x77x83", kind="shot", ex=80, ey=77, ez=83, order=5, steps=60, sponge=20, nrec=256,
             variant="default", field=False),
        # Batched shots: 64 sources on one mesh, all traces read (the 40^3 mesh of the batch profile).
        dict(name="shots64_q4_40", kind="batch", ex=40, ey=40, ez=40, order=4, steps=40, sponge=10, nrec=256,
             shots=64),
        # A batch of uneven problems (different sizes, orders 2-4, models) stepped as one group.
        dict(name="group32_8to24", kind="group", n=32, lo=8, hi=24, steps=100, nrec=64),
        # Gradient of one shot by the adjoint: forward, misfit, backward, gradient to the host (the
        # 96^3 order-3 configuration of the benchmark with fewer steps).
        dict(name="adjoint_q3_96", kind="adjoint", ex=96, ey=96, ez=96, order=3, steps=100, every=25, sponge=10,
             nrec=256),
        # A shot with the network as absorbing boundary around a 3-element sponge (86^3 order 4, the
        # size at which the benchmark reports its speed).
        dict(name="learned_q4_86", kind="learned", ex=86, ey=86, ez=86, order=4, steps=60, sponge=3, nrec=256),
        # Training the boundary network on samples: loss and gradient before, then epochs of
        # minibatches (the sample count of one teacher-forced run, the default batch of 2048).
        dict(name="train_60k", kind="train", n=60000, epochs=10, batch=2048),
        # Loss and gradient of a whole corrected run with respect to the network's parameters, through
        # the adjoint of the time loop (the training set-up: 12^3 order 4, region of interest 6^3).
        dict(name="bptt_q4_12", kind="bptt", interior=6, sponge=3, order=4, steps=100),
        # The allocation-free step on buffers that the caller owns (its own connectivity and mass
        # coefficients), in the time loop of a host code.
        dict(name="noalloc_q4_35x33x36", kind="noalloc", ex=35, ey=33, ez=36, order=4, steps=20, sponge=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["stream", "shot", "shot", "shot", "batch", "group", "adjoint", "learned", "train", "bptt",
                       "noalloc"])
    if kind == "stream":
        ex, ey, ez = (_log(rng, 4, 32) for _ in range(3))
        return dict(kind=kind, ex=ex, ey=ey, ez=ez, order=rng.choice([1, 2, 3, 4]), steps=rng.randint(4, 32),
                    sponge=rng.choice([0, 1]), nrec=_log(rng, 1, 256))
    if kind == "shot":
        order = rng.choice([1, 2, 2, 3, 3, 4, 4, 4, 5])
        nodes = math.exp(rng.uniform(math.log(2e4), math.log(3e8)))
        side = nodes ** (1.0 / 3.0) / order
        ex, ey, ez = (max(4, int(round(side * rng.uniform(0.7, 1.4)))) for _ in range(3))
        steps = max(10, min(300, int(4e9 / _nodes(ex, ey, ez, order))))
        small = _nodes(ex, ey, ez, order) < 2e6
        return dict(kind=kind, ex=ex, ey=ey, ez=ez, order=order, steps=steps,
                    sponge=rng.choice([0, 1]) * max(1, min(ex, ey, ez) // 4), nrec=_log(rng, 1, 1024),
                    variant=rng.choice(["default"] * 5 + ["reference", "difference", "element"]), field=small)
    if kind == "batch":
        order, shots = rng.choice([2, 3, 4, 5]), _log(rng, 2, 64)
        ex, ey, ez = (_log(rng, 10, 60) for _ in range(3))
        while _nodes(ex, ey, ez, order) * shots > 3e8:
            shots = max(2, shots // 2)
            ex, ey, ez = (max(6, v * 3 // 4) for v in (ex, ey, ez))
        return dict(kind=kind, ex=ex, ey=ey, ez=ez, order=order, steps=rng.randint(10, 40),
                    sponge=rng.choice([0, 2]), nrec=_log(rng, 1, 256), shots=shots)
    if kind == "group":
        lo = _log(rng, 4, 30)
        return dict(kind=kind, n=rng.randint(2, 32), lo=lo, hi=lo * 2 + rng.randint(1, 7), steps=rng.randint(20, 60),
                    nrec=_log(rng, 1, 64))
    if kind == "adjoint":
        order = rng.choice([2, 3, 4])
        ex, ey, ez = (_log(rng, 12, 240 // order) for _ in range(3))
        steps = rng.randint(40, 100)
        return dict(kind=kind, ex=ex, ey=ey, ez=ez, order=order, steps=steps, every=rng.randint(10, steps),
                    sponge=rng.choice([0, 2]), nrec=_log(rng, 4, 256))
    if kind == "learned":
        ex, ey, ez = (_log(rng, 10, 86) for _ in range(3))
        return dict(kind=kind, ex=ex, ey=ey, ez=ez, order=rng.choice([2, 3, 4]), steps=rng.randint(20, 60),
                    sponge=rng.choice([0, 3]), nrec=_log(rng, 4, 256))
    if kind == "train":
        return dict(kind=kind, n=_log(rng, 5000, 200000), epochs=rng.randint(1, 4), batch=_log(rng, 500, 8192))
    if kind == "bptt":
        return dict(kind=kind, interior=rng.randint(3, 7), sponge=rng.randint(2, 3), order=rng.choice([2, 3, 4]),
                    steps=rng.randint(40, 120))
    order = rng.choice([1, 2, 3, 4, 5])
    cap = 150 // order
    ex, ey, ez = (_log(rng, 4, cap) for _ in range(3))
    return dict(kind=kind, ex=ex, ey=ey, ez=ez, order=order, steps=rng.randint(4, 20), sponge=rng.choice([0, 1]))


# ---- bytes and operations -----------------------------------------------------------------------

def _nodes(ex, ey, ez, o):
    return (ex * o + 1) * (ey * o + 1) * (ez * o + 1)


def _step_flops(o):
    # per node: three axis rows (2o+1 entries on an element face, o+1 inside), scaling and update
    row = (2 * o + 1 + (o - 1) * (o + 1)) / o
    return 6.0 * row + 12.0


def _net_flops():
    return 2.0 * (N_IN * N_HID + N_HID * N_HID + N_HID)


def _surface(nx, ny, nz):
    return nx * ny * nz - (nx - 2) * (ny - 2) * (nz - 2)


def work(case):
    """A step reads p^n, p^{n-1} and dt^2/M once and writes p^{n+1} once: 16 bytes per node."""
    k = case["kind"]
    if k in ("stream", "shot", "noalloc", "learned", "batch", "adjoint"):
        n, o, st = _nodes(case["ex"], case["ey"], case["ez"], case["order"]), case["order"], case["steps"]
        b, f = 16.0 * n * st, _step_flops(o) * n * st
        if k == "batch":  # dt^2/M is shared by the shots
            b, f = (12.0 * case["shots"] + 4.0) * n * st, f * case["shots"]
            b += 4.0 * st * case["nrec"] * case["shots"]
        elif k == "adjoint":  # forward, recomputation and adjoint passes
            b, f = 3.0 * b + 8.0 * n, 3.0 * f
        elif k == "learned":  # three levels of the boundary's two-node shell, the network per boundary node
            s = _surface(case["ex"] * o + 1, case["ey"] * o + 1, case["ez"] * o + 1)
            b, f = b + 28.0 * s * st, f + _net_flops() * s * st
        if "nrec" in case:
            b += 4.0 * st * case["nrec"]
        return {"bytes": b, "flops": f}
    if k == "group":
        b = f = 0.0
        for ex, ey, ez, o in _members(case):
            n = _nodes(ex, ey, ez, o)
            b += 16.0 * n * case["steps"]
            f += _step_flops(o) * n * case["steps"]
        return {"bytes": b, "flops": f}
    if k == "train":  # loss and gradient once, then the epochs; no input gradient
        rows = case["n"] * (1 + case["epochs"])
        return {"bytes": 4.0 * (N_IN + 1) * rows, "flops": (2.0 * _net_flops() + 2.0 * (N_HID * N_HID + N_HID)) * rows}
    ne, o, st = case["interior"] + 2 * case["sponge"], case["order"], case["steps"]
    n, s = _nodes(ne, ne, ne, o), _surface(*[ne * o + 1] * 3)
    # forward step and its adjoint; network forward, forward again and both gradients
    return {"bytes": (2 * 16.0 * n + 2 * 28.0 * s) * st, "flops": (2 * _step_flops(o) * n + 4 * _net_flops() * s) * st}


# ---- inputs -------------------------------------------------------------------------------------

def _rng(seed, salt=0):
    return np.random.default_rng([int(seed), salt])


def _gll(o):
    from numpy.polynomial import legendre as L
    c = np.zeros(o + 1)
    c[-1] = 1.0
    xi = np.concatenate([[-1.0], np.sort(np.real(L.legroots(L.legder(c)))) if o > 1 else [], [1.0]])
    w = 2.0 / (o * (o + 1) * L.legval(xi, c) ** 2)
    d = np.array([[L.legval(xi[i], L.legder(_lagrange(xi, j))) for j in range(o + 1)] for i in range(o + 1)])
    return xi, w, d  # d[i][j] = phi_j'(xi_i)


def _lagrange(xi, j):
    """Legendre coefficients of the Lagrange polynomial of node j."""
    from numpy.polynomial import legendre as L
    return np.linalg.solve(L.legvander(xi, len(xi) - 1), np.eye(len(xi))[j])


def _velocity(rng, ex, ey, ez, lo=1500.0, hi=4500.0):
    """Five horizontal layers of random speeds times a smooth perturbation of up to 5 %."""
    v = np.sort(rng.uniform(lo, hi, 5))
    layer = np.minimum((np.arange(ez) + 0.5) / ez * 5, 4).astype(int)
    ph = rng.uniform(0, 2 * np.pi, 3)
    k = rng.uniform(0.05, 0.2, 3)
    wave = (np.sin(k[0] * np.arange(ey) + ph[0])[:, None, None] * np.sin(k[1] * np.arange(ez) + ph[1])[None, :, None]
            * np.sin(k[2] * np.arange(ex) + ph[2])[None, None, :])
    return (v[layer][None, :, None] * (1.0 + 0.05 * wave)).astype(np.float32).reshape(-1)


def _dt(o, vmax):
    return float(np.float32(0.4 * H * (_gll(o)[0][1] + 1.0) / 2.0 / vmax))


def _wavelet(rng, n, dt):
    """Ricker wavelets peaking 40 % into the run."""
    t0 = 0.4 * n * dt * rng.uniform(0.8, 1.2)
    u = (math.pi * (np.arange(n) * dt - t0) / t0) ** 2
    return ((1.0 - 2.0 * u) * np.exp(-u)).astype(np.float32)


def _sponge(ne, o, thickness, sigma=0.06):
    """Per-axis damping factors of a sponge `thickness` elements deep (float32)."""
    xi = _gll(o)[0]
    i = np.arange(ne * o + 1)
    e = np.minimum(i // o, ne - 1)
    x = e + 0.5 * (1.0 + xi[i - e * o])
    d = np.minimum(x, ne - x)
    r = np.clip((thickness - d) / max(thickness, 1), 0.0, None)
    return np.exp(-sigma * r ** 2).astype(np.float32)


def _box_inputs(case, seed):
    """Model, source, receivers and sponge of one shot on a box, as plain arrays."""
    rng = _rng(seed)
    ex, ey, ez, o, st = (case[k] for k in ("ex", "ey", "ez", "order", "steps"))
    nx, ny, nz = ex * o + 1, ey * o + 1, ez * o + 1
    vel = _velocity(rng, ex, ey, ez)
    dt = _dt(o, float(vel.max()))
    shots = case.get("shots", 1)
    mid = [max(1, v // 2) for v in (ex, ey, ez)]
    jit = [max(0, v // 6) for v in (ex, ey, ez)]
    src, nodes = [], []
    for _ in range(shots):
        e = [min(max(1, m + int(rng.integers(-j, j + 1))), max(1, v - 1)) for m, j, v in zip(mid, jit, (ex, ey, ez))]
        src.append(e[0] + e[2] * ex + e[1] * ex * ez)
    # half of the receivers around the (first) source where the wave gets in the run, half anywhere
    reach = max(2, int(min(4500.0 * dt * st / H * 0.3, max(ex, ey, ez)) * o))
    mid = [src[0] % ex, src[0] // (ex * ez), (src[0] // ex) % ez]
    for r in range(case.get("nrec", 0)):
        c = []
        for m, n in ((mid[0] * o, nx), (mid[1] * o, ny), (mid[2] * o, nz)):
            v = int(rng.integers(1, n - 1)) if r % 2 else m + int(rng.integers(-reach, reach + 1))
            c.append(min(max(1, v), n - 2))
        nodes.append(c[0] + c[2] * nx + c[1] * nx * nz)
    wav = np.stack([_wavelet(rng, st, dt) for _ in range(shots)])
    s = tuple(_sponge(n, o, case["sponge"]) for n in (ex, ey, ez)) if case["sponge"] else None
    return dict(ex=ex, ey=ey, ez=ez, o=o, steps=st, vel=vel, dt=dt, src=np.array(src, np.int64),
                rec=np.array(nodes, np.int64), wav=wav, sponge=s)


def _members(case):
    """Sizes and orders of a group's problems (the same for every seed: the work is)."""
    rng = _rng(case["n"] * 1000 + case["lo"] * 10 + case["hi"], 7)
    return [tuple(int(v) for v in rng.integers(case["lo"], case["hi"] + 1, 3)) + (int(rng.choice([2, 3, 4])),)
            for _ in range(case["n"])]


def _member_inputs(case, seed):
    return [_box_inputs(dict(ex=ex, ey=ey, ez=ez, order=o, steps=case["steps"], nrec=case["nrec"],
                             sponge=max(1, min(ex, ey, ez) // 4)), seed * 100 + i)
            for i, (ex, ey, ez, o) in enumerate(_members(case))]


def _net_params(rng, out=0.05):
    """He-normal hidden layers and a small output layer, as a network before or early in training."""
    p = np.zeros(N_HID * N_IN + N_HID + N_HID * N_HID + N_HID + N_HID + 1)
    a, b = N_HID * N_IN, N_HID * N_IN + N_HID
    p[:a] = rng.standard_normal(a) * math.sqrt(2.0 / N_IN)
    p[a:b] = rng.standard_normal(N_HID) * 0.05
    p[b:b + N_HID * N_HID] = rng.standard_normal(N_HID * N_HID) * math.sqrt(2.0 / N_HID)
    p[b + N_HID * N_HID:] = np.concatenate([rng.standard_normal(N_HID) * 0.05, rng.standard_normal(N_HID) * out,
                                            rng.standard_normal(1) * 0.01])
    return p.astype(np.float32)


def _train_inputs(case, seed):
    """Samples as the boundary gathers them: three time levels of a smooth field on a 3x3x3
    neighbourhood, divided by the largest magnitude; target: a value within it."""
    rng = _rng(seed)
    n = case["n"]
    g = np.array([-1.0, 0.0, 1.0])
    k = rng.uniform(-0.6, 0.6, (n, 3))
    ph, w = rng.uniform(0, 2 * np.pi, n), rng.uniform(0.1, 0.5, n)
    z, y, x = np.meshgrid(g, g, g, indexing="ij")
    phase = ph[:, None] + k @ np.stack([z.ravel(), y.ravel(), x.ravel()])
    f = np.concatenate([np.sin(phase - w[:, None] * l) for l in (0.0, -1.0, -2.0)], 1)
    f += 0.05 * rng.standard_normal(f.shape)
    sc = np.abs(f).max(1)
    t = np.sin(ph + w) / sc
    return dict(x=(f / sc[:, None]).astype(np.float32), t=np.clip(t, -1, 1).astype(np.float32), p=_net_params(rng))


def _bptt_inputs(case, seed):
    rng = _rng(seed)
    ne, o = case["interior"] + 2 * case["sponge"], case["order"]
    n = ne * o + 1
    lo, hi = case["sponge"] * o, (case["sponge"] + case["interior"]) * o
    i = np.arange(n)
    a = (i >= lo) & (i <= hi)
    roi = np.nonzero((a[:, None, None] & a[None, :, None] & a[None, None, :]).reshape(-1))[0]
    e = [int(rng.integers(case["sponge"], case["sponge"] + case["interior"])) for _ in range(3)]
    dt = _dt(o, 2000.0)
    b = dict(ex=ne, ey=ne, ez=ne, o=o, steps=case["steps"], vel=np.full(ne ** 3, 2000.0, np.float32), dt=dt,
             src=np.array([e[0] + e[2] * ne + e[1] * ne * ne], np.int64), rec=np.zeros(0, np.int64),
             wav=_wavelet(rng, case["steps"], dt)[None], sponge=tuple([_sponge(ne, o, case["sponge"], 0.015)] * 3))
    # the field to match: a spreading pulse of about the run's amplitude
    amp = 1e-3 * (dt * 2000.0) ** 2 * case["steps"]
    t = (np.arange(case["steps"]) + 1.0) / case["steps"]
    r = np.stack(np.unravel_index(roi, (n, n, n)), 1) / (n - 1.0) - 0.5
    rad = np.sqrt((r ** 2).sum(1))
    ref = amp * np.exp(-((rad[None] - 0.8 * t[:, None]) / 0.15) ** 2) * t[:, None]
    return b, roi, ref.astype(np.float32), _net_params(rng)


def _observed(b, rng):
    """Recorded traces for the misfit: the direct wave by straight rays at 2500 m/s."""
    o, nx, nz = b["o"], b["ex"] * b["o"] + 1, b["ez"] * b["o"] + 1
    r = b["rec"]
    pr = np.stack([r % nx, r // (nx * nz), (r // nx) % nz], 1) * (H / o)
    e = int(b["src"][0])
    ps = np.array([e % b["ex"], e // (b["ex"] * b["ez"]), (e // b["ex"]) % b["ez"]]) * H
    d = np.sqrt(((pr - ps) ** 2).sum(1)) + H
    t = np.arange(b["steps"])[:, None] * b["dt"] - d[None] / 2500.0
    t0 = 0.4 * b["steps"] * b["dt"]
    u = (math.pi * (t - t0) / t0) ** 2
    amp = (b["dt"] * 2500.0) ** 2 * b["steps"] * 1e-2
    return (amp * H / d[None] * (1.0 - 2.0 * u) * np.exp(-u) * rng.uniform(0.9, 1.1, len(r))).astype(np.float32)


def _noalloc_inputs(case, seed):
    rng = _rng(seed)
    ex, ey, ez, o = (case[k] for k in ("ex", "ey", "ez", "order"))
    nx, ny, nz = ex * o + 1, ey * o + 1, ez * o + 1
    vel = _velocity(rng, ex, ey, ez)
    dt = _dt(o, float(vel.max()))
    ph, k = rng.uniform(0, 2 * np.pi, 3), rng.uniform(0.1, 0.3, 3) * 4 / o
    base = (np.sin(k[0] * np.arange(ny) + ph[0])[:, None, None] * np.cos(k[1] * np.arange(nz) + ph[1])[None, :, None]
            * np.sin(k[2] * np.arange(nx) + ph[2])[None, None, :])
    b = dict(ex=ex, ey=ey, ez=ez, o=o, steps=case["steps"], vel=vel, dt=dt,
             sponge=tuple(_sponge(n, o, case["sponge"]) for n in (ex, ey, ez)) if case["sponge"] else None)
    return b, base.astype(np.float32).reshape(-1), (0.97 * base).astype(np.float32).reshape(-1)


def _solver(b, variant="default"):
    mesh = semgb.Mesh(b["ex"], b["ey"], b["ez"], b["ex"] * H, b["ey"] * H, b["ez"] * H, b["o"])
    mesh.set_velocity(b["vel"])
    s = semgb.Solver(mesh, b["dt"])
    if variant == "reference":
        s.set_rounding(semgb.ROUNDING_REFERENCE)
    elif variant == "difference":
        s.set_operator_form(semgb.FORM_DIFFERENCE)
    elif variant == "element":
        s.set_kernel(semgb.KERNEL_ELEMENT)
    if b["sponge"]:
        s.set_sponge_profile(*b["sponge"])
    s.set_sources(b["src"], b["wav"])
    s.set_receiver_nodes(b["rec"])
    return s


def prepare(case, seed):
    k = case["kind"]
    if k in ("stream", "shot"):
        b = _box_inputs(case, seed)
        return dict(k=k, s=_solver(b, case.get("variant", "default")), b=b, field=case.get("field", True))
    if k == "batch":
        b = _box_inputs(case, seed)
        mesh = semgb.Mesh(b["ex"], b["ey"], b["ez"], b["ex"] * H, b["ey"] * H, b["ez"] * H, b["o"])
        mesh.set_velocity(b["vel"])
        return dict(k=k, mesh=mesh, b=b)
    if k == "group":
        bs = _member_inputs(case, seed)
        s = [_solver(b) for b in bs]
        return dict(k=k, s=s, g=semgb.Group(s), steps=case["steps"])
    if k == "adjoint":
        b = _box_inputs(case, seed)
        mesh = semgb.Mesh(b["ex"], b["ey"], b["ez"], b["ex"] * H, b["ey"] * H, b["ez"] * H, b["o"])
        mesh.set_velocity(b["vel"])
        return dict(k=k, mesh=mesh, b=b, every=case["every"], obs=_observed(b, _rng(seed, 1)))
    if k == "learned":
        b = _box_inputs(case, seed)
        s = _solver(b)
        net = semgb.Mlp(0)
        net.params = _net_params(_rng(seed, 1))
        return dict(k=k, s=s, abc=semgb.Abc(s, net, 0), steps=case["steps"])
    if k == "train":
        return dict(k=k, net=semgb.Mlp(0), epochs=case["epochs"], batch=case["batch"], seed=int(seed),
                    **_train_inputs(case, seed))
    if k == "bptt":
        b, roi, ref, p = _bptt_inputs(case, seed)
        s = _solver(b)
        net = semgb.Mlp(0)
        net.params = p
        return dict(k=k, abc=semgb.Abc(s, net, 0), roi=roi, ref=ref)
    b, p, q = _noalloc_inputs(case, seed)
    dev = torch.device("cuda")
    ref = _Box(b, dev)
    buf = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    return dict(k=k, b=b, conn=_connectivity(b, dev), coef=ref.a.to(torch.float32).reshape(-1).contiguous(),
                p0=buf(p), q0=buf(q), cur=torch.empty(p.size, device=dev), prev=torch.empty(p.size, device=dev),
                sponge=[buf(x) for x in b["sponge"]] if b["sponge"] else [None] * 3)


def _connectivity(b, dev):
    """Node of (element, local node), element and local numbering as the package's, int32."""
    o, nx, nz = b["o"], b["ex"] * b["o"] + 1, b["ez"] * b["o"] + 1
    ar = lambda n: torch.arange(n, device=dev)  # noqa: E731
    e = (ar(b["ey"])[:, None, None] * nx * nz + ar(b["ez"])[None, :, None] * nx + ar(b["ex"])[None, None, :]) * o
    l = ar(o + 1)[:, None, None] * nx * nz + ar(o + 1)[None, :, None] * nx + ar(o + 1)[None, None, :]
    return (e.reshape(-1, 1) + l.reshape(1, -1)).to(torch.int32).contiguous()


# ---- one pass -----------------------------------------------------------------------------------

# A time loop starts from rest: reset, and a wait for it (synchronize) before the first step.  Batches
# and adjoints are made for each set of shots, as they have no reset of their own.
def run(st):
    k = st["k"]
    if k == "shot":
        s = st["s"]
        s.reset()
        s.synchronize()
        s.step(st["b"]["steps"])
        if not st["field"]:
            return [s.traces()]
        return [s.traces(), s.pressure(semgb.LEVEL_CURRENT), s.pressure(semgb.LEVEL_PREVIOUS)]
    if k == "stream":
        s, b = st["s"], st["b"]
        s.reset()
        s.synchronize()
        out = np.zeros((b["steps"], len(b["rec"])), np.float32)
        for n in range(b["steps"]):
            s.step_host(1, b["wav"][:, n], out[n])
        return [out, s.pressure(semgb.LEVEL_CURRENT), s.pressure(semgb.LEVEL_PREVIOUS)]
    if k == "batch":
        b = st["b"]
        bt = semgb.Batch(st["mesh"], b["dt"], len(b["src"]))
        if b["sponge"]:
            bt.set_sponge_profile(*b["sponge"])
        bt.set_sources(b["src"], b["wav"])
        bt.set_receiver_nodes(b["rec"])
        bt.step(b["steps"])
        out = [bt.traces()]
        bt.close()
        return out
    if k == "group":
        for s in st["s"]:
            s.reset()
        st["g"].synchronize()
        st["g"].step(st["steps"])
        return [s.traces() for s in st["s"]]
    if k == "adjoint":
        b = st["b"]
        a = semgb.Adjoint(st["mesh"], b["dt"], b["steps"], st["every"])
        if b["sponge"]:
            a.set_sponge_profile(*b["sponge"])
        a.set_sources(b["src"], b["wav"])
        a.set_receiver_nodes(b["rec"])
        d = a.forward()
        loss, g = a.gradient(st["obs"])
        a.close()
        return [d, loss, g]
    if k == "learned":
        st["s"].reset()
        st["abc"].reset()
        st["s"].synchronize()
        st["abc"].step(st["steps"])
        return [st["s"].traces()]
    if k == "train":
        net = st["net"]
        net.params = st["p"]
        loss, g = net.loss_grad(st["x"], st["t"])
        losses = net.train(st["x"], st["t"], st["epochs"], st["batch"], 1e-3, st["seed"])
        return [loss, g, losses, net.params]
    if k == "bptt":
        loss, g = st["abc"].bptt(st["roi"], st["ref"])
        return [loss, g]
    b, stream = st["b"], torch.cuda.current_stream().cuda_stream
    cur, prev = st["cur"], st["prev"]
    cur.copy_(st["p0"])
    prev.copy_(st["q0"])
    p = lambda t: None if t is None else ctypes.c_void_p(t.data_ptr())  # noqa: E731
    for _ in range(b["steps"]):
        rc = semgb.lib().sem_element_step_noalloc(b["ex"], b["ey"], b["ez"], b["ex"] * H, b["ey"] * H, b["ez"] * H,
                                                  b["o"], p(st["conn"]), p(cur), p(prev), p(st["coef"]),
                                                  *[p(s) for s in st["sponge"]], ctypes.c_void_p(stream))
        if rc != semgb.SEM_OK:
            raise RuntimeError(semgb.lib().sem_last_error_string().decode())
        cur, prev = prev, cur
    return [cur, prev]


# ---- the same in 64 bits --------------------------------------------------------------------------

class _Box:
    """The spectral-element step on a box in float64: K = sum over the axes of the assembled 1-D
    stiffness times the assembled weights of the other two, leapfrog, sponge on both levels."""

    def __init__(self, b, dev):
        o = b["o"]
        _, w, d = _gll(o)
        S = d.T @ np.diag(w) @ d
        self.o, self.n = o, [b[k] * o + 1 for k in ("ey", "ez", "ex")]  # [y][z][x]
        J = 0.5 * H
        self.band, self.W = [], []
        for ne in (b["ey"], b["ez"], b["ex"]):
            T, W = np.zeros((ne * o + 1, 2 * o + 1)), np.zeros(ne * o + 1)
            for e in range(ne):
                for i in range(o + 1):
                    W[e * o + i] += w[i]
                    T[e * o + i, o - i:2 * o + 1 - i] += S[i]
            self.band.append(torch.from_numpy(T * J).to(dev))  # detJ / J^2 = J
            self.W.append(torch.from_numpy(W).to(dev))
        v = torch.from_numpy(b["vel"].astype(np.float64)).to(dev).view(b["ey"], b["ez"], b["ex"])
        m = v.pow(-2) * J ** 3
        for dim in range(3):
            ne = m.shape[dim]
            shape = list(m.shape)
            shape[dim] = ne * o + 1
            out = torch.zeros(shape, dtype=torch.float64, device=dev)
            for i in range(o + 1):
                at = [slice(None)] * 3
                at[dim] = slice(i, i + (ne - 1) * o + 1, o)
                out[tuple(at)] += w[i] * m
            m = out
        dt2 = float(np.float32(b["dt"])) ** 2
        self.a = dt2 / m
        if b["sponge"]:
            sx, sy, sz = (torch.from_numpy(x.astype(np.float64)).to(dev) for x in b["sponge"])
            self.s = [sy.view(-1, 1, 1), sz.view(1, -1, 1), sx.view(1, 1, -1)]
        else:
            self.s = []
        if "src" in b:
            e = torch.as_tensor(b["src"])
            ix, iz, iy = e % b["ex"], (e // b["ex"]) % b["ez"], e // (b["ex"] * b["ez"])
            self.src = [(int(y) * o, int(z) * o, int(x) * o) for y, z, x in zip(iy, iz, ix)]
            c = b["vel"][b["src"]].astype(np.float64)
            self.b = (dt2 * c * c)[:, None] * b["wav"].astype(np.float64)
        self.dev = dev

    def zeros(self):
        return torch.zeros(self.n, dtype=torch.float64, device=self.dev)

    def along(self, v, dim):
        return v.view([-1 if k == dim else 1 for k in range(3)])

    def K(self, p):
        tot = torch.zeros_like(p)
        o = self.o
        for dim in range(3):
            n, r = self.n[dim], torch.zeros_like(p)
            for d in range(-min(o, n - 1), min(o, n - 1) + 1):
                lo, m = max(0, -d), n - abs(d)
                r.narrow(dim, lo, m).addcmul_(p.narrow(dim, lo + d, m), self.along(self.band[dim][lo:lo + m, d + o], dim))
            for k in range(3):
                if k != dim:
                    r *= self.along(self.W[k], k)
            tot += r
            del r
        return tot

    def damp(self, p):
        for s in self.s:
            p = p * s
        return p

    def interior(self, v, q):
        """v on interior nodes, q on the boundary."""
        out = q.clone()
        out[1:-1, 1:-1, 1:-1] = v[1:-1, 1:-1, 1:-1]
        return out

    def step(self, p, q, n=None, shot=None):
        """(p^{n+1}, damped p^n, K p^n) from the levels p^n and p^{n-1}; adds the sources of step n."""
        if n is not None:
            p = p.clone()
            for i, at in enumerate(self.src):
                if shot is None or shot == i:
                    p[at] += self.b[i, n]
        kp = self.K(p)
        v = self.interior(2.0 * p - q - self.a * kp, q)
        return self.damp(v), self.damp(p), kp


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _forward(b, dev, shot=None):
    box = _Box(b, dev)
    p, q = box.zeros(), box.zeros()
    rec = torch.from_numpy(b["rec"]).to(dev)
    tr = torch.zeros(b["steps"], len(b["rec"]), dtype=torch.float64, device=dev)
    for n in range(b["steps"]):
        p, q, _ = box.step(p, q, n, shot)
        tr[n] = p.reshape(-1)[rec]
    return tr, p.reshape(-1), q.reshape(-1)


def _net(params, x):
    """The network in float64 on the weights it runs with (BF16 matrices): y [n]."""
    w1, b1 = params[0].view(N_HID, N_IN), params[1]
    w2, b2, w3, b3 = params[2].view(N_HID, N_HID), params[3], params[4], params[5]
    g = lambda z: 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))  # noqa: E731
    return g(g(x @ w1.T + b1) @ w2.T + b2) @ w3 + b3


def _net_tensors(p, dev, grad=False):
    t = torch.from_numpy(p).to(dev)
    h, a = N_HID, N_HID * N_IN
    parts = [t[:a].bfloat16(), t[a:a + h], t[a + h:a + h + h * h].bfloat16(), t[a + h + h * h:a + 2 * h + h * h],
             t[a + 2 * h + h * h:a + 3 * h + h * h], t[-1:]]
    return [x.double().requires_grad_(grad) for x in parts]


class _Boundary:
    """The network on the boundary nodes: their new values from the 3x3x3 neighbourhoods at three
    time levels."""

    def __init__(self, box, params):
        self.box, self.params = box, params
        ny, nz, nx = box.n
        on = torch.ones(box.n, dtype=torch.bool, device=box.dev)
        on[1:-1, 1:-1, 1:-1] = False
        at = on.nonzero()
        self.flat = (at[:, 0] * nz + at[:, 1]) * nx + at[:, 2]
        off = [(dy, dz, dx) for dz in (0, 1, 2) for dy in (0, 1, 2) for dx in (0, 1, 2)]
        self.idx = torch.stack([((at[:, 0] + dy) * (nz + 2) + at[:, 1] + dz) * (nx + 2) + at[:, 2] + dx
                                for dy, dz, dx in off], 1)

    def apply(self, new, cur, prev):
        pad = lambda f: torch.nn.functional.pad(f, (1, 1, 1, 1, 1, 1)).reshape(-1)[self.idx]  # noqa: E731
        f = torch.cat([pad(new), pad(cur), pad(prev)], 1)
        sc = f.abs().amax(1) + 1e-30
        y = _net(self.params, f / sc[:, None])
        return new.reshape(-1).index_put((self.flat,), sc * y.clamp(-1.0, 1.0)).view(new.shape)


def exact(case, seed):
    k, dev = case["kind"], _device()
    with torch.no_grad():
        if k in ("stream", "shot"):
            tr, p, q = _forward(_box_inputs(case, seed), dev)
            return [tr, p, q] if case.get("field", True) else [tr]
        if k == "batch":
            if case["shots"] * _nodes(case["ex"], case["ey"], case["ez"], case["order"]) * case["steps"] > 2.5e10:
                return None
            b = _box_inputs(case, seed)
            return [torch.stack([_forward(b, dev, i)[0] for i in range(case["shots"])], 2)]
        if k == "group":
            return [_forward(b, dev)[0] for b in _member_inputs(case, seed)]
        if k == "adjoint":
            return _exact_adjoint(_box_inputs(case, seed), seed, dev)
        if k == "learned":
            b = _box_inputs(case, seed)
            box = _Box(b, dev)
            net = _Boundary(box, _net_tensors(_net_params(_rng(seed, 1)), dev))
            rec, p, q, tr = torch.from_numpy(b["rec"]).to(dev), box.zeros(), box.zeros(), []
            for n in range(b["steps"]):
                new, cur, _ = box.step(p, q, n)
                p, q = net.apply(new, cur, q), cur
                tr.append(p.reshape(-1)[rec])
            return [torch.stack(tr)]
        if k == "noalloc":
            b, p, q = _noalloc_inputs(case, seed)
            box = _Box(b, dev)
            p, q = (torch.from_numpy(x.astype(np.float64)).to(dev).view(box.n) for x in (p, q))
            for _ in range(case["steps"]):
                p, q, _ = box.step(p, q)
            return [p.reshape(-1), q.reshape(-1)]
    if k == "train":  # the order of the minibatches is the library's own: only the first two have a value here
        i = _train_inputs(case, seed)
        par = _net_tensors(i["p"], dev, True)
        x = torch.from_numpy(i["x"]).to(dev).bfloat16().double()
        loss = (_net(par, x) - torch.from_numpy(i["t"]).to(dev).double()).pow(2).mean()
        g = torch.autograd.grad(loss, par)
        return [float(loss.detach()), torch.cat([v.reshape(-1) for v in g]), None, None]
    b, roi, ref, p = _bptt_inputs(case, seed)
    return _exact_bptt(b, roi, ref, p, dev)


def _exact_adjoint(b, seed, dev):
    box = _Box(b, dev)
    p, q, kps, tr = box.zeros(), box.zeros(), [], []
    rec = torch.from_numpy(b["rec"]).to(dev)
    for n in range(b["steps"]):
        p, q, kp = box.step(p, q, n)
        kps.append(kp)
        tr.append(p.reshape(-1)[rec])
    tr = torch.stack(tr)
    res = tr - torch.from_numpy(_observed(b, _rng(seed, 1)).astype(np.float64)).to(dev)
    P, Q, g = box.zeros(), box.zeros(), box.zeros()
    for n in range(b["steps"] - 1, -1, -1):
        P.view(-1).index_add_(0, rec, res[n])
        V = box.damp(P)
        JV = box.interior(V, torch.zeros_like(V))
        g.addcmul_(box.a * JV, kps.pop())
        P, Q = 2.0 * JV - box.K(box.a * JV) + box.damp(Q), V - 2.0 * JV
    # 1/m per node, m the squared slowness: a = dt^2 / (m W) with W the assembled weights times detJ
    W = box.along(box.W[0], 0) * box.along(box.W[1], 1) * box.along(box.W[2], 2) * (0.5 * H) ** 3
    return [tr, float(0.5 * res.pow(2).sum()), (g * box.a * W / float(np.float32(b["dt"])) ** 2).reshape(-1)]


class _KFn(torch.autograd.Function):
    """The stiffness product (symmetric, linear) for autograd."""

    @staticmethod
    def forward(ctx, p, box):
        ctx.box = box
        return box.K(p)

    @staticmethod
    def backward(ctx, g):
        return ctx.box.K(g), None


def _exact_bptt(b, roi, ref, params, dev):
    box = _Box(b, dev)
    par = _net_tensors(params, dev, True)
    net = _Boundary(box, par)
    roi = torch.from_numpy(roi).to(dev)
    inner = torch.zeros(box.n, dtype=torch.bool, device=dev)
    inner[1:-1, 1:-1, 1:-1] = True
    p, q, loss = box.zeros(), box.zeros(), 0.0
    for n in range(b["steps"]):
        add = box.zeros()
        for i, at in enumerate(box.src):
            add[at] += box.b[i, n]
        c = p + add
        v = torch.where(inner, 2.0 * c - q - box.a * _KFn.apply(c, box), q)
        new, cur = box.damp(v), box.damp(c)
        p, q = net.apply(new, cur, q), cur
        loss = loss + (p.reshape(-1)[roi] - torch.from_numpy(ref[n].astype(np.float64)).to(dev)).pow(2).sum()
    g = torch.autograd.grad(loss, par)
    return [float(loss.detach()), torch.cat([x.reshape(-1) for x in g])]
