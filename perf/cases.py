"""The work a user of this library has it do, as cases that can be timed and checked.

A case is a dict of plain values.  prepare(case, seed) makes what a program has
in hand before the call (fields, models, handles; all from the seed), run(state)
is one pass through the public Python entry points, exact(case, seed) the same
results in 64 bits by plain torch, work(case) the bytes and operations of a pass.

Kinds:
  wave     one acoustic step, FP32 fields (sb.wave_step), any extents
  exact    one acoustic step in the reference's operation order (sb.wave_step_exact)
  heat     one heat step, FP32 (sb.heat_step)
  half     one acoustic step with FP16 storage (sb.wave_step_f16)
  run      a whole simulation through sb.Run: fields in from pinned host memory,
           the steps, the final field and the source trace out
  shots    steps of a tuned sb.Batch of uneven shots, then every shot's trace and
           one shot's field
  learned  one coarse step with the learned correction (Mlp.learned_step), on a
           field that is active everywhere, behind the composition pre-pass, or on
           a compact pulse with activity flags
  train    Adam steps of the correction network over mini-batches (Mlp.train_step)
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import stencil_solver_b200 as sb

DX = 10.0
V_TOP, V_BOTTOM, V_PERT = 1500.0, 4500.0, 0.05
DT = float(np.float32(0.4 * DX / (V_BOTTOM * (1.0 + V_PERT))))  # Courant 0.4 at the fastest cell
FD8 = (-205.0 / 72, 8.0 / 5, -1.0 / 5, 8.0 / 315, -1.0 / 560)
SRC_FREQ = 15.0
HEAT_DT, HEAT_ALPHA = 1.0, 0.05 * DX * DX  # alpha dt / dx^2 = 0.05
HALF_SCALE = 1024.0
OUT_SCALE, FLOOR = 0.05, 2.0 ** -24  # of the learned correction
BETA = 1.0 / 16.0                    # the composition pre-pass' term of two half steps
MAX_BATCH_STEPS = 1 << 18


def listed():
    return [
        # one step of the 128^3 point-source case: launch latency counts
        {"name": "acoustic_128", "kind": "wave", "nx": 128, "ny": 128, "nz": 128, "source": True},
        # a survey box of odd extents: rows that start on no 16-byte boundary
        {"name": "acoustic_odd", "kind": "wave", "nx": 401, "ny": 357, "nz": 301, "source": True},
        # the plain step at scale
        {"name": "acoustic_1024", "kind": "wave", "nx": 1024, "ny": 1024, "nz": 1024, "source": True},
        # the parity mode: the reference's operation order, bit for bit
        {"name": "exact_384", "kind": "exact", "nx": 384, "ny": 384, "nz": 384, "source": True},
        # the small simulation whole: 300 steps, host to host
        {"name": "run_128x300", "kind": "run", "nx": 128, "ny": 128, "nz": 128, "steps": 300,
         "half": False},
        # the heat configuration
        {"name": "heat_512", "kind": "heat", "nx": 512, "ny": 512, "nz": 512},
        # FP16 storage at scale
        {"name": "half_1024", "kind": "half", "nx": 1024, "ny": 1024, "nz": 1024},
        # FP16 storage with its renormalisation and monitor
        {"name": "run_half_256x100", "kind": "run", "nx": 256, "ny": 256, "nz": 256, "steps": 100,
         "half": True},
        # uneven shots in one persistent launch per step, both storages
        {"name": "shots_16", "kind": "shots", "shots": 16, "extents": 1, "steps": 100, "half": False},
        {"name": "shots_half_16", "kind": "shots", "shots": 16, "extents": 1, "steps": 100,
         "half": True},
        # the learned coarse step with the correction active everywhere
        {"name": "learned_260", "kind": "learned", "nx": 260, "ny": 260, "nz": 260, "compose": False,
         "pulse": False},
        # eight mini-batches of the network's training
        {"name": "train_8192x8", "kind": "train", "rows": 8192, "batches": 8},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _extents(rng, lo, hi, multiple):
    """Three extents around one log-uniform size, each off it by up to a fifth."""
    n = _log_uniform(rng, lo, hi)
    out = []
    for _ in range(3):
        e = min(hi, max(lo, int(n * rng.uniform(0.8, 1.2))))
        out.append(max(lo, e // multiple * multiple))
    return dict(zip(("nx", "ny", "nz"), out))


def draw(rng):
    kind = rng.choice(["wave", "wave", "wave", "exact", "heat", "heat", "half", "half", "run",
                       "shots", "learned", "train"])
    if kind in ("wave", "exact", "heat"):
        hi = {"wave": 1024, "exact": 512, "heat": 640}[kind]
        # half of the grids have rows of whole 16-byte chunks, the others any length
        c = {"kind": kind, **_extents(rng, 64, hi, 1)}
        if rng.random() < 0.5:
            c["nx"] = c["nx"] // 4 * 4
        if kind != "heat":
            c["source"] = rng.random() < 0.5
        return c
    if kind == "half":
        c = {"kind": kind, **_extents(rng, 64, 1024, 1)}
        c["nx"] = c["nx"] // 8 * 8
        return c
    if kind == "run":
        half = rng.random() < 0.5
        c = {"kind": kind, **_extents(rng, 64, 256, 1), "steps": 10 * rng.randint(5, 30), "half": half}
        c["nx"] = c["nx"] // 8 * 8 if half or rng.random() < 0.5 else c["nx"]
        return c
    if kind == "shots":
        c = {"kind": kind, "shots": rng.randint(4, 16), "extents": rng.randrange(1000),
             "steps": 50 * rng.randint(1, 2), "half": rng.random() < 0.5}
        most = _points(listed()[8]) * 100
        while _points(c) * c["steps"] > most:
            c["shots"] -= 1
        return c
    if kind == "learned":
        c = {"kind": kind, **_extents(rng, 64, 388, 1), "compose": rng.random() < 0.5,
             "pulse": rng.random() < 0.5}
        c["nx"] = c["nx"] // 4 * 4
        return c
    return {"kind": kind, "rows": _log_uniform(rng, 1000, 65536), "batches": rng.randint(2, 8)}


# ── inputs ────────────────────────────────────────────────────────────────────


def _shots(case):
    """(nx, ny, nz) of each shot: 96..320 in steps of 8, from the case's extents seed."""
    r = random.Random(case["extents"])
    return [tuple(8 * r.randint(12, 40) for _ in range(3)) for _ in range(case["shots"])]


def _points(case):
    return sum((x - 8) * (y - 8) * (z - 8) for x, y, z in _shots(case))


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _walls(t):
    t[:4], t[-4:] = 0, 0
    t[:, :4], t[:, -4:] = 0, 0
    t[:, :, :4], t[:, :, -4:] = 0, 0
    return t


def _waves(shape, r, n=4):
    """(p, p_prev): a developed field, n plane waves of 8 to 24 cells, walls zero."""
    z, y, x = (torch.arange(k, device="cuda", dtype=torch.float32) for k in shape)
    p = torch.zeros(shape, device="cuda")
    q = torch.zeros(shape, device="cuda")
    for _ in range(n):
        d = np.array([r.gauss(0, 1) for _ in range(3)])
        k = d / np.linalg.norm(d) * 2 * math.pi / r.uniform(8, 24)
        phase, back = r.uniform(0, 2 * math.pi), 0.3 * float(np.linalg.norm(k))
        amp = r.uniform(0.2, 1.0)
        arg = (k[0] * x + phase)[None, None, :] + ((k[1] * y)[:, None] + (k[2] * z)[:, None, None])
        q.add_(torch.sin(arg + back), alpha=amp)
        p.add_(arg.sin_(), alpha=amp)
        del arg
    return _walls(p), _walls(q)


def _pulse(shape, r):
    """(p, p_prev): a Gaussian pulse of 6 cells away from the walls, at rest, exactly
    zero beyond 24 cells."""
    at = [r.uniform(0.4, 0.6) * n for n in shape]
    d2 = sum((torch.arange(n, device="cuda", dtype=torch.float32) - a).square().reshape(
        [-1 if i == ax else 1 for i in range(3)]) for ax, (n, a) in enumerate(zip(shape, at)))
    p = torch.exp(-d2 / 72.0)
    p[d2 > 24.0 ** 2] = 0
    p = _walls(p)
    return p, p.clone()


def _model(shape, r, layers=8):
    """v^2: horizontal layers, speeds rising with depth, times 1 + 0.05 g, g smooth."""
    nz, ny, nx = shape
    cuts = sorted(r.uniform(0, nz) for _ in range(layers - 1))
    speeds = [V_TOP + (V_BOTTOM - V_TOP) * i / (layers - 1) for i in range(layers)]
    v = torch.tensor([speeds[sum(c <= z for c in cuts)] for z in range(nz)], device="cuda",
                     dtype=torch.float32)
    g = [torch.sin(torch.arange(k, device="cuda", dtype=torch.float32) * (2 * math.pi / r.uniform(40, 80))
                   + r.uniform(0, 6)) for k in (nx, ny, nz)]
    f = (V_PERT * g[1])[None, :, None] * g[0][None, None, :] * g[2][:, None, None]
    return f.add_(1.0).mul_(v[:, None, None]).square_()


def _shape(case):
    return (case["nz"], case["ny"], case["nx"])


def _grid(shape, dt=DT):
    nz, ny, nx = shape
    return sb.Grid(nx, ny, nz, DX, DX, DX, dt)


def _source(shape, r):
    """Flat index of a random interior cell."""
    z, y, x = (r.randrange(4, n - 4) for n in shape)
    return (z * shape[1] + y) * shape[2] + x


def _step_inputs(case, seed):
    """Fields, model and source of a single-step case."""
    r = random.Random(int(seed))
    shape = _shape(case)
    p, q = _waves(shape, r)
    v = _model(shape, r)
    src = _source(shape, r) if case.get("source") else -1
    return p, q, v, src, 0.5 / (DT * DT * 3000.0 ** 2)


def _run_inputs(case, seed):
    r = random.Random(int(seed))
    shape = _shape(case)
    return _model(shape, r), _source(shape, r)


def _shot_inputs(case, seed):
    """Per shot (shape, v^2, source index, source frequency)."""
    r = random.Random(int(seed))
    out = []
    for x, y, z in _shots(case):
        shape = (z, y, x)
        out.append((shape, _model(shape, r), _source(shape, r), r.uniform(10.0, 25.0)))
    return out


def _learned_inputs(case, seed):
    r = random.Random(int(seed))
    shape = _shape(case)
    p, q = _pulse(shape, r) if case["pulse"] else _waves(shape, r)
    v = _model(shape, r)
    g = np.random.default_rng(int(seed))
    w = np.zeros(sb.MLP_NPARAM)
    w[:1024].reshape(32, 32)[:, :26] = g.standard_normal((32, 26)) * math.sqrt(2.0 / 26)
    w[1024:1056] = 0.1 * g.standard_normal(32)
    w[1056:2080] = g.standard_normal(1024) * math.sqrt(2.0 / 32)
    w[2080:2112] = 0.1 * g.standard_normal(32)
    w[2112:2144] = g.standard_normal(32) * math.sqrt(1.0 / 32)
    w[2144] = 0.05
    return p, q, v, w.astype(np.float32)


def _train_inputs(case, seed):
    """Feature rows (BF16), targets of order one, network parameters."""
    gen = _gen(seed)
    b, n = case["batches"], case["rows"]
    X = torch.randn((b, n, 32), generator=gen, device="cuda").mul_(0.4).clamp_(-2, 2)
    X[:, :, 25] = torch.rand((b, n), generator=gen, device="cuda") * 0.3 + 0.1
    X[:, :, 26:] = 0
    X = X.to(torch.bfloat16)
    a = torch.randn((32,), generator=gen, device="cuda")
    t = torch.tanh(X.float() @ a) + 0.1 * torch.randn((b, n), generator=gen, device="cuda")
    g = np.random.default_rng(int(seed))
    w = np.zeros(sb.MLP_NPARAM)
    w[:1024].reshape(32, 32)[:, :26] = g.standard_normal((32, 26)) * math.sqrt(2.0 / 26)
    w[1056:2080] = g.standard_normal(1024) * math.sqrt(2.0 / 32)
    w[2112:2144] = g.standard_normal(32) * 0.1
    return X, t.contiguous(), w.astype(np.float32)


LR = 1e-3


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("wave", "exact"):
        p, q, v, src, amp = _step_inputs(case, seed)
        return {"case": case, "g": _grid(_shape(case)), "p": p, "q": q, "v": v, "src": src, "amp": amp}
    if kind == "heat":
        shape = _shape(case)
        u = torch.zeros(shape, device="cuda")
        u[4:-4, 4:-4, 4:-4] = torch.rand([n - 8 for n in shape], generator=_gen(seed), device="cuda")
        return {"case": case, "g": _grid(shape, HEAT_DT), "u": u, "un": torch.zeros_like(u)}
    if kind == "half":
        p, q, v, _, _ = _step_inputs(case, seed)
        g = _grid(_shape(case))
        P, Q, K = (torch.empty(p.shape, dtype=torch.int16, device="cuda") for _ in range(3))
        sb.f16_pack(p, P, g.size, HALF_SCALE)
        sb.f16_pack(q, Q, g.size, HALF_SCALE)
        sb.k_field_bf16(v, K, g)
        return {"case": case, "g": g, "p": P, "q": Q, "k": K,
                "scale": torch.tensor([HALF_SCALE, 1.0], device="cuda")}
    if kind == "run":
        v, src = _run_inputs(case, seed)
        run_ = sb.Run(_grid(v.shape), src_index=src, src_freq=SRC_FREQ,
                      precision=sb.PRECISION_F16 if case["half"] else sb.PRECISION_F32)
        return {"case": case, "run": run_, "v": v.cpu().pin_memory(),
                "rest": torch.zeros(v.shape).pin_memory(), "out": torch.empty(v.shape).pin_memory()}
    if kind == "shots":
        inputs = _shot_inputs(case, seed)
        batch = sb.Batch([(_grid(shape), src) for shape, _, src, _ in inputs],
                         max_steps=MAX_BATCH_STEPS,
                         precision=sb.PRECISION_F16 if case["half"] else sb.PRECISION_F32)
        batch.tune(2)
        for i, (shape, v, _, f) in enumerate(inputs):
            batch.set_fields(i, np.zeros(shape, np.float32), None, v.cpu().numpy())
            batch.set_wavelet(i, sb.ricker(f, 1.0 / f, DT, 400))
        return {"case": case, "batch": batch}
    if kind == "learned":
        p, q, v, w = _learned_inputs(case, seed)
        g = _grid(p.shape)
        mlp = sb.Mlp()
        mlp.set_params(w)
        mlp.output_scale, mlp.min_scale = OUT_SCALE, FLOOR
        s = {"case": case, "g": g, "p": p, "q": q, "v": v, "mlp": mlp, "flags": None, "r": None}
        if case["compose"]:
            s["r"] = torch.zeros_like(p)
        if case["pulse"]:
            # one step with every flag set leaves the flags of its result
            n = mlp.flags_bytes(g)
            fl = [torch.full((n,), 255, dtype=torch.uint8, device="cuda") for _ in range(3)]
            mlp.learned_step(p, q, v, g, flags=(fl[0], fl[1]))
            s.update(p=q, q=p, flags=(fl[1], fl[0], fl[2]))
        return s
    X, t, w = _train_inputs(case, seed)
    mlp = sb.Mlp()
    mlp.set_params(w)
    return {"case": case, "mlp": mlp, "X": X.view(torch.int16), "t": t,
            "loss": torch.zeros(1, device="cuda")}


def run(s):
    kind = s["case"]["kind"]
    if kind in ("wave", "exact"):
        step = sb.wave_step if kind == "wave" else sb.wave_step_exact
        p, q = s["p"], s["q"]
        step(p, q, s["v"], q, s["g"], s["src"], s["amp"])
        s["p"], s["q"] = q, p
        return q
    if kind == "heat":
        u, un = s["u"], s["un"]
        sb.heat_step(u, un, s["g"], HEAT_ALPHA)
        s["u"], s["un"] = un, u
        return un
    if kind == "half":
        p, q = s["p"], s["q"]
        sb.wave_step_f16(p, q, s["k"], s["g"], s["scale"])
        s["p"], s["q"] = q, p
        return q.view(torch.float16)
    if kind == "run":
        r, n = s["run"], s["case"]["steps"]
        r.set_fields(s["rest"], s["rest"], s["v"])
        r.steps(n)
        return {"field": r.field(s["out"]), "trace": r.trace(n)}
    if kind == "shots":
        b, n = s["batch"], s["case"]["steps"]
        b.steps(n)
        b.synchronize()
        done = b.steps_done
        return {"traces": [b.trace(i, done)[-n:] for i in range(s["case"]["shots"])],
                "field": b.field(0)}
    if kind == "learned":
        # p stays: every pass steps the same state, over the level the last one left
        mlp, g, p, q, r, fl = s["mlp"], s["g"], s["p"], s["q"], s["r"], s["flags"]
        cur, flags = p, None if fl is None else (fl[0], fl[1])
        if r is not None:
            sb.wave_prepass(p, q, s["v"], r, g, BETA)
            cur = r
            if fl is not None:
                mlp.flags_compose(g, fl[0], fl[2])
                flags = (fl[2], fl[1])
        mlp.learned_step(cur, q, s["v"], g, flags=flags)
        return q
    mlp = s["mlp"]
    for X, t in zip(s["X"], s["t"]):
        mlp.train_step(X, t, LR, s["loss"])
    return {"loss": s["loss"], "params": mlp.params()}


def work(case):
    """Bytes and operations of one pass: each step reads its fields and its model and
    writes one field, once per interior point."""
    kind = case["kind"]
    if kind == "train":
        n = case["rows"] * case["batches"]
        return {"bytes": 68 * n, "flops": 3 * 4160 * n}
    pts = _points(case) if kind == "shots" else (case["nx"] - 8) * (case["ny"] - 8) * (case["nz"] - 8)
    n = case.get("steps", 1)
    size = 8 if kind in ("heat", "half") or case.get("half") else 16
    if kind == "learned":
        net = 0 if case["pulse"] else 4160
        return {"bytes": (36 if case["compose"] else 16) * pts, "flops": (42 + net) * pts}
    return {"bytes": size * pts * n, "flops": (40 if kind == "heat" else 42) * pts * n}


# ── the same in 64 bits ───────────────────────────────────────────────────────


def _lap64(p):
    """Laplacian x dx^2 of the interior of a slab (4 halo cells on each side)."""
    c = p[4:-4, 4:-4, 4:-4]
    out = c * (3 * FD8[0])
    nz, ny, nx = c.shape
    for r in range(1, 5):
        out.add_(p[4 + r:4 + r + nz, 4:-4, 4:-4], alpha=FD8[r]).add_(
            p[4 - r:4 - r + nz, 4:-4, 4:-4], alpha=FD8[r])
        out.add_(p[4:-4, 4 + r:4 + r + ny, 4:-4], alpha=FD8[r]).add_(
            p[4:-4, 4 - r:4 - r + ny, 4:-4], alpha=FD8[r])
        out.add_(p[4:-4, 4:-4, 4 + r:4 + r + nx], alpha=FD8[r]).add_(
            p[4:-4, 4:-4, 4 - r:4 - r + nx], alpha=FD8[r])
    return out


def _slabs(nz, n=64):
    return [(z, min(z + n, nz - 4)) for z in range(4, nz - 4, n)]


def _step64(p, q, k, src=-1, add=0.0, scale=1.0):
    """q with its interior replaced by 2p - q + scale k dx^2 lap(p) (k a field), plus
    the source; p, q, k of any floating type."""
    out = q.double()
    for z0, z1 in _slabs(p.shape[0]):
        lap = _lap64(p[z0 - 4:z1 + 4].double())
        i = (slice(z0, z1), slice(4, -4), slice(4, -4))
        out[i] = 2 * p[i].double() - out[i] + scale * k[i].double() * lap
    if src >= 0:
        out.view(-1)[src] += add
    return out


def _sim64(shape, v, src, f, steps):
    """(field, trace) of a run from rest with a Ricker source."""
    p = torch.zeros(shape, device="cuda", dtype=torch.float64)
    q = torch.zeros_like(p)
    k = v.double() * (DT * DT / (DX * DX))
    vs = float(v.view(-1)[src]) * DT * DT
    trace = torch.zeros(steps, device="cuda", dtype=torch.float64)
    for n in range(steps):
        a = (math.pi * f * (n * DT - 1.0 / f)) ** 2
        out = _step64(p, q, k, src, vs * (1.0 - 2.0 * a) * math.exp(-a))
        trace[n] = out.view(-1)[src]
        p, q = out, p
    return p, trace


def _net64(p, k, w, shape):
    """The correction of one step of p (64 bits): s c y at every interior point whose
    star reaches the floor."""
    w = torch.from_numpy(w).cuda().double()
    w1, b1 = w[:1024].view(32, 32)[:, :26], w[1024:1056]
    w2, b2, w3, b3 = w[1056:2080].view(32, 32), w[2080:2112], w[2112:2144], w[2144]
    out = torch.zeros(shape, device="cuda", dtype=torch.float64)
    for z0, z1 in _slabs(shape[0], 4):
        s = p[z0 - 4:z1 + 4]
        c = s[4:-4, 4:-4, 4:-4]
        nz, ny, nx = c.shape
        mag, feats = c.abs(), []
        for ax, n in ((2, nx), (1, ny), (0, nz)):
            for r in range(1, 5):
                at = [slice(4, -4)] * 3
                at[ax] = slice(4 + r, 4 + r + n)
                up = s[tuple(at)]
                at[ax] = slice(4 - r, 4 - r + n)
                dn = s[tuple(at)]
                mag = torch.maximum(mag, torch.maximum(up.abs(), dn.abs()))
                feats += [up - dn, up + dn - 2 * c]
        on = (mag > 0) & (mag >= FLOOR)
        scale = torch.where(on, torch.exp2(torch.floor(torch.log2(torch.clamp(mag, min=1e-30))) + 1),
                            torch.ones_like(mag))
        f = torch.stack([x / scale for x in feats + [c]] + [k[z0:z1, 4:-4, 4:-4].sqrt()], -1)
        h = torch.relu(f @ w1.T + b1)
        h = torch.relu(h @ w2.T + b2)
        y = h @ w3 + b3
        out[z0:z1, 4:-4, 4:-4] = torch.where(on, scale * OUT_SCALE * y, torch.zeros_like(y))
    return out


def _learned64(case, seed):
    p, q, v, w = _learned_inputs(case, seed)
    shape = tuple(p.shape)
    k = v.double() * (DT * DT / (DX * DX))
    p, q = p.double(), q.double()
    if case["pulse"]:  # the step that prepare() makes
        p, q = _step64(p, q, k) + _net64(p, k, w, shape), p
    cur = p
    if case["compose"]:
        lap = torch.zeros_like(p)
        for z0, z1 in _slabs(shape[0]):
            lap[z0:z1, 4:-4, 4:-4] = k[z0:z1, 4:-4, 4:-4] * _lap64(p[z0 - 4:z1 + 4])
        q = q + 2 * BETA * lap
        cur = _walls(p + BETA * lap)
    return _step64(cur, q, k) + _net64(cur, k, w, shape)


def _train64(case, seed):
    X, t, w = _train_inputs(case, seed)
    w = torch.from_numpy(w).cuda().double()
    m, u = torch.zeros_like(w), torch.zeros_like(w)
    live = torch.ones_like(w)
    live[:1024].view(32, 32)[:, 26:] = 0
    for i in range(case["batches"]):
        x = X[i].double()
        z = w.clone().requires_grad_()
        h = torch.relu(x @ z[:1024].view(32, 32).T + z[1024:1056])
        h = torch.relu(h @ z[1056:2080].view(32, 32).T + z[2080:2112])
        loss = (h @ z[2112:2144] + z[2144] - t[i].double()).square().mean()
        (g,) = torch.autograd.grad(loss, z)
        g = g * live
        m = 0.9 * m + 0.1 * g
        u = 0.999 * u + 0.001 * g * g
        w = w - LR * (m / (1 - 0.9 ** (i + 1))) / ((u / (1 - 0.999 ** (i + 1))).sqrt() + 1e-8)
    return {"loss": loss.detach().reshape(1), "params": w}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("wave", "exact"):
        p, q, v, src, amp = _step_inputs(case, seed)
        c = DT * DT
        add = c * float(v.view(-1)[src]) * amp if src >= 0 else 0.0
        return _step64(p, q, v, src, add, c / (DX * DX))
    if kind == "heat":
        u = prepare(case, seed)["u"]
        out = torch.zeros(u.shape, device="cuda", dtype=torch.float64)
        for z0, z1 in _slabs(u.shape[0]):
            slab = u[z0 - 4:z1 + 4].double()
            out[z0:z1, 4:-4, 4:-4] = slab[4:-4, 4:-4, 4:-4] + _lap64(slab) * (
                HEAT_DT * HEAT_ALPHA / (DX * DX))
        return out
    if kind == "half":
        p, q, v, _, _ = _step_inputs(case, seed)
        P, Q = ((x * HALF_SCALE).to(torch.float16) for x in (p, q))
        del p, q
        return _step64(P, Q, (v * (DT * DT / (DX * DX))).to(torch.bfloat16))
    if kind == "run":
        v, src = _run_inputs(case, seed)
        field, trace = _sim64(tuple(v.shape), v, src, SRC_FREQ, case["steps"])
        return {"field": field, "trace": trace}
    if kind == "shots":
        traces, field = [], None
        for i, (shape, v, src, f) in enumerate(_shot_inputs(case, seed)):
            p, trace = _sim64(shape, v, src, f, case["steps"])
            traces.append(trace)
            field = p if i == 0 else field
        return {"traces": traces, "field": field}
    if kind == "learned":
        return _learned64(case, seed)
    return _train64(case, seed)
