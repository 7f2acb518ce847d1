"""Reference-order steps on the kernels that stage planes by TMA (5 x 2^16 interior points
and more, 7 x 2^16 where rows are ragged): grids of any row length (rows as lines of
four), and the pencil tiles in that order on aligned grids; below, the one-thread-per-point kernel.  Bit for bit the
oracle, halos (and everything outside the interior) untouched."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import stencil_solver_b200 as sb

pytestmark = pytest.mark.gpu

# (nz, ny, nx): one interior plane and column-thin grids; rows of every residue modulo
# 4 words and planes of every residue; one below, at and above both ragged tiles
# (64 x 16, 32 x 32); the last sizes of the one-thread-per-point kernel and the first
# staged ones
RAGGED = [(9, 733, 741), (10, 520, 521), (2060, 9, 265), (900, 603, 9), (137, 72, 71),
          (133, 72, 73), (71, 137, 74), (75, 90, 105), (41, 250, 73), (12, 23, 41),
          (9, 9, 9), (88, 88, 89), (89, 89, 89), (85, 85, 85), (85, 85, 86)]
ALIGNED = [(9, 733, 740), (133, 72, 72), (75, 90, 108), (12, 24, 40), (2060, 9, 264), (76, 76, 76),
           (76, 76, 80)]


def case(shape, seed):
    rng = np.random.default_rng(seed)
    cur, prev = (rng.standard_normal(shape).astype(np.float32) for _ in range(2))
    vel2 = rng.uniform(1500.0, 4500.0, shape).astype(np.float32) ** 2
    return cur, prev, vel2


@pytest.mark.parametrize("shape", RAGGED + ALIGNED, ids=str)
def test_steps_bit_for_bit(torch_cuda, shape):
    nz, ny, nx = shape
    d, dt = (10.0, 7.5, 12.0), np.float32(1e-3)
    g = sb.Grid(nx, ny, nz, *d, float(dt))
    cur, prev, vel2 = case(shape, nx * ny + nz)
    dev = [torch_cuda.from_numpy(a).cuda() for a in (cur, prev, vel2)]
    ref = oracle.wave_step(cur, prev, vel2, *d, dt, out=prev.copy())
    # the source at the far interior corner; in place over p_prev
    src, amp = g.index(nx - 5, ny - 5, nz - 5), np.float32(0.37)
    ref.reshape(-1)[src] += np.float32(dt * dt) * vel2.reshape(-1)[src] * amp
    for step in (sb.wave_step_exact, sb.wave_step) if nx % 4 else (sb.wave_step_exact,):
        out = dev[1].clone()
        step(dev[0], out, dev[2], out, g, src, float(amp))
        assert np.array_equal(out.cpu().numpy(), ref)
    # an output that no 16-byte store could reach
    room = torch_cuda.zeros(cur.size + 1, device="cuda")
    out = room[1:].view(shape)
    sb.launch_naive(*dev, out, g)
    assert np.array_equal(out.cpu().numpy(), oracle.wave_step(cur, prev, vel2, *d, dt))
    # u + (alpha dt) lap: the wave arithmetic with p_prev = u, dt = 1 and v^2 = alpha dt
    k = np.full(shape, np.float32(900.0) * dt, np.float32)
    heat = oracle.wave_step(cur, cur, k, *d, np.float32(1.0), out=prev.copy())
    for step in (sb.heat_step_exact, sb.heat_step) if nx % 4 else (sb.heat_step_exact,):
        out = dev[1].clone()
        step(dev[0], out, g, 900.0)
        assert np.array_equal(out.cpu().numpy(), heat)
    assert sb.device_error() == 0


@pytest.mark.parametrize("heat", [False, True], ids=["acoustic", "heat"])
def test_every_tile_and_split_bit_for_bit(torch_cuda, heat):
    """Each tile of the table in the reference order, over chunks of 67, 23, 9, 8 and 1
    planes (a whole unroll of 8, one more, remainders, and less than the rings hold)."""
    shape = (75, 90, 108)
    nz, ny, nx = shape
    d, dt = (10.0, 7.5, 12.0), np.float32(1e-3)
    g = sb.Grid(nx, ny, nz, *d, float(dt))
    cur, prev, vel2 = case(shape, 5)
    dev = [torch_cuda.from_numpy(a).cuda() for a in (cur, prev, vel2)]
    if heat:
        k = np.full(shape, np.float32(900.0) * dt, np.float32)
        ref = oracle.wave_step(cur, cur, k, *d, np.float32(1.0), out=prev.copy())
    else:
        ref = oracle.wave_step(cur, prev, vel2, *d, dt, out=prev.copy())
    kind = sb.KIND_HEAT_F32 if heat else sb.KIND_WAVE_F32
    try:
        for v in range(len(sb.variant_names(kind))):
            for zchunks in (1, 3, 8, 9, 67):
                sb.set_pencil_override(kind, v, zchunks)
                out = dev[1].clone()
                if heat:
                    sb.heat_step_exact(dev[0], out, g, 900.0)
                else:
                    sb.wave_step_exact(dev[0], out, dev[2], out, g)
                assert np.array_equal(out.cpu().numpy(), ref), (v, zchunks)
    finally:
        sb.set_pencil_override(kind, -1, 1)
    assert sb.device_error() == 0


# rows on both sides of the line between one thread per point and staged planes (aligned:
# 4 and 5 rows; ragged, by covered columns: 5 and 6 rows of 257, 7 and 8 of 65), a single
# row, and the grids too tall for the former's launch
THIN = [(2060, 12, 264), (2060, 13, 264), (2060, 13, 265), (2060, 14, 265), (1900, 15, 73),
        (1900, 16, 73), (5000, 9, 265), (131090, 9, 40), (131090, 9, 41)]


@pytest.mark.parametrize("shape", THIN, ids=str)
def test_grids_of_few_rows_bit_for_bit(torch_cuda, shape):
    test_steps_bit_for_bit(torch_cuda, shape)


@pytest.mark.parametrize("shape", [(5000, 9, 264), (5000, 9, 265), (12000, 12, 73)], ids=str)
def test_few_rows_take_no_longer_than_one_thread_per_point(torch_cuda, shape):
    """Fields off a 16-byte boundary always run one thread per point: steps of the same
    grid from aligned fields (which tiles of 16 rows would make 1.8 to 4.6 times as
    long) take no more than 1.4 times theirs."""
    nz, ny, nx = shape
    g = sb.Grid(nx, ny, nz, 10.0, 7.5, 12.0, 1e-3)
    n = nx * ny * nz

    def step_us(offset):
        p, q, v = (torch_cuda.zeros(n + 4, device="cuda")[offset:offset + n].view(shape)
                   for _ in range(3))
        e0, e1 = (torch_cuda.cuda.Event(enable_timing=True) for _ in range(2))
        best = float("inf")
        for _ in range(6):
            e0.record()
            for _ in range(50):
                sb.wave_step_exact(p, q, v, q, g)
            e1.record()
            e1.synchronize()
            best = min(best, e0.elapsed_time(e1) * 20.0)
        return best

    assert step_us(0) <= 1.4 * step_us(1)


# both tiles of the ragged kernel: 32 x 32 and 64 x 16
@pytest.mark.parametrize("nx, ny, nz", [(89, 88, 88), (69, 88, 110)], ids=["32x32", "64x16"])
@pytest.mark.parametrize("heat", [False, True], ids=["acoustic", "heat"])
def test_ragged_splits_bit_for_bit(torch_cuda, heat, nx, ny, nz):
    """Chunks of 1, 2, 3, 7, 8, 9, 16, 17 planes (around its groups of 4 and unroll of 8) and
    one of all."""
    d, dt = (10.0, 7.5, 12.0), np.float32(1e-3)
    g = sb.Grid(nx, ny, nz, *d, float(dt))
    cur, prev, vel2 = case(g.shape, nx)
    dev = [torch_cuda.from_numpy(a).cuda() for a in (cur, prev, vel2)]
    if heat:
        k = np.full(g.shape, np.float32(900.0) * dt, np.float32)
        ref = oracle.wave_step(cur, cur, k, *d, np.float32(1.0), out=prev.copy())
    else:
        ref = oracle.wave_step(cur, prev, vel2, *d, dt, out=prev.copy())
    kind = sb.KIND_HEAT_F32 if heat else sb.KIND_WAVE_F32
    inz = nz - 8
    try:
        for planes in (1, 2, 3, 7, 8, 9, 16, 17, inz):
            sb.set_pencil_override(kind, 0, -(-inz // planes))
            out = dev[1].clone()
            if heat:
                sb.heat_step(dev[0], out, g, 900.0)
            else:
                sb.wave_step(dev[0], out, dev[2], out, g)
            assert np.array_equal(out.cpu().numpy(), ref), planes
    finally:
        sb.set_pencil_override(kind, -1, 1)
    assert sb.device_error() == 0


@pytest.mark.parametrize("nx, ny, nz", [(89, 88, 88), (69, 88, 110), (41, 40, 44)],
                         ids=["32x32", "64x16", "one thread per point"])
def test_ragged_runs_bit_for_bit(torch_cuda, nx, ny, nz):
    """Whole runs on ragged rows: the source's sample and the trace through the device's step
    counter, eager and in graphs entered at both parities, against the oracle; heat alike."""
    d, dt = (10.0, 7.5, 12.0), np.float32(7e-4)
    g = sb.Grid(nx, ny, nz, *d, float(dt))
    cur, prev, vel2 = case(g.shape, nz)
    src = g.index(nx - 6, 5, nz // 2)
    pieces = (3, 20, 1, 21, 4)
    n = sum(pieces)
    w = np.random.default_rng(2).uniform(-1, 1, n).astype(np.float32)
    a, b = cur.copy(), prev.copy()
    trace = np.zeros(n, np.float32)
    for k in range(n):
        out = oracle.wave_step(a, b, vel2, *d, dt, out=b.copy())
        out.reshape(-1)[src] += np.float32(dt * dt) * vel2.reshape(-1)[src] * w[k]
        trace[k] = out.reshape(-1)[src]
        a, b = out, a
    kv = np.full(g.shape, np.float32(900.0) * dt, np.float32)
    u = cur
    for k in range(n):
        u = oracle.wave_step(u, u, kv, *d, np.float32(1.0), out=u.copy())
    for chunk in (0, 20):
        with sb.Run(g, src_index=src, graph_chunk=chunk) as r:
            r.set_fields(cur, prev, vel2)
            r.set_wavelet(w)
            for k in pieces:
                r.steps(k)
            assert np.array_equal(r.field(), a) and np.array_equal(r.trace(n), trace), chunk
        with sb.Run(g, physics=sb.PHYSICS_HEAT, diffusivity=900.0, graph_chunk=chunk) as r:
            r.set_fields(cur)
            for k in pieces:
                r.steps(k)
            assert np.array_equal(r.field(), u), chunk
    assert sb.device_error() == 0
