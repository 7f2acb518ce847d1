"""Steps that follow work of several streams: the library's kernels begin as the last one on
their stream ends, and have to wait for everything else their stream waits for.  Eager and
captured, behind kernels, copies and fills of another stream; bits of the same calls in one
stream with a wait after each."""
from __future__ import annotations

import pytest

import stencil_solver_b200 as sb

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _clean(torch_cuda):
    yield
    torch_cuda.cuda.synchronize()
    assert sb.device_error() == 0


def fields(torch, g, seed, n):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return [torch.randn(g.shape, generator=gen, device="cuda") for _ in range(n)]


# a branch's last piece of work before the join
BRANCHES = ["step", "copy", "fill", "torch kernel"]


@pytest.mark.parametrize("branch", BRANCHES)
@pytest.mark.parametrize("kind", ["wave", "exact", "heat"])
@pytest.mark.parametrize("captured", [False, True], ids=["eager", "captured"])
def test_steps_behind_a_join_of_two_streams(torch_cuda, captured, kind, branch):
    """A long step on a second stream, then `branch`, joins a short step on the first; the
    step behind the join reads what both wrote, and a third one follows it at once."""
    torch = torch_cuda
    small, big = sb.Grid(96, 80, 72, 10.0, 10.0, 10.0, 7e-4), sb.Grid(256, 256, 256, 10.0, 10.0, 10.0, 7e-4)
    p, q, v, a, b = fields(torch, small, 1, 5)
    P, Q, V = fields(torch, big, 2, 3)
    v.square_().add_(1.0).mul_(1e6)
    V.square_().add_(1.0).mul_(1e6)
    out, last = torch.zeros_like(p), torch.zeros_like(p)
    n = p.numel()

    def step(x, y, z, g, s):
        """z = a step of x and y (heat: of x)."""
        if kind == "wave":
            sb.wave_step(x, y, v if g is small else V, z, g, stream=s)
        elif kind == "exact":
            sb.wave_step_exact(x, y, v if g is small else V, z, g, stream=s)
        else:
            sb.heat_step(x, z, g, 1.0, stream=s)

    def pieces(s1, s2):
        """(stream, call) in order; None: the join of s2 into s1."""
        def last_of_branch():
            part = Q.view(-1)[:n].view(p.shape)
            if branch == "step":
                step(part, q, b, small, s2)
            elif branch == "copy":
                b.copy_(part)
            elif branch == "fill":
                b.fill_(0.5)
            else:
                torch.mul(part, 2.0, out=b)

        return [(s2, lambda: step(P, Q, Q, big, s2)), (s2, last_of_branch),
                (s1, lambda: step(p, q, a, small, s1)), None,
                (s1, lambda: step(a if kind != "heat" else b, b, out, small, s1)),
                (s1, lambda: step(out, a, last, small, s1))]

    state = [t.clone() for t in (p, q, a, b, P, Q, out, last)]

    def reset():
        for t, w in zip((p, q, a, b, P, Q, out, last), state):
            t.copy_(w)
        torch.cuda.synchronize()

    one = torch.cuda.Stream()
    torch.cuda.synchronize()  # the fields come from the default stream
    for piece in pieces(one, one):
        if piece:
            with torch.cuda.stream(one):
                piece[1]()
            torch.cuda.synchronize()
    want = [t.clone() for t in (a, b, out, last)]
    reset()

    def run(s1, s2):
        s2.wait_stream(s1)
        for piece in pieces(s1, s2):
            if piece:
                with torch.cuda.stream(piece[0]):
                    piece[1]()
            else:
                s1.wait_stream(s2)

    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    if captured:
        run(s1, s2)
        torch.cuda.synchronize()
        reset()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s1):
            run(s1, s2)
    for _ in range(10):
        reset()
        if captured:
            graph.replay()
        else:
            run(s1, s2)
        torch.cuda.synchronize()
        for got, w in zip((a, b, out, last), want):
            assert torch.equal(got, w)


@pytest.mark.parametrize("kind", ["wave", "exact", "heat", "half", "ragged"])
def test_steps_on_five_streams_give_the_bits_of_one(torch_cuda, kind):
    """Rounds of steps of unlike grids, each on its own stream (beside two others they take
    another tile and split than alone), against each grid by itself."""
    torch = torch_cuda
    shapes = [(96, 88, 80), (128, 64, 100), (160, 72, 61), (64, 120, 90), (200, 48, 77)]
    sets = []
    for k, (nx, ny, nz) in enumerate(shapes):
        g = sb.Grid(nx + (kind == "ragged"), ny, nz, 10.0, 10.0, 10.0, 7e-4)
        p, q, v = fields(torch, g, k, 3)
        v.square_().add_(1.0).mul_(1e6)
        if kind == "half":
            halves = [torch.empty(g.shape, dtype=torch.int16, device="cuda") for _ in range(3)]
            sb.f16_pack(p, halves[0], g.size, 256.0)
            sb.f16_pack(q, halves[1], g.size, 256.0)
            sb.k_field_bf16(v, halves[2], g)
            p, q, v = halves
        sets.append((g, p, q, v, torch.tensor([256.0, 1.0], device="cuda")))

    def run(g, p, q, v, scale, stream, rounds=7):
        for _ in range(rounds):
            if kind == "half":
                sb.wave_step_f16(p, q, v, g, scale, stream=stream)
            elif kind == "heat":
                sb.heat_step(p, q, g, 1.0, stream=stream)
            else:
                (sb.wave_step_exact if kind == "exact" else sb.wave_step)(p, q, v, q, g, stream=stream)
            p, q = q, p
        return p

    want = []
    for g, p, q, v, scale in sets:
        want.append(run(g, p.clone(), q.clone(), v, scale, None))
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in sets]
    state = [[p.clone(), q.clone()] for _, p, q, _, _ in sets]
    torch.cuda.synchronize()
    for _ in range(7):
        for (g, _, _, v, scale), s, pq in zip(sets, streams, state):
            run(g, pq[0], pq[1], v, scale, s, 1)
            pq.reverse()
    torch.cuda.synchronize()
    for pq, w in zip(state, want):
        assert torch.equal(pq[0], w)
