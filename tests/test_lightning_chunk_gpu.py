"""Lightning attention and retention in chunks: closer to float64 than the walk token by token, each
request by its own length, and numbers that are not finite stay behind their token."""

import pytest
import torch

from hetero_serve_b200.kernels.ops import CudaOps

pytestmark = pytest.mark.gpu
DEV = "cuda"


def inputs(lens, H, D, V, rot, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    T, R = sum(lens), len(lens)
    proj = torch.randn(T, 2 + H * (2 * D + V), device=DEV, generator=g)
    state = torch.randn(R + 1, H * D * V, device=DEV, generator=g)
    pos = [100 * r + t for r, n in enumerate(lens) for t in range(n)]
    freq = 10000.0 ** (-torch.arange(max(rot // 2, 1), device=DEV) * 2.0 / max(rot, 1))
    return proj, state, pos, freq.float()


def walk(lens, proj, state, pos, freq, decay, H, D, V, rot, act, scale):
    """The recurrence in float64; angles from the float32 frequencies."""
    x = proj.double()
    x = torch.nn.functional.silu(x) if act == "silu" else x
    q, k, v = x[:, 2:2 + H * D], x[:, 2 + H * D:2 + 2 * H * D], x[:, 2 + 2 * H * D:]
    q, k, v = q.view(-1, H, D).clone(), k.view(-1, H, D).clone(), v.view(-1, H, V)
    if rot:
        angle = torch.tensor(pos, device=DEV).double()[:, None] * freq.double()[:rot // 2]
        c, s = torch.cos(angle)[:, None], torch.sin(angle)[:, None]
        for u in (q, k):
            a, b = u[..., :rot // 2].clone(), u[..., rot // 2:rot].clone()
            u[..., :rot // 2], u[..., rot // 2:rot] = a * c - b * s, b * c + a * s
        k = k * scale
    o, S, at = torch.zeros_like(v), state.double().view(-1, H, D, V).clone(), 0
    for r, n in enumerate(lens):
        slot = len(lens) - r
        for t in range(at, at + n):
            S[slot] = S[slot] * decay.double()[:, None, None] + k[t, :, :, None] * v[t, :, None]
            o[t] = torch.einsum("hdv,hd->hv", S[slot], q[t])
        at += n
    return o.flatten(1), S.flatten(1)


def run(ops, lens, proj, state, pos, freq, decay, H, D, V, rot, act, scale, chunks):
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    o, S, R = torch.full((sum(lens), H * V), float("nan"), device=DEV), state.clone(), len(lens)
    more = dict(tok_pos=i32(pos), freq=freq, rot_dims=rot, k_scale=scale) if rot else {}
    ops.lightning_recurrence(o, S, proj, decay, i32([sum(lens[:r]) for r in range(R)]), i32(lens),
                             i32(list(range(R, 0, -1))), q_off=2, k_off=2 + H * D, v_off=2 + 2 * H * D, heads=H,
                             dim=D, vdim=V, act=act, chunks=chunks, **more)
    return o, S


@pytest.mark.parametrize("rot, act", [(128, "none"), (0, "silu"), (64, "silu"), (4, "none")])
@pytest.mark.parametrize("lens", [(512,), (513, 3, 0, 511), (64, 575, 576), (600, 1, 1025)])
def test_against_float64(rot, act, lens):
    D, V = 128, 128
    H, decay = 3, torch.tensor([0.9961, 0.55, 0.93], device=DEV)
    ops = CudaOps(DEV)
    proj, state, pos, freq = inputs(lens, H, D, V, rot, D + V + sum(lens))
    args = (lens, proj, state, pos, freq, decay, H, D, V, rot, act, 0.125)
    want_o, want_S = walk(*args)
    (o, S), (po, pS) = run(ops, *args, chunks=True), run(ops, *args, chunks=False)
    err = lambda a, b: float((a.double() - b).norm() / b.norm())  # noqa: E731
    # sequential sums round every token: the chunks are to be no further off (a few roundings of 2^-24 where
    # a portion has only a handful of chunks)
    assert err(o, want_o) <= err(po, want_o) * 1.02 + 2e-8 and err(S, want_S) <= err(pS, want_S) * 1.02 + 2e-8
    assert err(o, want_o) < 1e-6 and err(S, want_S) < 1e-6
    at = 0
    for r, n in enumerate(lens):               # short portions and their states: the same bits
        if n < 512:
            assert torch.equal(o[at:at + n], po[at:at + n])
            assert torch.equal(S[len(lens) - r], pS[len(lens) - r])
        at += n
    assert torch.equal(S[0], state[0])         # nobody's slot
    # a request's chunks do not depend on its neighbours
    n = max(lens)
    at = sum(lens[:lens.index(n)])
    alone = (proj[at:at + n].clone(), state[[0, len(lens) - lens.index(n)]].clone(), pos[at:at + n])
    ao, aS = run(ops, (n,), *alone, freq, decay, H, D, V, rot, act, 0.125, chunks=True)
    assert torch.equal(ao, o[at:at + n]) and torch.equal(aS[1], S[len(lens) - lens.index(n)])
    assert ops.status.item() == 0


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), 3.3e38])
@pytest.mark.parametrize("where", ["q", "k", "v", "state"])
def test_numbers_that_are_not_finite_stay_behind_their_token(bad, where):
    H, D, V, lens, t = 2, 128, 128, (576,), 100
    ops, decay = CudaOps(DEV), torch.tensor([0.99, 0.5], device=DEV)
    proj, state, pos, freq = inputs(lens, H, D, V, 0, 7)
    args = lambda p, s: (lens, p, s, pos, freq, decay, H, D, V, 0, "none", 1.0)  # noqa: E731
    clean, _ = run(ops, *args(proj, state), chunks=True)
    p, s = proj.clone(), state.clone()
    if where == "state":
        s[1, 5 * V + 3] = bad
    else:
        p[t, 2 + {"q": 0, "k": H * D, "v": 2 * H * D}[where] + 3] = bad
    (o, S), (po, pS) = run(ops, *args(p, s), chunks=True), run(ops, *args(p, s), chunks=False)
    if where != "state":
        assert torch.equal(o[:64], clean[:64])             # the chunk before keeps its bits
        assert o[:t].isfinite().all()
    assert torch.equal(o.isnan(), po.isnan()) and torch.equal(S.isnan(), pS.isnan())
    assert torch.equal(o.isfinite(), po.isfinite()) and torch.equal(S.isfinite(), pS.isfinite())
    fine = po.isfinite() & (po.abs() < 1e30)
    assert bool(((o - po)[fine].abs() <= 1e-3 + 1e-4 * po[fine].abs()).all())


def test_decays_at_the_ends():
    H, D, V, lens = 3, 128, 128, (550,)
    ops, decay = CudaOps(DEV), torch.tensor([0.0, 1.0, 1e-3], device=DEV)
    proj, state, pos, freq = inputs(lens, H, D, V, 0, 8)
    args = (lens, proj, state, pos, freq, decay, H, D, V, 0, "none", 1.0)
    want_o, want_S = walk(*args)
    o, S = run(ops, *args, chunks=True)
    assert float((o.double() - want_o).norm() / want_o.norm()) < 1e-6
    assert float((S.double() - want_S).norm() / want_S.norm()) < 1e-6


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf")])
@pytest.mark.parametrize("where", ["k", "v", "state"])
def test_infinities_under_decays_whose_powers_vanish(bad, where):
    """The 64th power of these decays is zero or nearly; an infinity of the state is what the walk makes of it:
    itself as long as the decay is not zero."""
    H, D, V, lens, t = 4, 128, 128, (700,), 100
    ops, decay = CudaOps(DEV), torch.tensor([0.0, 1e-3, 0.1, 0.3], device=DEV)
    proj, state, pos, freq = inputs(lens, H, D, V, 0, 11)
    for h in range(H):
        if where == "state":
            state[1, h * D * V + 5 * V + 3] = bad
        else:
            proj[t, 2 + h * 128 + {"k": H * D, "v": 2 * H * D}[where] + 3] = bad
    args = (lens, proj, state, pos, freq, decay, H, D, V, 0, "none", 1.0)
    (o, S), (po, pS) = run(ops, *args, chunks=True), run(ops, *args, chunks=False)
    for got, want in ((o, po), (S, pS)):
        assert torch.equal(got.isnan(), want.isnan())
        assert torch.equal(got.isinf(), want.isinf()) and torch.equal(got[got.isinf()], want[want.isinf()])
    assert bool(S.view(2, H, D * V)[1, 1:].isinf().any()) == (bad == bad)   # (a NaN leaves no infinity)


@pytest.mark.parametrize("rot, act", [(128, "none"), (0, "silu"), (4, "silu")])
def test_chunks_without_numbers_take_no_longer_than_the_recurrence(rot, act):
    """A prompt of NaNs from its middle on (what a layer before makes of one) in chunks, against the same prompt
    token by token: the same entries are finite, and the walk of such chunks is no slower than that."""
    H, D, V, lens = 8, 128, 128, (1024, 1024)
    ops, decay = CudaOps(DEV), torch.linspace(0.9, 0.99, H, device=DEV)
    proj, state, pos, freq = inputs(lens, H, D, V, rot, 3)
    proj[700:1024] = float("nan")
    proj[1500:, 2 + H * D + 5] = float("nan")                  # one entry of k of every later token
    args = (lens, proj, state, pos, freq, decay, H, D, V, rot, act, 0.1)
    (o, S), (po, pS) = run(ops, *args, chunks=True), run(ops, *args, chunks=False)
    assert torch.equal(o.isnan(), po.isnan()) and torch.equal(S.isnan(), pS.isnan())
    fine = po.isfinite()
    assert bool(((o - po).abs()[fine] <= 1e-4 * po.abs()[fine] + 1e-4 * po[fine].abs().mean()).all())

    def best(chunks):
        graph, times = torch.cuda.CUDAGraph(), []
        more = dict(tok_pos=i32(pos), freq=freq, rot_dims=rot, k_scale=0.1) if rot else {}
        o, S, a = torch.empty_like(po), state.clone(), (i32([0, 1024]), i32(lens), i32([2, 1]))
        with torch.cuda.graph(graph):
            for _ in range(4):
                ops.lightning_recurrence(o, S, proj, decay, *a, q_off=2, k_off=2 + H * D, v_off=2 + 2 * H * D,
                                         heads=H, dim=D, vdim=V, act=act, chunks=chunks, **more)
        for _ in range(6):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            graph.replay()
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    assert best(True) <= 1.25 * best(False)


@pytest.mark.parametrize("lens", [(8,) * 64, (600, 700), (511, 1, 512)])
@pytest.mark.parametrize("rot", [0, 128])
def test_only_the_forms_of_the_step_are_launched(lens, rot):
    """A plan says which lengths there are: the same bits as without one, and no kernel that has no request."""
    H, D, V = 2, 128, 128
    proj, state, pos, freq = inputs(lens, H, D, V, rot, 5)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    ops, decay = CudaOps(DEV), torch.tensor([0.9, 0.99], device=DEV)
    start = [sum(lens[:r]) for r in range(len(lens))]
    plan = ops.make_plan([(r, r, 0, n) for r, n in enumerate(lens)], sum(lens), 16)
    more = dict(tok_pos=i32(pos), freq=freq, rot_dims=rot) if rot else {}
    got, graph = [], []
    for p in (None, plan):
        o, S = torch.full((sum(lens), H * V), float("nan"), device=DEV), state.clone()
        call = lambda: ops.lightning_recurrence(  # noqa: E731
            o, S, proj, decay, i32(start), i32(lens), i32(list(range(len(lens)))), q_off=2, k_off=2 + H * D,
            v_off=2 + 2 * H * D, heads=H, dim=D, vdim=V, act="silu", chunks=True, plan=p, **more)
        before = ops.launches
        call()
        got.append((o.clone(), S.clone(), ops.launches - before))
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            call()
            torch.cuda.synchronize()
        graph.append([e.key for e in prof.key_averages() if "lightning" in e.key])
    (a, sa, _), (b, sb, launches) = got
    assert torch.equal(a, b) and torch.equal(sa, sb)
    chunked, walked = max(lens) >= 512, min(lens) < 512
    assert launches == (3 + (rot > 0)) * chunked + 2 * walked
    if graph[1]:                                             # (where the profiler can see kernels)
        assert any("chunk" in k for k in graph[1]) == chunked
        assert any("chunk" not in k and "turns" not in k for k in graph[1]) == walked


def test_requests_in_chunks_among_many():
    """More requests than can go in chunks, before, between and behind those that do: each has the bits it has
    alone."""
    H, D, V, lens = 2, 128, 128, (3,) * 40 + (600, 0, 0, 5, 700) + (1,) * 70 + (512,)
    ops, decay = CudaOps(DEV), torch.tensor([0.9, 0.99], device=DEV)
    proj, state, pos, freq = inputs(lens, H, D, V, 0, 13)
    rest = (freq, decay, H, D, V, 0, "silu", 1.0)
    o, S = run(ops, lens, proj, state, pos, *rest, chunks=True)
    for r in (0, 40, 43, 44, 60, len(lens) - 1):
        n, at, slot = lens[r], sum(lens[:r]), len(lens) - r
        one, sone = run(ops, (n,), proj[at:at + n].clone(), state[[0, slot]].clone(), pos[at:at + n], *rest, chunks=True)
        assert torch.equal(one, o[at:at + n]) and torch.equal(sone[1], S[slot])
    assert torch.equal(S[0], state[0])


@pytest.mark.parametrize("rot", [0, 128])
def test_heads_that_take_turns_with_the_scratch(rot):
    """More heads than the scratch holds states of: bounded, and each head has the bits it has in a part of them."""
    H, D, V, lens = 40, 128, 128, (4096, 20, 513)
    ops, decay = CudaOps(DEV), torch.linspace(0.5, 0.999, H, device=DEV)
    proj, state, pos, freq = inputs(lens, H, D, V, rot, 17)
    o, S = run(ops, lens, proj, state, pos, freq, decay, H, D, V, rot, "none", 0.5, chunks=True)
    held = sum(t.numel() for (name, _), t in ops._scratch.items() if name == "lightning_chunks")
    assert 0 < held <= 2 ** 25 + sum(lens) * rot
    for h0 in (0, 15, 35):                                  # five heads at a time
        cols = torch.cat([torch.arange(2 + b + h0 * 128, 2 + b + (h0 + 5) * 128) for b in (0, H * D, 2 * H * D)])
        part = torch.cat([proj[:, :2], proj[:, cols.to(DEV)]], 1).contiguous()
        st = state.view(-1, H, D * V)[:, h0:h0 + 5].reshape(-1, 5 * D * V).contiguous()
        po, pS = run(CudaOps(DEV), lens, part, st, pos, freq, decay[h0:h0 + 5].contiguous(), 5, D, V, rot, "none", 0.5,
                     chunks=True)
        assert torch.equal(po, o[:, h0 * V:(h0 + 5) * V])
        assert torch.equal(pS, S.view(-1, H, D * V)[:, h0:h0 + 5].reshape(-1, 5 * D * V))
