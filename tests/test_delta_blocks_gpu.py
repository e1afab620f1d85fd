"""The delta rule's portions four tokens at a time: lengths around the blocks and stages, requests
without tokens, value columns that end inside a warp, decays of 0 and 1, values that are not finite,
against float64 and beside the kernel that goes token after token; which requests take that form, and
that a request's bits are those it has alone."""

import json

import pedorax_cases as pc
import pytest
import torch

from hetero_serve_b200.engine.loading import load_model
from hetero_serve_b200.engine.step import Runner, StepEntry
from hetero_serve_b200.kernels.ops import CudaOps
from hetero_serve_b200.weights import write_model_dir

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dim,vdim,heads,kv_heads", [(64, 128, 2, 1), (128, 20, 3, 3), (256, 33, 1, 1)])
@pytest.mark.parametrize("lens", [(31,), (32,), (63, 1), (64,), (9, 70), (1, 31, 4, 0, 65, 101),
                                  (33, 64, 5, 2, 127, 66)])
def test_blocks_of_four(dim, vdim, heads, kv_heads, lens):
    ops = CudaOps(DEV)
    g = torch.Generator(device=DEV).manual_seed(dim + sum(lens))
    T, R, taps = sum(lens), len(lens), 2
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)  # noqa: E731
    qn = (unit(rnd(T, kv_heads, dim)) * dim ** -0.5).flatten(1).contiguous()
    kn = unit(rnd(T, kv_heads, dim)).flatten(1).contiguous()
    vv, beta = rnd(T, heads * vdim), torch.sigmoid(rnd(T, heads))
    decay = torch.sigmoid(2.0 * rnd(T, heads * dim) + 2.0)
    decay[:, 0], decay[:, 1] = 0.0, 1.0
    shape = dict(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, taps=taps, a_rank=4, g_rank=4)
    channels = 2 * kv_heads * dim + heads * vdim
    state0 = rnd(R + 1, heads * dim * vdim + (taps - 1) * channels) * 0.3
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    start = [sum(lens[:i]) for i in range(R)]
    slots = list(range(R, 0, -1))
    got = {}
    for blocks in (True, False):
        ops.delta_blocks = blocks
        o, state = torch.full((T, heads * vdim), float("nan"), device=DEV), state0.clone()
        before = ops.launches
        ops.delta_recurrence(o, state, qn, kn, vv, beta, decay, i32(start), i32(list(lens)),
                             i32(slots), shape)
        assert ops.launches - before == (3 if blocks and T >= ops.DELTA_LONG[dim] else 1)
        got[blocks] = o, state
    want_o, want_s = torch.empty(T, heads * vdim, dtype=torch.float64, device=DEV), state0.double()
    rep = heads // kv_heads
    for r, n in enumerate(lens):
        S = want_s[slots[r], :heads * dim * vdim].view(heads, dim, vdim)
        for t in range(start[r], start[r] + n):
            k = kn[t].double().view(kv_heads, dim).repeat_interleave(rep, 0)
            q = qn[t].double().view(kv_heads, dim).repeat_interleave(rep, 0)
            S.mul_(decay[t].double().view(heads, dim, 1))
            u = beta[t].double().view(heads, 1) * (vv[t].double().view(heads, vdim)
                                                   - torch.einsum("hdv,hd->hv", S, k))
            S.add_(k[:, :, None] * u[:, None])
            want_o[t] = torch.einsum("hdv,hd->hv", S, q).flatten()
    def off(o, s):
        return max(float((o.double() - want_o).norm() / want_o.norm()),
                   float((s.double() - want_s).norm() / want_s.norm()))
    short = [t for r, n in enumerate(lens) if n < ops.DELTA_LONG[dim]
             for t in range(start[r], start[r] + n)]
    assert torch.equal(got[True][0][short], got[False][0][short])
    # sums of dim products in float32, a few per token, through a state that the rule contracts:
    # sqrt(dim) + 2 roundings of 2^-24 and as many again for what earlier tokens left
    bound = 2.0 * (dim ** 0.5 + 2.0) * 2.0 ** -24
    assert off(*got[True]) <= bound and off(*got[False]) <= bound
    assert ops.status.item() == 0


@pytest.mark.parametrize("dim", [64, 128, 256])
@pytest.mark.parametrize("n", [64, 65, 66, 67])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_values_that_are_not_finite_stay_behind_their_token(dim, n, bad):
    """A token that brings an infinity or a NaN in one value column, or in its key or query: the
    outputs in front of it, the other columns and, behind the last token, the infinities of the state
    are those of the kernel that goes token after token."""
    ops, vdim = CudaOps(DEV), 24
    g = torch.Generator(device=DEV).manual_seed(dim + n)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)  # noqa: E731
    shape = dict(heads=1, kv_heads=1, dim=dim, vdim=vdim, taps=1, a_rank=4, g_rank=4)
    qn, kn, vv = unit(rnd(n, dim)) * dim ** -0.5, unit(rnd(n, dim)), rnd(n, vdim)
    beta, decay = torch.sigmoid(rnd(n, 1)), torch.sigmoid(rnd(n, dim) + 2.0)
    state0 = rnd(1, dim * vdim) * 0.3
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    bound = 4.0 * (dim ** 0.5 + 2.0) * 2.0 ** -24          # of either kernel off the exact result

    def both(q, k, v, s0):
        got = []
        for blocks in (True, False):
            ops.delta_blocks = blocks
            o, state = torch.zeros(n, vdim, device=DEV), s0.clone()
            before = ops.launches
            ops.delta_recurrence(o, state, q, k, v, beta, decay, i32([0]), i32([n]), i32([0]), shape)
            assert (ops.launches - before > 1) == blocks
            got.append((o, state.view(dim, vdim)))
        return got

    def close(a, b):
        assert torch.isfinite(b).all() and float((a - b).norm()) <= bound * float(b.norm())
    for at in range(n - 7, n):                             # every place of a block, and its end
        v = vv.clone()
        v[at, 3] = bad
        (o, s), (o1, s1) = both(qn, kn, v, state0)
        close(o[:at], o1[:at])
        others = [c for c in range(vdim) if c != 3]
        close(o[:, others], o1[:, others])
        close(s[:, others], s1[:, others])
        assert not torch.isfinite(o[at, 3])
        if at == n - 1 and bad == float("inf"):            # nothing behind it: infinities of k's signs
            assert torch.isinf(s1[:, 3]).all() and torch.equal(s[:, 3], s1[:, 3])
        else:
            assert not torch.isfinite(s[:, 3]).any()
        for name in ("q", "k"):
            x = (qn if name == "q" else kn).clone()
            x[at, 5] = bad
            (o, s), (o1, s1) = both(x if name == "q" else qn, x if name == "k" else kn, vv, state0)
            close(o[:at], o1[:at])
            if name == "q":                                # only this token's output reads it
                close(o[at + 1:], o1[at + 1:])
                close(s, s1)


@pytest.mark.parametrize("tokens,requests,plan,launches", [(4, 1, False, 1), (63, 1, False, 1),
                                                           (64, 1, False, 3), (64, 1, True, 2),
                                                           (64, 64, True, 1), (160, 10, True, 1)])
def test_steps_of_one_kind_of_request_launch_that_kind(tokens, requests, plan, launches):
    ops = CudaOps(DEV)
    shape = dict(heads=1, kv_heads=1, dim=64, vdim=8, taps=1, a_rank=4, g_rank=4)
    z = lambda *s: torch.ones(*s, device=DEV)  # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    n = tokens // requests
    more = {"plan": ops.make_plan([(r, r, 0, n) for r in range(requests)], tokens, 16)} if plan else {}
    before = ops.launches
    ops.delta_recurrence(z(tokens, 8), z(requests, 512), z(tokens, 64), z(tokens, 64), z(tokens, 8),
                         z(tokens, 1), z(tokens, 64), i32([n * r for r in range(requests)]),
                         i32([n] * requests), i32(list(range(requests))), shape, **more)
    assert ops.launches == before + launches


@pytest.mark.parametrize("dim", [64, 128, 256])
def test_a_request_has_the_bits_it_has_alone(dim):
    """Portions on both sides of the limit and a single token, each alone and beside the others."""
    ops, heads, vdim = CudaOps(DEV), 2, 40
    g = torch.Generator(device=DEV).manual_seed(dim)
    lens = [1, 200, 5, ops.DELTA_LONG[dim], 1, ops.DELTA_LONG[dim] - 1, 30] + [1] * 40
    lens += [0] * 30 + [ops.DELTA_LONG[dim] + 2]           # (more than the requests of one warp)
    T, R = sum(lens), len(lens)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    qn, kn, vv = 0.1 * rnd(T, heads * dim), 0.1 * rnd(T, heads * dim), rnd(T, heads * vdim)
    beta, decay = torch.sigmoid(rnd(T, heads)), torch.sigmoid(rnd(T, heads * dim) + 2.0)
    shape = dict(heads=heads, kv_heads=heads, dim=dim, vdim=vdim, taps=1, a_rank=4, g_rank=4)
    state0 = rnd(R, heads * dim * vdim) * 0.3
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    start = [sum(lens[:r]) for r in range(R)]
    o, state = torch.zeros(T, heads * vdim, device=DEV), state0.clone()
    ops.delta_recurrence(o, state, qn, kn, vv, beta, decay, i32(start), i32(lens),
                         i32(list(range(R))), shape)
    for r in [*range(7), R - 1]:
        at, n = start[r], lens[r]
        part = lambda x: x[at:at + n].contiguous()  # noqa: E731
        o1, s1 = torch.zeros(n, heads * vdim, device=DEV), state0.clone()
        ops.delta_recurrence(o1, s1, part(qn), part(kn), part(vv), part(beta), part(decay), i32([0]),
                             i32([n]), i32([r]), shape)
        assert torch.equal(o1, o[at:at + n]) and torch.equal(s1[r], state[r]), (r, n)
    assert ops.status.item() == 0


# layers whose delta heads are of the sizes that go four tokens at a time
CONFIG = {
    "architecture": "Pedorax", "vocab": 70, "width": 48, "embedding": {"scale": 1.0},
    "logit_scale": 0.5, "norm": {"eps": 1e-5},
    "layers": [
        {"type": "channel_delta", "mixer": pc._delta(2, 1, 64, 24, 4, 5, 7), "mlp": None},
        {"type": "channel_delta", "mixer": pc._delta(1, 1, 128, 20, 3, 4, 4), "mlp": None},
    ],
}


@pytest.mark.parametrize("graphs", [False, True])
def test_the_engine_with_heads_of_these_sizes(tmp_path, graphs):
    """Float32: the plain model's logits, and those of a request alone beside others."""
    write_model_dir(tmp_path, CONFIG, 21, "float32")
    case = pc.Case("wide", tmp_path, json.loads((tmp_path / "config.json").read_text()), 21)

    def runner():
        model, _ = load_model(case.dir, "float32", DEV)
        return Runner(model, num_pages=80, page_size=16, max_requests=40, dtype=model.dtype,
                      device=DEV, cuda_graphs=graphs)
    a, b, c = case.tokens(230, 1), case.tokens(140, 2), case.tokens(61, 3)
    alone = runner()
    want = alone.step([StepEntry("a", a[:150], want=[10, 149])]).logits.clone()
    want2 = alone.step([StepEntry("a", a[150:229], want=[78])]).logits.clone()
    want3 = alone.step([StepEntry("a", a[229:], want=[0])]).logits.clone()
    rn = runner()
    rn.step([StepEntry("c", c)])
    singles = [StepEntry(f"s{i}", [i % case.vocab]) for i in range(30)]
    got = rn.step([StepEntry("b", b[:7]), *singles, StepEntry("a", a[:150], want=[10, 149]),
                   StepEntry("c", [5])]).logits.clone()
    got2 = rn.step([StepEntry("a", a[150:229], want=[78]), StepEntry("b", b[7:]), *singles]).logits.clone()
    got3 = rn.step([*singles, StepEntry("a", a[229:], want=[0])]).logits.clone()
    for x, y in ((got, want), (got2, want2), (got3, want3)):
        assert torch.equal(x, y)
    plain = case.logits(a)
    for row, at in ((got[0], 10), (got[1], 149), (got2[0], 228), (got3[0], 229)):
        assert pc.rms_error(row.cpu(), plain[at]) < 2e-5
