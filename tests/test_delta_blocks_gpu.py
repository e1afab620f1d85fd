"""The delta rule's portions four tokens at a time: lengths around the blocks and stages, requests
without tokens, value columns that end inside a warp, decays of 0 and 1, against float64 and beside
the kernel that goes token after token."""

import pytest
import torch

from hetero_serve_b200.kernels.ops import CudaOps

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dim,vdim,heads,kv_heads", [(64, 128, 2, 1), (128, 20, 3, 3), (256, 33, 1, 1)])
@pytest.mark.parametrize("lens", [(8,), (9, 30), (1, 31, 4, 0, 40), (33, 64, 5, 2)])
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
        assert ops.launches - before == (2 if blocks and T >= 8 * R else 1)
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


def test_few_tokens_a_request_go_token_after_token():
    ops = CudaOps(DEV)
    shape = dict(heads=1, kv_heads=1, dim=64, vdim=8, taps=1, a_rank=4, g_rank=4)
    z = lambda *s: torch.ones(*s, device=DEV)  # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    before = ops.launches
    ops.delta_recurrence(z(4, 8), z(1, 512), z(4, 64), z(4, 64), z(4, 8), z(4, 1), z(4, 64),
                         i32([0]), i32([4]), i32([0]), shape)
    assert ops.launches == before + 1
