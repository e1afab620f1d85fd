"""Prompt portions of latent attention with a sink per head: the expanded form against float64
softmax with the sink in its denominator; the mixer over portions behind positions of their own and
single tokens between them, with a window and a gate, in both forms; which of them a step takes."""

from types import SimpleNamespace

import pytest
import torch

from hetero_serve_b200.engine.step import CacheView
from hetero_serve_b200.kernels.ops import CudaOps
from hetero_serve_b200.parts import Model  # noqa: F401  (registers the parts)
from hetero_serve_b200.parts.latent_attention import LatentAttention

pytestmark = pytest.mark.gpu
DEV = "cuda"
PAGE = 16


@pytest.mark.parametrize("n,sinks", [(5, (0.0, 3.0)), (128, (-4.0, 30.0)), (300, (1.0, -30.0))])
def test_sink_in_the_denominator(n, sinks):
    H, D, P, V, R = 2, 64, 64, 64, 64
    ops = CudaOps(DEV)
    g = torch.Generator(device=DEV).manual_seed(n)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g).bfloat16()  # noqa: E731
    q, kv, rope = rnd(n, H * (D + P)), rnd(n, H * (D + V)), rnd(n, 64)
    out = torch.zeros(n, H * V, dtype=torch.bfloat16, device=DEV)
    plan = ops.make_plan([(0, 0, 0, n)], n, 16)
    base = torch.zeros(1, dtype=torch.int32, device=DEV)
    sink = torch.tensor(sinks, device=DEV)
    scale = (D + P) ** -0.5
    ops.latent_prompt_attention(out, q, kv, rope, base, plan, n_heads=H, dim=D, rot_dim=P, vdim=V,
                                rank=R, window=0, scale=scale, status=ops.status, sink=sink)
    qd = q.double().view(n, H, D + P)
    k = kv[:, :H * D].double().view(n, H, D)
    v = kv[:, H * D:].double().view(n, H, V)
    s = (torch.einsum("nhd,mhd->hnm", qd[..., :D], k)
         + torch.einsum("nhp,mp->hnm", qd[..., D:], rope.double())) * scale
    s = s.masked_fill(torch.ones(n, n, device=DEV).triu(1).bool(), float("-inf"))
    s = torch.cat([s, sink.double().view(H, 1, 1).expand(H, n, 1)], -1)
    want = torch.einsum("hnm,mhv->nhv", torch.softmax(s, -1)[..., :-1], v).flatten(1)
    # weights and outputs are rounded to bfloat16: two roundings of 2^-9 of values that the sum of
    # the weights' magnitudes bounds
    assert float((out.double() - want).abs().max()) <= 2 * 2.0 ** -9 * float(v.abs().max())
    assert ops.status.item() == 0


def _mixer(sizes, batch, window, gate, seed):
    """A mixer, a step's context, its input rows, its cache, and the float64 result of the step."""
    H, D, P, V, R = sizes
    W, T, scale = 96, sum(n for _, n in batch), (sizes[1] + sizes[2]) ** -0.5
    g = torch.Generator(device=DEV).manual_seed(seed)
    rnd = lambda *s, std=1.0: torch.randn(*s, device=DEV, generator=g) * std  # noqa: E731
    t = {"q": rnd(H * (D + P), W, std=W ** -0.5), "dkv": rnd(R + P, W, std=W ** -0.5),
         "uk": rnd(H * D, R, std=R ** -0.5), "uv": rnd(H * V, R, std=R ** -0.5),
         "o": rnd(W, H * V, std=(H * V) ** -0.5)}
    if gate:
        t["g"] = rnd(H * V, W, std=W ** -0.5)
    t = {n: v.bfloat16() for n, v in t.items()}
    t["norm"], t["sink"] = 1.0 + 0.1 * rnd(R), 3.0 + rnd(H)           # (a sink that matters)
    mixer = LatentAttention(width=W, n_heads=H, dim=D, rot_dim=P, vdim=V, kv_rank=R, scale=scale,
                            rot_base=10000.0, rot_dims=0, eps=1e-6, q_weight="q",
                            latent_weight="dkv", latent_norm="norm", key_up="uk", value_up="uv",
                            sink="sink", out_weight="o", window=window, gate="g" if gate else None)
    mixer.bind(t)
    ops = CudaOps(DEV)
    need = [-(-(p + n) // PAGE) for p, n in batch]
    pages, width = sum(need) + 1, max(need)
    order = torch.randperm(pages, generator=torch.Generator().manual_seed(seed)).tolist()
    table = torch.full((len(batch), width), -1, dtype=torch.int32)
    for r, k in enumerate(need):
        table[r, :k] = torch.tensor([order.pop() for _ in range(k)], dtype=torch.int32)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    buffers = {}

    def buffer(name, shape, dtype):
        key = (name, tuple(shape), dtype)
        if key not in buffers:
            buffers[key] = torch.zeros(*shape, dtype=dtype, device=DEV)
        return buffers[key]
    ctx = SimpleNamespace(
        ops=ops, status=ops.status, dtype=torch.bfloat16, n_requests=len(batch), buffer=buffer,
        tok_pos=i32([p + i for p, n in batch for i in range(n)]),
        tok_req=i32([r for r, (_, n) in enumerate(batch) for _ in range(n)]),
        req_start=i32([sum(n for _, n in batch[:r]) for r in range(len(batch))]),
        req_len=i32([n for _, n in batch]),
        plan=ops.make_plan([(r, r, p, n) for r, (p, n) in enumerate(batch)], T, PAGE))
    h = rnd(T, W).bfloat16()
    pool = rnd(pages, 1, 1, PAGE, R + P).bfloat16()
    cache = CacheView(pool=pool, table=table.to(DEV), page_size=PAGE, num_pages=pages, writes=True,
                      group=0)
    d = {n: v.double() for n, v in t.items()}
    hd = h.double()
    row = hd @ d["dkv"].T
    c = row[:, :R] / torch.sqrt((row[:, :R] ** 2).mean(-1, keepdim=True) + 1e-6) * d["norm"]
    rows, out, at = torch.cat([c, row[:, R:]], -1), [], 0
    q = (hd @ d["q"].T).view(T, H, D + P)
    for r, (p, n) in enumerate(batch):
        seen = pool[table[r, :need[r]].long()].double().reshape(-1, R + P)[:p + n].clone()
        seen[p:] = rows[at:at + n]
        k = torch.cat([(seen[:, :R] @ d["uk"].T).view(-1, H, D),
                       seen[:, None, R:].expand(-1, H, P)], -1)
        v = (seen[:, :R] @ d["uv"].T).view(-1, H, V)
        s = torch.einsum("nhd,mhd->hnm", q[at:at + n], k) * scale
        back = (torch.arange(p, p + n, device=DEV)[:, None]
                - torch.arange(p + n, device=DEV)[None])
        s = s.masked_fill((back < 0) | ((back >= window) if window else False), float("-inf"))
        s = torch.cat([s, d["sink"].view(H, 1, 1).expand(H, n, 1)], -1)
        out.append(torch.einsum("hnm,mhv->nhv", torch.softmax(s, -1)[..., :-1], v).flatten(1))
        at += n
    want = torch.cat(out)
    if gate:
        want = want * torch.sigmoid(hd @ d["g"].T)
    return mixer, ctx, h, cache, want @ d["o"].T


def _run(mixer, ctx, h, cache, expanded):
    ctx.ops.latent_expanded = expanded
    x = torch.zeros(h.shape[0], mixer.width, device=DEV)
    mixer.forward(ctx, h, x, cache)
    assert ctx.ops.status.item() == 0
    return x


@pytest.mark.parametrize("sizes", [(2, 64, 32, 64, 64), (3, 128, 64, 128, 256), (2, 128, 64, 128, 512)])
@pytest.mark.parametrize("window,gate", [(0, False), (0, True), (50, False)])
@pytest.mark.parametrize("batch", [[(0, 40), (70, 33), (300, 1), (20, 3)], [(700, 6), (0, 129)],
                                   [(90, 1)] * 64 + [(33, 9)]])
def test_portions_behind_positions_of_their_own(sizes, window, gate, batch):
    made = _mixer(sizes, batch, window, gate, len(batch) + sizes[4])
    mixer, ctx, h, cache, want = made
    assert mixer._prompt_rows(ctx, h.shape[0]) > 0
    off = [float((_run(*made[:4], form).double() - want).norm() / want.norm()) for form in (True, False)]
    # queries, keys (or absorbed queries), values (or mixed latents), weights and head rows are each
    # rounded to bfloat16 once: five relative errors of at most 2^-9
    assert off[0] <= 5 * 2.0 ** -9 and off[1] <= 5 * 2.0 ** -9, off
    assert off[0] <= 1.1 * off[1], off         # (the forms round as often: the same but for chance)


@pytest.mark.parametrize("sizes,batch", [((2, 64, 32, 64, 64), [(0, 7), (300, 20), (41, 1)]),
                                         ((2, 64, 32, 64, 64), [(100, 63)]),
                                         ((3, 128, 64, 128, 256), [(500, 5)]),
                                         ((2, 48, 32, 64, 64), [(0, 80)])])
def test_steps_in_which_the_latent_form_rounds_less_keep_it(sizes, batch):
    mixer, ctx, h, cache, want = _mixer(sizes, batch, 0, False, 5)
    assert mixer._prompt_rows(ctx, h.shape[0]) == 0
    got = _run(mixer, ctx, h, cache, True)
    assert torch.equal(got, _run(mixer, ctx, h, cache, False))
    assert float((got.double() - want).norm() / want.norm()) <= 5 * 2.0 ** -9
