"""Prompt portions of latent attention in expanded form with a sink per head, against the kernel
that works on the latent itself and against float64 softmax with the sink in its denominator."""

import pytest
import torch

from hetero_serve_b200.kernels.ops import CudaOps

pytestmark = pytest.mark.gpu
DEV = "cuda"


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
