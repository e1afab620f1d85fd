"""Top-k sampling where the threshold is hard to find: many equal logits at it, more of them than the
list of candidates holds, k around the number of threads, all logits equal, infinite logits; and rows
close to the longest that fits shared memory."""

import plain_ops
import pytest
import torch

from hetero_serve_b200.kernels.ops import CudaOps

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("vocab,step", [(50257, 0.25), (50257, 2.0), (50257, 0.0), (5000, 1.0),
                                        (56320, 0.5), (12000, 1.0), (11999, 0.05)])
@pytest.mark.parametrize("top_k", [1, 40, 511, 512, 513, 1023, 1024, 1025])
def test_threshold_among_equal_logits(vocab, step, top_k):
    ops, plain = CudaOps(DEV), plain_ops.PlainOps()
    g = torch.Generator(device=DEV).manual_seed(vocab + top_k)
    rows = 4
    lg = torch.randn(rows, vocab, device=DEV, generator=g) * 3.0
    if step:
        lg = torch.round(lg / step) * step         # ties everywhere
    lg[1] = 0.5                                    # nothing but ties
    lg[2, ::3] = -float("inf")
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    temp = torch.tensor([0.9, 1.0, 0.4, 2.0], device=DEV)
    k, lo, hi = i32([top_k] * rows), i32([7, 8, 9, 10]), i32([0] * rows)
    for pos in range(3):
        p = i32([pos] * rows)
        out, want = torch.empty(rows, dtype=torch.int32, device=DEV), torch.empty(rows, dtype=torch.int32)
        ops.sample(out, lg, temp, k, lo, hi, p)
        plain.sample(want, lg.cpu(), temp.cpu(), k.cpu(), lo.cpu(), hi.cpu(), p.cpu())
        assert out.tolist() == want.tolist(), (pos, out.tolist(), want.tolist())
