"""Sampling with a row over a cluster of blocks: the tokens of the kernel with a block a row, which more
rows than a launch of clusters takes go to."""

import pytest
import torch

from hetero_serve_b200.kernels.ops import CudaOps

pytestmark = pytest.mark.gpu
DEV = "cuda"
MOST = 64                                    # rows the clusters take


def rows_of(kind, n, vocab, g):
    x = torch.randn(n, vocab, device=DEV, generator=g) * 2.5
    if kind == "rounded":                    # ties everywhere
        x = x.round()
    elif kind == "equal":
        x = torch.zeros_like(x)
    elif kind == "masked":                   # most of the row at the lowest value or minus infinity
        x[:, 50:] = torch.finfo(torch.float32).min
        x[1::2, 40:] = -float("inf")
    elif kind == "nan":
        x[:, 5::977] = float("nan")
        x[1::2, :4000] = -float("nan")
        x[2::3] = float("nan")
    elif kind == "inf":
        x[:, 77] = float("inf")
        x[1::2, 78] = float("inf")
    elif kind == "sorted":
        x = x.sort(-1, descending=True).values
    return x


@pytest.mark.parametrize("kind", ["normal", "rounded", "equal", "masked", "nan", "inf", "sorted"])
@pytest.mark.parametrize("vocab", [24576, 24577, 32000, 50257, 55000])
def test_same_tokens_as_a_block_a_row(vocab, kind):
    ops, n = CudaOps(DEV), 14
    g = torch.Generator(device=DEV).manual_seed(vocab)
    x = rows_of(kind, n, vocab, g)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    temp = torch.tensor([0.0, 0.8, 1.0, 0.3, 0.9, 1.5, 0.7] * 2, device=DEV)
    k = i32([0, 0, 40, 1, 2048, 2049, vocab - 1, 7, 512, 0, 600, 10, vocab, 3])
    lo, hi, pos = i32([7 * i + 1 for i in range(n)]), i32([i for i in range(n)]), i32([i + 5 for i in range(n)])
    got = torch.full((n,), -1, dtype=torch.int32, device=DEV)
    ops.sample(got, x, temp, k, lo, hi, pos)
    times = MOST // n + 1
    many = lambda t: t.repeat(times, *[1] * (t.dim() - 1)).contiguous()  # noqa: E731
    want = torch.full((n * times,), -1, dtype=torch.int32, device=DEV)
    assert n * times > MOST
    ops.sample(want, many(x), many(temp), many(k), many(lo), many(hi), many(pos))
    assert torch.equal(want.view(times, n)[0], want.view(times, n)[-1])
    assert torch.equal(got, want[:n])
    # one row at a time
    for r in (0, 2, 5):
        one = torch.full((1,), -1, dtype=torch.int32, device=DEV)
        ops.sample(one, x[r:r + 1].contiguous(), temp[r:r + 1], k[r:r + 1], lo[r:r + 1], hi[r:r + 1], pos[r:r + 1])
        assert one.item() == got[r].item()


def test_feedback_and_status_word():
    ops, n, vocab = CudaOps(DEV), 3, 30000
    g = torch.Generator(device=DEV).manual_seed(3)
    x = torch.randn(n, vocab, device=DEV, generator=g)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    out, back, word = torch.full((n + 1,), -1, dtype=torch.int32, device=DEV), i32([-9] * 4), i32([6])
    ops.sample(out, x, torch.tensor([0.0, 1.0, 0.7], device=DEV), i32([0, 0, 5]), i32([1] * 3), i32([0] * 3),
               i32([2] * 3), feedback=back, feedback_slot=i32([2, -1, 0]), status_word=word)
    t = out.tolist()
    assert t[0] == int(x[0].argmax()) and t[3] == 6
    assert back.tolist() == [t[2], -9, t[0], -9]
