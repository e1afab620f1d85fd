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


@pytest.mark.parametrize("kind", ["normal", "rounded", "masked", "nan"])
@pytest.mark.parametrize("vocab", [24576, 50257])
def test_lists_of_every_length(vocab, kind):
    """k around the lines between the ways its threshold is found: the tokens of a block a row."""
    ops, ks = CudaOps(DEV), [1, 63, 64, 65, 66, 100, 129, 200, 255, 256, 257, 400, 511, 512, 513, 700]
    g, n = torch.Generator(device=DEV).manual_seed(vocab + 1), len(ks)
    x = rows_of(kind, n, vocab, g)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    times = MOST // n + 1
    for draw in range(4):
        args = (x, torch.full((n,), 1.3, device=DEV), i32(ks), i32([draw] * n), i32(list(range(n))), i32([3] * n))
        got = torch.full((n,), -1, dtype=torch.int32, device=DEV)
        ops.sample(got, *args)
        want = torch.full((n * times,), -1, dtype=torch.int32, device=DEV)
        ops.sample(want, *(t.repeat(times, *[1] * (t.dim() - 1)).contiguous() for t in args))
        assert torch.equal(got, want[:n])


@pytest.mark.parametrize("k", [40, 100, 256, 400])
@pytest.mark.parametrize("vocab", [32000, 50257])
def test_clusters_take_no_longer_than_a_block_a_row(vocab, k):
    """Against one row more than clusters take, which goes a block a row, an SM each either way."""
    ops, g = CudaOps(DEV), torch.Generator(device=DEV).manual_seed(k)
    times = []
    for n in (32, MOST + 1):
        x = torch.randn(n, vocab, device=DEV, generator=g) * 3
        zero = torch.zeros(n, dtype=torch.int32, device=DEV)
        out, temp, graph = torch.empty(n, dtype=torch.int32, device=DEV), torch.full((n,), 0.8, device=DEV), None
        ops.sample(out, x, temp, zero + k, zero, zero, zero)
        kk, graph = zero + k, torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(10):
                ops.sample(out, x, temp, kk, zero, zero, zero)
        best = []
        for _ in range(8):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            graph.replay()
            b.record()
            b.synchronize()
            best.append(a.elapsed_time(b))
        times.append(min(best))
    assert times[0] <= 1.15 * times[1]
