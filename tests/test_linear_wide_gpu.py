"""Very wide bfloat16 layers of few rows: the tile chosen is about as fast as the best of those there are."""

import pytest
import torch

from hetero_serve_b200.kernels.ops import CudaOps

pytestmark = pytest.mark.gpu
DEV = "cuda"


def time_of(ops, out, a, ws, tile):
    ops.tile_n = tile
    graph, best = torch.cuda.CUDAGraph(), []
    ops.linear(out, a, ws[0])
    with torch.cuda.graph(graph):
        for w in ws:                                   # together larger than the L2
            ops.linear(out, a, w)
    for _ in range(8):
        x, y = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        x.record()
        graph.replay()
        y.record()
        y.synchronize()
        best.append(x.elapsed_time(y))
    return min(best)


@pytest.mark.parametrize("n", [18944, 22016, 28160, 32000, 37888, 40000, 50257])
@pytest.mark.parametrize("m, k", [(32, 1024), (64, 768), (100, 1280)])
def test_the_width_chosen(m, k, n):
    ops, g = CudaOps(DEV), torch.Generator(device=DEV).manual_seed(n)
    a = torch.randn(m, k, device=DEV, generator=g).bfloat16()
    ws = [(torch.randn(n, k, device=DEV, generator=g) * 0.03).bfloat16() for _ in range(max(2, 260_000_000 // (2 * n * k) + 1))]
    out = torch.empty(m, n, device=DEV)
    times = {tile: time_of(ops, out, a, ws, tile) for tile in (0, 128, 192, 256)}
    assert times.pop(0) <= 1.12 * min(times.values())
    want = a.float() @ ws[-1].float().T
    ops.tile_n = 0
    ops.linear(out, a, ws[-1])
    # k products of bfloat16 numbers summed in float32 on both sides
    assert bool(((out - want).abs() <= 2 * k * 2.0 ** -24 * (a.float().abs() @ ws[-1].float().abs().T)).all())
