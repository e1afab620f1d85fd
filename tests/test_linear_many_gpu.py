"""bfloat16 layers of thousands of rows: the tile chosen, single or paired, is about as fast as the best."""

import pytest
import torch

from hetero_serve_b200.kernels.ops import CudaOps

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n, k", [(4096, 1024), (1024, 4096), (1280, 1280), (5120, 1280), (768, 3072), (3072, 1024)])
@pytest.mark.parametrize("m", [4096, 8192, 16384])
def test_the_tile_chosen(m, n, k):
    ops, g = CudaOps(DEV), torch.Generator(device=DEV).manual_seed(n)
    a = torch.randn(m, k, device=DEV, generator=g).bfloat16()
    ws = [(torch.randn(n, k, device=DEV, generator=g) * 0.03).bfloat16() for _ in range(4)]
    out, times = torch.empty(m, n, device=DEV, dtype=torch.bfloat16), {}
    for tile, pairs in ((0, -1), (128, 0), (192, 0), (256, 0), (128, 1), (256, 1)):
        ops.tile_n, ops.cta_pairs = tile, pairs
        ops.linear(out, a, ws[0])
        graph, best = torch.cuda.CUDAGraph(), []
        with torch.cuda.graph(graph):
            for w in ws * 2:
                ops.linear(out, a, w)
        for _ in range(6):
            x, y = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            x.record()
            graph.replay()
            y.record()
            y.synchronize()
            best.append(x.elapsed_time(y))
        times[tile, pairs] = min(best)
    assert times.pop((0, -1)) <= 1.12 * min(times.values()), times
