"""The tcgen05 linear where rows of the output do not start on 16 bytes: the bits of the same columns of
a layer whose rows do."""

import pytest
import torch

from hetero_serve_b200.kernels.ops import CudaOps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("m", [17, 31, 32, 33, 129, 200])
@pytest.mark.parametrize("n", [257, 259, 1001, 1004])
@pytest.mark.parametrize("tile", [64, 128, 192, 256])
def test_same_bits_as_aligned_rows(tile, n, m, dtype):
    ops, k = CudaOps("cuda"), 64                 # one step of the summed index: nothing is split
    ops.tile_n, ops.skinny_max_rows = tile, 0
    ops.status = torch.zeros(1, dtype=torch.int32, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(n + m)
    pad = -n % 8
    a = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    w = torch.randn(n + pad, k, device="cuda", generator=g).bfloat16()
    bias = torch.randn(n + pad, device="cuda", generator=g)
    for b, act in ((None, "none"), (bias, "gelu_tanh")):
        whole = torch.full((m, n + pad), float("nan"), device="cuda", dtype=dtype)
        part = torch.full((m * n + 8,), 7.0, device="cuda", dtype=dtype)
        ops.linear(whole, a, w, b, act=act)
        ops.linear(part[:m * n].view(m, n), a, w[:n].contiguous(), None if b is None else b[:n].clone(), act=act)
        assert torch.equal(part[:m * n].view(m, n), whole[:, :n])
        assert bool((part[m * n:] == 7.0).all())             # nothing behind the last row
    assert ops.status.item() == 0
