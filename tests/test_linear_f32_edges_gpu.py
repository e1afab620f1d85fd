"""The 32-bit linear at the row counts, widths and lengths where one kernel hands over to the next:
a row's bits are the same in every batch, and off float64 by no more than one rounding a product."""

import pytest
import torch

from hetero_serve_b200.kernels.ops import CudaOps

pytestmark = pytest.mark.gpu
ROWS = (1, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 100, 257)


@pytest.mark.parametrize("n,k", [(1024, 1024), (40, 132), (2400, 64), (63, 70), (33, 1023), (8, 4)])
def test_rows_keep_their_bits(n, k):
    ops = CudaOps("cuda")
    g = torch.Generator(device="cuda").manual_seed(n + k)
    a = torch.randn(max(ROWS), k, device="cuda", generator=g)
    w = torch.randn(n, k, device="cuda", generator=g)
    bias = torch.randn(n, device="cuda", generator=g)
    res = torch.randn(max(ROWS), n, device="cuda", generator=g)
    exact = a.double() @ w.double().T + bias.double() + res.double()
    # a chain of k fused multiply-adds and two additions, each off by half a unit of 2^-23 of a
    # running value that the sum of magnitudes bounds
    bound = (k + 2) * 2.0 ** -24 * (a.abs().double() @ w.abs().double().T + bias.abs() + res.abs())
    first = None
    for m in ROWS:
        out = torch.full((m, n), float("nan"), device="cuda")
        ops.linear(out, a[:m].contiguous(), w, bias, residual=res[:m].contiguous())
        assert bool(((out.double() - exact[:m]).abs() <= bound[:m]).all()), m
        first = out[0].clone() if first is None else first
        assert torch.equal(out[0], first), m
    whole = out
    for m in ROWS:
        part = torch.empty(m, n, device="cuda")
        ops.linear(part, a[:m].contiguous(), w, bias, residual=res[:m].contiguous())
        assert torch.equal(part, whole[:m]), m
    assert ops.status.item() == 0


def test_bfloat16_rows_on_the_cuda_cores():
    ops = CudaOps("cuda")
    ops.tensor_cores = False
    g = torch.Generator(device="cuda").manual_seed(3)
    for k in (96, 70, 33):
        w = torch.randn(200, k, device="cuda", generator=g).bfloat16()
        a = torch.randn(300, k, device="cuda", generator=g).bfloat16()
        whole = torch.empty(300, 200, device="cuda")
        ops.linear(whole, a, w)
        want = a.double() @ w.double().T
        assert float((whole.double() - want).abs().max()) <= k * 2.0 ** -24 * float(
            (a.abs().double() @ w.abs().double().T).max())
        for m in ROWS[:-1]:
            part = torch.empty(m, 200, device="cuda")
            ops.linear(part, a[:m].contiguous(), w)
            assert torch.equal(part, whole[:m]), (k, m)
