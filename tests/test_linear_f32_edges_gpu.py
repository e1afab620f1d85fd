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


@pytest.mark.parametrize("dtype,m,n,k", [(torch.float32, 1601, 1537, 70), (torch.float32, 1601, 1540, 33),
                                         (torch.bfloat16, 1601, 1537, 70), (torch.bfloat16, 1601, 1540, 100),
                                         (torch.bfloat16, 1601, 1537, 97), (torch.bfloat16, 200, 9477, 70),
                                         (torch.bfloat16, 200, 9480, 100),
                                         # 247 and 126 tiles of 128 x 128
                                         (torch.bfloat16, 1601, 2393, 100), (torch.bfloat16, 1100, 1700, 97)])
def test_rows_keep_their_bits_in_the_large_tiles(dtype, m, n, k):
    """Enough 64 x 64 tiles that the large ones are taken, with remainders in every direction: a row's
    bits are those it has in the small tiles and among few rows."""
    ops = CudaOps("cuda")
    ops.tensor_cores = False
    assert -(-m // 64) * -(-n // 64) >= (4 if m != 1100 else 3) * ops.sm_count
    g = torch.Generator(device="cuda").manual_seed(n + k)
    a = torch.randn(m, k, device="cuda", generator=g).to(dtype)
    w = torch.randn(n, k, device="cuda", generator=g).to(dtype)
    bias, res = (torch.randn(*s, device="cuda", generator=g) for s in ((n,), (m, n)))
    exact = a.double() @ w.double().T + bias.double() + res.double()
    bound = (k + 2) * 2.0 ** -24 * (a.abs().double() @ w.abs().double().T + bias.abs() + res.abs())
    whole = torch.full((m, n), float("nan"), device="cuda")
    ops.linear(whole, a, w, bias, residual=res)
    assert bool(((whole.double() - exact).abs() <= bound).all())
    for rows in (r for r in (1, 33, 65, 257) if r <= m):
        for first in (0, m - rows):
            part = torch.full((rows, n), float("nan"), device="cuda")
            ops.linear(part, a[first:first + rows].clone(), w, bias, residual=res[first:first + rows].clone())
            assert torch.equal(part, whole[first:first + rows]), (rows, first)
    if dtype == torch.bfloat16:                              # outputs rounded once, from the same sums
        out = torch.empty(m, n, device="cuda", dtype=dtype)
        ops.linear(out, a, w, bias, residual=res)
        assert torch.equal(out, whole.bfloat16())
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
