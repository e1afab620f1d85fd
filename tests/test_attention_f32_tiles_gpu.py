"""Float32 prompt portions as tiles of queries and single tokens with chunks fetched ahead: the same
bits as the kernel that takes up to four tokens a block, at lengths around its tiles and chunks, behind earlier positions, with heads that share
keys, beside single tokens, and with an infinite value behind a query's own position."""

import pytest
import torch

from hetero_serve_b200.kernels.ops import AttentionGeometry, CudaOps

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("heads,kv_heads,page", [(2, 2, 16), (4, 2, 32)])
@pytest.mark.parametrize("batch", [[(0, 5)], [(0, 64), (31, 65)], [(7, 1), (0, 33), (200, 3), (96, 128)],
                                   [(100, 300)], [(0, 129), (511, 1), (33, 31)], [(0, 1)],
                                   [(p, 1) for p in (31, 32, 127, 128, 160, 511, 900, 1500)],
                                   [(5 * i, 1) for i in range(90)]])
def test_same_bits_as_token_by_token(heads, kv_heads, page, batch):
    ops, D = CudaOps(DEV), 64
    g = torch.Generator(device=DEV).manual_seed(len(batch) + heads)
    T, R = sum(n for _, n in batch), len(batch)
    need = [-(-(p + n) // page) for p, n in batch]
    pages, width = sum(need) + 1, max(need) + 1
    order = torch.randperm(pages, generator=torch.Generator().manual_seed(1)).tolist()
    table = torch.full((R, width), -1, dtype=torch.int32)
    for r, k in enumerate(need):
        table[r, :k] = torch.tensor([order.pop() for _ in range(k)], dtype=torch.int32)
    qkv_w = (heads + 2 * kv_heads) * D
    qkv = torch.randn(T, qkv_w, device=DEV, generator=g)
    pool = torch.randn(pages, 2, kv_heads, page, D, device=DEV, generator=g)
    pos, req = [], []
    for r, (p, n) in enumerate(batch):
        pos += range(p, p + n)
        req += [r] * n
    # a value no earlier query may see: the last position of the first request
    p, n = batch[0]
    last = p + n - 1
    pool[table[0, last // page], 1, :, last % page] = float("inf")
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    geo = AttentionGeometry(heads, kv_heads, D, page, pages, width, 0, heads * D,
                            (heads + kv_heads) * D, qkv_w)
    plan = ops.make_plan([(r, r, p, n) for r, (p, n) in enumerate(batch)], T, page)
    outs = []
    for tiles in (True, False):
        ops.f32_tiles = ops.f32_single = tiles
        out = torch.zeros(T, heads * D, device=DEV)
        ops.attention(out, qkv, pool, table.to(DEV), i32(pos), i32(req), geo, 0.13, ops.status, plan)
        outs.append(out)
    assert torch.equal(torch.nan_to_num(outs[0], nan=-77.0), torch.nan_to_num(outs[1], nan=-77.0))
    assert torch.isfinite(outs[0][:n - 1]).all() and not torch.isfinite(outs[0][n - 1]).any()
    assert ops.status.item() == 0


@pytest.mark.parametrize("start,tokens", [(0, 200), (130, 70), (40, 1), (64, 33)])
@pytest.mark.parametrize("scale", [0.125, -0.125])
def test_chunks_in_which_no_score_is_above_minus_infinity(start, tokens, scale):
    """Keys of whole chunks whose scores overflow to minus infinity, for some queries or for all, with
    values that are infinite or NaN there: a query leaves such a chunk out."""
    ops, D, page = CudaOps(DEV), 64, 16
    g = torch.Generator(device=DEV).manual_seed(start + tokens)
    end = start + tokens
    n_pages = -(-end // page)
    pool = torch.randn(n_pages, 2, 1, page, D, device=DEV, generator=g)
    qkv = torch.randn(tokens, 3 * D, device=DEV, generator=g)
    keys = lambda a, b: (slice(a // page, b // page), 0, 0)  # noqa: E731
    vals = lambda a, b: (slice(a // page, b // page), 1, 0)  # noqa: E731
    sign = 1.0 if scale > 0 else -1.0
    qkv[:, 0] = 2.0 * sign * torch.where(torch.arange(tokens, device=DEV) % 3 == 0, -1.0, 1.0)
    for a, bad in ((0, float("inf")), (96, float("nan"))):   # one chunk of two streams
        if a + 32 <= end:
            pool[keys(a, a + 32)][..., 0] = -3e38            # every third query: + infinity
            pool[vals(a, a + 32)][..., 5] = bad
    table = torch.arange(n_pages, dtype=torch.int32, device=DEV).view(1, -1)
    geo = AttentionGeometry(1, 1, D, page, n_pages, n_pages, 0, D, 2 * D, 3 * D)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    plan = ops.make_plan([(0, 0, start, tokens)], tokens, page)
    outs = []
    for tiles in (True, False):
        ops.f32_tiles = ops.f32_single = tiles
        out = torch.zeros(tokens, D, device=DEV)
        ops.attention(out, qkv, pool, table, i32(list(range(start, end))), i32([0] * tokens), geo,
                      scale, ops.status, plan)
        outs.append(torch.nan_to_num(out, nan=-77.0, posinf=-78.0, neginf=-79.0))
    assert torch.equal(*outs)
    rest = outs[0][torch.arange(tokens, device=DEV) % 3 != 0]
    if end > 160 and start > 31:                             # those that skip both chunks are finite
        assert (rest > -70.0).all()


@pytest.mark.parametrize("batch", [[(0, 40)], [(0, 40), (9, 1)], [(0, 9), (100, 140), (3, 1), (50, 3)]])
def test_rows_of_no_request_become_zeros(batch):
    """Padding behind the tokens of a step, as captured steps have it, beside portions and singles."""
    ops, D, H, page = CudaOps(DEV), 64, 2, 16
    T, R, pad = sum(n for _, n in batch), len(batch), 700
    width = max(-(-(p + n) // page) for p, n in batch)
    table = torch.arange(R * width, dtype=torch.int32, device=DEV).view(R, width)
    geo = AttentionGeometry(H, H, D, page, R * width, width, 0, H * D, 2 * H * D, 3 * H * D)
    g = torch.Generator(device=DEV).manual_seed(T)
    qkv = torch.randn(T + pad, 3 * H * D, device=DEV, generator=g)
    pool = torch.randn(R * width, 2, H, page, D, device=DEV, generator=g)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    pos = i32([p + i for p, n in batch for i in range(n)] + [0] * pad)
    req = i32([r for r, (_, n) in enumerate(batch) for _ in range(n)] + [-1] * pad)
    plan = ops.make_plan([(r, r, p, n) for r, (p, n) in enumerate(batch)], T + pad, page)
    outs = []
    for tiles in (True, False):
        ops.f32_tiles = ops.f32_single = tiles
        out = torch.full((T + pad, H * D), float("nan"), device=DEV)
        ops.attention(out, qkv, pool, table, pos, req, geo, 0.125, ops.status, plan)
        outs.append(out)
    assert torch.equal(*outs) and not outs[0][T:].any() and ops.status.item() == 0


@pytest.mark.parametrize("tokens", [20, 3])
def test_refused_page_is_reported(tokens):
    ops, D = CudaOps(DEV), 64
    table = torch.tensor([[0, 9]], dtype=torch.int32, device=DEV)
    geo = AttentionGeometry(1, 1, D, 16, 2, 2, 0, D, 2 * D, 3 * D)
    qkv, pool = torch.randn(20, 3 * D, device=DEV), torch.randn(2, 2, 1, 16, D, device=DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    start = 20 - tokens
    plan = ops.make_plan([(0, 0, start, tokens)], tokens, 16)
    outs = []
    for tiles in (True, False):
        ops.f32_tiles = ops.f32_single = tiles
        ops.status.zero_()
        out = torch.zeros(tokens, D, device=DEV)
        ops.attention(out, qkv[:tokens].contiguous(), pool, table, i32(list(range(start, 20))),
                      i32([0] * tokens), geo, 0.1, ops.status, plan)
        assert ops.status.item() == 4
        outs.append(out)
    assert torch.equal(*outs)
