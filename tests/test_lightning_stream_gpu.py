"""Lightning attention's and retention's steps of many tokens as a stream (heads of 64, 128, 256): the
bits of the kernel for few tokens, at lengths around its stages, with value columns that end inside a
group, with and without rotation."""

import pytest
import torch

from hetero_serve_b200.kernels.ops import CudaOps

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dim,vdim,rot,act", [(64, 64, 64, "none"), (128, 20, 0, "silu"),
                                              (128, 128, 64, "none"), (256, 33, 256, "silu")])
@pytest.mark.parametrize("lens", [(64,), (1, 70, 0, 9), (8, 12, 3, 45)])
def test_same_bits_as_few_tokens(dim, vdim, rot, act, lens):
    ops, H = CudaOps(DEV), 2
    g = torch.Generator(device=DEV).manual_seed(dim + rot + sum(lens))
    T, R = sum(lens), len(lens)
    stride = 3 + H * (2 * dim + vdim)
    proj = torch.randn(T, stride, device=DEV, generator=g)
    decay = torch.tensor([0.97, 0.6], device=DEV)
    state0 = torch.randn(R + 1, H * dim * vdim, device=DEV, generator=g)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    start = [sum(lens[:i]) for i in range(R)]
    pos = i32([1000 * r + t for r, n in enumerate(lens) for t in range(n)])
    freq = torch.rand(max(rot // 2, 1), device=DEV, generator=g)
    more = dict(tok_pos=pos, freq=freq, rot_dims=rot, k_scale=0.3) if rot else {}
    got = []
    for bulk in (64, 10 ** 9):
        ops.lightning_bulk_rows = bulk
        o, state = torch.full((T, H * vdim), float("nan"), device=DEV), state0.clone()
        before = ops.launches
        ops.lightning_recurrence(o, state, proj, decay, i32(start), i32(list(lens)),
                                 i32(list(range(R, 0, -1))), q_off=3, k_off=3 + H * dim,
                                 v_off=3 + 2 * H * dim, heads=H, dim=dim, vdim=vdim, act=act, **more)
        assert ops.launches - before == (2 if bulk == 64 else 1)
        got.append((o, state))
    assert torch.isfinite(got[0][0]).all()
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert ops.status.item() == 0


@pytest.mark.parametrize("dim,vdim", [(64, 64), (128, 30), (256, 12)])
@pytest.mark.parametrize("heads", [1, 5])
def test_steps_of_few_tokens_a_request_do_not_stream(dim, vdim, heads):
    """Single tokens beside each other: the kernel for few tokens, and the bits of the stream that the
    same tokens take as parts of longer portions."""
    ops = CudaOps(DEV)
    g = torch.Generator(device=DEV).manual_seed(dim + heads)
    T = 70
    proj = torch.randn(T, heads * (2 * dim + vdim), device=DEV, generator=g)
    decay = torch.rand(heads, device=DEV, generator=g)
    state0 = torch.randn(T, heads * dim * vdim, device=DEV, generator=g)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731

    def run(lens, rows):
        o, state = torch.zeros(len(rows), heads * vdim, device=DEV), state0.clone()
        before = ops.launches
        ops.lightning_recurrence(o, state, proj[rows].contiguous(), decay,
                                 i32([sum(lens[:r]) for r in range(len(lens))]), i32(lens),
                                 i32(list(range(len(lens)))), q_off=0, k_off=heads * dim,
                                 v_off=2 * heads * dim, heads=heads, dim=dim, vdim=vdim, act="silu")
        return o, state, ops.launches - before
    o, state, launches = run([1] * T, list(range(T)))
    assert launches == (2 if vdim % 4 == 0 else 1)
    # each of the first eight tokens at the head of a portion of its own
    rows = [r if i == 0 else (r + 9 * i) % T for r in range(8) for i in range(9)]
    want, _, launches = run([9] * 8, rows)
    assert launches == 2
    for r in range(8):
        assert torch.equal(o[r], want[9 * r])
    assert ops.status.item() == 0
