"""The tcgen05 tiles of the routed feed-forward at their edges: segments of one row, of whole and
broken steps of 16, of one tile exactly and one row more; summed indexes that end inside a step of 64;
feature counts that end inside a tile of 128; more experts than the sorting block has threads."""

import pytest
import torch

from hetero_serve_b200.kernels.ops import CudaOps

pytestmark = pytest.mark.gpu
DEV = "cuda"


def reference(h, wg, wu, wd, idx, wts, req, limit, act):
    """float64 sums; activated rows rounded to bfloat16 as between the two kernels."""
    out = torch.zeros(h.shape, dtype=torch.float64, device=h.device)
    for e in range(wu.shape[0]):
        rows, place = ((idx == e) & (req >= 0)[:, None]).nonzero(as_tuple=True)
        if not rows.numel():
            continue
        a = h[rows].double()
        u = a @ wu[e].double().T
        if act == "relu2":
            y = u.clamp(min=0) ** 2
        else:
            g = a @ wg[e].double().T
            if act == "silu":
                y = g * torch.sigmoid(g) * u
            else:
                g = g.clamp(max=limit)
                y = g * torch.sigmoid(1.702 * g) * (u.clamp(-limit, limit) + 1.0)
        y = y.to(torch.bfloat16).double() @ wd[e].double().T
        out.index_add_(0, rows, y * wts[rows, place, None].double())
    return out


@pytest.mark.parametrize("act", ["clamped", "silu", "relu2"])
@pytest.mark.parametrize("width, ff", [(96, 32), (64, 160), (256, 128), (320, 288)])
@pytest.mark.parametrize("counts", [[1, 16, 17, 222], [256, 257, 0, 31], [512, 513, 33, 2], [700]])
def test_segments(counts, width, ff, act):
    ops, g = CudaOps(DEV), torch.Generator(device=DEV).manual_seed(width + ff + len(counts))
    ops.status = torch.zeros(1, dtype=torch.int32, device=DEV)
    E, T = len(counts), sum(counts) + 3
    rnd = lambda *s, std: (torch.randn(*s, device=DEV, generator=g) * std).to(torch.bfloat16)  # noqa: E731
    h, wu = rnd(T, width, std=1.0), rnd(E, ff, width, std=width ** -0.5)
    wg = None if act == "relu2" else rnd(E, ff, width, std=width ** -0.5)
    wd = rnd(E, width, ff, std=ff ** -0.5)
    idx = torch.full((T, 1), -1, dtype=torch.int32, device=DEV)
    order, at = torch.randperm(T, device=DEV, generator=g), 0
    for e, n in enumerate(counts):
        idx[order[at:at + n], 0] = e
        at += n
    req = torch.zeros(T, dtype=torch.int32, device=DEV)
    req[order[0]] = -1                                          # a padding row with a choice
    wts = torch.rand(T, 1, device=DEV, generator=g)
    x = torch.full((T, width), 0.5, device=DEV)
    y = torch.zeros(T, ff, device=DEV)
    ops.moe_experts(x, y, h, wg, wu, wd, idx, wts, req, limit=1.5, act=act)
    assert ops.status.item() == 0
    want = reference(h, wg, wu, wd, idx, wts, req, 1.5, act)
    # float32 sums against float64: an activation may fall on the other side of a bfloat16 boundary
    # (2^-8 of itself), so a row differs by 2^-8 of a few of its ff terms
    diff = (x.double() - 0.5 - want).norm() / want.norm()
    assert diff < 2e-3, diff
    assert (x.double() - 0.5 - want).abs().max() < 0.03 * want.abs().max()
    assert torch.equal(x[order[0]], torch.full((width,), 0.5, device=DEV))


def test_more_experts_than_sorting_threads():
    E, T, top, width, ff = 1500, 300, 2, 64, 32
    ops, g = CudaOps(DEV), torch.Generator(device=DEV).manual_seed(5)
    ops.status = torch.zeros(1, dtype=torch.int32, device=DEV)
    rnd = lambda *s, std: (torch.randn(*s, device=DEV, generator=g) * std).to(torch.bfloat16)  # noqa: E731
    h, wg, wu = rnd(T, width, std=1.0), rnd(E, ff, width, std=0.125), rnd(E, ff, width, std=0.125)
    wd = rnd(E, width, ff, std=0.2)
    idx = torch.stack([torch.arange(T, device=DEV) * 5 % E, 1499 - torch.arange(T, device=DEV)], 1).int()
    req, wts = torch.zeros(T, dtype=torch.int32, device=DEV), torch.rand(T, top, device=DEV, generator=g)
    x = torch.zeros(T, width, device=DEV)
    ops.moe_experts(x, torch.zeros(T * top, ff, device=DEV), h, wg, wu, wd, idx.contiguous(), wts, req,
                    limit=7.0, act="silu", fresh=True)
    assert ops.status.item() == 0
    want = reference(h, wg, wu, wd, idx, wts, req, 7.0, "silu")
    assert (x.double() - want).norm() / want.norm() < 2e-3


@pytest.mark.parametrize("act", ["silu", "clamped"])
def test_gates_whose_exponential_is_near_the_end_of_the_range(act):
    """Tiles and single pairs form the same quotient, up to where the exponential leaves the range."""
    T, width, ff = 300, 32, 64
    gates = -(80.0 + 0.5 * torch.arange(ff, device=DEV)) / (1.0 if act == "silu" else 1.702)
    h = torch.zeros(T, width, device=DEV, dtype=torch.bfloat16)
    h[:, 0] = 1.0
    wg, wu = (torch.zeros(1, ff, width, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    wg[0, :, 0], wu[0, :, 0] = gates.to(torch.bfloat16), 2.0 ** 60
    wd = torch.zeros(1, width, ff, device=DEV, dtype=torch.bfloat16)
    idx, req = (torch.zeros(s, dtype=torch.int32, device=DEV) for s in ((T, 1), (T,)))
    for first in (0, 32):                         # a feature an output
        wd[0, :, first:first + 32] = torch.eye(32, device=DEV)
        outs = []
        for tiles in (True, False):
            ops = CudaOps(DEV)
            ops.sorted_experts = tiles
            x = torch.zeros(T, width, device=DEV)
            ops.moe_experts(x, torch.zeros(T, ff, device=DEV), h, wg, wu, wd, idx, torch.ones(T, 1, device=DEV), req,
                            limit=2.0 ** 60, act=act, fresh=True)
            outs.append(x)
        wd.zero_()
        # the tiles' activated rows are rounded to bfloat16: half a step of 2^-7 at most
        assert bool(((outs[0] - outs[1]).abs() <= 2.0 ** -8 * outs[1].abs()).all())
        assert bool((outs[1] != 0).any()) or first == 32
