"""The delta rule's pre-pass of eight tokens a warp and its finish of a warp a head: the bits of the kernels
of few tokens, with blocks of eight that straddle requests, begin behind a portion's start or hold padding."""

import pytest
import torch

from hetero_serve_b200.kernels.ops import CudaOps

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("H, HK, D, V", [(3, 3, 128, 128), (8, 4, 64, 96), (5, 5, 96, 256), (9, 9, 32, 64)])
@pytest.mark.parametrize("lens", [(600,), (1, 2, 3, 250, 9, 263), (517, 11)])
@pytest.mark.parametrize("product", [True, False])
def test_same_bits_as_token_by_token(H, HK, D, V, lens, product):
    g = torch.Generator(device=DEV).manual_seed(H * D + V + len(lens))
    rnd = lambda *s, std=1.0: torch.randn(*s, device=DEV, generator=g) * std  # noqa: E731
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    T, R, ra, rg, taps = sum(lens) + 3, len(lens), 6, 5, 4
    C = 2 * HK * D + H * V
    proj = rnd(T, C + H + ra + rg)
    conv, a2, g2 = rnd(C, taps, std=0.5), rnd(ra, H * D), rnd(rg, H * V)
    dt, A, norm = rnd(H * D, std=0.5), rnd(H, std=0.5), rnd(V)
    z_a = rnd(T, H * D) if product else None
    z_g = rnd(T, H * V) if product else None
    state = rnd(R, H * D * V + (taps - 1) * C)
    req = i32([r for r, n in enumerate(lens) for _ in range(n)] + [-1] * 3)
    start = [sum(lens[:r]) for r in range(R)]
    z = dict(heads=H, kv_heads=HK, dim=D, vdim=V, taps=taps, a_rank=ra, g_rank=rg)

    def prepare(ops, first, n, lens_, starts, slots, st):
        outs = [torch.full((n, w), 7.0, device=DEV) for w in (HK * D, HK * D, H * V, H, H * D)]
        ops.delta_prepare(*outs, proj[first:first + n].contiguous(), conv, a2, dt, A, st,
                          req[first:first + n].contiguous() if len(lens_) == R else i32([0] * n), i32(starts),
                          i32(lens_), i32(slots), z, z_a=None if z_a is None else z_a[first:first + n].contiguous())
        return outs
    ops = CudaOps(DEV)
    ops.delta_rows = 1                   # whatever the step's size
    st = state.clone()
    got = prepare(ops, 0, T, list(lens), start, list(range(R)), st)
    for x in got:
        assert bool((x[T - 3:] == 7.0).all())                # rows of no request are left alone
    # portions of up to 37 tokens, each request in turn, a block a token
    ops.delta_rows = 0
    for r, n in enumerate(lens):
        mine = state[r:r + 1].clone()
        for a in range(0, n, 37):
            k = min(37, n - a)
            part = prepare(ops, start[r] + a, k, [k], [0], [0], mine) if R > 1 else None
            if part is None:
                outs = [torch.full((k, x.shape[1]), 7.0, device=DEV) for x in got]
                ops.delta_prepare(*outs, proj[a:a + k].contiguous(), conv, a2, dt, A, mine, i32([0] * k), i32([0]),
                                  i32([k]), i32([0]), z, z_a=None if z_a is None else z_a[a:a + k].contiguous())
                part = outs
            for x, y in zip(got, part):
                assert torch.equal(x[start[r] + a:start[r] + a + k], y)
        assert torch.equal(mine[0], st[r])
    o = rnd(T, H * V)
    for dt_ in (torch.float32, torch.bfloat16):
        out, other = (torch.full((T, H * V), 3.0, device=DEV, dtype=dt_) for _ in range(2))
        for ops.delta_rows, dst in ((1, out), (0, other)):
            ops.delta_finish(dst, o, proj, g2, norm, req, 1e-6, z, z_g=z_g)
        assert torch.equal(out, other)
        # by the formula; without z_g the gates' logits are formed from the projection's last columns
        gate = proj[:, C + H + ra:].double() @ g2.double() if z_g is None else z_g.double()
        x = o.double().view(T, H, V)
        y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-6) * norm.double()
        y = (y * torch.sigmoid(gate).view(T, H, V)).flatten(1)
        tol = 2.0 ** -8 if dt_ == torch.bfloat16 else 1e-5
        live = slice(0, T - 3)
        assert bool(((out.double() - y)[live].abs() <= tol * y[live].abs() + 1e-6).all())
        assert bool((out[T - 3:] == 3.0).all())


@pytest.mark.parametrize("V", [32, 64, 96, 128, 160, 224, 256])
@pytest.mark.parametrize("dt_", [torch.float32, torch.bfloat16])
def test_finish_has_the_same_bits_by_warps_and_by_blocks(V, dt_):
    ops, g = CudaOps(DEV), torch.Generator(device=DEV).manual_seed(V)
    T, H = 77, 3
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    o, z_g, norm, req = rnd(T, H * V), rnd(T, H * V), rnd(V), torch.zeros(T, dtype=torch.int32, device=DEV)
    z = dict(heads=H, kv_heads=H, dim=64, vdim=V, taps=4, a_rank=5, g_rank=6)
    proj, g2 = rnd(T, 2 * H * 64 + H * V + H + 11), rnd(6, H * V)
    outs = [torch.empty(T, H * V, device=DEV, dtype=dt_) for _ in range(2)]
    for ops.delta_rows, out in enumerate(outs):
        ops.delta_finish(out, o, proj, g2, norm, req, 1e-6, z, z_g=z_g)
    assert torch.equal(*outs)


@pytest.mark.parametrize("H, D, lens, product", [
    (8, 128, (512,), True), (8, 128, (8,) * 64, True), (8, 128, (13,) * 100, True), (32, 32, (2048,), True),
    (8, 128, (512,), False), (32, 32, (1000, 24), False)])
def test_the_form_chosen_is_no_slower_than_a_block_a_token(H, D, lens, product):
    g = torch.Generator(device=DEV).manual_seed(1)
    rnd = lambda *s, std=1.0: torch.randn(*s, device=DEV, generator=g) * std  # noqa: E731
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    T, R, C = sum(lens), len(lens), 3 * H * D
    z = dict(heads=H, kv_heads=H, dim=D, vdim=D, taps=4, a_rank=64, g_rank=64)
    outs = [torch.empty(T, w, device=DEV) for w in (H * D, H * D, H * D, H, H * D)]
    args = (*outs, rnd(T, C + H + 128), rnd(C, 4), rnd(64, H * D, std=0.1), rnd(H * D), rnd(H),
            rnd(R, H * D * D + 3 * C), i32([r for r, n in enumerate(lens) for _ in range(n)]),
            i32([sum(lens[:r]) for r in range(R)]), i32(lens), i32(list(range(R))), z)
    more = dict(z_a=rnd(T, H * D) if product else None)
    ops, times = CudaOps(DEV), []
    for ops.delta_rows in (-1, 0):
        ops.delta_prepare(*args, **more)
        graph, best = torch.cuda.CUDAGraph(), []
        with torch.cuda.graph(graph):
            for _ in range(10):
                ops.delta_prepare(*args, **more)
        for _ in range(8):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            graph.replay()
            b.record()
            b.synchronize()
            best.append(a.elapsed_time(b))
        times.append(min(best))
    assert times[0] <= 1.15 * times[1]
