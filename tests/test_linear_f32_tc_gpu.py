"""The float32 linear on the tensor cores: the same bits in every tile and share of the work, closer to
float64 than a chain of FMAs, and the results a chain gives where numbers are not finite."""

import pytest
import torch

from hetero_serve_b200.kernels.ops import CudaOps

pytestmark = pytest.mark.gpu
DEV = "cuda"


def run(ops, rows, a, w, bias=None, act="none", residual=None):
    ops.f32_rows = rows
    out = torch.full((a.shape[0], w.shape[0]), float("nan"), device=DEV)
    ops.linear(out, a, w, bias, act=act, residual=residual)
    ops.f32_rows = 0
    return out


def chain(ops, a, w, *args, **kw):
    ops.tensor_cores = False
    out = run(ops, 0, a, w, *args, **kw)
    ops.tensor_cores = True
    return out


@pytest.mark.parametrize("n, k", [(1, 4), (127, 60), (128, 64), (129, 68), (300, 260), (640, 1024), (257, 2052)])
@pytest.mark.parametrize("m", [1, 15, 16, 17, 63, 65, 129, 300])
def test_tiles_and_shares_give_the_same_bits(m, n, k):
    ops, g = CudaOps(DEV), torch.Generator(device=DEV).manual_seed(m + n + k)
    ops.status = torch.zeros(1, dtype=torch.int32, device=DEV)
    a, w = (torch.randn(s, k, device=DEV, generator=g) for s in (m, n))
    bias, res = torch.randn(n, device=DEV, generator=g), torch.randn(m, n, device=DEV, generator=g)
    first = run(ops, 16, a, w, bias, "gelu_tanh", res)
    for rows in (0, 32, 64, 128):
        assert torch.equal(run(ops, rows, a, w, bias, "gelu_tanh", res), first), rows
    # a row alone: its segments are shared out otherwise
    assert torch.equal(run(ops, 0, a[m - 1:].clone(), w, bias, "gelu_tanh", res[m - 1:].clone()), first[m - 1:])
    exact = a.double() @ w.double().T
    plain = run(ops, 0, a, w)
    # cut-off sums: 2^-23 of a running value a product at most, as many as a segment's chunks are deep,
    # and a rounding a chunk: below a chain of k roundings
    bound = (min(k, 64) / 4 + k / 64 + 2) * 2.0 ** -23 * (a.abs().double() @ w.abs().double().T)
    assert bool(((plain.double() - exact).abs() <= bound).all())
    if k >= 256:
        err = lambda x: float((x.double() - exact).norm())  # noqa: E731
        assert err(plain) <= err(chain(ops, a, w))
    assert ops.status.item() == 0


@pytest.mark.parametrize("act", ["gelu_erf", "relu2", "silu", "none"])
def test_activations(act):
    ops, g = CudaOps(DEV), torch.Generator(device=DEV).manual_seed(1)
    a, w = torch.randn(70, 128, device=DEV, generator=g), torch.randn(200, 128, device=DEV, generator=g) * 0.1
    bias, res = torch.randn(200, device=DEV, generator=g), torch.randn(70, 200, device=DEV, generator=g)
    got, want = run(ops, 64, a, w, bias, act, res), chain(ops, a, w, bias, act, res)
    # both sums are off by no more than k + 2 roundings; no activation is steeper than 2 |u| + 1.2
    u = (a.double() @ w.double().T + bias.double()).abs()
    bound = 2 * (128 + 2) * 2.0 ** -24 * (a.abs() @ w.abs().T + bias.abs() + res.abs()).double() * (2 * u + 1.2)
    assert bool(((got - want).abs().double() <= bound).all())
    assert torch.equal(run(ops, 0, a, w, bias, act, res), got)


@pytest.mark.parametrize("m, rows", [(3, 16), (70, 64), (130, 128)])
def test_numbers_that_are_not_finite(m, rows):
    """Infinities, numbers that are none, products beyond the range and numbers that round up to an
    infinity as bfloat16: what a chain of FMAs gives; every other output keeps its bits."""
    n, k = 160, 320
    ops, g = CudaOps(DEV), torch.Generator(device=DEV).manual_seed(m)
    a, w = torch.randn(m, k, device=DEV, generator=g), torch.randn(n, k, device=DEV, generator=g)
    clean = run(ops, rows, a, w)
    a[1, 7], w[5, 9], w[6, 7] = float("inf"), float("nan"), 0.0     # inf x 0 in one output
    a[2, 3], w[9, 3] = 1e30, 1e30                                    # a product beyond the range
    a[0, 100] = 3.4e38                                               # finite, an infinity as bfloat16
    w[:, 100] = torch.rand(n, device=DEV, generator=g) * 0.5
    got, want = run(ops, rows, a, w), chain(ops, a, w)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    inf = want.isinf()
    assert torch.equal(got[inf], want[inf])
    fine = want.isfinite()
    assert bool(((got - want).abs()[fine] <= 1e-4 * want.abs()[fine] + 1e-3).all())
    assert torch.equal(run(ops, 0, a, w).nan_to_num(), got.nan_to_num())
    # untouched rows and features: as before
    w2 = w.clone()
    w2[:, 100] = 0.0
    rest = run(ops, rows, a, w2)
    a0 = a.clone()
    a0[:, 100] = 0.0
    same = run(ops, rows, a0, w2)
    assert torch.equal(rest[3:, 10:], same[3:, 10:]) and clean.isfinite().all()


def test_small_and_large_numbers_keep_their_digits():
    """Rows scaled by powers of two give outputs scaled by them, bit for bit, far from the ends of the range."""
    ops, g = CudaOps(DEV), torch.Generator(device=DEV).manual_seed(9)
    a, w = torch.randn(20, 256, device=DEV, generator=g), torch.randn(130, 256, device=DEV, generator=g)
    base = run(ops, 0, a, w)
    for e in (-60, -30, 30, 60):
        assert torch.equal(run(ops, 0, a * 2.0 ** e, w), base * 2.0 ** e), e


def test_shapes_it_refuses_go_to_the_cuda_cores():
    ops, g = CudaOps(DEV), torch.Generator(device=DEV).manual_seed(2)
    a, w = torch.randn(40, 70, device=DEV, generator=g), torch.randn(50, 70, device=DEV, generator=g)
    assert torch.equal(run(ops, 0, a, w), chain(ops, a, w))              # k not a multiple of four
    buf = torch.randn(50 * 64 + 1, device=DEV, generator=g)
    a, w = torch.randn(40, 64, device=DEV, generator=g), buf[1:].view(50, 64)
    assert torch.equal(run(ops, 0, a, w), chain(ops, a, w))              # weights off a 16-byte boundary


def time_of(call):
    graph, best = torch.cuda.CUDAGraph(), []
    call()
    with torch.cuda.graph(graph):
        for _ in range(4):
            call()
    for _ in range(6):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        graph.replay()
        b.record()
        b.synchronize()
        best.append(a.elapsed_time(b))
    return min(best)


@pytest.mark.parametrize("what", ["row", "number", "rows", "weight"])
@pytest.mark.parametrize("m, n, k", [(8, 1024, 4096), (1024, 1024, 4096), (1024, 4096, 1024)])
def test_numbers_that_are_none_take_no_longer_than_chains(m, n, k, what):
    """A row of NaNs, one NaN in a row, all rows, one NaN among the weights: as the CUDA cores answer and, since
    those take as long as for other numbers, not slower than them by much."""
    ops, g = CudaOps(DEV), torch.Generator(device=DEV).manual_seed(k)
    a, w = torch.randn(m, k, device=DEV, generator=g), torch.randn(n, k, device=DEV, generator=g) * 0.03
    if what == "row":
        a[1] = float("nan")
    elif what == "number":
        a[1, k - 2] = float("nan")
    elif what == "rows":
        a[:] = float("nan")
    else:
        w[7, k // 2] = float("nan")
    got, want = run(ops, 0, a, w), chain(ops, a, w)
    assert torch.equal(got.isnan(), want.isnan()) and got.isfinite().equal(want.isfinite())
    times = []
    for ops.tensor_cores in (True, False):
        out = torch.empty(m, n, device=DEV)
        times.append(time_of(lambda: ops.linear(out, a, w)))
    assert times[0] <= 2 * times[1]


@pytest.mark.parametrize("m", [1, 2, 8, 16, 17, 40])
@pytest.mark.parametrize("n, k", [(768, 768), (64, 768), (1024, 1028), (6400, 1600), (130, 132), (200, 8192)])
def test_chunks_and_segments_shared_out(m, n, k):
    """Few rows: a tile's single chunks or its segments go to blocks, whichever fills the device; the bits of a
    row do not show it."""
    ops, g = CudaOps(DEV), torch.Generator(device=DEV).manual_seed(m * n + k)
    ops.status = torch.zeros(1, dtype=torch.int32, device=DEV)
    a, w = torch.randn(300, k, device=DEV, generator=g), torch.randn(n, k, device=DEV, generator=g)
    bias, res = torch.randn(n, device=DEV, generator=g), torch.randn(300, n, device=DEV, generator=g)
    whole = run(ops, 128, a, w, bias, "silu", res)
    assert torch.equal(run(ops, 0, a[:m].clone(), w, bias, "silu", res[:m].clone()), whole[:m])
    assert torch.equal(run(ops, 16, a[:m].clone(), w, bias, "silu", res[:m].clone()), whole[:m])
    assert ops.status.item() == 0


@pytest.mark.parametrize("k", [4, 8, 12, 20, 36, 64, 68, 100, 128, 192])
def test_short_sums_are_no_further_off_than_chains(k):
    ops, g = CudaOps(DEV), torch.Generator(device=DEV).manual_seed(k)
    for shape in (torch.randn, torch.rand):                # (sums that cancel and sums that do not)
        a, w = shape(300, k, device=DEV, generator=g), shape(640, k, device=DEV, generator=g)
        exact = a.double() @ w.double().T
        err = lambda x: float((x.double() - exact).norm())  # noqa: E731
        assert err(run(ops, 0, a, w)) <= err(chain(ops, a, w))


@pytest.mark.parametrize("m, n, k", [(1, 768, 768), (1, 1024, 1024), (8, 768, 768), (1, 6400, 1600), (1024, 1024, 16),
                                     (64, 1024, 64), (4096, 1024, 32)])
def test_few_rows_and_short_sums_take_about_as_long_as_chains(m, n, k):
    ops, g = CudaOps(DEV), torch.Generator(device=DEV).manual_seed(k)
    a, w = torch.randn(m, k, device=DEV, generator=g), torch.randn(n, k, device=DEV, generator=g)
    out, times = torch.empty(m, n, device=DEV), []
    for ops.tensor_cores in (True, False):
        times.append(time_of(lambda: ops.linear(out, a, w)))
    assert times[0] <= 1.35 * times[1]


@pytest.mark.parametrize("e", [-100, -108, -112, -120, -126])
def test_numbers_near_the_end_of_the_range(e):
    """A third term below bfloat16's range is lost: 2^-134 of the other operand a product, nothing above 2^-109."""
    ops, g = CudaOps(DEV), torch.Generator(device=DEV).manual_seed(-e)
    a, w = torch.randn(64, 256, device=DEV, generator=g) * 2.0 ** e, torch.randn(128, 256, device=DEV, generator=g)
    exact = a.double() @ w.double().T
    # the bound of the sums as above, half a step of bfloat16's smallest a product, float32's own last step
    sums = (64 / 4 + 4 + 2) * 2.0 ** -23 * (a.abs().double() @ w.abs().double().T)
    lost = 2.0 ** -134 * w.abs().double().sum(1) + 2.0 ** -149
    assert bool(((run(ops, 0, a, w).double() - exact).abs() <= sums + lost).all())
    if e >= -108:
        err = lambda x: float((x.double() - exact).norm())  # noqa: E731
        assert err(run(ops, 0, a, w)) <= err(chain(ops, a, w))
