"""GPU: f32 products on the tensor cores (three bf16 terms per operand, sums of 64 k) against float64: tile widths, K splits, ragged edges
and numbers that the split does not hold."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from teenygrad_b200 import ops as o
    return o


def bound(x, w, K):
    """Per element: a sum of 64 k is cut off at most 24 times by 2^-23 of the products' sizes, the sums of K / 64 such and of up to eight parts
    are rounded, and the terms left out are below 3 * 2^-24."""
    return (48 + K // 64 + 12) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)


@pytest.mark.parametrize("M,N,K", [(17, 1000, 1000), (4, 4096, 4096), (64, 4096, 2052), (300, 700, 2000), (2000, 100, 4000), (512, 512, 512), (129, 4100, 68),
                                   (1000, 4096, 1024), (1100, 2300, 36), (4000, 64, 516)])
def test_shapes(ops, M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    wide = [torch.full((r, K + 4), float("nan"), device="cuda") for r in (M, N)]  # what lies between the rows is not read
    x, w = wide[0][:, :K], wide[1][:, :K]
    x.copy_(torch.randn(M, K, generator=g, device="cuda"))
    w.copy_(torch.randn(N, K, generator=g, device="cuda"))
    bias = torch.randn(N, generator=g, device="cuda")
    e, b = x.double() @ w.double().T, bound(x, w, K)
    out = torch.empty(M, N, device="cuda")
    ops.linear_forward(x, w, bias, out=out)
    assert bool(((out.double() - e - bias.double()).abs() <= b + 2.0 ** -23 * (e.abs() + bias.abs())).all())
    kn = w.T.contiguous()
    assert bool(((ops.matmul_forward(x.contiguous(), kn).double() - e).abs() <= b).all())
    rel = float((out.double() - e - bias.double()).norm() / e.norm())
    assert rel < 3e-7  # f32 multiply-adds in one chain: 2.4e-7 at K = 1000, 1.2e-6 at K = 4096
    assert ops.device_error() == 0


@pytest.mark.parametrize("M,N,K", [(200, 1500, 320), (40, 1000, 1600)])
@pytest.mark.parametrize("kn", [False, True])
def test_numbers_at_the_limits(ops, M, N, K, kn):
    g = torch.Generator(device="cuda").manual_seed(K)
    x, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda")
    x[3, 7] = float("inf")
    x[5, 9] = float("nan")
    x[7, 1], w[:, 1] = 3.4028e38, w[:, 1].clamp(-0.9, 0.9)  # rounds to infinity as bf16
    x[9] *= 1e-36
    x[11] = 0.0
    w[4, 7] = 0.0
    w[6, 3] = -float("inf")
    w[8] = 1e-3
    w[12] *= 1e20
    y = ops.matmul_forward(x, w.T.contiguous()) if kn else ops.linear_forward(x, w, None)
    e = x.double() @ w.double().T
    f = e.float()
    assert torch.equal(torch.isnan(y), torch.isnan(f)) and torch.equal(torch.isinf(y), torch.isinf(f))
    ok = torch.isfinite(f)
    # products below the smallest number that f32 holds with all its bits are off by up to 2^-149 each
    b = (48 + K // 64 + 12) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T) + K * 2.0 ** -149
    assert bool(((y.double() - e).abs() <= b)[ok].all())
    assert ops.device_error() == 0


@pytest.mark.parametrize("M,N,K", [(2048, 2304, 64), (600, 1500, 320), (200, 1500, 1600), (512, 512, 512)])
@pytest.mark.parametrize("kn", [False, True])
@pytest.mark.parametrize("lo,hi,wlo,whi", [(-149, -126, 60, 127), (-134, -110, 20, 120), (-126, -90, -10, 90), (-100, -60, -48, -20), (90, 127, -149, -100), (100, 127, -90, -20),
                                           (70, 110, -30, 17)])
def test_single_products_over_all_exponents(ops, M, N, K, kn, lo, hi, wlo, whi):
    """One product per result, down to the subnormals on one side and up to the largest numbers on the other: no sum hides what the split of
    an operand loses."""
    g = torch.Generator(device="cuda").manual_seed(K + lo)

    def numbers(shape, lo, hi):
        e = torch.randint(lo, hi + 1, shape, generator=g, device="cuda").double()
        m = 1.0 + torch.randint(0, 1 << 23, shape, generator=g, device="cuda").double() * 2.0 ** -23
        return (m * torch.where(torch.rand(shape, generator=g, device="cuda") < 0.5, -1.0, 1.0).double() * torch.exp2(e)).float()

    x, w = torch.zeros(M, K, device="cuda"), numbers((N, K), wlo, whi)
    at = torch.randint(0, K, (M,), generator=g, device="cuda")
    x[torch.arange(M, device="cuda"), at] = numbers((M,), lo, hi)
    y = ops.matmul_forward(x, w.T.contiguous()) if kn else ops.linear_forward(x, w, None)
    e = x[torch.arange(M, device="cuda"), at].double()[:, None] * w[:, at].T.double()
    # three products of 2^-24 each left out, five roundings of 2^-24, a half subnormal step
    b = 8 * 2.0 ** -24 * e.abs() + 2.0 ** -149
    over = e.abs() >= 2.0 ** 128 * (1 - 2.0 ** -25)
    assert bool(torch.isinf(y)[over].all()) and bool(((y.double() - e).abs() <= b)[~over].all())
    assert ops.device_error() == 0


@pytest.mark.parametrize("M,N,K", [(1000, 2048, 2048), (512, 512, 512), (64, 4096, 2048), (40, 300, 4000)])
@pytest.mark.parametrize("kn", [False, True])
def test_numbers_out_of_range_cost_a_second_pass_at_most(ops, M, N, K, kn):
    """Results that overflow, operands full of infinities, sums beyond what tensor memory holds at the split's scale and tiny results: right,
    and in the time of a few finite products."""
    g = torch.Generator(device="cuda").manual_seed(N)
    x, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda")
    run = (lambda a, b: ops.matmul_forward(a, b)) if kn else (lambda a, b: ops.linear_forward(a, b, None))

    def passes(a, b):
        b = b.T.contiguous() if kn else b
        for _ in range(3):
            y = run(a, b)
        t = []
        for _ in range(5):
            t0, t1 = torch.cuda.Event(True), torch.cuda.Event(True)
            t0.record()
            for _ in range(10):
                run(a, b)
            t1.record()
            torch.cuda.synchronize()
            t.append(t0.elapsed_time(t1))
        return y, min(t)

    usual = passes(x, w)[1]
    for a, b in ((x * 1e30, w * 1e6), (x * 1e-30, w * 1e-3), (x * 1e18, w * 1e17)):
        y, t = passes(a, b)
        e = a.double() @ b.double().T
        bound = (48 + K // 64 + 12) * 2.0 ** -24 * (a.double().abs() @ b.double().abs().T) + K * 2.0 ** -149
        if float(e.abs().max()) > 1e30:  # these are sums of K multiply-adds, any order
            bound = bound + K * 2.0 ** -24 * (a.double().abs() @ b.double().abs().T)
        fits = e.abs() < 3e38
        assert bool(((y.double() - e).abs() <= bound)[fits].all())
        assert t < 8 * usual + 0.3, (t, usual)
    a = x.clone()
    a[:, 5] = float("inf")
    y, t = passes(a, w)
    assert bool((y == torch.where(w[:, 5] > 0, float("inf"), -float("inf"))).all())
    assert t < 8 * usual + 0.3, (t, usual)
    a[:, 7] = float("nan")
    assert bool(torch.isnan(passes(a, w)[0]).all())
    # one bad row leaves the others what they are without it
    a = x.clone()
    a[M // 2, 3] = float("inf")
    y, clean = passes(a, w)[0], passes(x, w)[0]
    rows = torch.arange(M, device="cuda") != M // 2
    assert torch.equal(y[rows], clean[rows]) and bool(torch.isinf(y[M // 2]).all())
    assert ops.device_error() == 0
