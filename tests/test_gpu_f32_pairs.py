"""GPU: f32 products by pairs of CTAs, and of rows that a tensor map cannot describe, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from teenygrad_b200 import ops as o
    return o


def rows(M, K, ld, first, seed):
    """[M, K] with row stride `ld`, beginning `first` numbers into its memory; what lies between is NaN."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    mem = torch.full((first + M * max(ld, 1) + K,), float("nan"), device="cuda")
    x = mem.as_strided((M, K), (ld, 1), first)
    if ld:
        x.copy_(torch.randn(M, K, generator=g, device="cuda"))
    else:
        x[0].copy_(torch.randn(K, generator=g, device="cuda"))
    return x


@pytest.mark.parametrize("M,N,K,lda,ldb,first", [
    (1024, 4096, 320, 320, 320, 0), (1290, 4100, 580, 580, 584, 0), (1281, 4097, 516, 516, 520, 4),  # pairs
    (300, 1000, 1001, 1001, 1001, 0), (257, 900, 960, 961, 960, 0), (257, 900, 960, 960, 960, 1), (200, 1025, 1300, 0, 1303, 0),  # copies of four bytes
])
@pytest.mark.parametrize("kn", [False, True])
def test_products(ops, M, N, K, lda, ldb, first, kn):
    x, w = rows(M, K, lda, first, K), rows(N, K, ldb, first, N)
    if kn:  # [K, N] with a row stride of its own, as the transposed view that the linear entry takes
        held = rows(K, N, N + ldb - K, first, N)
        w = held.T
    bias = torch.randn(N, device="cuda")
    e = x.double() @ w.double().T
    # a sum of 64 k is cut off at most 24 times by 2^-23 of the products' sizes, the sums of K / 64 such and of up to eight parts are rounded, and the
    # terms left out are below 3 * 2^-24; f32 multiply-adds in one chain round K times
    b = max(48 + K // 64 + 12, K) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    for ldc in (N, N + 3, (N + 15) // 8 * 8):
        mem = torch.full((M, ldc), 7.0, device="cuda")
        out = mem[:, :N]
        ops.linear_forward(x, w, bias, out=out)
        assert bool(((out.double() - e - bias.double()).abs() <= b + 2.0 ** -23 * (e.abs() + bias.abs())).all())
        assert bool((mem[:, N:] == 7.0).all())
    assert float((out.double() - e - bias.double()).norm() / e.norm()) < 6e-7
    assert ops.device_error() == 0


@pytest.mark.parametrize("M,N,K", [(1290, 4100, 580), (300, 1000, 1001)])
@pytest.mark.parametrize("kn", [False, True])
def test_results_that_are_not_finite(ops, M, N, K, kn):
    x, w = rows(M, K, K, 0, 1), rows(N, K, K, 0, 2)
    x[3, 7], x[M - 1, K - 1], w[N - 1, 5], x[9, 1] = float("inf"), float("nan"), -float("inf"), 3.4028e38
    w[:, 1] = w[:, 1].clamp(-0.9, 0.9)
    x[200] *= 1e-36
    y = ops.matmul_forward(x, w.T.contiguous()) if kn else ops.linear_forward(x, w, None)
    e = x.double() @ w.double().T
    f = e.float()
    assert torch.equal(torch.isnan(y), torch.isnan(f)) and torch.equal(torch.isinf(y), torch.isinf(f))
    some = torch.isfinite(f)
    b = max(48 + K // 64 + 12, K) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T) + K * 2.0 ** -149
    assert bool(((y.double() - e).abs() <= b)[some].all())


@pytest.mark.parametrize("M,N", [(1290, 4100), (300, 1002), (130, 70)])  # pairs, single CTAs, K over a cluster
@pytest.mark.parametrize("K", [1001, 1002, 1003])
@pytest.mark.parametrize("kn", [False, True])
def test_results_that_are_not_finite_between_padded_rows(ops, M, N, K, kn):
    """Rows that start on 16 bytes with lengths that are no multiple of four: what is summed again ends at a row's last number as well."""
    x = rows(M, K, 1004, 0, 1)
    w = rows(K, N, (N + 3) // 4 * 4 + 4, 0, 2).T if kn else rows(N, K, 1004, 0, 2)
    x[3, 7], x[M - 1, K - 1], w[N - 1, 5] = float("inf"), float("nan"), -float("inf")
    x[9] *= 2.0 ** 50  # finite sums from 2^80 on overflow on their way
    w[11] *= 2.0 ** 45
    y = ops.linear_forward(x, w, None)
    e = x.double() @ w.double().T
    f = e.float()
    assert torch.equal(torch.isnan(y), torch.isnan(f)) and torch.equal(torch.isinf(y), torch.isinf(f))
    some = torch.isfinite(f)
    assert bool(some[9, 11]) and abs(float(e[9, 11])) > 2.0 ** 90
    b = max(48 + K // 64 + 12, K) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)  # (as above)
    assert bool(((y.double() - e).abs() <= b)[some].all())
    assert ops.device_error() == 0
