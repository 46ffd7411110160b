"""GPU: the CUDA-core GEMM (f32, and bf16 layouts that TMA cannot describe) against float64, over its four tiles, its operand layouts and
ragged edges."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from teenygrad_b200 import ops as o
    return o


def off(t, n):
    """The same values in a storage that starts ``n`` elements later and has rows of an odd length."""
    w = torch.full((t.shape[0], t.shape[1] + n + 1), float("nan"), dtype=t.dtype, device=t.device)
    w[:, n:n + t.shape[1]] = t
    return w[:, n:n + t.shape[1]]


@pytest.mark.parametrize("M,N,K", [
    (1, 1, 1), (3, 33, 17), (16, 32, 96), (17, 100, 1000), (33, 65, 15), (130, 260, 300), (64, 64, 64), (257, 129, 100), (1000, 1030, 64),
    (1100, 2300, 36),
])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_every_layout_and_edge(ops, M, N, K, dtype):
    g = torch.Generator().manual_seed(M * 7 + N * 3 + K)
    x, w, bias = (torch.randn(*s, generator=g).to(dtype).cuda() for s in ((M, K), (N, K), (N,)))
    e = x.double() @ w.double().T
    # sums of K products in any order: at most K half-ulps of the products' sizes; bf16 results are rounded once
    size = x.double().abs() @ w.double().abs().T + bias.double().abs()
    bound = (K + 2) * 2.0 ** -24 * size + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0) * (e.abs() + bias.double().abs())
    views = [(x, w), (off(x, 1), off(w, 3)), (x.T.contiguous().T, w), (x, w.T.contiguous().T), (x.T.contiguous().T, w.T.contiguous().T)]
    for a, b in views:
        out = torch.empty(M, N, dtype=dtype, device="cuda")
        ops.linear_forward(a, b, bias, out=out)
        assert bool(((out.double() - e - bias.double()).abs() <= bound).all())
        out_t = torch.empty(N, M, dtype=dtype, device="cuda").T  # a transposed result
        ops.linear_forward(a, b, None, out=out_t)
        assert bool(((out_t.double() - e).abs() <= bound).all())
    if dtype == torch.float32:
        assert bool(((ops.matmul_forward(x, w.T.contiguous()).double() - e).abs() <= bound).all())
    assert ops.device_error() == 0
