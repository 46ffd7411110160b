"""The decode GEMM for few rows (M <= 16): edges of its units (8 weight rows), of its 64-k blocks and of its groups, plain, gated and with
norm and residual folded in (the latter through a model's decode step), against f32 products of the same operands."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _close(y, ref):
    # one rounding to bf16 (2^-9 of the value) behind f32 sums of at most a few thousand products
    assert torch.isfinite(y).all()
    d = (y.double() - ref).abs()
    assert float((d / (ref.abs() * 2 ** -8 + 1e-3 * ref.pow(2).mean().sqrt())).max()) <= 1.0


@pytest.mark.parametrize("M", [1, 3, 8, 9, 16])
@pytest.mark.parametrize("N,K,pad,bias", [(8, 8, 0, False), (1, 64, 0, True), (1024, 1024, 0, False), (1187, 72, 8, True), (4096, 520, 0, False),
                                          (2367, 1032, 16, True), (12345, 256, 0, False), (72, 4096, 0, False)])
def test_linear_few_rows(M, N, K, pad, bias):
    from teenygrad_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N + K)
    x = torch.full((M, K + pad), float("nan"), device="cuda", dtype=torch.bfloat16)[:, :K]  # what lies between the rows is not read
    w = torch.full((N, K + pad), float("nan"), device="cuda", dtype=torch.bfloat16)[:, :K]
    x.copy_(torch.randn(M, K, generator=g, device="cuda"))
    w.copy_(torch.randn(N, K, generator=g, device="cuda") * K ** -0.5)
    b = torch.randn(N, generator=g, device="cuda").bfloat16() if bias else None
    y = ops.linear_forward(x, w, b)
    ref = x.double() @ w.double().t() + (b.double() if bias else 0.0)
    _close(y, ref)
    assert ops.device_error() == 0


@pytest.mark.parametrize("M,C,K", [(1, 64, 64), (5, 3072, 1024), (16, 1600, 136), (8, 12288, 512)])
def test_swiglu_few_rows(M, C, K):
    from teenygrad_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + C + K)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    gate, up = ((torch.randn(C, K, generator=g, device="cuda") * K ** -0.5).bfloat16() for _ in range(2))
    w = torch.stack([gate.view(-1, 64, K), up.view(-1, 64, K)], 1).reshape(2 * C, K).contiguous()
    y = ops.linear_swiglu(x, w)
    a, b = (x.float() @ gate.float().t()).bfloat16().double(), (x.float() @ up.float().t()).bfloat16().double()
    ref = torch.nn.functional.silu(a) * b
    # the projections, silu and the product are bf16 tensors: four roundings
    d = (y.double() - ref).abs()
    assert float((d / (ref.abs() * 2 ** -6 + 2e-2 * ref.pow(2).mean().sqrt())).max()) <= 1.0
    assert ops.device_error() == 0
