"""bf16 linear layers of more than 128 rows: every kernel that the choice by size can take (narrow and wide tiles, CTA pairs, token tiles with K
over a cluster), at ragged sizes and with a gated unit, against f64 products."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(129, 520, 8192), (200, 4096, 4096), (300, 1000, 3080), (513, 1024, 3072), (255, 136, 72), (800, 4096, 1032), (300, 12288, 1024),
                                   (1000, 2056, 520), (129, 8, 4096), (2000, 300, 264)])
def test_linear_any_kernel(M, N, K):
    from teenygrad_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    b = torch.randn(N, generator=g, device="cuda").bfloat16()
    y = ops.linear_forward(x, w, b)
    ref = x.double() @ w.double().t() + b.double()
    # one rounding to bf16 behind f32 sums
    assert float(((y.double() - ref).abs() / (ref.abs() * 2 ** -8 + 1e-3 * ref.pow(2).mean().sqrt())).max()) <= 1.0
    assert ops.device_error() == 0


@pytest.mark.parametrize("M,C,K", [(130, 64, 4096), (300, 512, 3072), (700, 3072, 1024), (129, 1600, 520)])
def test_swiglu_any_kernel(M, C, K):
    from teenygrad_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + C + K)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    gate, up = ((torch.randn(C, K, generator=g, device="cuda") * K ** -0.5).bfloat16() for _ in range(2))
    w = torch.stack([gate.view(-1, 64, K), up.view(-1, 64, K)], 1).reshape(2 * C, K).contiguous()
    y = ops.linear_swiglu(x, w)
    a, b = (x.float() @ gate.float().t()).bfloat16().double(), (x.float() @ up.float().t()).bfloat16().double()
    ref = torch.nn.functional.silu(a) * b
    # the projections, silu and the product are bf16 tensors: four roundings
    assert float(((y.double() - ref).abs() / (ref.abs() * 2 ** -6 + 2e-2 * ref.pow(2).mean().sqrt())).max()) <= 1.0
    assert ops.device_error() == 0


@pytest.mark.parametrize("M,N,K", [(17, 136, 520), (33, 8, 4096), (64, 1000, 72), (65, 129, 8200), (128, 520, 8200), (100, 4096, 1000), (31, 12288, 512), (127, 700, 136),
                                   (16, 640, 11160), (190, 2000, 1032), (257, 3000, 4104), (385, 6144, 1024), (193, 8200, 512)])
@pytest.mark.parametrize("pad", [0, 3])
def test_resident_tiles_and_their_clusters(M, N, K, pad):
    """K of few tiles over clusters of one to eight CTAs, 32 to 256 tokens wide: ragged tokens, weight rows and k, rows of Y that take 8-byte stores and
    rows that do not."""
    from teenygrad_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    b = torch.randn(N, generator=g, device="cuda").bfloat16()
    out = torch.full((M, N + pad), 7.0, dtype=torch.bfloat16, device="cuda")
    ops.linear_forward(x, w, b, out=out[:, :N])
    ref = x.double() @ w.double().t() + b.double()
    assert float(((out[:, :N].double() - ref).abs() / (ref.abs() * 2 ** -8 + 1e-3 * ref.pow(2).mean().sqrt())).max()) <= 1.0
    assert bool((out[:, N:] == 7.0).all()) and ops.device_error() == 0
    again = torch.empty_like(out)
    ops.linear_forward(x, w, b, out=again[:, :N])
    assert torch.equal(out[:, :N], again[:, :N])
