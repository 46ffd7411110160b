"""GPU: bf16 GEMMs of many rows store their results through shared memory and clipped TMA stores: ragged edges, bias, rows with a
stride of their own, and outputs that such a store cannot describe."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from teenygrad_b200 import ops as o
    return o


@pytest.mark.parametrize("M,N,K", [(1300, 5000, 200), (4500, 2056, 136), (2049, 4104, 72)])
@pytest.mark.parametrize("extra", [0, 8, 3])
def test_edges(ops, M, N, K, extra):
    g = torch.Generator(device="cuda").manual_seed(M + N + extra)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    bias = torch.randn(N, generator=g, device="cuda").bfloat16()
    e, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    slack = K * 2.0 ** -23 * size  # f32 sums, cut off or rounded at each of K steps; the result is rounded to bf16 once
    mem = torch.full((M, N + extra), 7.0, device="cuda", dtype=torch.bfloat16)
    out = mem[:, :N]
    for b in (None, bias):
        ops.linear_forward(x, w, b, out=out)
        want = e if b is None else e + b.double()
        assert bool(((out.double() - want).abs() <= slack + 2.0 ** -8 * want.abs()).all())
        assert bool((mem[:, N:] == 7.0).all())
    y = ops.matmul_forward(x, w.T.contiguous())
    assert bool(((y.double() - e).abs() <= slack + 2.0 ** -8 * e.abs()).all())
    assert ops.device_error() == 0
