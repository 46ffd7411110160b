"""GPU: attention with f32 sums on the tensor cores (f32 operands, bf16 head sizes outside the bf16 kernel) against float64, at the edges of its tiles of
128 query rows and 128 (head size up to 64) or 64 keys, on sizes that its estimate takes from the CUDA-core kernel."""
import pytest
import torch

from test_gpu_simt_attention import reference

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from teenygrad_b200 import ops as o
    return o


@pytest.mark.parametrize("H,Sq,Skv,D,scale", [
    (1, 1, 257, 64, 0.125), (2, 128, 256, 64, 0.125), (3, 129, 511, 64, 1.0), (40, 127, 128, 64, 0.125), (150, 130, 129, 64, 0.125), (5, 300, 300, 8, 0.5),
    (4, 257, 385, 40, 0.3), (2, 128, 320, 128, 0.1), (3, 255, 191, 128, 0.0884), (5, 1, 257, 72, 0.1), (149, 64, 128, 128, 0.0884), (7, 100, 1000, 120, 2.0),
])
def test_f32_within_the_error_of_f32_sums(ops, H, Sq, Skv, D, scale):
    g = torch.Generator().manual_seed(H + Sq * Skv + D)
    q, k, v = (torch.randn(1, H, n, D, generator=g).cuda() for n in (Sq, Skv, Skv))
    e, el, bound, lbound = reference(q, k, v, scale, False)
    o, l = ops.flash_attention2_forward(q[0], k[0], v[0], scale)
    assert float((o.double() - e[0]).abs().max()) <= bound
    assert float((l.double() - el[0]).abs().max()) <= lbound + 2.0 ** -22 * float(el.abs().max())
    assert ops.device_error() == 0


@pytest.mark.parametrize("B,H,G,Sq,Skv,D,causal", [
    (1, 8, 2, 300, 300, 64, True), (2, 6, 3, 129, 400, 64, True), (1, 4, 4, 257, 257, 96, True), (1, 5, 1, 128, 700, 32, False), (2, 3, 3, 513, 640, 80, True),
    (1, 2, 2, 1, 300, 16, True),
])
@pytest.mark.parametrize("out_pad", [0, 4])
def test_bf16_heads_of_other_sizes(ops, B, H, G, Sq, Skv, D, causal, out_pad):
    g = torch.Generator().manual_seed(B + H * Sq + Skv * D)
    # views of the layout [B, S, H, D], as a projection leaves them
    q, k, v = (torch.randn(B, n, h, D, generator=g).bfloat16().cuda().transpose(1, 2) for h, n in ((H, Sq), (G, Skv), (G, Skv)))
    e, el, bound, lbound = reference(q, k, v, D ** -0.5, causal)
    out = torch.zeros(B, Sq, H, D + out_pad, dtype=torch.bfloat16, device="cuda")
    o, l = ops.flash_attn_fwd(q, k, v, D ** -0.5, causal=causal, out=out[..., :D].transpose(1, 2), want_lse=True)
    assert float((o.double() - e).abs().max()) <= bound + 2.0 ** -8 * float(e.abs().max())  # and one rounding to bf16
    assert float((l.double() - el).abs().max()) <= lbound + 2.0 ** -22 * float(el.abs().max())
    assert not out[..., D:].any() and ops.device_error() == 0


@pytest.mark.parametrize("D", [64, 128])
def test_f32_values_outside_the_range_of_the_terms(ops, D):
    """Rows that meet infinities, NaNs or numbers whose terms or sums overflow are those of a loop over the keys, the others are not touched."""
    g = torch.Generator().manual_seed(D)
    q, k, v = (torch.randn(6, 260, D, generator=g).cuda() for _ in range(3))
    k[0, 200] = float("inf")
    v[1, 3, 5] = float("nan")
    q[2, 7] = 2.0 ** 105
    k[3, 11] *= 2.0 ** 90
    v[4] *= 2.0 ** 110
    o, l = ops.flash_attention2_forward(q, k, v, D ** -0.5)
    e, el, bound, _ = reference(q[None], k[None], v[None], D ** -0.5, False)
    e, el = e[0], el[0]
    for h in (0, 1, 3, 4):  # (head 3: scores of 1e27, a key or none decides)
        want = e[h].float()
        assert torch.equal(torch.isfinite(o[h]), torch.isfinite(want)), h
        ok = torch.isfinite(want)
        scale = float(v[h][torch.isfinite(v[h])].abs().max())
        assert float((o[h].double() - e[h])[ok].abs().max() if ok.any() else 0.0) <= 1e-5 * scale, h
    rows = torch.arange(260, device="cuda") != 7
    assert float((o[2, rows].double() - e[2, rows]).abs().max()) <= 1e-5
    assert float((o[5].double() - e[5]).abs().max()) <= 1e-5 and float((l[5].double() - el[5]).abs().max()) <= 1e-5
    # the row with huge queries: one key takes it all
    assert float((o[2, 7].double() - e[2, 7]).abs().max()) <= 1e-5
    tiny = ops.flash_attention2_forward(q[5:], k[5:] * 2.0 ** -120, v[5:] * 2.0 ** -110, 1.0)[0].double()
    mean = torch.softmax(q[5:].double() @ (k[5:] * 2.0 ** -120).double().transpose(1, 2), -1) @ (v[5:] * 2.0 ** -110).double()
    assert float((tiny - mean).abs().max()) <= 1e-6 * float(mean.abs().max())
    assert ops.device_error() == 0


@pytest.mark.parametrize("D", [64, 96])
def test_values_behind_the_causal_edge_do_not_count(ops, D):
    g = torch.Generator().manual_seed(1)
    q, k, v = (torch.randn(1, 2, 300, D, generator=g).bfloat16().cuda() for _ in range(3))
    v[:, :, 299] = float("nan")
    o = ops.flash_attn_fwd(q, k, v, 0.125, causal=True)
    assert torch.isfinite(o[:, :, :299]).all() and torch.isnan(o[:, :, 299]).all()
    e, _, bound, _ = reference(q[:, :, :299], k[:, :, :299], v[:, :, :299], 0.125, True)
    assert float((o[:, :, :299].double() - e).abs().max()) <= bound + 2.0 ** -8 * float(e.abs().max())
    k[:, :, 130] = float("inf")
    o = ops.flash_attn_fwd(q, k, v, 0.125, causal=True)
    assert torch.isfinite(o[:, :, :130]).all() and torch.isnan(o[:, :, 130:]).all()
    assert ops.device_error() == 0
