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


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D", [8, 16, 32, 48, 64, 80, 96, 112, 128])
def test_scores_are_not_off_to_one_side(ops, dtype, D):
    """Mean error of logsumexp over many rows, relative to the largest scores, which decide it: a score times the scale in f32 may be off by the scale's
    rounding, a half-ulp (2^-24), for all keys alike; the mean over 30000 rows of what else is rounded stays well below a third of that."""
    if dtype == torch.bfloat16 and D == 128:
        pytest.skip("the bf16 kernel's head size")
    g = torch.Generator(device="cuda").manual_seed(D)
    q, k, v = (torch.randn(32, 1000, D, generator=g, device="cuda").to(dtype) for _ in range(3))
    off = []
    for scale in (4.0, 3.7, 3.1, 2.6):
        scale = float(torch.tensor(scale * D ** -0.5))  # as the f32 number that the kernel gets
        s = q.double() @ k.double().transpose(1, 2) * scale
        l = ops.flash_attention2_forward(q, k, v, scale)[1]
        off.append(float((l.double() - torch.logsumexp(s, -1)).mean() / s.amax(-1).mean()))
    assert max(map(abs, off)) <= 2.0 ** -24 * 4 / 3 and abs(sum(off)) / len(off) <= 2.0 ** -24, off


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D", [8, 16, 64, 120])
def test_exact_scores(ops, dtype, D):
    """Scores of one product of powers of two: nothing is cut off, and what the kernel allows for on average (up to 6.5e-8) and the roundings of scale and result
    stay within 1.5 ulps of 2^-23."""
    i = torch.arange(300, device="cuda")
    q, k = (torch.zeros(40, 300, D, device="cuda", dtype=dtype) for _ in range(2))
    q[:, i, i % D], k[:, i, i % D] = 8.0, 4.0
    l = ops.flash_attention2_forward(q, k, torch.ones_like(k), 1.0)[1]
    e = torch.logsumexp(q.double() @ k.double().transpose(1, 2), -1)
    assert float(((l.double() - e) / e).abs().max()) <= 1.5 * 2.0 ** -23
    assert ops.device_error() == 0
