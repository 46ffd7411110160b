"""GPU: the CUDA-core attention kernel (f32, and bf16 head sizes outside the tcgen05 kernel) against float64, at the edges of its tiles of
16 R query rows and 64 keys and of its head-size classes 64 / 128 / 256."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from teenygrad_b200 import ops as o
    return o


def reference(q, k, v, scale, causal):
    """(output, logsumexp, bound on an f32 evaluation's error) in float64; q [B, H, Sq, D], k / v [B, G, Skv, D]."""
    q, k, v = q.double(), k.double(), v.double()
    per = q.shape[1] // k.shape[1]
    k, v = k.repeat_interleave(per, 1), v.repeat_interleave(per, 1)
    s = q @ k.transpose(-1, -2) * scale
    size = q.abs() @ k.abs().transpose(-1, -2) * scale
    if causal:
        hidden = torch.ones(s.shape[-2:], dtype=torch.bool, device=s.device).triu(1 + s.shape[-1] - s.shape[-2])
        s = s.masked_fill(hidden, -float("inf"))
    # every score is off by at most (D + 2) half-ulps of its products' size, an exponential by that and two ulps, a weighted mean of
    # Skv terms by twice the largest such error and Skv half-ulps more
    eps = 2.0 ** -24
    err = (q.shape[-1] + 2) * eps * float(size.max()) + 6 * eps
    bound = (2 * err + (k.shape[2] + 8) * eps) * float(v.abs().max())
    return torch.softmax(s, -1) @ v, torch.logsumexp(s, -1), bound, err + (k.shape[2] + 8) * eps


@pytest.mark.parametrize("B,H,G,Sq,Skv,D,causal", [
    (1, 1, 1, 1, 1, 8, False), (1, 3, 3, 17, 65, 64, False), (1, 40, 40, 130, 200, 64, False), (1, 64, 64, 700, 63, 64, False),
    (2, 33, 11, 64, 128, 128, True), (1, 64, 64, 129, 129, 128, True), (1, 2, 1, 40, 70, 200, True), (1, 40, 8, 65, 190, 256, False),
    (1, 5, 5, 7, 64, 3, False), (2, 6, 2, 33, 97, 65, True), (3, 64, 32, 257, 320, 40, True),
])
def test_f32_attention_stays_within_the_error_of_f32_sums(ops, B, H, G, Sq, Skv, D, causal):
    g = torch.Generator().manual_seed(B + H * Sq + Skv * D)
    q, k, v = (torch.randn(B, h, n, D, generator=g).cuda() for h, n in ((H, Sq), (G, Skv), (G, Skv)))
    e, el, bound, lbound = reference(q, k, v, D ** -0.5, causal)
    if G == H and not causal:
        o, l = ops.flash_attention2_forward(q.flatten(0, 1), k.flatten(0, 1), v.flatten(0, 1), D ** -0.5)
        assert float((o.view_as(e).double() - e).abs().max()) <= bound
        assert float((l.view_as(el).double() - el).abs().max()) <= lbound + 2.0 ** -22 * float(el.abs().max())
    # bf16 views whose rows no vector load may touch: one element off, a row stride that is no multiple of 4
    wide = [torch.zeros(B, t.shape[1], t.shape[2], D + 3, dtype=torch.bfloat16, device="cuda") for t in (q, k, v)]
    for w, t in zip(wide, (q, k, v)):
        w.fill_(float("nan"))[..., 1:D + 1] = t.bfloat16()
    qb, kb, vb = (w[..., 1:D + 1] for w in wide)
    e, el, bound, lbound = reference(qb, kb, vb, D ** -0.5, causal)
    o, l = ops.flash_attn_fwd(qb, kb, vb, D ** -0.5, causal=causal, want_lse=True)
    assert float((o.double() - e).abs().max()) <= bound + 2.0 ** -8 * float(e.abs().max())  # and one rounding to bf16
    assert float((l.double() - el).abs().max()) <= lbound + 2.0 ** -22 * float(el.abs().max())
    assert ops.device_error() == 0


def test_masked_and_infinite_values_behave_as_in_a_loop_over_the_keys(ops):
    """A NaN in a value row past the causal edge or in the padding of a tile must not reach a result; a NaN or an infinite score
    that a row does see must."""
    g = torch.Generator().manual_seed(1)
    q, k, v = (torch.randn(1, 2, 70, 64, generator=g).bfloat16().cuda() for _ in range(3))
    v[:, :, 69] = float("nan")
    o = ops.flash_attn_fwd(q, k, v, 0.125, causal=True)
    assert torch.isfinite(o[:, :, :69]).all() and torch.isnan(o[:, :, 69]).all()
    k[:, :, 3] = float("inf")
    o = ops.flash_attn_fwd(q, k, v, 0.125, causal=True)
    assert torch.isfinite(o[:, :, :3]).all() and torch.isnan(o[:, :, 3:]).all()
