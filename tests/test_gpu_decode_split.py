"""Decode attention with a sequence over the CTAs of a cluster: live lengths at the edges of the 64-key tiles and of the parts, parts without
keys, one to eight parts; and, through a model's decode steps, the newest key written into a tile that was requested before it existed."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Hq,Hkv,cap", [(1, 16, 8, 576), (1, 8, 8, 100), (2, 16, 2, 320), (4, 32, 8, 1024), (8, 32, 8, 200), (3, 8, 1, 4096), (5, 40, 5, 640)])
@pytest.mark.parametrize("which", ["one", "tile-1", "tile", "tile+1", "half", "full"])
def test_lengths_at_the_edges(B, Hq, Hkv, cap, which):
    from teenygrad_b200 import ops
    n = {"one": 1, "tile-1": 63, "tile": 64, "tile+1": 65, "half": cap // 2 + 1, "full": cap}[which]
    g = torch.Generator(device="cuda").manual_seed(B + Hq + cap + n)
    q = torch.randn(B, Hq, 1, 128, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(B, Hkv, cap, 128, generator=g, device="cuda").bfloat16() for _ in range(2))
    k[:, :, n:] = float("nan")
    v[:, :, n:] = float("nan")  # rows behind the live length are never part of a result
    y = ops.flash_attn_decode(q, k, v, n, 128 ** -0.5).view(B, Hq, 128)
    kk, vv = (t[:, :, :n].double().repeat_interleave(Hq // Hkv, 1) for t in (k, v))
    p = torch.softmax(torch.einsum("bhd,bhkd->bhk", q.view(B, Hq, 128).double(), kk) * 128 ** -0.5, -1)
    ref = torch.einsum("bhk,bhkd->bhd", p, vv)
    # probabilities and the output are rounded to bf16 (2^-9 each, the former averaged over the keys)
    assert float((y.double() - ref).norm() / ref.norm()) < 4e-3
    assert ops.device_error() == 0


@pytest.mark.parametrize("B,prompt,cap", [(1, 60, 600), (1, 122, 200), (2, 250, 300), (1, 4, 64)])
def test_steps_across_tiles(B, prompt, cap):
    """Logits of decode steps against those of one prefill over the same tokens."""
    from teenygrad_b200 import qwen3
    cfg = qwen3.Qwen3Config(2, 256, 4, 2, 128, 512, 1024, tied=False)
    r = qwen3.Qwen3Runner(cfg, max_batch=B, max_len=cap, max_tokens=B * cap, max_new_tokens=16)
    qwen3.load_random_weights(r, 3)
    ids = torch.randint(0, cfg.vocab, (B, prompt), generator=torch.Generator().manual_seed(prompt), dtype=torch.int32)
    for graph in (False, True):
        got = r.generate(ids, 9, use_graph=graph).cpu()
        last = r.logits().float().cpu()
        r.prefill(torch.cat([ids, got[:, :8]], 1))
        want = r.logits().float().cpu()
        # the same weights and tokens, sums in another order with bf16 tensors in between: a few rounding steps of 2^-9
        assert float((last - want).norm() / want.norm()) < 2e-2
    assert r.device_error() == 0
