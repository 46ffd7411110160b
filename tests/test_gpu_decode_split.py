"""Decode attention with a sequence over the CTAs of a cluster: live lengths at the edges of the 64-key tiles and of the parts, parts without
keys, one to eight parts; the same over more parts than a cluster has CTAs, merged by a second kernel or by the last CTA to arrive; and, through
a model's decode steps, the newest key written into a tile that was requested before it existed."""
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


def reference(q, k, v, n, scale):
    """[B, Hq, 128] in 64 bits over the first n rows of the caches."""
    rep = q.shape[1] // k.shape[1]
    kk, vv = (t[:, :, :n].double().repeat_interleave(rep, 1) for t in (k, v))
    return torch.einsum("bhk,bhkd->bhd", torch.softmax(torch.einsum("bhd,bhkd->bhk", q.double(), kk) * scale, -1), vv)


# clusters that the GPU holds at once and ones that it does not (then fewer parts), one CTA for few live keys
@pytest.mark.parametrize("B,Hq,Hkv,cap", [(2, 32, 8, 2048), (3, 32, 8, 1600), (6, 32, 8, 1024), (7, 40, 5, 700), (4, 32, 4, 1100), (12, 32, 8, 512), (3, 64, 8, 900)])
@pytest.mark.parametrize("n", [1, 191, 192, 193, 255, 256, 257, 320, 500])
def test_parts_by_residency_and_live_length(B, Hq, Hkv, cap, n):
    from teenygrad_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(B + Hq + cap + n)
    q = torch.randn(B, Hq, 1, 128, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(B, Hkv, cap, 128, generator=g, device="cuda").bfloat16() for _ in range(2))
    k[:, :, n:] = v[:, :, n:] = float("nan")
    ref = reference(q.view(B, Hq, 128), k, v, n, 128 ** -0.5)
    y = ops.flash_attn_decode(q, k, v, n, 128 ** -0.5).view(B, Hq, 128)
    assert float((y.double() - ref).norm() / ref.norm()) < 4e-3  # as above
    c = ops.cached_attention(q.view(B, Hq, 128), k, v, 128 ** -0.5, [(b, n - 1, b, 1) for b in range(B)])
    assert float((c.double() - ref).norm() / ref.norm()) < 4e-3
    assert ops.device_error() == 0


MANY = [(1, 8, 1, 8192), (1, 16, 8, 4609), (2, 32, 8, 6000), (1, 4, 4, 8192), (4, 8, 2, 5121), (2, 16, 2, 4700), (16, 8, 1, 4673)]


@pytest.mark.parametrize("B,Hq,Hkv,cap", MANY)
@pytest.mark.parametrize("which", ["one", "tile", "tile+1", "few", "part-1", "part", "part+1", "half", "full-1", "full"])
def test_more_parts_than_a_cluster(B, Hq, Hkv, cap, which):
    """Capacities of nine and more parts: partial results through scratch, merged by a second kernel (the operator over whole caches) or
    by the last CTA of a head to arrive, which re-arms its counter (the operator over slots, several calls on one scratch)."""
    from teenygrad_b200 import ops
    parts = min(148 // (B * Hkv), (cap + 511) // 512)
    span = ((cap + parts - 1) // parts + 63) // 64 * 64
    n = {"one": 1, "tile": 64, "tile+1": 65, "few": 700, "part-1": span - 1, "part": span, "part+1": span + 1, "half": cap // 2 + 1, "full-1": cap - 1,
         "full": cap}[which]
    g = torch.Generator(device="cuda").manual_seed(B + Hq + cap + n)
    q = torch.randn(B, Hq, 1, 128, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(B, Hkv, cap, 128, generator=g, device="cuda").bfloat16() for _ in range(2))
    q3, scale = q.view(B, Hq, 128), 128 ** -0.5
    y = ops.flash_attn_decode(q, k, v, n, scale).view(B, Hq, 128)
    dev = ops.flash_attn_decode(q, k, v, torch.tensor([n], dtype=torch.int32, device="cuda"), scale).view(B, Hq, 128)
    ref = reference(q3, k, v, n, scale)
    assert float((y.double() - ref).norm() / ref.norm()) < 4e-3 and torch.equal(y, dev)
    scratch = (torch.full((ops.lib.teeny_attn_decode_scratch_bytes(B, Hq, 128, cap),), 255, dtype=torch.uint8, device="cuda"),  # NaNs
               torch.zeros(B * Hkv, dtype=torch.int32, device="cuda"))
    for m in (n, max(1, n - 70), n):  # another number of parts with keys in between
        c = ops.cached_attention(q3, k, v, scale, [(b, m - 1, b, 1) for b in range(B)], scratch=scratch)
        ref = reference(q3, k, v, m, scale)
        assert float((c.double() - ref).norm() / ref.norm()) < 4e-3
        assert not scratch[1].any()
    assert ops.device_error() == 0


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("cap", [1000, 6000])
def test_slots_with_sink_gate_and_cap(dim, cap):
    """The form over slots: entries of unequal lengths in other slots than their number, sinks, a gate and a soft cap; eight parts and more."""
    from teenygrad_b200 import ops
    H, G = 8, 2
    lens, slots = [cap, 1, 65, cap // 2], [3, 0, 4, 2]
    g = torch.Generator(device="cuda").manual_seed(cap + dim)
    q = torch.randn(4, H, dim, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(5, G, cap, dim, generator=g, device="cuda").bfloat16() for _ in range(2))
    sink, gate = torch.randn(H, generator=g, device="cuda"), torch.randn(4, H * dim, generator=g, device="cuda").bfloat16()
    out = ops.cached_attention(q, k, v, dim ** -0.5, [(s, n - 1, i, 1) for i, (s, n) in enumerate(zip(slots, lens))], softcap=8.0, sink=sink, gate=gate)
    for i, (s, n) in enumerate(zip(slots, lens)):
        kk, vv = (t[s, :, :n].double().repeat_interleave(H // G, 0) for t in (k, v))
        x = 8.0 * torch.tanh(torch.einsum("hd,hkd->hk", q[i].double(), kk) * dim ** -0.5 / 8.0)
        p = torch.softmax(torch.cat([x, sink.double()[:, None]], 1), -1)[:, :-1]
        ref = torch.einsum("hk,hkd->hd", p, vv) * torch.sigmoid(gate[i].double()).view(H, dim)
        # probabilities and the output are rounded to bf16
        assert float((out[i].double() - ref).norm() / ref.norm()) < 4e-3
    assert ops.device_error() == 0


@pytest.mark.parametrize("B,prompt,cap", [(1, 600, 8192), (2, 1000, 5000), (1, 4600, 4700)])
def test_steps_with_more_parts_than_a_cluster(B, prompt, cap):
    """Decode steps of a model whose caches have nine parts or more (counters, newest key by the fused front end): every step's logits
    against those of a prefill over the same tokens, eager and by graph replay."""
    from teenygrad_b200 import qwen3
    cfg = qwen3.Qwen3Config(2, 256, 8, 8, 128, 512, 1024, tied=False)
    r = qwen3.Qwen3Runner(cfg, max_batch=B, max_len=cap, max_tokens=B * (prompt + 16), max_new_tokens=16)
    qwen3.load_random_weights(r, 3)
    ids = torch.randint(0, cfg.vocab, (B, prompt), generator=torch.Generator().manual_seed(prompt), dtype=torch.int32)
    for graph in (False, True):
        for steps in (2, 3, 9):
            got = r.generate(ids, steps, use_graph=graph).cpu()
            last = r.logits().float().cpu()
            r.prefill(torch.cat([ids, got[:, :steps - 1]], 1))
            want = r.logits().float().cpu()
            # the same weights and tokens, sums in another order with bf16 tensors in between: a few rounding steps of 2^-9
            assert float((last - want).norm() / want.norm()) < 2e-2
    assert r.device_error() == 0
