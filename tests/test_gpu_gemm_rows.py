"""The decode GEMM for few rows (M <= 16): edges of its units (8 weight rows), of its 64-k blocks and of its groups, plain and gated against f32
products of the same operands; with FP8 weights, and with the norm in front and the residual behind folded in, through decode steps of single
layers against the oracle."""
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


# ---- with norm and residual folded in, and with FP8 weights: a decode step of one layer ----
def _layer(hidden, ff, weights, seed):
    """(oracle's configuration, its bf16 weights, a runner's tensors): every matrix as E4M3 bytes with power-of-two scales that differ from
    channel to channel, so that both see the same numbers and a scale taken from elsewhere shows; sublayers as large as the residual."""
    from oracle import qwen3 as oq
    cfg = oq.OracleQwen3Config(1, hidden, 4, 2, 128, ff, 256, tied=False)
    g = torch.Generator().manual_seed(seed)
    sd, q8 = {}, {}
    for name, t in oq.make_weights(cfg, seed).items():
        if t.dim() < 2 or "embed" in name or "lm_head" in name:
            sd[name] = q8[name] = (1.0 + 0.2 * torch.randn(t.shape, generator=g)).bfloat16() if t.dim() < 2 else torch.randn(t.shape, generator=g).bfloat16()
            continue
        scale = torch.full((1,), 0.25) if weights == "tensor" else 2.0 ** torch.randint(-4, 0, (t.shape[0],), generator=g).float()
        b = (torch.randn(t.shape, generator=g) * 4 * t.shape[1] ** -0.5).to(torch.float8_e4m3fn)
        sd[name] = (b.float() * scale[:, None]).bfloat16()
        q8[name], q8[name + "_scale"] = b, scale
    return cfg, sd, q8


@pytest.mark.parametrize("batch", [1, 3, 8, 9, 13, 16])
@pytest.mark.parametrize("weights", ["bf16", "channel", "tensor"])
@pytest.mark.parametrize("hidden,ff", [(208, 64), (336, 192), (1040, 1600), (528, 2880)])  # K = 16 x odd; last CTAs of the gated unit partly filled
def test_decode_step_of_one_layer(batch, weights, hidden, ff):
    from oracle import qwen3 as oq
    from teenygrad_b200 import ops, quant, qwen3
    cfg, sd, q8 = _layer(hidden, ff, weights, hidden + ff)
    r = qwen3.Qwen3Runner(qwen3.Qwen3Config(1, hidden, 4, 2, 128, ff, 256, tied=False), max_batch=batch, max_len=24, max_tokens=batch * 20, max_new_tokens=4)
    if weights == "bf16":
        r.load_state_dict(sd)
    else:
        r.load_quantized(q8, quant.Fp8Scheme(weights))
    ids = torch.randint(0, 256, (batch, 20), generator=torch.Generator().manual_seed(batch))
    o = oq.OracleQwen3(cfg, sd, f32_twin=True)
    for graph in (False, True):
        o.reset()
        r.prefill(ids)
        o.forward(ids)
        for _ in range(2):
            nxt = r.next_ids().cpu().long()
            r.decode_step(graph=graph)
            logits = o.forward(nxt[:, None])
            want = o.last_residual[:, 0].double()
            h, d = r.residual_stream(batch)
            d = (h.double().cpu() - want).abs()
            # the same rounding points, sums in another order: single roundings of 2^-9 that fall the other way, carried through two sublayers
            assert float(d.norm() / want.norm()) < 6e-3
            assert float((d / (want.abs() * 2 ** -6 + 4e-2 * want.pow(2).mean().sqrt())).max()) <= 1.0
            assert float((r.logits().double().cpu() - logits.double()).norm() / logits.double().norm()) < 1e-2
    assert ops.device_error() == 0


@pytest.mark.parametrize("batch", [1, 3, 9, 13, 16])
@pytest.mark.parametrize("width,ff", [(96, 100), (328, 136), (1032, 1544)])
def test_step_of_a_hybrid_decoder(batch, width, ff):
    """Norms of f32 rows in front and sums into the f32 residual behind: single tokens of every sequence in one step, against the same tokens
    as part of prompts (more than 16 rows: other kernels) and against 64 bits."""
    from oracle import fiferax as of
    from teenygrad_b200 import fiferax, ops
    cfg = of.make_config(width, 200, [of.gru_layer(width - 8, ff=ff), of.delta_layer(2, 32, ff=ff),
                                      of.parallel_layer(4, 2, 32, 16, 32, 1000.0, 0.25, 2, 16, 24, [0.9, 0.6], ff=ff)])
    w = of.make_weights(cfg, 3)
    toks = [torch.randint(0, 200, (21 + i % 3,), generator=torch.Generator().manual_seed(i)).tolist() for i in range(batch)]
    r = fiferax.build(cfg, w, max_batch=16, max_len=32, max_rows=32 * 16)

    def run(cut):
        seqs = [r.open() for _ in toks]
        r.step([(s, t[:-cut], []) for s, t in zip(seqs, toks)])
        for j in range(cut, 0, -1):
            out = r.step([(s, t[len(t) - j:len(t) - j + 1], [0]) for s, t in zip(seqs, toks)])
        for s in seqs:
            r.close(s)
        return torch.cat(out).double().cpu()

    got = run(3)
    want = torch.stack([of.forward(cfg, w, t)[-1] for t in toks])
    seqs = [r.open() for _ in toks]
    whole = torch.cat(r.step([(s, t, [len(t) - 1]) for s, t in zip(seqs, toks)])).double().cpu()
    size = want.pow(2).mean().sqrt()
    # bf16 tensors between the kernels on either way: within the scatter that the prompt's way has around 64 bits
    err, scatter = float((got - want).pow(2).mean().sqrt() / size), float((whole - want).pow(2).mean().sqrt() / size)
    assert err < max(1.5 * scatter, 1e-2) and err < 4e-2
    assert ops.device_error() == 0
