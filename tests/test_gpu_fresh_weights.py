"""Weights that another operator of the library has written just before: an operator must not fetch them ahead of that.  Every launch is
asynchronous, so each chain below runs many times over new contents without a synchronisation in between, and has to give what the same
operator gives once its weights are known to be in place."""
import pytest
import torch

pytestmark = pytest.mark.gpu

ROUNDS = 24
# rows on both sides of every choice by rows; weights that the kernel for few rows takes and ones that it does not
SHAPES = [(1, 1024, 1024), (16, 1024, 3072), (16, 4096, 4096), (17, 1024, 1024), (64, 4096, 1024), (128, 2048, 4096), (200, 520, 8192), (3, 72, 48)]


def _fp8(g, N, K):
    bits = torch.randint(0, 256, (N, K), generator=g, dtype=torch.uint8, device="cuda")
    bits[(bits & 0x7F) == 0x7F] = 0x08  # no NaN encodings
    return bits


def _chain(write, use, same):
    """``write(i, buffer)`` then ``use(buffer)``, back to back; against ``use`` on finished contents."""
    outs = [None] * ROUNDS
    for i in range(ROUNDS):
        write(i)
        outs[i] = use().clone()  # (torch's copy waits for the operator in front of it, the next write for the copy)
    torch.cuda.synchronize()
    for i in range(ROUNDS):
        write(i)
        torch.cuda.synchronize()
        want = use()
        torch.cuda.synchronize()
        assert same(outs[i], want), f"pass {i} differs"


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_dequantised_just_before(M, N, K):
    from teenygrad_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    src = [_fp8(g, N, K) for _ in range(3)]
    scale = torch.rand(N, generator=g, device="cuda") * 0.01 + 0.001
    w, y = torch.zeros(N, K, dtype=torch.bfloat16, device="cuda"), torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    _chain(lambda i: ops.dequant_fp8(src[i % 3], scale, out=w), lambda: ops.linear_forward(x, w, out=y), torch.equal)
    # an independent value, so that both sides cannot be wrong alike: f32 sums of exact products, one rounding
    ref = x.double() @ w.double().t()
    assert float((y.double() - ref).norm() / ref.norm()) < 2 ** -8
    assert ops.device_error() == 0


@pytest.mark.parametrize("M,N,K", [(1, 1024, 1024), (16, 512, 2048), (17, 1024, 1024), (128, 128, 4096)])
def test_computed_by_a_linear_just_before(M, N, K):
    """w = b a^T by the kernels for few rows (N <= 16 rows of w would be too few to tell: several of them make one w)."""
    from teenygrad_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M * N + K)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    a = [(torch.randn(K, 256, generator=g, device="cuda") / 16).bfloat16() for _ in range(3)]
    b = torch.randn(N, 256, generator=g, device="cuda").bfloat16()
    w, y = torch.zeros(N, K, dtype=torch.bfloat16, device="cuda"), torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    last = (N - 1) // 16 * 16

    def write(i):
        ops.linear_forward(b, a[i % 3], out=w)
        ops.linear_forward(b[last:], a[i % 3], out=w[last:])  # the same values again, by the kernel that lets the next one in at once
    _chain(write, lambda: ops.linear_forward(x, w, out=y), torch.equal)
    assert ops.device_error() == 0


@pytest.mark.parametrize("M,N,K", [(1, 1024, 2048), (16, 2048, 4096), (40, 512, 1024), (128, 1024, 4096)])
def test_fp8_weights_split_just_before(M, N, K):
    """FP8 weight bytes that split_fp8 has written: by the converting kernel and by the FP8 x FP8 one."""
    from teenygrad_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + 3 * N + K)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    src = [torch.randn(N // 2, K, generator=g, device="cuda").bfloat16() for _ in range(3)]
    w8, s8 = torch.zeros(N, K, dtype=torch.uint8, device="cuda"), torch.empty(N // 2, device="cuda")
    one = torch.full((N,), 0.01, device="cuda")
    y = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    x8, xs = ops.split_fp8(x)
    torch.cuda.synchronize()

    def write(i):
        ops.split_fp8(src[i % 3], out=w8, scale=s8)
    _chain(write, lambda: ops.linear_w8a16(x, w8, one, out=y), torch.equal)
    _chain(write, lambda: ops.linear_w8a8x2(x8, xs, w8, one, out=y), torch.equal)
    assert ops.device_error() == 0


@pytest.mark.parametrize("M", [1, 16, 100])
def test_gated_unit_just_before(M):
    from teenygrad_b200 import ops
    N, K = 1024, 1024
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    src = [_fp8(g, N, K) for _ in range(3)]
    scale = torch.full((N,), 0.001, device="cuda")
    w, y = torch.zeros(N, K, dtype=torch.bfloat16, device="cuda"), torch.empty(M, N // 2, dtype=torch.bfloat16, device="cuda")
    _chain(lambda i: ops.dequant_fp8(src[i % 3], scale, out=w), lambda: ops.linear_swiglu(x, w, out=y), torch.equal)
    assert ops.device_error() == 0


@pytest.mark.parametrize("batch,prompt", [(1, 130), (2, 100), (1, 500)])
def test_fp8_prefill_converts_each_matrix_in_front_of_its_product(batch, prompt):
    """A prefill of more than 128 rows with an FP8 checkpoint, at sizes whose products share K over clusters of the decode kernel:
    the same logits as a bf16 checkpoint of the dequantised weights."""
    from teenygrad_b200 import quant, qwen3
    cfg = qwen3.Qwen3Config(3, 1024, 8, 4, 128, 3072, 1024, tied=False)
    make = lambda: qwen3.Qwen3Runner(cfg, max_batch=batch, max_len=prompt + 8, max_tokens=batch * prompt, max_new_tokens=4)
    g = torch.Generator(device="cuda").manual_seed(prompt)
    t = {"model.embed_tokens.weight": torch.randn(cfg.vocab, 1024, generator=g, device="cuda").bfloat16()}
    shapes = {"self_attn.q_proj": (1024, 1024), "self_attn.k_proj": (512, 1024), "self_attn.v_proj": (512, 1024), "self_attn.o_proj": (1024, 1024),
              "mlp.gate_proj": (3072, 1024), "mlp.up_proj": (3072, 1024), "mlp.down_proj": (1024, 3072)}
    for i in range(3):
        p = f"model.layers.{i}."
        for n, s in shapes.items():
            t[p + n + ".weight"] = (torch.randn(*s, generator=g, device="cuda") * 0.02).bfloat16()
        for n, d in (("self_attn.q_norm", 128), ("self_attn.k_norm", 128), ("input_layernorm", 1024), ("post_attention_layernorm", 1024)):
            t[p + n + ".weight"] = torch.ones(d, device="cuda").bfloat16()
    t["model.norm.weight"] = torch.ones(1024, device="cuda").bfloat16()
    t["lm_head.weight"] = (torch.randn(cfg.vocab, 1024, generator=g, device="cuda") * 0.02).bfloat16()
    q8, plain = {}, {}
    for name, w in t.items():
        if w.dim() < 2 or "embed" in name or "lm_head" in name:
            q8[name] = plain[name] = w
            continue
        scale = 2.0 ** torch.ceil(torch.log2(w.float().abs().amax(1) / 448.0))  # powers of two: the dequantised weights are bf16 numbers
        q8[name] = (w.float() / scale[:, None]).to(torch.float8_e4m3fn)
        q8[name + "_scale"] = scale
        plain[name] = (q8[name].float() * scale[:, None]).bfloat16()
    a, b = make(), make()
    a.load_quantized(q8, quant.Fp8Scheme("channel"))
    b.load_state_dict(plain)
    ids = torch.randint(0, cfg.vocab, (batch, prompt), generator=torch.Generator().manual_seed(prompt), dtype=torch.int32).cuda()
    b.prefill(ids)
    want = b.logits().clone()
    for _ in range(8):
        a.prefill(ids)
        # the head's few rows run in other kernels for other weight types: sums in another order, one rounding of 2^-9
        assert float((a.logits().float() - want.float()).norm() / want.float().norm()) < 2 ** -8
    assert a.device_error() == 0


@pytest.mark.parametrize("rows", [1, 16, 40])
def test_head_linear_weights_just_before(rows):
    """The matrices of a per-head product that dequant_fp8 has written."""
    from teenygrad_b200 import ops
    H, n, k = 16, 512, 128
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, H, k, generator=g, device="cuda").bfloat16()
    src = [_fp8(g, H * n, k) for _ in range(3)]
    scale = torch.full((H * n,), 0.001, device="cuda")
    w, y = torch.zeros(H * n, k, dtype=torch.bfloat16, device="cuda"), torch.zeros(rows, H, n, dtype=torch.bfloat16, device="cuda")
    _chain(lambda i: ops.dequant_fp8(src[i % 3], scale, out=w), lambda: ops.head_linear(x, w.view(H, n, k), out=y), torch.equal)
    assert ops.device_error() == 0


@pytest.mark.parametrize("post", [False, True])
def test_norm_weights_just_before(post):
    """The weights of the residual norm that the sum of two vectors has made."""
    from teenygrad_b200 import ops
    rows, n = 600, 4096
    g = torch.Generator(device="cuda").manual_seed(7)
    x0 = torch.randn(rows, n, generator=g, device="cuda")
    delta = torch.randn(rows, n, generator=g, device="cuda").bfloat16()
    src = [torch.randn(rows, n, generator=g, device="cuda") for _ in range(3)]
    zero, x, none = torch.zeros(rows, n, device="cuda"), x0.clone(), torch.zeros(rows, n, device="cuda").bfloat16()
    w = torch.zeros(rows, n, device="cuda")

    def write(i):
        # one norm in front whose f32 rows w (the last one is used) become src: it lets the next kernel in before it writes
        w.copy_(src[i % 3])
        ops.residual_rms_norm(w, delta, zero[0], 1e-6)

    def use():
        y = ops.residual_rms_norm(x, none, w[rows - 1], 1e-6, w[rows - 2] if post else None)
        return y
    _chain(write, use, torch.equal)
    assert ops.device_error() == 0


@pytest.mark.parametrize("rows,cached", [(1, 700), (4, 300)])
def test_latent_cache_written_just_before(rows, cached):
    """The cached rows of an entry that latent_prepare has written, with nothing between it and the attention."""
    from teenygrad_b200 import ops
    H, rank, rot = 16, 256, 64
    dim, n = rank + rot, cached + rows
    g = torch.Generator(device="cuda").manual_seed(cached)
    q = torch.randn(rows, H, dim, generator=g, device="cuda").bfloat16()
    src = [torch.randn(n, 64 + rank + rot, generator=g, device="cuda").bfloat16() for _ in range(3)]
    qw, cw = torch.ones(64, device="cuda"), torch.ones(rank, device="cuda")
    freq = 1.0 / 1e4 ** (torch.arange(rot // 2, device="cuda").float() / (rot // 2))
    cache = torch.zeros(1, n, dim, dtype=torch.bfloat16, device="cuda")
    whole, last = ops.seq_table([(0, 0, 0, n)]), ops.seq_table([(0, cached, 0, rows)])
    scratch = torch.empty(ops.lib.teeny_latent_attention_scratch_bytes(rank), dtype=torch.uint8, device="cuda")
    y = torch.zeros(rows, H, rank, dtype=torch.bfloat16, device="cuda")

    def write(i):
        ops.latent_prepare(src[i % 3], (0, 64, 64 + rank), 64, rank, qw, cw, freq, 1e-6, cache, whole, n)
    _chain(write, lambda: ops.latent_attention(q, cache, rank, dim ** -0.5, last, rows, out=y, scratch=scratch), torch.equal)
    assert ops.device_error() == 0


@pytest.mark.parametrize("cached,cap", [(300, 512), (1500, 1600), (5000, 5120)])
def test_cached_rows_written_just_before(cached, cap):
    """All cached rows of an entry, and not only the newest, from the operator in front of its attention (rope_cache over a whole prompt)."""
    from teenygrad_b200 import ops
    H, G, D = 16, 8, 128
    g = torch.Generator(device="cuda").manual_seed(cached)
    q = torch.randn(1, H, D, generator=g, device="cuda").bfloat16()
    src = [(torch.randn(cached, G, D, generator=g, device="cuda").bfloat16(), torch.randn(cached, G, D, generator=g, device="cuda").bfloat16()) for _ in range(3)]
    qs = torch.zeros(cached, H, D, dtype=torch.bfloat16, device="cuda")
    freq = 1.0 / 1e4 ** (torch.arange(D // 2, device="cuda").float() / (D // 2))
    kc, vc = (torch.zeros(1, G, cap, D, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    whole = ops.seq_table([(0, 0, 0, cached)])
    last = (ops.seq_table([(0, cached - 1, 0, 1)]), ops.seq_table([(0, cached - 1, 0, 1)], "cpu"))
    scratch = (torch.empty(ops.lib.teeny_attn_decode_scratch_bytes(1, H, 128, cap), dtype=torch.uint8, device="cuda"), torch.zeros(G, dtype=torch.int32, device="cuda"))
    y = torch.zeros(1, H, D, dtype=torch.bfloat16, device="cuda")

    def write(i):
        ops.rope_cache(qs, *src[i % 3], kc, vc, freq, D, whole, cached)
    _chain(write, lambda: ops.cached_attention(q, kc, vc, D ** -0.5, last, out=y, scratch=scratch), torch.equal)
    assert ops.device_error() == 0


def test_bf16_norm_weights_just_before():
    """The weights of the bf16 norms and of the head norms, from a norm in front whose rows they are."""
    from teenygrad_b200 import ops
    rows, n, H, G = 600, 2048, 4, 2
    g = torch.Generator(device="cuda").manual_seed(9)
    src = [torch.randn(rows, n, generator=g, device="cuda").bfloat16() for _ in range(3)]
    x = torch.randn(rows, n, generator=g, device="cuda").bfloat16()
    w, zero, one = (torch.zeros(rows, n, device="cuda").bfloat16() for _ in range(3))
    one += 1
    qkv0 = torch.randn(8, (H + 2 * G) * 128, generator=g, device="cuda").bfloat16()
    cos, sin = ops.rope_table(1.0 / 1e4 ** (torch.arange(64, device="cuda").float() / 64), 16)
    kc, vc = (torch.zeros(1, G, 16, 128, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    qkv, res = qkv0.clone(), zero.clone()

    def write(i):
        w.copy_(src[i % 3])
        qkv.copy_(qkv0)
        res.copy_(zero)
        ops.add_rms_norm(zero, w, one[0], 1e-6)  # w <- w + 0, by the kernel that lets the next one in before it stores

    def heads():
        ops.qk_norm_rope_kv(qkv, w[rows - 1, :128], w[rows - 1, 128:256], cos, sin, kc, vc, 8, H, G, 0, 1e-6)
        return torch.cat([qkv[:, :H * 128].flatten(), kc.flatten()])
    _chain(write, lambda: ops.rms_norm_forward(x, w[rows - 1], 1e-6), torch.equal)
    _chain(write, lambda: ops.add_rms_norm(x, res, w[rows - 1], 1e-6), torch.equal)
    _chain(write, heads, torch.equal)
    assert ops.device_error() == 0
