"""GPU: kernels that a choice by size takes, each at ragged sizes that reach it (checked by its name) against float64."""
import pytest
import torch

from kernel_names import kernels

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from teenygrad_b200 import ops as o
    return o


def check_product(y, x, w, bias=None):
    """y = x w^T (+ bias) in bf16: f32 sums, cut off or rounded at each of K steps, rounded to bf16 once."""
    K = x.shape[1]
    e, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    if bias is not None:
        e = e + bias.double()
    assert bool(((y.double() - e).abs() <= K * 2.0 ** -23 * size + 2.0 ** -8 * e.abs()).all())


@pytest.mark.parametrize("kernel,M,N,K", [
    ("gemm_bf16_kernelILi128ELb0ELb0EE", 1290, 6152, 264), ("gemm_bf16_kernelILi128ELb0ELb0EE", 4100, 3000, 72), ("gemm_bf16_kernelILi128ELb0ELb0EE", 257, 6152, 4104),
    ("gemm_bf16_kernelILi256ELb0ELb0EE", 257, 12296, 2056), ("gemm_bf16_kernelILi256ELb0ELb0EE", 1290, 6152, 520),
    ("gemm_bf16_2cta_kernel", 700, 9224, 1032), ("gemm_bf16_2cta_kernel", 2000, 2056, 8200), ("gemm_bf16_2cta_kernel", 3001, 3000, 264),
    ("gemm_bf16_2cta_kernel", 350, 6464, 8104), ("gemm_bf16_2cta_kernel", 1278, 2384, 3464),  # rows off the 32-byte sectors, which pairs mind least
    ("gemm_bf16_skinny_kernelILi16ELb0ELb0EE", 3, 10816, 4032), ("gemm_bf16_skinny_kernelILi16ELb0ELb0EE", 16, 9601, 2696),
    ("gemm_bf16_split_kernelILi32EE", 17, 9601, 2696), ("gemm_bf16_split_kernelILi32EE", 129, 1000, 1032), ("gemm_bf16_split_kernelILi32EE", 200, 136, 2056),
    ("gemm_bf16_split_kernelILi64EE", 257, 520, 2056), ("gemm_bf16_split_kernelILi64EE", 129, 520, 8200), ("gemm_bf16_split_kernelILi64EE", 999, 1000, 264),
    ("gemm_bf16_split_kernelILi128EE", 700, 2056, 264), ("gemm_bf16_split_kernelILi128EE", 385, 520, 4104), ("gemm_bf16_split_kernelILi128EE", 200, 6152, 520),
    ("gemm_bf16_split_kernelILi192EE", 129, 3000, 4104), ("gemm_bf16_split_kernelILi192EE", 257, 4104, 2056), ("gemm_bf16_split_kernelILi192EE", 1290, 2056, 520),
    ("gemm_bf16_split_kernelILi256EE", 200, 6152, 8200), ("gemm_bf16_split_kernelILi256EE", 1000, 4104, 520),
])
def test_bf16_linears_of_many_rows(ops, kernel, M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    bias = torch.randn(N, generator=g, device="cuda").bfloat16()
    out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    names = kernels(lambda: ops.linear_forward(x, w, bias, out=out))
    assert len(names) == 1 and kernel in names[0], names
    check_product(ops.linear_forward(x, w, bias), x, w, bias)
    assert ops.device_error() == 0


@pytest.mark.parametrize("hidden,vocab", [(520, 1000), (1032, 4104), (4104, 520), (72, 8), (2056, 20008)])
@pytest.mark.parametrize("batch", [9, 16, 17, 32, 33, 64, 65, 100, 128])
def test_bf16_steps_of_9_to_128_rows(ops, hidden, vocab, batch):
    """The decode GEMM with K over a cluster, which only the runners call: the LM head of a step, whose input and output both stay in the workspace."""
    from teenygrad_b200 import qwen3
    cfg = qwen3.Qwen3Config(1, hidden, 2, 1, 128, 64, vocab, tied=False)
    r = qwen3.Qwen3Runner(cfg, max_batch=128, max_len=4, max_tokens=128, max_new_tokens=2)
    tensors = dict(qwen3.random_weights_device(cfg, hidden, r.device))
    r.load_state_dict(tensors)
    ids = torch.arange(batch, device="cuda", dtype=torch.int32)[:, None] % vocab
    tokens = 16 if batch <= 16 else (32 if batch <= 32 else (64 if batch <= 64 else 128))
    names = kernels(lambda: r.prefill(ids))
    assert sum(f"gemm_bf16_skinny_kernelILi{tokens}ELb0ELb0EE" in n for n in names) == 5, names  # four projections and the head
    seen = []
    for graph in (None, False, True):
        r.prefill(ids) if graph is None else r.decode_step(graph=graph)
        x = r._view(qwen3.BUF_HIDDEN, (batch, hidden), torch.bfloat16)
        seen.append(r.logits().clone())
        check_product(seen[-1], x, tensors["lm_head.weight"])
    r.prefill(ids)
    assert torch.equal(r.logits(), seen[0]) and r.device_error() == 0


def padded(M, K, ld, first, seed):
    """[M, K] with row stride `ld`, beginning `first` numbers into its memory; what lies between is NaN.  ld 0: one row M times."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.full((first + M * ld + K,), float("nan"), device="cuda").as_strided((M, K), (ld, 1), first)
    (x if ld else x[0]).copy_(torch.randn(M if ld else 1, K, generator=g, device="cuda").view_as(x if ld else x[0]))
    return x


@pytest.mark.parametrize("kernel,M,N,K,lda,ldb,first", [
    # [N][K]: pairs, tiles of 128, 64 and 32 columns; then copies of four bytes: odd rows, rows that start off 16 bytes, one row M times
    ("gemm_f32_pair_kernelILb0EE", 1290, 4097, 579, 580, 584, 0), ("gemm_f32_tc_kernelILi128ELb0ELb0EE", 300, 1002, 1001, 1004, 1004, 0),
    ("gemm_f32_tc_kernelILi64ELb0ELb0EE", 130, 1000, 2003, 2004, 2008, 4), ("gemm_f32_tc_kernelILi32ELb0ELb0EE", 40, 70, 4001, 4004, 4004, 0),
    ("gemm_f32_tc_kernelILi128ELb0ELb1EE", 600, 1000, 1001, 1001, 1004, 0), ("gemm_f32_tc_kernelILi128ELb0ELb1EE", 1290, 4100, 515, 515, 515, 3),
    ("gemm_f32_tc_kernelILi64ELb0ELb1EE", 300, 300, 2003, 2004, 2004, 1), ("gemm_f32_tc_kernelILi64ELb0ELb1EE", 300, 300, 2003, 0, 2003, 0),
    ("gemm_f32_tc_kernelILi32ELb0ELb1EE", 17, 70, 4001, 4005, 4001, 2), ("gemm_f32_tc_kernelILi32ELb0ELb1EE", 130, 70, 2003, 2003, 2003, 0),
    # few chunks, where a launch's start and end decide; results that are not whole sectors
    ("gemm_f32_tc_kernelILi64ELb1ELb0EE", 3490, 136, 136, 136, 136, 0), ("gemm_simt_kernel", 1325, 801, 88, 88, 88, 0), ("gemm_simt_kernel", 10, 776, 488, 488, 488, 0),
    # [K][N]: ldb is the stride of k
    ("gemm_f32_pair_kernelILb1EE", 1290, 4097, 579, 580, 4100, 0), ("gemm_f32_tc_kernelILi128ELb1ELb0EE", 300, 1002, 1001, 1004, 1004, 0),
    ("gemm_f32_tc_kernelILi64ELb1ELb0EE", 130, 1001, 2003, 2004, 1004, 4),
    ("gemm_f32_tc_kernelILi128ELb1ELb1EE", 600, 1000, 1001, 1001, 1001, 0), ("gemm_f32_tc_kernelILi128ELb1ELb1EE", 1290, 4100, 515, 0, 4101, 3),
    ("gemm_f32_tc_kernelILi64ELb1ELb1EE", 300, 300, 2003, 2003, 301, 1), ("gemm_f32_tc_kernelILi64ELb1ELb1EE", 17, 70, 4001, 4001, 70, 2),
])
def test_f32_linears(ops, kernel, M, N, K, lda, ldb, first):
    kn = "pair_kernelILb1" in kernel or "ELb1ELb" in kernel
    x = padded(M, K, lda, first, K)
    w = padded(K, N, ldb, first, N).T if kn else padded(N, K, ldb, first, N)
    bias = torch.randn(N, device="cuda")
    out = torch.empty(M, N, device="cuda")
    names = kernels(lambda: ops.linear_forward(x, w, bias, out=out))
    assert len(names) == 1 and kernel in names[0], names
    ops.linear_forward(x, w, bias, out=out)
    e, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    # a sum of 64 k is cut off at most 24 times by 2^-23 of the products' sizes, the sums of K / 64 such and of up to eight parts are rounded, and the
    # terms left out are below 3 * 2^-24; f32 multiply-adds in one chain round K times
    assert bool(((out.double() - e - bias.double()).abs() <= max(48 + K // 64 + 12, K if "simt" in kernel else 0) * 2.0 ** -24 * size + 2.0 ** -23 * (e.abs() + bias.double().abs())).all())
    assert ops.device_error() == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,Sq,Skv,D", [(1, 1, 257, 64), (2, 128, 256, 64), (3, 129, 511, 64), (40, 127, 128, 64), (150, 130, 129, 64), (5, 300, 300, 8), (4, 257, 385, 40),
                                        (5, 1, 257, 72), (7, 100, 1000, 120), (2, 128, 320, 128), (3, 255, 191, 128), (149, 64, 128, 128), (6, 260, 260, 64),
                                        (6, 260, 260, 128), (1, 260, 260, 128)])
def test_sizes_of_the_f32_attention_tests(ops, dtype, H, Sq, Skv, D):
    """The sizes that its own tests compare with float64 run in the tensor-core kernel (bf16 with a head size of 128 has another one)."""
    q, k, v = (torch.randn(H, n, D, device="cuda").to(dtype) for n in (Sq, Skv, Skv))
    names = kernels(lambda: ops.flash_attention2_forward(q, k, v, 0.1))
    other = dtype == torch.bfloat16 and D == 128
    assert len(names) == 1 and ("attention_prefill_kernel" if other else "attention_f32_tc_kernel") in names[0], names


@pytest.mark.parametrize("hidden,inter,batch,split", [(1024, 3072, 16, False), (3072, 9216, 12, False), (4096, 12288, 1, True), (4096, 12288, 16, True), (4096, 12288, 17, False),
                                                      (4096, 12288, 128, False), (4096, 9728, 9, True), (4096, 9664, 9, False)])
def test_fp8_down_projection(hidden, inter, batch, split):
    """Up to 16 rows in front of a large weight are split into two FP8 terms; a model with FP8 weights that bf16 holds gives what the bf16 model gives."""
    from teenygrad_b200 import quant, qwen3
    cfg = qwen3.Qwen3Config(1, hidden, 2, 1, 128, inter, 264, tied=False)
    fp8, bf16 = {}, {}
    for name, t in qwen3.random_weights_device(cfg, hidden + inter, "cuda"):
        fp8[name] = bf16[name] = t
        if t.dim() == 2:
            fp8[name], fp8[name + "_scale"] = (t.float() * 2.0 ** 10).to(torch.float8_e4m3fn), torch.full((t.shape[0],), 2.0 ** -10, device="cuda")
            bf16[name] = (fp8[name].float() * 2.0 ** -10).bfloat16()
    ids = torch.arange(batch, device="cuda", dtype=torch.int32)[:, None]
    first, picked, step = [], [], []
    for tensors in (fp8, bf16):
        r = qwen3.Qwen3Runner(cfg, max_batch=batch, max_len=4, max_tokens=128, max_new_tokens=2)
        r.load_quantized(tensors, quant.Fp8Scheme("channel")) if tensors is fp8 else r.load_state_dict(tensors)
        if tensors is fp8:
            assert any("split_e4m3_vec_kernel" in n for n in kernels(lambda: r.prefill(ids))) == split  # noqa: B023
        r.prefill(ids)
        first.append(r.logits().double())
        picked.append(r.next_ids().clone())
        r.decode_step()
        step.append(r.logits().double())
        assert r.device_error() == 0
    same = picked[0] == picked[1]  # (near ties may go to another token, which the step then goes on from)
    assert int(same.sum()) >= 0.9 * batch
    for a, b in (first, [x[same] for x in step]):
        # eight bf16 tensors from the first kernel to the last, each rounded by 2^-9 at most from sums in another order
        assert float((a - b).norm() / b.norm()) < 8 * 2.0 ** -9
