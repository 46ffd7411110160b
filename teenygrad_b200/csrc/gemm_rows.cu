// Linear layers of a decode step with few sequences on a small model: y[M, N] = f(x)[M, K] W[N, K]^T, M <= 8 (16 as an operator).
//
// What bounds these calls is the way from one kernel to the next, not the bytes: at M = 1 a layer of a 1024-wide model has 31 MB of
// weights, 5 us at HBM rate, and its seven kernels took 33 us.  So the kernel is built for a short chain:
//   * the weights of a CTA (all of them: at most kMaxSmem) are requested by bulk copies at its very start, before the wait for
//     the kernel in front, so that only the activations are left to fetch when that has ended (weights that the kernel in front may
//     have computed are asked into L2 instead, and copied behind the wait);
//   * what stood between two GEMMs is part of them: the RMSNorm of the input rows in front (every CTA norms the few rows for
//     itself), bias, gated linear unit or the addition into the residual stream behind;
//   * little code: a short rolled loop of mma.m16n8k16 with the tokens as the 16-row A operand and 8 weight rows as B; no tensor
//     memory, no tensor maps, no cluster reduction.
// Measured (graph of back-to-back calls, weights from HBM, M = 1, against the 128-row kernel with its cluster reduction): 1024 x 1024
// 5.5 -> 3.0 us, 1024 x 3072 6.5 -> 4.0, 4096 x 1024 6.5 -> 4.3, 6144 x 1024 7.5 -> 5.2; weights read behind the wait, as an operator
// does it, 3.0, 4.0, 4.7, 5.5, and at M = 16 5.6 -> 4.6, 6.7 -> 6.7, 6.6 -> 6.5, 7.8 -> 7.3.  Decode step of a 28-layer, 1024-wide model at batch 1: 944 -> 663 us; of a 24-layer recurrent hybrid at batch 4 1010 ->
// 805.  A first version that kept the weights in registers (16 loads of a thread in flight, loops unrolled to match) took 822 us:
// its code was five times as long, and every launch fetches it anew.
// The eight warps of a CTA share the K range (64 k each in turn) and add their sums through shared memory.  Unit = 8 weight rows
// (gated: 4 gate rows and the 4 up rows of the same channels); a CTA takes UPC of them, which share the activation fragments.
// Within a 64-k block lane c of a quad holds k 8c .. 8c+7 and 32 + 8c .. of its row (FP8: k 16c .. 16c+15), and MMA j takes the
// lane's elements 4j .. 4j+3; A is read with the same numbering, so any order of k gives the same sum.
#include <atomic>

#include "common.cuh"
#include "kernels.h"
#include "mma.cuh"

namespace teeny {

namespace {

constexpr int kThreads = 256, kWarps = 8;
constexpr int kMaxSmem = 108 << 10;  // two CTAs (of neighbouring kernels) share an SM

// Bytes from one row to the next in shared memory.  Eight lanes of a 16-byte fragment load are two rows of four lanes, 16 bytes
// apart (activations beside FP8 weights: 32 bytes), so the rows lie 64 (16) bytes apart modulo the 128 bytes of all banks.
__host__ __device__ constexpr int x_pitch(int K, bool w8) { return (K + 63) / 64 * 128 + (w8 ? 16 : 64); }
__host__ __device__ constexpr int w_pitch(int K, bool w8) { return w8 ? (K + 127) / 128 * 128 + 64 : (K + 63) / 64 * 128 + 64; }
// f32 partial sums [warp][token][weight row]: token rows 8 mod 32 words apart, so that a quarter of a warp's stores hits all banks
__host__ __device__ constexpr int part_pitch(int upc) { return upc * 8 + (upc % 2 ? 0 : 8); }
__host__ __device__ constexpr int weight_bytes(int upc, int K, bool w8, bool two) {
  const int w = upc * 8 * w_pitch(K, w8), p = kWarps * (two ? 16 : 8) * part_pitch(upc) * 4;  // the sums reuse the weights' place
  return w > p ? w : p;
}

size_t smem_bytes(int upc, int M, int K, bool w8, int norm) {
  size_t n = static_cast<size_t>(weight_bytes(upc, K, w8, M > 8)) + static_cast<size_t>(M) * x_pitch(K, w8);
  if (norm == kRowsNormBf16) n += static_cast<size_t>(K) * 2;
  if (norm == kRowsNormF32) n += static_cast<size_t>(K) * 4 * (M + 1);
  return n;
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               :: "r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

// UPC: units of a CTA.  TWO: more than 8 tokens (the upper half of the A operand is used).  W8: FP8 E4M3 weight bytes.
template <int UPC, bool TWO, bool W8>
__global__ void __launch_bounds__(kThreads, 3) gemm_rows_kernel(const __grid_constant__ RowsGemm g, int* err) {
  constexpr int kEs = W8 ? 1 : 2;
  constexpr int kSecond = W8 ? 16 : 64;  // bytes between a lane's two activation vectors of a block
  constexpr int kTok = TWO ? 16 : 8;
  constexpr int kChains = UPC == 1 ? 4 : (UPC == 2 ? 2 : 1);  // independent sums per unit: few units, short chains of MMAs
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ float red[kWarps];
  __shared__ __align__(8) uint64_t bar_mem;
  const int pitch = x_pitch(g.K, W8), wp = w_pitch(g.K, W8);
  uint8_t* xs = smem + weight_bytes(UPC, g.K, W8, TWO);  // [M][pitch]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = lane >> 2, c = lane & 3;
  const int unit0 = blockIdx.x * UPC;
  const uint32_t bar = smem_u32(&bar_mem);

  // weight row of row lr of this CTA
  auto w_row = [&](int lr) {
    if (!g.glu) return unit0 * 8 + lr;
    const int ch = (unit0 + (lr >> 3)) * 4 + (lr & 3);
    return (ch >> 6) * 128 + (ch & 63) + ((lr >> 2) & 1) * 64;
  };
  if (warp == 0) {
    static_assert(UPC * 8 <= 32, "a lane per row");
    const int n = w_row(lane);
    const bool mine = lane < UPC * 8 && n < g.N;
    const unsigned rows = __popc(__ballot_sync(0xffffffffu, mine));
    if (lane == 0) {
      mbar_init(bar, 1);
      mbar_fence_init();
      mbar_expect_tx(bar, rows * g.K * kEs);
    }
    __syncwarp();
    const uint8_t* src = static_cast<const uint8_t*>(g.w) + static_cast<size_t>(n) * g.ldw * kEs;
    if (!g.w_early) {
      if (mine) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" :: "l"(src), "r"(g.K * kEs) : "memory");
      pdl_wait();
    }
    if (mine) bulk_load(smem_u32(smem) + lane * wp, src, g.K * kEs, bar);
  }
  // columns behind K up to a whole block: zeros on both sides
  if (g.K & 63) {
    const int from = g.K * kEs / 16, tail = (g.K + 63) / 64 * 64 * kEs / 16 - from;
    for (int i = tid; i < UPC * 8 * tail; i += kThreads) *reinterpret_cast<uint4*>(smem + i / tail * wp + (from + i % tail) * 16) = make_uint4(0u, 0u, 0u, 0u);
  }

  // ---- the input rows into shared memory, normed where asked for; `tpr` threads share a row ----
  int lg = 8;
  for (int m = 1; m < g.M; m <<= 1) --lg;
  const int tpr = 1 << lg, row = tid >> lg, at = tid & (tpr - 1);
  const bool has_row = row < g.M;
  const int nv8 = g.K >> 3;
  // The next kernel may come in as soon as this one's input is there, under its products: 570 us a step against 681 behind the products
  // (28 layers, batch 1).  With few k there is nothing to hide, and its CTAs only come in between (4096-wide recurrent hybrid, batch
  // 1, four calls of K = 128 a step: 890 us early, 868 late).
  const bool early = g.K >= 256;
  if (has_row)
    for (int i = nv8 + at; i < (g.K + 63) / 64 * 8; i += tpr) *reinterpret_cast<uint4*>(xs + row * pitch + i * 16) = make_uint4(0u, 0u, 0u, 0u);
  if (g.norm == kRowsNormNone) {
    pdl_wait();
    if (early) pdl_trigger();
    if (has_row) {
      const uint4* src = reinterpret_cast<const uint4*>(static_cast<const bf16*>(g.x) + static_cast<size_t>(row) * g.ldx);
#pragma unroll 4
      for (int i = at; i < nv8; i += tpr) *reinterpret_cast<uint4*>(xs + row * pitch + i * 16) = __ldcg(src + i);
    }
  } else {
    // the norm's weights wait in shared memory (they come from HBM, in the shadow of the kernel in front), the raw rows where
    // the normed ones will be (f32 rows: behind everything else), so that no registers are held beside the weights in flight
    const bool f32 = g.norm == kRowsNormF32;
    const int nv = f32 ? g.K >> 2 : nv8;  // 16-byte vectors of a row
    uint4* ws = reinterpret_cast<uint4*>(xs + g.M * pitch);
    uint4* stage = f32 ? ws + nv + row * nv : reinterpret_cast<uint4*>(xs + row * pitch);
    for (int i = tid; i < nv; i += kThreads) ws[i] = __ldg(static_cast<const uint4*>(g.norm_w) + i);
    pdl_wait();
    if (early) pdl_trigger();
    float sq = 0.0f;
    if (has_row) {
      const uint4* src = reinterpret_cast<const uint4*>(static_cast<const uint8_t*>(g.x) + static_cast<size_t>(row) * g.ldx * (f32 ? 4 : 2));
#pragma unroll 4
      for (int i = at; i < nv; i += tpr) {
        const uint4 v = __ldcg(src + i);
        stage[i] = v;
        const uint32_t e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (f32) sq = fmaf(__uint_as_float(e[j]), __uint_as_float(e[j]), sq);
          else sq = fmaf(bf16_lo(e[j]), bf16_lo(e[j]), fmaf(bf16_hi(e[j]), bf16_hi(e[j]), sq));
        }
      }
    }
    for (int o = (tpr < 32 ? tpr : 32) >> 1; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if (lane == 0) red[warp] = sq;
    __syncthreads();  // (the norm's weights are there, too)
    if (tpr > 32) {
      sq = 0.0f;
      for (int i = 0; i < tpr / 32; ++i) sq += red[row * (tpr / 32) + i];
    }
    const float rr = 1.0f / sqrtf(sq / static_cast<float>(g.K) + g.eps);
    if (has_row)
      for (int i = at; i < nv; i += tpr) {
        const uint4 v = stage[i], w = ws[i];
        const uint32_t e[4] = {v.x, v.y, v.z, v.w}, q[4] = {w.x, w.y, w.z, w.w};
        if (f32) {
          float o[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) o[j] = __uint_as_float(e[j]) * rr * __uint_as_float(q[j]);
          *reinterpret_cast<uint2*>(xs + row * pitch + i * 8) = make_uint2(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]));
        } else {
          uint32_t o[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            o[j] = pack_bf16x2(bf16_round(bf16_lo(e[j]) * rr) * bf16_lo(q[j]), bf16_round(bf16_hi(e[j]) * rr) * bf16_hi(q[j]));
          stage[i] = make_uint4(o[0], o[1], o[2], o[3]);
        }
      }
  }

  // Outputs: (token, unit, weight row of the unit or channel), the last fastest.  The residual value of this thread's first output
  // is requested now: its way from L2 would be the last wait of the kernel.
  const int lg_unit = g.glu ? 2 : 3, per_tok = UPC << lg_unit, n_out = g.glu ? g.N >> 1 : g.N, n0 = unit0 << lg_unit;
  float res0 = 0.0f;
  if (g.add32 || g.add16) {
    const int m = tid / per_tok, n = n0 + tid - m * per_tok;
    if (m < g.M && n < n_out) {
      const size_t off = static_cast<size_t>(m) * g.ldy + n;
      res0 = g.add32 ? __ldcg(g.add32 + off)
                     : __uint_as_float(static_cast<uint32_t>(__ldcg(reinterpret_cast<const unsigned short*>(g.add16) + off)) << 16);
    }
  }
  __syncthreads();
  TRACE_MARK(1, tid == 0);  // activations are there

  const uint8_t* xa = xs + (r < g.M ? r : g.M - 1) * pitch + c * (W8 ? 32 : 16);
  const uint8_t* xb = xs + (r + 8 < g.M ? r + 8 : g.M - 1) * pitch + c * (W8 ? 32 : 16);
  const uint8_t* wa = smem + r * wp + c * 16;
  float acc[UPC][kChains][4] = {};
  const int kb_count = (g.K + 63) >> 6;
  const bool ok = mbar_wait(bar, 0, err, DEVERR_GEMM_ROWS);
  TRACE_MARK(2, tid == 0);  // weights are there
  if (ok) {
#pragma unroll 1
    for (int kb = warp; kb < kb_count; kb += kWarps) {
      const uint4 q0 = *reinterpret_cast<const uint4*>(xa + kb * 128), q1 = *reinterpret_cast<const uint4*>(xa + kb * 128 + kSecond);
      uint4 p0 = make_uint4(0u, 0u, 0u, 0u), p1 = p0;
      if (TWO) { p0 = *reinterpret_cast<const uint4*>(xb + kb * 128); p1 = *reinterpret_cast<const uint4*>(xb + kb * 128 + kSecond); }
#pragma unroll
      for (int u = 0; u < UPC; ++u) {
        const uint8_t* src = wa + u * 8 * wp + kb * 64 * kEs;
        uint32_t w[8];
        const uint4 t0 = *reinterpret_cast<const uint4*>(src);
        if constexpr (W8) {
          e4m3x4_to_bf16x4(t0.x, g.w_mul16, w[0], w[1]);
          e4m3x4_to_bf16x4(t0.y, g.w_mul16, w[2], w[3]);
          e4m3x4_to_bf16x4(t0.z, g.w_mul16, w[4], w[5]);
          e4m3x4_to_bf16x4(t0.w, g.w_mul16, w[6], w[7]);
        } else {
          const uint4 t1 = *reinterpret_cast<const uint4*>(src + 64);
          w[0] = t0.x; w[1] = t0.y; w[2] = t0.z; w[3] = t0.w;
          w[4] = t1.x; w[5] = t1.y; w[6] = t1.z; w[7] = t1.w;
        }
        mma_bf16_16816(acc[u][0], q0.x, p0.x, q0.y, p0.y, w[0], w[1]);
        mma_bf16_16816(acc[u][1 % kChains], q0.z, p0.z, q0.w, p0.w, w[2], w[3]);
        mma_bf16_16816(acc[u][2 % kChains], q1.x, p1.x, q1.y, p1.y, w[4], w[5]);
        mma_bf16_16816(acc[u][3 % kChains], q1.z, p1.z, q1.w, p1.w, w[6], w[7]);
      }
    }
  }
  if (!ok) {  // a wait gave up: let the copies that may still be in flight land before their memory is used again
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
  if (!early) pdl_trigger();
  __syncthreads();  // everyone is done with the weights: the sums take their place
  float* part = reinterpret_cast<float*>(smem);
  constexpr int kPp = part_pitch(UPC);
  // C fragment: [0..1] = (token r, weight rows 2c, 2c + 1), [2..3] = token r + 8
#pragma unroll
  for (int u = 0; u < UPC; ++u) {
#pragma unroll
    for (int ch = 1; ch < kChains; ++ch)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[u][0][e] += acc[u][ch][e];
    float* p = part + (warp * kTok + r) * kPp + u * 8 + 2 * c;
    *reinterpret_cast<float2*>(p) = make_float2(acc[u][0][0], acc[u][0][1]);
    if (TWO) *reinterpret_cast<float2*>(p + 8 * kPp) = make_float2(acc[u][0][2], acc[u][0][3]);
  }
  __syncthreads();
  TRACE_MARK(3, tid == 0);  // all warps' sums are there
  for (int idx = tid; idx < per_tok * g.M; idx += kThreads) {
    const int m = idx / per_tok, o = idx - m * per_tok, n = n0 + o;
    if (n >= n_out) continue;
    const float* p = part + m * kPp + (g.glu ? (o >> 2) * 8 + (o & 3) : o);
    float v = 0.0f, up = 0.0f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      v += p[w * kTok * kPp];
      if (g.glu) up += p[w * kTok * kPp + 4];
    }
    if constexpr (W8) {
      const int wn = g.glu ? (n >> 6) * 128 + (n & 63) : n;
      v *= __ldg(g.w_scale + (g.w_scale_kind ? wn : 0));
      if (g.glu) up *= __ldg(g.w_scale + (g.w_scale_kind ? wn + 64 : 0));
    }
    if (g.glu) v = glu_f(g.glu, v, up);
    else if (g.bias) v += __bfloat162float(g.bias[n]);
    const size_t off = static_cast<size_t>(m) * g.ldy + n;
    if (g.add32) {  // the sublayer's output is a bf16 tensor before it joins the f32 residual stream
      g.add32[off] = (idx == tid ? res0 : g.add32[off]) + bf16_round(v);
    } else if (g.add16) {
      g.add16[off] = __float2bfloat16_rn((idx == tid ? res0 : __bfloat162float(g.add16[off])) + bf16_round(v));
    } else {
      g.y[off] = __float2bfloat16_rn(v);
    }
  }
  TRACE_END();
}

template <int UPC, bool TWO, bool W8>
int prepare_rows() {
  static std::atomic<unsigned long long> done{0};  // one bit per device; threads may race to set it
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && (done.load(std::memory_order_acquire) >> dev) & 1ull) return 0;
  const cudaError_t e = cudaFuncSetAttribute(gemm_rows_kernel<UPC, TWO, W8>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
  if (e != cudaSuccess) return static_cast<int>(e);
  if (dev < 64) done.fetch_or(1ull << dev, std::memory_order_release);
  return 0;
}

template <int UPC, bool TWO, bool W8>
int launch_rows(const RowsGemm& g, int units, int* err, cudaStream_t st) {
  const int rc = prepare_rows<UPC, TWO, W8>();
  if (rc) return rc;
  return launch_kernel(gemm_rows_kernel<UPC, TWO, W8>, dim3((units + UPC - 1) / UPC), dim3(kThreads), smem_bytes(UPC, g.M, g.K, W8, g.norm), st, 1,
                       g, err);
}

template <bool TWO, bool W8>
int launch_rows_upc(const RowsGemm& g, int upc, int units, int* err, cudaStream_t st) {
  if (upc == 1) return launch_rows<1, TWO, W8>(g, units, err, st);
  if (upc == 2) return launch_rows<2, TWO, W8>(g, units, err, st);
  return launch_rows<4, TWO, W8>(g, units, err, st);
}

// Units of a CTA: as many as give every SM one CTA or a little more.
int rows_upc(int N) {
  const int units = (N + 7) / 8, sms = sm_count();
  return units <= sms ? 1 : (units <= 2 * sms ? 2 : 4);
}

}  // namespace

bool gemm_rows_takes(int M, int N, int K, int ldw, bool w8, int norm) {
  if (M < 1 || M > (w8 ? kRowsStepM : kRowsMaxM) || N < 1 || K < 8 || K % (w8 ? 16 : 8) || ldw % (w8 ? 16 : 8)) return false;
  // All weights at once in the shared memory of the GPU, half of it left for the kernel behind: about 14 MB.  Beyond that a call
  // lasts long enough for HBM to bound it, and the 128-row kernel's ring streams better (24576 x 4096 at M = 1: 35.9 us there, 46.1 in
  // a variant of this kernel with several passes).
  const int upc = rows_upc(N);
  if (static_cast<long long>(N) * w_pitch(K, w8) > static_cast<long long>(kMaxSmem) * sm_count()) return false;
  return smem_bytes(upc, M, K, w8, norm) <= kMaxSmem;
}

int gemm_rows_prepare() {
  int rc = 0;
  if ((rc = prepare_rows<1, false, false>()) || (rc = prepare_rows<2, false, false>()) || (rc = prepare_rows<4, false, false>()) ||
      (rc = prepare_rows<1, true, false>()) || (rc = prepare_rows<2, true, false>()) || (rc = prepare_rows<4, true, false>()) ||
      (rc = prepare_rows<1, false, true>()) || (rc = prepare_rows<2, false, true>()) || (rc = prepare_rows<4, false, true>()))
    return rc;
  return 0;
}

int gemm_rows(const RowsGemm& in, cudaStream_t st) {
  RowsGemm g = in;
  const bool two = g.M > 8, w8 = g.w_scale != nullptr;
  if (!g.x || !g.w || !(g.y || g.add16 || g.add32) || !gemm_rows_takes(g.M, g.N, g.K, g.ldw, w8, g.norm)) return TEENY_ERR_BAD_ARG;
  if (g.norm != kRowsNormNone && (!g.norm_w || !g.w_early)) return TEENY_ERR_BAD_ARG;  // norm_w is always read ahead of the wait
  if (g.glu && (g.bias || g.add16 || g.add32 || g.N % 128)) return TEENY_ERR_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(g.x) | reinterpret_cast<uintptr_t>(g.w) | reinterpret_cast<uintptr_t>(g.norm_w)) & 15 || g.ldx % 8) return TEENY_ERR_ALIGNMENT;
  g.w_mul16 = 16u;
  int* err = device_error_word();
  if (!err) return TEENY_ERR_DRIVER;
  const int units = (g.N + 7) / 8, upc = rows_upc(g.N);
  if (two) return launch_rows_upc<true, false>(g, upc, units, err, st);
  return w8 ? launch_rows_upc<false, true>(g, upc, units, err, st) : launch_rows_upc<false, false>(g, upc, units, err, st);
}

}  // namespace teeny
