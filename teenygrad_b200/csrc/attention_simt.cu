// Attention with f32 scores, probabilities and sums on the CUDA cores: the f32 entry points, and bf16 problems that the tcgen05
// kernels do not take (head dims other than 128, unaligned views).  Any head_dim <= 256, grouped-query, optionally causal.
//
// Bound: the FP32 pipe, 4 D multiply-adds per query and key.  A CTA of 128 threads owns 16 R query rows of one head and walks the
// keys in tiles of 64; a thread keeps an R x 8 block of scores and an R x (8 DN) block of the output in registers, so an operand
// word read from shared memory feeds R or 8 multiply-adds.  K is transposed on its way into shared memory (key index fastest)
// and the multiply-adds are packed pairs of keys (or of output dimensions), which halves their issue slots.  A row's eight
// threads sit side by side in one warp: the probabilities pass through shared memory behind a __syncwarp, the row maximum takes
// three shuffles, the row sum is only added up at the end.  Two or more CTAs per SM hide each other's tile loads, which hit L2.
// Measured on B200, f32, 32 heads x 1000 x 1000: 279 us at D = 64 (29 TFLOP/s of the pipe's 74), 562 us at D = 128 (error against 64 bits
// 6.0e-7 either way; what the tensor-core kernel does not take goes here); a warp per query row
// with a chain of shuffles and exponentials per key took 6250 us at D = 64 (7.4e-7).
#include <atomic>
#include <cmath>

#include "attention_simt.cuh"

namespace teeny {

namespace {

using namespace attn_simt;

template <typename T, int R, int DN>
__global__ void __launch_bounds__(kThreads)
attention_simt_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, T* __restrict__ o,
                      float* __restrict__ lse, const AttnShape s, const int row_tiles, const bool vec) {
  pdl_wait();
  extern __shared__ __align__(16) float smem[];
  // the longest rows (causal) start first
  const int tile = row_tiles - 1 - static_cast<int>(blockIdx.x % row_tiles);
  const int h = static_cast<int>(blockIdx.x / row_tiles) % s.Hq, b = static_cast<int>(blockIdx.x / row_tiles) / s.Hq;
  attention_tile<T, R, DN, false>(q, k, v, o, lse, s, tile * TileCfg<R, DN>::kRows, h, b, vec, threadIdx.x, smem, 0, 0u);
}

template <typename T, int R, int DN>
int launch(const T* q, const T* k, const T* v, T* o, float* lse, const AttnShape& s, bool vec, cudaStream_t st) {
  using Cfg = TileCfg<R, DN>;
  static std::atomic<unsigned long long> done{0};  // one bit per device; threads may race to set it
  int dev = 0;
  cudaGetDevice(&dev);
  if (Cfg::kSmemBytes > 48 * 1024 && !(dev < 64 && (done.load(std::memory_order_acquire) >> dev) & 1ull)) {
    const cudaError_t e = cudaFuncSetAttribute(attention_simt_kernel<T, R, DN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (dev < 64) done.fetch_or(1ull << dev, std::memory_order_release);
  }
  const int row_tiles = (s.Sq + Cfg::kRows - 1) / Cfg::kRows;
  const long long blocks = static_cast<long long>(row_tiles) * s.Hq * s.B;
  if (blocks > 0x7fffffffLL) return TEENY_ERR_BAD_ARG;
  launch_kernel(attention_simt_kernel<T, R, DN>, dim3(static_cast<unsigned>(blocks)), dim3(kThreads), Cfg::kSmemBytes, st, 1, q, k, v, o,
                lse, s, row_tiles, vec);
  return static_cast<int>(cudaGetLastError());
}

// Estimated time on the CUDA cores with 16 r rows a CTA, head sizes up to 128: a CTA by itself takes what the chain through its tiles
// takes (start, tile, key: measured with one CTA on an SM, 16 to 640 keys), more rows on an SM share its pipes.
double simt_us(bool f32, const AttnShape& s, int r) {
  const bool wide = s.D > 64;
  const double start = f32 ? (wide ? 2.3 : 1.25) : (wide ? 2.0 : 1.0), tile = f32 ? (wide ? 4.55 : 2.6) : (wide ? 6.3 : 3.36),
               key = f32 ? (wide ? 0.053 : 0.032) : (wide ? 0.078 : 0.046);
  const double keys = attention_mean_keys(s), ctas = static_cast<double>(s.B) * s.Hq * ((s.Sq + 16 * r - 1) / (16 * r)), per_sm = ctas / sm_count();
  const double share = (r == 1 ? 0.45 : (r == 2 ? 0.37 : (r == 4 ? 0.26 : 0.22))) * (wide ? 1.25 : 1.0) * ((per_sm > 1.0 ? per_sm : 1.0) * r - 1.0);
  return 1.5 + 1.6e-3 * ctas * r + (1.0 + share) * (start + tile * std::ceil(keys / kTile) + key * keys);
}

}  // namespace

template <typename T>
int attention_generic(const T* q, const T* k, const T* v, T* o, float* lse, const AttnShape& s, cudaStream_t stream) {
  if (!q || !k || !v || !o || s.B <= 0 || s.Hq <= 0 || s.Hkv <= 0 || s.Sq <= 0 || s.Skv <= 0 || s.D <= 0)
    return TEENY_ERR_BAD_ARG;
  if (s.D > 256 || s.Hq % s.Hkv != 0 || (s.causal && s.Skv < s.Sq)) return TEENY_ERR_BAD_ARG;
  const uintptr_t align = 4 * sizeof(T) - 1;
  const long long strides = s.q_sb | s.q_sh | s.q_ss | s.k_sb | s.k_sh | s.k_ss | s.v_sb | s.v_sh | s.v_ss;
  const bool vec = s.D % 4 == 0 && strides % 4 == 0 &&
                   !((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v)) & align);
  // Rows per CTA: as many as the registers hold (more multiply-adds per word read), fewer where the rows would not fill the SMs
  // twice or most of a tile would be padding: 16 heads x 128 rows x 1024 keys, D = 128, takes 136 us with 16-row tiles on 128 SMs.
  const long long bh = static_cast<long long>(s.B) * s.Hq, want = 2LL * sm_count();
  auto fills = [&](int r) { return s.Sq > 8 * r && bh * ((s.Sq + 16 * r - 1) / (16 * r)) >= want; };
  const int most = s.D <= 64 ? 8 : (s.D <= 128 ? 4 : 2);
  int r = most;
  while (r > 1 && !fills(r)) r >>= 1;
  if (attention_f32_tc_takes(q, k, v, s) && attention_f32_tc_us(sizeof(T) == 4, s) < simt_us(sizeof(T) == 4, s, r)) return attention_f32_tc(q, k, v, o, lse, s, stream);
  if (s.D <= 64) {
    if (r == 8) return launch<T, 8, 1>(q, k, v, o, lse, s, vec, stream);
    if (r == 4) return launch<T, 4, 1>(q, k, v, o, lse, s, vec, stream);
    if (r == 2) return launch<T, 2, 1>(q, k, v, o, lse, s, vec, stream);
    return launch<T, 1, 1>(q, k, v, o, lse, s, vec, stream);
  }
  if (s.D <= 128) {
    if (r == 4) return launch<T, 4, 2>(q, k, v, o, lse, s, vec, stream);
    if (r == 2) return launch<T, 2, 2>(q, k, v, o, lse, s, vec, stream);
    return launch<T, 1, 2>(q, k, v, o, lse, s, vec, stream);
  }
  if (r == 2) return launch<T, 2, 4>(q, k, v, o, lse, s, vec, stream);
  return launch<T, 1, 4>(q, k, v, o, lse, s, vec, stream);
}
template int attention_generic<float>(const float*, const float*, const float*, float*, float*, const AttnShape&, cudaStream_t);
template int attention_generic<bf16>(const bf16*, const bf16*, const bf16*, bf16*, float*, const AttnShape&, cudaStream_t);

}  // namespace teeny
