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
// 6.0e-7 either way); a warp per query row
// with a chain of shuffles and exponentials per key took 6250 us at D = 64 (7.4e-7).
#include <atomic>

#include "common.cuh"
#include "kernels.h"

namespace teeny {

namespace {

constexpr int kThreads = 128;
constexpr int kTile = 64;  // keys per tile

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const bf16* p) {
  const uint2 v = *reinterpret_cast<const uint2*>(p);
  return make_float4(bf16_lo(v.x), bf16_hi(v.x), bf16_lo(v.y), bf16_hi(v.y));
}
__device__ __forceinline__ float load1(const float* p) { return *p; }
__device__ __forceinline__ float load1(const bf16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ void store1(float* p, float v) { *p = v; }
__device__ __forceinline__ void store1(bf16* p, float v) { *p = __float2bfloat16_rn(v); }

// Elements [d, d + 4) of a row of D, zero beyond it.  `vec`: every row starts on a 4-element boundary and D % 4 == 0.
template <typename T>
__device__ __forceinline__ float4 row4(const T* row, int d, int D, bool vec) {
  if (vec) return d < D ? load4(row + d) : make_float4(0.f, 0.f, 0.f, 0.f);
  float v[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) v[e] = d + e < D ? load1(row + d + e) : 0.0f;
  return make_float4(v[0], v[1], v[2], v[3]);
}

template <int R, int DN>
struct TileCfg {
  static constexpr int kRows = 16 * R;
  static constexpr int kD = 64 * DN;
  static constexpr int kPCols = R >= 4 ? kRows : 32;  // a key's probabilities: at least eight 16-byte chunks to swizzle over
  static constexpr int kFloats = kD * kRows + 2 * kD * kTile + kTile * kPCols;
  static constexpr int kSmemBytes = kFloats * 4;
};

// R consecutive floats of shared memory (R = 1, 2, 4, 8; the address is a multiple of min(R, 4) floats)
template <int R>
__device__ __forceinline__ void read_rows(float (&v)[R], const float* p) {
  if constexpr (R >= 4) {
#pragma unroll
    for (int i = 0; i < R; i += 4) {
      const float4 t = *reinterpret_cast<const float4*>(p + i);
      v[i] = t.x; v[i + 1] = t.y; v[i + 2] = t.z; v[i + 3] = t.w;
    }
  } else if constexpr (R == 2) {
    const float2 t = *reinterpret_cast<const float2*>(p);
    v[0] = t.x; v[1] = t.y;
  } else {
    v[0] = *p;
  }
}

template <typename T, int R, int DN>
__global__ void __launch_bounds__(kThreads)
attention_simt_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, T* __restrict__ o,
                      float* __restrict__ lse, const AttnShape s, const int row_tiles, const bool vec) {
  using Cfg = TileCfg<R, DN>;
  pdl_wait();
  extern __shared__ __align__(16) float smem[];
  float* qt = smem;                       // [kD][kRows]
  float* kt = qt + Cfg::kD * Cfg::kRows;  // [kD][64]
  float* vs = kt + Cfg::kD * kTile;       // [64][kD]
  float* ps = vs + Cfg::kD * kTile;       // [64][kPCols], the 16-byte chunks of a key's row permuted by the key (see below)
  const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
  // the longest rows (causal) start first
  const int tile = row_tiles - 1 - static_cast<int>(blockIdx.x % row_tiles);
  const int h = static_cast<int>(blockIdx.x / row_tiles) % s.Hq, b = static_cast<int>(blockIdx.x / row_tiles) / s.Hq;
  const int hk = h / (s.Hq / s.Hkv);
  const int row0 = tile * Cfg::kRows;
  const T* qb = q + b * s.q_sb + h * s.q_sh;
  const T* kb = k + b * s.k_sb + hk * s.k_sh;
  const T* vb = v + b * s.v_sb + hk * s.v_sh;

  for (int e = tid; e < Cfg::kRows * (Cfg::kD / 4); e += kThreads) {
    const int r = e % Cfg::kRows, d = e / Cfg::kRows * 4;
    const int i = min(row0 + r, s.Sq - 1);
    const float4 x = row4(qb + static_cast<long long>(i) * s.q_ss, d, s.D, vec);
    qt[d * Cfg::kRows + r] = x.x; qt[(d + 1) * Cfg::kRows + r] = x.y;
    qt[(d + 2) * Cfg::kRows + r] = x.z; qt[(d + 3) * Cfg::kRows + r] = x.w;
  }

  // keys of a thread within a tile: {4 tx + e, 32 + 4 tx + e}; its output dimensions likewise, 8 per 64 of D
  f32x2 acc[R][4 * DN];
  float m[R], l[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    m[r] = -INFINITY;
    l[r] = 0.0f;
#pragma unroll
    for (int j = 0; j < 4 * DN; ++j) acc[r][j] = pack2(0.0f, 0.0f);
  }
  const int shift = s.Skv - s.Sq;
  const int last_row = min(row0 + Cfg::kRows, s.Sq) - 1;
  const int keys = s.causal ? min(s.Skv, last_row + shift + 1) : s.Skv;
  // a chunk of 4 rows of key kk's probabilities lies at (chunk ^ swizzle(kk)): the eight threads of a row write and read
  // eight different bank groups
  auto p_at = [&](int kk, int r) {
    const int chunk = (r >> 2) ^ ((kk >> 2) & 7);
    return ps + kk * Cfg::kPCols + chunk * 4 + (r & 3);
  };

  for (int k0 = 0; k0 < keys; k0 += kTile) {
    __syncthreads();  // the previous tile has been read
    // eight loads in flight per thread
#pragma unroll 1
    for (int e0 = tid; e0 < kTile * (Cfg::kD / 4); e0 += 8 * kThreads) {
      float4 x[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int e = e0 + i * kThreads, kk = e & (kTile - 1), d = e / kTile * 4;
        x[i] = row4(kb + static_cast<long long>(min(k0 + kk, s.Skv - 1)) * s.k_ss, d, s.D, vec);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int e = e0 + i * kThreads, kk = e & (kTile - 1), d = e / kTile * 4;
        float* t = kt + d * kTile + kk;
        t[0] = x[i].x; t[kTile] = x[i].y; t[2 * kTile] = x[i].z; t[3 * kTile] = x[i].w;
      }
    }
#pragma unroll 1
    for (int e0 = tid; e0 < kTile * (Cfg::kD / 4); e0 += 8 * kThreads) {
      float4 x[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int e = e0 + i * kThreads, d = e % (Cfg::kD / 4) * 4, kk = e / (Cfg::kD / 4);
        x[i] = row4(vb + static_cast<long long>(min(k0 + kk, s.Skv - 1)) * s.v_ss, d, s.D, vec);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int e = e0 + i * kThreads, d = e % (Cfg::kD / 4) * 4, kk = e / (Cfg::kD / 4);
        *reinterpret_cast<float4*>(vs + kk * Cfg::kD + d) = x[i];
      }
    }
    __syncthreads();

    f32x2 sc[R][4];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int j = 0; j < 4; ++j) sc[r][j] = pack2(0.0f, 0.0f);
    // 32 dimensions at a time: a shorter chain of roundings than the whole head
#pragma unroll 1
    for (int d0 = 0; d0 < Cfg::kD; d0 += 32) {
      f32x2 part[R][4];
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int j = 0; j < 4; ++j) part[r][j] = pack2(0.0f, 0.0f);
#pragma unroll 4
      for (int d = d0; d < d0 + 32; ++d) {
        float a[R];
        read_rows<R>(a, qt + d * Cfg::kRows + ty * R);
        const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(kt + d * kTile + 4 * tx);
        const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(kt + d * kTile + 32 + 4 * tx);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const f32x2 aa = pack2(a[r], a[r]);
          part[r][0] = fma2(aa, b0.x, part[r][0]);
          part[r][1] = fma2(aa, b0.y, part[r][1]);
          part[r][2] = fma2(aa, b1.x, part[r][2]);
          part[r][3] = fma2(aa, b1.y, part[r][3]);
        }
      }
      const f32x2 one = pack2(1.0f, 1.0f);
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int j = 0; j < 4; ++j) sc[r][j] = fma2(part[r][j], one, sc[r][j]);
    }

    const bool edge = k0 + kTile > s.Skv || (s.causal && k0 + kTile - 1 > row0 + shift);
    float p[R][8];
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 t = unpack2(sc[r][j]);
        p[r][2 * j] = t.x * s.scale;
        p[r][2 * j + 1] = t.y * s.scale;
      }
      if (edge) {
        const int last = s.causal ? min(s.Skv - 1, row0 + ty * R + r + shift) : s.Skv - 1;
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (k0 + (j >> 2) * 32 + 4 * tx + (j & 3) > last) p[r][j] = -INFINITY;
      }
      float top = p[r][0];
#pragma unroll
      for (int j = 1; j < 8; ++j) top = fmaxf(top, p[r][j]);
#pragma unroll
      for (int off = 4; off > 0; off >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, off));
      const float m_new = fmaxf(m[r], top);
      const float corr = expf(m[r] - m_new);
      m[r] = m_new;
      float sum = 0.0f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        p[r][j] = expf(p[r][j] - m_new);
        sum += p[r][j];
      }
      l[r] = corr * l[r] + sum;
      const f32x2 cc = pack2(corr, corr);
#pragma unroll
      for (int j = 0; j < 4 * DN; ++j) acc[r][j] = mul2(acc[r][j], cc);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int kk = (j >> 2) * 32 + 4 * tx + (j & 3);
      if constexpr (R >= 4) {
#pragma unroll
        for (int r = 0; r < R; r += 4)
          *reinterpret_cast<float4*>(p_at(kk, ty * R + r)) = make_float4(p[r][j], p[r + 1][j], p[r + 2][j], p[r + 3][j]);
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) *p_at(kk, ty * R + r) = p[r][j];
      }
    }
    __syncwarp();

    auto probabilities = [&](int kk, float (&a)[R]) {
      if constexpr (R == 8) {
        float a0[4], a1[4];
        read_rows<4>(a0, p_at(kk, ty * R));
        read_rows<4>(a1, p_at(kk, ty * R + 4));
#pragma unroll
        for (int r = 0; r < 4; ++r) { a[r] = a0[r]; a[r + 4] = a1[r]; }
      } else {
        read_rows<R>(a, p_at(kk, ty * R));
      }
    };
    const int live = min(kTile, keys - k0);
    if (s.causal && edge) {
      // a row's sums end at its own last key: 0 times a NaN or an infinity beyond it would spoil them
#pragma unroll 1
      for (int kk = 0; kk < live; ++kk) {
        float a[R];
        probabilities(kk, a);
#pragma unroll
        for (int j = 0; j < 2 * DN; ++j) {
          const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(vs + kk * Cfg::kD + j * 32 + 4 * tx);
#pragma unroll
          for (int r = 0; r < R; ++r) {
            if (k0 + kk > row0 + ty * R + r + shift) continue;
            const f32x2 aa = pack2(a[r], a[r]);
            acc[r][2 * j] = fma2(aa, x.x, acc[r][2 * j]);
            acc[r][2 * j + 1] = fma2(aa, x.y, acc[r][2 * j + 1]);
          }
        }
      }
      continue;
    }
#pragma unroll 4
    for (int kk = 0; kk < live; ++kk) {
      float a[R];
      probabilities(kk, a);
#pragma unroll
      for (int j = 0; j < 2 * DN; ++j) {
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(vs + kk * Cfg::kD + j * 32 + 4 * tx);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const f32x2 aa = pack2(a[r], a[r]);
          acc[r][2 * j] = fma2(aa, x.x, acc[r][2 * j]);
          acc[r][2 * j + 1] = fma2(aa, x.y, acc[r][2 * j + 1]);
        }
      }
    }
  }

#pragma unroll
  for (int r = 0; r < R; ++r) {
    float sum = l[r];
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    const int i = row0 + ty * R + r;
    if (i >= s.Sq) continue;
    T* orow = o + b * s.o_sb + h * s.o_sh + static_cast<long long>(i) * s.o_ss;
#pragma unroll
    for (int j = 0; j < 2 * DN; ++j) {
      const float2 lo = unpack2(acc[r][2 * j]), hi = unpack2(acc[r][2 * j + 1]);
      const float x[4] = {lo.x / sum, lo.y / sum, hi.x / sum, hi.y / sum};
      const int d = j * 32 + 4 * tx;
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (d + e < s.D) store1(orow + d + e, x[e]);
    }
    if (lse && tx == 0) lse[(static_cast<long long>(b) * s.Hq + h) * s.Sq + i] = m[r] + logf(sum);
  }
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
  if (s.D <= 64) {
    if (fills(8)) return launch<T, 8, 1>(q, k, v, o, lse, s, vec, stream);
    if (fills(4)) return launch<T, 4, 1>(q, k, v, o, lse, s, vec, stream);
    if (fills(2)) return launch<T, 2, 1>(q, k, v, o, lse, s, vec, stream);
    return launch<T, 1, 1>(q, k, v, o, lse, s, vec, stream);
  }
  if (s.D <= 128) {
    if (fills(4)) return launch<T, 4, 2>(q, k, v, o, lse, s, vec, stream);
    if (fills(2)) return launch<T, 2, 2>(q, k, v, o, lse, s, vec, stream);
    return launch<T, 1, 2>(q, k, v, o, lse, s, vec, stream);
  }
  if (fills(2)) return launch<T, 2, 4>(q, k, v, o, lse, s, vec, stream);
  return launch<T, 1, 4>(q, k, v, o, lse, s, vec, stream);
}
template int attention_generic<float>(const float*, const float*, const float*, float*, float*, const AttnShape&, cudaStream_t);
template int attention_generic<bf16>(const bf16*, const bf16*, const bf16*, bf16*, float*, const AttnShape&, cudaStream_t);

}  // namespace teeny
