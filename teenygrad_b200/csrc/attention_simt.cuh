// The tile of the CUDA-core attention (attention_simt.cu), shared with the tensor-core kernel (attention_f32_tc.cu), which makes rows
// with results that are not finite again with it.
#pragma once

#include "common.cuh"
#include "kernels.h"

namespace teeny {

namespace attn_simt {

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

// One tile of 16 R query rows from `row0` on, head h of batch entry b, by 128 threads that meet at barrier `bar`.  MASKED: only rows whose bit
// in `rows` (counted from row0) is set are stored.
template <typename T, int R, int DN, bool MASKED>
__device__ __forceinline__ void attention_tile(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, T* __restrict__ o,
                                               float* __restrict__ lse, const AttnShape& s, const int row0, const int h, const int b,
                                               const bool vec, const int tid, float* smem, const int bar, const unsigned rows) {
  using Cfg = TileCfg<R, DN>;
  float* qt = smem;                       // [kD][kRows]
  float* kt = qt + Cfg::kD * Cfg::kRows;  // [kD][64]
  float* vs = kt + Cfg::kD * kTile;       // [64][kD]
  float* ps = vs + Cfg::kD * kTile;       // [64][kPCols], the 16-byte chunks of a key's row permuted by the key (see below)
  const int tx = tid & 7, ty = tid >> 3;
  const int hk = h / (s.Hq / s.Hkv);
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
    named_barrier_sync(bar, kThreads);  // the previous tile has been read
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
    named_barrier_sync(bar, kThreads);

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
    if (i >= s.Sq || (MASKED && !((rows >> (ty * R + r)) & 1u))) continue;
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

}  // namespace attn_simt

}  // namespace teeny
