// f32 GEMM on the tensor cores with the accuracy of f32 multiply-adds: C[M, N] = A[M, K] B (+ bias), B as [N, K] or [K, N].
//
// An f32 number is the sum of three bf16 numbers, x = hi + mid + lo (8 + 8 + 8 bits, each the rounded rest of the one before), so a
// product is nine bf16 products, all exact in f32; the six largest are taken, the other three are below 2^-24 of the product.  What
// would lose accuracy is the tensor core's accumulator, which cuts off instead of rounding: after 1024 k the result would be off by
// 1e-6.  So the sum stays in it for 64 k only (smallest products first) and is then added to f32 registers, rounded.
//
// The split runs beside the products: the f32 numbers come by TMA, warps 0-7 split them and store the terms of A in tensor memory (the MMA
// reads A from there) and those of B as swizzled tiles (two stages of each), warps 8-15 move finished 64-k sums from
// tensor memory (two accumulators) into registers; warp 8 issues the MMAs of a chunk before it turns to the sums of the chunk before.
// Bound: for 64 k of a 128 x 128 tile the tensor pipe takes 1536 clocks (24 MMAs of 64) and the splitting warps 2170, which is the latency of a chunk's way
// through them as much as their 900 instructions; 2680 were measured.  With A's terms in shared memory too and f32 rows loaded by the
// splitting warps 3100: 3300 clocks of shared memory.  So large products are made by pairs of CTAs, 256 x 256, where a CTA splits as much for twice
// the products: 3260 clocks against 3072 of the tensor pipe.
// Tried: the splitting warps in two teams of four, each every other chunk, to hide the latency: 64 k of 128, 64 and 32 columns 2400, 1540 and 1200 clocks instead
// of 2680, 1670 and 1560, but a launch's first chunk later, 1000 x 4096 x 1024 40.6 us for 38.2, 512^3 9.3 for 8.8.  Two terms of B as one MMA of
// twice the columns in narrow tiles: no faster, errors up to 15 % larger.
// Measured back to back (f32 rows split by the warps that loaded them, one CTA to a tile -> now): 1000 x 4096 x 1024 63 -> 39 us (with bias called alone 74 -> 50),
// 2048 x 4096 x 4096 478 -> 273, 2048 x 2048 x 2048 [K][N] 123 -> 72, 594 x 780 x 652 25 -> 13.3, 300 x 700 x 2000 16.8 -> 15.1, 512^3 9.6 -> 8.8; error against 64 bits the
// same or smaller (8e-8 to 1.3e-7; f32 multiply-adds 1.2e-6 for 2048 x 4096 x 4096).  Tensor pipe 92 % active with 128 tiles on 74 pairs.  The pairs' kernel spills
// 112 bytes a thread (stored; 284 loaded) with B as [N][K], 56 (96) with [K][N]: their roles have 80 and 176 registers.
//
// bf16 has the exponents of f32 but only eight bits, so the terms of a small number would run out of exponent: the third below 2^-110, all
// three below 2^-134.  Both operands are therefore taken times 2^24, with which every term of every f32 number, the smallest subnormal
// included, is a normal bf16 number or zero, and the sums leave tensor memory times 2^-48.  What that costs is at the other end: from
// 2^104 on an operand, and from 2^80 on a sum, may overflow, infinities and NaNs split into NaNs, and the sums of a tile with results that
// are not finite are made again for these, with f32 multiply-adds (every result infinite: 2048 x 4096 x 4096 2.9 ms, 512^3 34 us).
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace teeny {

namespace {

constexpr int kBM = 128, kBK = 64;
constexpr int kSplitWarps = 8, kSumWarps = 8, kSplit = 32 * kSplitWarps;
constexpr int kThreads = kSplit + 32 * kSumWarps;  // 16 warps: 128 registers each (two more, for the loads and the MMAs: 96)
constexpr int kPairSplitRegs = 80, kPairSumRegs = 176;  // of a pair's 16 warps, 128 at launch
constexpr float kUp = 0x1p24f, kDown = 0x1p-48f;  // of the operands, of the sums
constexpr int kTermColumns = kBK / 2, kTmemA = 256;  // tensor memory columns of a bf16 term of 64 k of A (two k each); where they begin
template <int BN> struct Cfg {
  static constexpr int kBoxA = kBM * 128, kRawA = 2 * kBoxA, kRaw = kRawA + BN * kBK * 4;  // f32 numbers of 64 k: boxes of 128-byte rows
  static constexpr int kTermB = BN * 128, kTerms = 3 * kTermB;                              // bf16 terms of B
  static constexpr int kRawStages = BN == 128 ? 2 : (BN == 64 ? 3 : 4);  // what there is room for: the loads' latency is what narrow tiles wait for
  static constexpr int kStages = kRawStages * kRaw + 2 * kTerms;
  static constexpr int kSmem = kStages + 1024 + 256;
  static_assert(2 * BN <= kTmemA && kTmemA + 6 * kTermColumns <= 512, "two accumulators, two times three terms of A");
  static constexpr int kPitch = BN + 4;             // floats of a row of sums in shared memory (split K)
  static constexpr int kPart = kBM * kPitch * 4;
  static_assert(2 * kPart <= kStages, "a CTA's sums, and behind them those that the others send, in the place of the stages");
};

struct F32Args {
  const float *a, *b, *bias;
  float* c;
  long long lda, ldb;  // row strides: A [M][K]; B [N][K], or [K][N] (KN)
  long long scm, scn;
  int M, N, K, tiles_m, tiles;
  int split, per;  // CTAs (of a cluster) that share the K range of a tile, 64-k chunks of each
  int* err;
};

template <int OA, int OB>
__device__ __forceinline__ void umma_ts_pair_at(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\t.reg .b32 x;\n\t.reg .b64 y;\n\tadd.u32 x, %1, %5;\n\tadd.u64 y, %2, %6;\n\tsetp.ne.b32 p, %4, 0;\n\t"
               "tcgen05.mma.cta_group::2.kind::f16 [%0], [x], y, %3, p;\n\t}"
               ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate), "n"(OA), "n"(OB) : "memory");
}
// Arrives on the barrier in both CTAs of the pair once all MMAs issued so far have completed.
__device__ __forceinline__ void commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"(static_cast<uint16_t>(3)) : "memory");
}

// the three terms of kUp times two numbers
__device__ __forceinline__ void split3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  bf16_terms3(mul2(pack2(x, y), pack2(kUp, kUp)), hi, mid, lo);
}

// Results (m, n .. n + 3); whether one of them is not finite.
__device__ __forceinline__ bool store4(const F32Args& g, int m, int n, float4 v) {
  if (m >= g.M) return false;
  const float x[4] = {v.x, v.y, v.z, v.w};
  float y[4];
  bool again = false;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    again |= !isfinite(x[q]) && n + q < g.N;
    y[q] = x[q] + (g.bias && n + q < g.N ? __ldg(g.bias + n + q) : 0.0f);
  }
  float* out = g.c + m * g.scm + n * g.scn;
  if (g.scn == 1 && n + 4 <= g.N && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
    *reinterpret_cast<float4*>(out) = make_float4(y[0], y[1], y[2], y[3]);
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (n + q < g.N) out[q * g.scn] = y[q];
  }
  return again;
}

// Results of a row, COUNT neighbours; whether one of them is not finite.  Whole rows of 32-byte sectors where C is so aligned (1000 x 4096 x 1024:
// pieces of 16 bytes, each tested and biased by itself, 45.4 us; these 40.9; pieces turned between eight lanes into lines 46.6).
template <int COUNT>
__device__ __forceinline__ bool store_columns(const F32Args& g, int m, int n, const f32x2 (&acc)[COUNT / 2]) {
  if (m >= g.M || n >= g.N) return false;
  float* out = g.c + m * g.scm + n * g.scn;
  if (g.scn != 1 || n + COUNT > g.N || ((reinterpret_cast<uintptr_t>(g.c) | static_cast<uintptr_t>(g.scm) * 4) & 31)) {
    bool again = false;
#pragma unroll
    for (int e = 0; e < COUNT; e += 4) {
      const float2 x = unpack2(acc[e / 2]), y = unpack2(acc[e / 2 + 1]);
      again |= store4(g, m, n + e, make_float4(x.x, x.y, y.x, y.y));
    }
    return again;
  }
  const bool biased = g.bias, wide = !(reinterpret_cast<uintptr_t>(g.bias) & 15);
  f32x2 seen = pack2(0.0f, 0.0f);  // a number that is not finite times zero is not zero
#pragma unroll
  for (int e = 0; e < COUNT; e += 8) {
    f32x2 v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      v[q] = acc[e / 2 + q];
      seen = fma2(v[q], pack2(0.0f, 0.0f), seen);
    }
    if (biased) {
      const float* p = g.bias + n + e;
      float4 b[2];
      if (wide) {
        b[0] = __ldg(reinterpret_cast<const float4*>(p));
        b[1] = __ldg(reinterpret_cast<const float4*>(p) + 1);
      } else {
        b[0] = make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
        b[1] = make_float4(__ldg(p + 4), __ldg(p + 5), __ldg(p + 6), __ldg(p + 7));
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        v[2 * q] = fma2(v[2 * q], pack2(1.0f, 1.0f), pack2(b[q].x, b[q].y));
        v[2 * q + 1] = fma2(v[2 * q + 1], pack2(1.0f, 1.0f), pack2(b[q].z, b[q].w));
      }
    }
    const float2 x = unpack2(v[0]), y = unpack2(v[1]), z = unpack2(v[2]), w = unpack2(v[3]);
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"l"(out + e), "f"(x.x), "f"(x.y), "f"(y.x), "f"(y.y), "f"(z.x), "f"(z.y), "f"(w.x), "f"(w.y) : "memory");
  }
  const float2 f = unpack2(seen);
  return !(f.x == 0.0f && f.y == 0.0f);
}

// The first `count` of four numbers (none where it is not positive) and zeros behind them.
__device__ __forceinline__ void copy16(uint32_t dst, const float* src, int count) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(4 * max(0, min(4, count))) : "memory");
}
__device__ __forceinline__ void copy4(uint32_t dst, const float* src, bool there) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(there ? 4 : 0) : "memory");
}

// The results of rows m0 .. m0 + 16 TM - 1 and columns n0 .. n0 + BN - 1 that are not finite, in f32 multiply-adds in the order of k, by all
// threads of the CTA: a warp has TM rows, a lane BN / 32 columns.  32 k at a time in two buffers; the next are on their way while one is
// multiplied.  The whole tile is summed whatever the number of such results, at about the rate of the CUDA-core kernel, and the finite
// ones keep what the tensor cores gave.
template <int BN, bool KN, bool FILL, int TM, int WARPS>
__device__ __forceinline__ void sum_again_here(const F32Args& g, float* sm, int m0, int n0, int tid) {
  constexpr int kThreads = 32 * WARPS, kK = 32, kLd = kK + 4, kRows = WARPS * TM, kA = kRows * kLd, kBuffer = kA + (KN ? kK * BN : BN * kLd), TN = BN / 32;
  static_assert(2 * kBuffer * 4 <= Cfg<BN>::kStages, "in the place of the terms");
  const int warp = tid >> 5, lane = tid & 31;
  const uint32_t base = smem_u32(sm);
  auto request = [&](int k0, int buf) {
    const uint32_t d = base + buf * kBuffer * 4;
    if constexpr (FILL) {
      for (int i = tid; i < kRows * kK; i += kThreads) {
        const int r = i / kK, k = k0 + i % kK;
        const bool there = m0 + r < g.M && k < g.K;
        copy4(d + (r * kLd + i % kK) * 4, there ? g.a + (m0 + r) * g.lda + k : g.a, there);
      }
      for (int i = tid; i < BN * kK; i += kThreads) {
        const int r = KN ? i / BN : i / kK, c = KN ? i % BN : i % kK, k = k0 + (KN ? r : c), n = n0 + (KN ? c : r);
        const bool there = k < g.K && n < g.N;
        copy4(d + (kA + (KN ? r * BN : r * kLd) + c) * 4, there ? g.b + (KN ? k * g.ldb + n : n * g.ldb + k) : g.b, there);
      }
    } else {
      // 16 bytes at a time, cut off at the row's last number: rows that a tensor map describes start on 16 bytes, but K and N need not be multiples of
      // four, and what lies behind a row belongs to nobody
      for (int i = tid; i < kRows * (kK / 4); i += kThreads) {
        const int r = i / (kK / 4), k = k0 + i % (kK / 4) * 4, count = m0 + r < g.M ? g.K - k : 0;
        copy16(d + (r * kLd + i % (kK / 4) * 4) * 4, count > 0 ? g.a + (m0 + r) * g.lda + k : g.a, count);
      }
      for (int i = tid; i < BN * (kK / 4); i += kThreads) {
        if constexpr (KN) {
          const int r = i / (BN / 4), n = i % (BN / 4) * 4, count = k0 + r < g.K ? g.N - n0 - n : 0;
          copy16(d + (kA + r * BN + n) * 4, count > 0 ? g.b + (k0 + r) * g.ldb + n0 + n : g.b, count);
        } else {
          const int r = i / (kK / 4), k = k0 + i % (kK / 4) * 4, count = n0 + r < g.N ? g.K - k : 0;
          copy16(d + (kA + r * kLd + i % (kK / 4) * 4) * 4, count > 0 ? g.b + (n0 + r) * g.ldb + k : g.b, count);
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;
  named_barrier_sync(1, kThreads);  // the buffers are free
  request(0, 0);
  for (int k0 = 0, buf = 0; k0 < g.K; k0 += kK, buf ^= 1) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    named_barrier_sync(1, kThreads);
    if (k0 + kK < g.K) request(k0 + kK, buf ^ 1);
    const float* as = sm + buf * kBuffer + warp * TM * kLd;
    const float* bs = sm + buf * kBuffer + kA;
#pragma unroll 2
    for (int k = 0; k < kK; k += 4) {
      float b[TN][4];
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        if constexpr (KN) {
#pragma unroll
          for (int e = 0; e < 4; ++e) b[j][e] = bs[(k + e) * BN + j * 32 + lane];
        } else {
          const float4 v = *reinterpret_cast<const float4*>(bs + (j * 32 + lane) * kLd + k);
          b[j][0] = v.x; b[j][1] = v.y; b[j][2] = v.z; b[j][3] = v.w;
        }
      }
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const float4 v = *reinterpret_cast<const float4*>(as + i * kLd + k);
        const float a[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[e], b[j][e], acc[i][j]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int m = m0 + warp * TM + i, n = n0 + j * 32 + lane;
      if (m >= g.M || n >= g.N) continue;
      float* out = g.c + m * g.scm + n * g.scn;
      if (!isfinite(*out)) *out = acc[i][j] + (g.bias ? g.bias[n] : 0.0f);
    }
}

template <int BN, bool KN, bool FILL, int TM>
__device__ __noinline__ void sum_again(const F32Args& g, float* sm, int m0, int n0) {
  sum_again_here<BN, KN, FILL, TM, kThreads / 32>(g, sm, m0, n0, threadIdx.x);
}

// The f32 numbers of a chunk -> bf16 terms, A's in tensor memory and B's in shared memory as swizzled tiles, by the splitting warps.  A thread has
// half of a row of A (its lane of tensor memory) and BN / 4 numbers of a row of B, in pieces of 16 bytes; eight lanes' pieces of the
// swizzled rows lie in different banks.
template <int BN, bool KN>
__device__ __forceinline__ void split_chunk(const uint8_t* raw, uint8_t* terms, uint32_t tmem_a) {
  using C = Cfg<BN>;
  constexpr int kRowsB = KN ? kBK : BN, kBoxB = kRowsB * 128;
  const int tid = threadIdx.x, warp = tid >> 5, quarter = warp & 3, half = warp >> 2, row = quarter * 32 + (tid & 31);
  const int row_b = tid % kRowsB, first_b = tid / kRowsB * (BN / 4);
  const uint8_t* from = raw + half * C::kBoxA + row * 128;
  const uint32_t to = tmem_a + (static_cast<uint32_t>(quarter * 32) << 16) + half * 16;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t hi[8], mid[8], lo[8];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float4 x = *reinterpret_cast<const float4*>(from + (((h * 4 + q) ^ (row & 7)) << 4));
      split3(x.x, x.y, hi[2 * q], mid[2 * q], lo[2 * q]);
      split3(x.z, x.w, hi[2 * q + 1], mid[2 * q + 1], lo[2 * q + 1]);
    }
    tmem_st_32x8(to + h * 8, hi);
    tmem_st_32x8(to + kTermColumns + h * 8, mid);
    tmem_st_32x8(to + 2 * kTermColumns + h * 8, lo);
  }
  from = raw + C::kRawA + row_b * 128;
  uint8_t* place = terms + row_b * 128;
#pragma unroll
  for (int p = 0; p < BN / 32; ++p) {
    const int f = first_b + p * 8;  // k of the row, n with KN
    const uint8_t* box = from + (f >> 5) * kBoxB;
    const float4 x = *reinterpret_cast<const float4*>(box + ((((f >> 2) & 7) ^ (row_b & 7)) << 4));
    const float4 y = *reinterpret_cast<const float4*>(box + ((((f >> 2) & 7 | 1) ^ (row_b & 7)) << 4));
    uint4 hi, mid, lo;
    split3(x.x, x.y, hi.x, mid.x, lo.x);
    split3(x.z, x.w, hi.y, mid.y, lo.y);
    split3(y.x, y.y, hi.z, mid.z, lo.z);
    split3(y.z, y.w, hi.w, mid.w, lo.w);
    uint8_t* d = place + (KN ? (f >> 6) * (kBK * 128) : 0) + ((((f >> 3) & 7) ^ (row_b & 7)) << 4);
    *reinterpret_cast<uint4*>(d) = hi;
    *reinterpret_cast<uint4*>(d + C::kTermB) = mid;
    *reinterpret_cast<uint4*>(d + 2 * C::kTermB) = lo;
  }
}

// FILL: operands that a tensor map cannot describe (rows that do not start on 16 bytes, strides below a row's length): the splitting warps
// bring the numbers in by copies of four bytes, a row's 32 side by side, as far ahead as there are stages.
template <int BN, bool KN, bool FILL>
__global__ void __launch_bounds__(kThreads, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ F32Args g) {
  using C = Cfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bars = base + C::kStages;
  auto full = [&](int s) { return bars + 8u * s; };              // a stage's terms are in place
  auto empty = [&](int s) { return bars + 16u + 8u * s; };       // the MMAs have read them
  auto acc_full = [&](int s) { return bars + 32u + 8u * s; };
  auto acc_empty = [&](int s) { return bars + 48u + 8u * s; };
  auto raw_full = [&](int s) { return bars + 64u + 8u * s; };    // a stage's f32 numbers are in place
  auto raw_empty = [&](int s) { return bars + 96u + 8u * s; };   // the splitting warps have read them
  const uint32_t received = bars + 128u, tmem_slot = bars + 136u;
  constexpr int R = C::kRawStages;
  auto raw = [&](int s) { return base + s * C::kRaw; };
  auto terms = [&](int s) { return base + R * C::kRaw + s * C::kTerms; };
  // bit i: a result of this CTA's tile number i (modulo the bits) is not finite and its sums are made again
  __shared__ unsigned again[32], gave_up;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = blockIdx.x % g.split, chunk0 = rank * g.per, chunks = min(g.per, (g.K + kBK - 1) / kBK - chunk0);
  const int tile0 = blockIdx.x / g.split, tile_step = gridDim.x / g.split;
  const int total = (g.tiles - tile0 + tile_step - 1) / tile_step * chunks;  // chunks of all of this CTA's tiles
  const int rows = kBM / g.split;  // of a tile with split K, that a CTA finishes
  const bool one = elect_one();
  if (tid < 32) again[tid] = 0;
  if (tid == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(full(s), kSplitWarps);
      mbar_init(empty(s), 1);
      mbar_init(acc_full(s), 1);
      mbar_init(acc_empty(s), kSumWarps);
    }
    for (int s = 0; s < R; ++s) {
      mbar_init(raw_full(s), FILL ? kSplit : 1);
      mbar_init(raw_empty(s), kSplitWarps);
    }
    mbar_init(received, 1);
    mbar_fence_init();
    if (g.split > 1) mbar_expect_tx(received, (g.split - 1) * rows * C::kPitch * 4);
  }
  if (warp == kSplitWarps) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(gen + C::kStages + 136);
  pdl_wait();

  if (warp < kSplitWarps) {
    // ---- split ----
    constexpr int kRowsB = KN ? kBK : BN, kBoxB = kRowsB * 128;
    int fill_tile = tile0, fill_chunk = 0;
    auto fill = [&](int s) {  // the next chunk's numbers
      if constexpr (!FILL) {
        if (warp == 0 && fill_tile < g.tiles) {
          const int tn = fill_tile / g.tiles_m, k0 = (chunk0 + fill_chunk) * kBK, m0 = (fill_tile - tn * g.tiles_m) * kBM, n0 = tn * BN;
          if (one) {
            mbar_expect_tx(raw_full(s), C::kRaw);
            const uint32_t a = raw(s), b = a + C::kRawA;
            tma_load_2d(a, &map_a, raw_full(s), k0, m0);
            tma_load_2d(a + C::kBoxA, &map_a, raw_full(s), k0 + 32, m0);
#pragma unroll
            for (int q = 0; q < (KN ? BN / 32 : 2); ++q)
              tma_load_2d(b + q * kBoxB, &map_b, raw_full(s), KN ? n0 + q * 32 : k0 + q * 32, KN ? k0 : n0);
          }
          if (++fill_chunk == chunks) { fill_chunk = 0; fill_tile += tile_step; }
        }
        return;
      }
      if (fill_tile < g.tiles) {
        const int tn = fill_tile / g.tiles_m, k0 = (chunk0 + fill_chunk) * kBK, m = (fill_tile - tn * g.tiles_m) * kBM + warp, n0 = tn * BN;
        const uint32_t at = raw(s) + warp * 128 + (((lane >> 2) ^ warp) << 4) + (lane & 3) * 4;  // row number warp + 8 j: j KB on
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          const int k = k0 + b * 32 + lane;
          const float* p = g.a + m * g.lda + k;
#pragma unroll 4
          for (int j = 0; j < kBM / 8; ++j) {
            const bool there = k < g.K && m + j * 8 < g.M;
            copy4(at + b * C::kBoxA + j * 1024, there ? p + j * 8 * g.lda : g.a, there);
          }
        }
#pragma unroll
        for (int b = 0; b < (KN ? BN / 32 : 2); ++b) {
          const int x = (KN ? n0 : k0) + b * 32 + lane, y = (KN ? k0 : n0) + warp;
          const float* p = g.b + y * g.ldb + x;
#pragma unroll 4
          for (int j = 0; j < kRowsB / 8; ++j) {
            const bool there = x < (KN ? g.N : g.K) && y + j * 8 < (KN ? g.K : g.N);
            copy4(at + C::kRawA + b * kBoxB + j * 1024, there ? p + j * 8 * g.ldb : g.b, there);
          }
        }
        if (++fill_chunk == chunks) { fill_chunk = 0; fill_tile += tile_step; }
      }
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(raw_full(s)) : "memory");
    };
    for (int r = 0; r < R; ++r) fill(r);
    for (int it = 0, r = 0, raw_ph = 0; it < total; ++it) {
      const int s = it & 1, ph = (it >> 1) & 1;
      if (!mbar_wait(raw_full(r), raw_ph, g.err, DEVERR_GEMM_PRODUCER) || !mbar_wait(empty(s), ph ^ 1, g.err, DEVERR_GEMM_PRODUCER)) break;
      tc_fence_after();
      split_chunk<BN, KN>(gen + r * C::kRaw, gen + R * C::kRaw + s * C::kTerms, tmem + kTmemA + s * (3 * kTermColumns));
      tmem_wait_st();
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(full(s));
        mbar_arrive(raw_empty(r));
      }
      if ((FILL || warp == 0) && it + R < total) {
        if (!mbar_wait(raw_empty(r), raw_ph, g.err, DEVERR_GEMM_PRODUCER)) break;
        fill(r);
      }
      if (++r == R) { r = 0; raw_ph ^= 1; }
    }
    if (FILL) asm volatile("cp.async.wait_all;" ::: "memory");
  } else {
    // ---- sums: a warp owns 32 rows (TMEM lanes of its quarter) and half of the columns ----
    constexpr int kCols = BN / 2, kStep = kCols < 32 ? 16 : 32;
    const int w = warp - kSplitWarps, quarter = warp & 3, col0 = (w >> 2) * kCols;
    // Products of a chunk, the largest last: what is cut off is relative to the sum so far.
    auto issue = [&](int n) {  // the whole warp, one lane issues: descriptors stay in uniform registers
      const int s = n & 1, ph = (n >> 1) & 1;
      if (!mbar_wait(acc_empty(s), ph ^ 1, g.err, DEVERR_GEMM_MMA) || !mbar_wait(full(s), ph, g.err, DEVERR_GEMM_MMA)) return;
      tc_fence_after();
      const uint32_t a = tmem + kTmemA + s * (3 * kTermColumns), d = tmem + s * BN;
      const uint64_t b = make_smem_desc_sw128(terms(s), KN ? kBK * 128 : 16, 1024);
      constexpr uint32_t idesc = make_idesc_bf16(kBM, BN, false, KN);
      auto step = [&](auto ta, auto tb, uint32_t first) {  // 16 k: 8 columns of A, 32 bytes of a K-major row of B, 16 rows of an N-major tile
        constexpr int A = decltype(ta)::value * kTermColumns, B = decltype(tb)::value * (C::kTermB / 16), kK = KN ? 128 : 2;
        umma_ts_at<A, B>(d, a, b, idesc, first);
        umma_ts_at<A + 8, B + kK>(d, a, b, idesc, 1);
        umma_ts_at<A + 16, B + 2 * kK>(d, a, b, idesc, 1);
        umma_ts_at<A + 24, B + 3 * kK>(d, a, b, idesc, 1);
      };
      using std::integral_constant;
      constexpr integral_constant<int, 0> c0;
      constexpr integral_constant<int, 1> c1;
      constexpr integral_constant<int, 2> c2;
      if (one) {
        step(c0, c2, 0);
        step(c2, c0, 1);
        step(c1, c1, 1);
        step(c1, c0, 1);
        step(c0, c1, 1);
        step(c0, c0, 1);
        umma_commit(empty(s));
        umma_commit(acc_full(s));
      }
    };
    const f32x2 down = pack2(kDown, kDown);
    if (w == 0 && total > 0) issue(0);
    int it = 0, number = 0;
    bool ok = true;
    for (int t = tile0; ok && t < g.tiles; t += tile_step, ++number) {
      f32x2 acc[kCols / 2];
#pragma unroll
      for (int e = 0; e < kCols / 2; ++e) acc[e] = pack2(0.0f, 0.0f);
      for (int i = 0; i < chunks; ++i, ++it) {
        const int s = it & 1;
        if (w == 0 && it + 1 < total) issue(it + 1);
        if (!mbar_wait(acc_full(s), (it >> 1) & 1, g.err, DEVERR_GEMM_EPILOGUE)) { ok = false; break; }
        tc_fence_after();
        const uint32_t addr = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + s * BN + col0;
#pragma unroll
        for (int c = 0; c < kCols; c += kStep) {
          uint32_t r[kStep];
          if constexpr (kStep == 32) tmem_ld_32x32(addr + c, r); else tmem_ld_32x16(addr + c, r);
          tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < kStep; e += 2) acc[(c + e) / 2] = fma2(pack2(__uint_as_float(r[e]), __uint_as_float(r[e + 1])), down, acc[(c + e) / 2]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty(s));
      }
      if (!ok) break;
      if (g.split > 1) {  // (one tile) the stages' place takes the sums: every MMA that read it is done
        float* dst = reinterpret_cast<float*>(gen) + (quarter * 32 + lane) * C::kPitch + col0;
#pragma unroll
        for (int e = 0; e < kCols; e += 4) {
          const float2 x = unpack2(acc[e / 2]), y = unpack2(acc[e / 2 + 1]);
          *reinterpret_cast<float4*>(dst + e) = make_float4(x.x, x.y, y.x, y.y);
        }
        fence_proxy_async_smem();
        continue;
      }
      const int tn = t / g.tiles_m, m = (t - tn * g.tiles_m) * kBM + quarter * 32 + lane, n0 = tn * BN + col0;
      const bool bad = store_columns<kCols>(g, m, n0, acc);
      if (bad) atomicOr(&again[(number >> 5) & 31], 1u << (number & 31));
    }
  }
  __syncwarp();
  tc_fence_before();
  if (tid == 0) gave_up = *reinterpret_cast<volatile int*>(g.err) != 0;
  __syncthreads();
  if (g.split > 1) {
    // Every CTA is behind its main loop, so what the others send may take the place of its stages: a CTA finishes kBM / split rows of
    // the tile and gets them from the others by bulk copies (remote loads took 2000 clocks), relaxed arrivals: the barrier above
    // has seen every reader.
    cluster_arrive_relaxed();
    cluster_wait();
    const int bytes = rows * C::kPitch * 4;
    if (warp == kSplitWarps && lane < g.split && lane != rank && !gave_up)
      send_bulk(map_rank(base + C::kPart + (rank - (rank > lane)) * bytes, lane), base + lane * bytes, bytes, map_rank(received, lane));
    __syncwarp();
    if (mbar_wait(received, 0, g.err, DEVERR_GEMM_EPILOGUE)) {
      // the parts added in the order of k
      const int tn = tile0 / g.tiles_m, m0 = (tile0 - tn * g.tiles_m) * kBM + rank * rows;
      const uint8_t* own = gen + rank * bytes;
      const uint8_t* got = gen + C::kPart;
      for (int u = tid; u < rows * (BN / 4); u += kThreads) {
        const int r = u / (BN / 4), n = u % (BN / 4) * 4, at = (r * C::kPitch + n) * 4;
        float4 v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (q < g.split) v[q] = *reinterpret_cast<const float4*>((q == rank ? own : got + (q - (q > rank)) * bytes) + at);
        float4 x = v[0];
#pragma unroll
        for (int q = 1; q < 8; ++q)
          if (q < g.split) x = make_float4(x.x + v[q].x, x.y + v[q].y, x.z + v[q].z, x.w + v[q].w);
        if (store4(g, m0 + r, tn * BN + n, x)) atomicOr(&again[0], 1u);
      }
    }
    __syncwarp();
    cluster_arrive_relaxed();
    cluster_wait();  // nobody leaves, or takes its shared memory for something else, while what it sent is on its way
    if (tid == 0) gave_up = *reinterpret_cast<volatile int*>(g.err) != 0;
    __syncthreads();
  }
  if (warp == kSplitWarps) {
    if (gave_up) {
      // a wait gave up: let MMAs that are still in flight drain before the memory is released
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 2000000ull) __nanosleep(1000);
    }
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
  if (gave_up) return;
  // (the barrier above: every result is stored, every MMA and every CTA of the cluster is done with this shared memory)
  for (int t = tile0, number = 0; t < g.tiles; t += tile_step, ++number) {
    if (!((again[(number >> 5) & 31] >> (number & 31)) & 1u)) continue;
    const int tn = t / g.tiles_m, m0 = (t - tn * g.tiles_m) * kBM + rank * rows, n0 = tn * BN;
    float* sm = reinterpret_cast<float*>(gen);
    switch (g.split) {
      case 1: sum_again<BN, KN, FILL, 8>(g, sm, m0, n0); break;
      case 2: sum_again<BN, KN, FILL, 4>(g, sm, m0, n0); break;
      case 4: sum_again<BN, KN, FILL, 2>(g, sm, m0, n0); break;
      default: sum_again<BN, KN, FILL, 1>(g, sm, m0, n0); break;
    }
  }
}

// 256 x 256 tiles by pairs of CTAs (cta_group::2): a CTA splits 128 rows of A and 128 of B for twice as many products.  Each MMA is 256 x 128: the
// rows of A of both CTAs (each CTA's terms in its own tensor memory) and 64 rows of B of each, so that the sums of one half of the columns are
// moved while the other half is multiplied: two accumulators, as many tensor memory columns as a CTA's 128 x 128 tile takes with two.
template <bool KN>
__global__ void __launch_bounds__(kThreads, 1)
gemm_f32_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ F32Args g) {
  constexpr int BN = 128;  // rows of B of a CTA
  using C = Cfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bars = base + C::kStages;
  auto raw_full = [&](int s) { return bars + 8u * s; };
  auto raw_empty = [&](int s) { return bars + 16u + 8u * s; };
  auto full = [&](int s) { return bars + 32u + 8u * s; };        // in the leader: the terms of both CTAs are in place
  auto empty = [&](int s) { return bars + 48u + 8u * s; };       // in both CTAs, as acc_full
  auto acc_full = [&](int h) { return bars + 64u + 8u * h; };
  auto acc_empty = [&](int h) { return bars + 80u + 8u * h; };   // in the leader
  const uint32_t tmem_slot = bars + 104u;
  __shared__ unsigned again[32], gave_up;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rank = blockIdx.x & 1;
  const int tile0 = blockIdx.x >> 1, tile_step = gridDim.x >> 1, chunks = (g.K + kBK - 1) / kBK;
  const int total = (g.tiles - tile0 + tile_step - 1) / tile_step * chunks;
  const bool one = elect_one();
  if (tid < 32) again[tid] = 0;
  if (tid == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(raw_full(s), 1);
      mbar_init(raw_empty(s), kSplitWarps);
      mbar_init(full(s), 2 * kSplitWarps);
      mbar_init(empty(s), 1);
      mbar_init(acc_full(s), 1);
      mbar_init(acc_empty(s), 2 * kSumWarps);
    }
    mbar_fence_init();
  }
  if (warp == kSplitWarps) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_arrive_relaxed();
  cluster_wait();  // both CTAs' barriers exist
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(gen + C::kStages + 104);
  pdl_wait();

  if (warp < kSplitWarps) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kPairSplitRegs));
    int fill_tile = tile0, fill_chunk = 0;
    auto fill = [&](int s) {
      if (warp != 0 || fill_tile >= g.tiles) return;
      const int tn = fill_tile / g.tiles_m, k0 = fill_chunk * kBK, m0 = (fill_tile - tn * g.tiles_m) * (2 * kBM) + rank * kBM, n0 = tn * (2 * BN) + rank * BN;
      if (one) {
        mbar_expect_tx(raw_full(s), C::kRaw);
        const uint32_t a = base + s * C::kRaw, b = a + C::kRawA;
        tma_load_2d(a, &map_a, raw_full(s), k0, m0);
        tma_load_2d(a + C::kBoxA, &map_a, raw_full(s), k0 + 32, m0);
#pragma unroll
        for (int q = 0; q < (KN ? BN / 32 : 2); ++q)
          tma_load_2d(b + q * ((KN ? kBK : BN) * 128), &map_b, raw_full(s), KN ? n0 + q * 32 : k0 + q * 32, KN ? k0 : n0);
      }
      if (++fill_chunk == chunks) { fill_chunk = 0; fill_tile += tile_step; }
    };
    fill(0);
    fill(1);
    const uint32_t there = map_rank(full(0), 0);
    for (int it = 0; it < total; ++it) {
      const int s = it & 1, ph = (it >> 1) & 1;
      if (!mbar_wait(raw_full(s), ph, g.err, DEVERR_GEMM_PRODUCER) || !mbar_wait(empty(s), ph ^ 1, g.err, DEVERR_GEMM_PRODUCER)) break;
      tc_fence_after();
      split_chunk<BN, KN>(gen + s * C::kRaw, gen + 2 * C::kRaw + s * C::kTerms, tmem + kTmemA + s * (3 * kTermColumns));
      tmem_wait_st();
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(raw_empty(s));
        asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(there + 8 * s) : "memory");
      }
      if (warp == 0 && it + 2 < total) {
        if (!mbar_wait(raw_empty(s), ph, g.err, DEVERR_GEMM_PRODUCER)) break;
        fill(s);
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kPairSumRegs));
    // a warp owns 32 rows and the 64 columns of each half that are rows of one CTA's B: 128 neighbours
    const int w = warp - kSplitWarps, quarter = warp & 3, side = w >> 2;
    const bool issuer = w == 0 && rank == 0;
    auto issue = [&](int n) {  // step n: half n & 1 of chunk n / 2
      const int h = n & 1, i = n >> 1, s = i & 1;
      if (!mbar_wait(acc_empty(h), (i & 1) ^ 1, g.err, DEVERR_GEMM_MMA)) return;
      if (h == 0 && !mbar_wait(full(s), (i >> 1) & 1, g.err, DEVERR_GEMM_MMA)) return;
      tc_fence_after();
      const uint32_t a = tmem + kTmemA + s * (3 * kTermColumns), d = tmem + h * 128;
      const uint64_t b = make_smem_desc_sw128(base + 2 * C::kRaw + s * C::kTerms + h * 8192, KN ? kBK * 128 : 16, 1024);
      constexpr uint32_t idesc = make_idesc_bf16(2 * kBM, 128, false, KN);
      auto step = [&](auto ta, auto tb, uint32_t first) {
        constexpr int A = decltype(ta)::value * kTermColumns, B = decltype(tb)::value * (C::kTermB / 16), kK = KN ? 128 : 2;
        umma_ts_pair_at<A, B>(d, a, b, idesc, first);
        umma_ts_pair_at<A + 8, B + kK>(d, a, b, idesc, 1);
        umma_ts_pair_at<A + 16, B + 2 * kK>(d, a, b, idesc, 1);
        umma_ts_pair_at<A + 24, B + 3 * kK>(d, a, b, idesc, 1);
      };
      using std::integral_constant;
      constexpr integral_constant<int, 0> c0;
      constexpr integral_constant<int, 1> c1;
      constexpr integral_constant<int, 2> c2;
      if (one) {
        step(c0, c2, 0);  // the order of the other kernel
        step(c2, c0, 1);
        step(c1, c1, 1);
        step(c1, c0, 1);
        step(c0, c1, 1);
        step(c0, c0, 1);
        if (h) commit_pair(empty(s));
        commit_pair(acc_full(h));
      }
    };
    const uint32_t there = map_rank(acc_empty(0), 0);
    const f32x2 down = pack2(kDown, kDown);
    if (issuer && total > 0) issue(0);
    int it = 0, number = 0;
    bool ok = true;
    for (int t = tile0; ok && t < g.tiles; t += tile_step, ++number) {
      f32x2 acc[2][32];
#pragma unroll
      for (int e = 0; e < 32; ++e) acc[0][e] = acc[1][e] = pack2(0.0f, 0.0f);
      for (int i = 0; ok && i < chunks; ++i, ++it) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (issuer && 2 * it + h + 1 < 2 * total) issue(2 * it + h + 1);
          if (ok && !mbar_wait(acc_full(h), it & 1, g.err, DEVERR_GEMM_EPILOGUE)) ok = false;
          if (ok) {
            tc_fence_after();
            const uint32_t addr = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + h * 128 + side * 64;
#pragma unroll
            for (int c = 0; c < 64; c += 16) {
              uint32_t r[16];
              tmem_ld_32x16(addr + c, r);
              tmem_wait_ld();
#pragma unroll
              for (int e = 0; e < 16; e += 2)
                acc[h][(c + e) / 2] = fma2(pack2(__uint_as_float(r[e]), __uint_as_float(r[e + 1])), down, acc[h][(c + e) / 2]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(there + 8 * h) : "memory");
          }
        }
      }
      if (!ok) break;
      const int tn = t / g.tiles_m, m = (t - tn * g.tiles_m) * (2 * kBM) + rank * kBM + quarter * 32 + lane, n0 = tn * (2 * BN) + side * BN;
      bool bad = store_columns<64>(g, m, n0, acc[0]);
      bad |= store_columns<64>(g, m, n0 + 64, acc[1]);
      if (bad) atomicOr(&again[(number >> 5) & 31], 1u << (number & 31));
    }
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(128));
  }
  if (warp < kSplitWarps) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(128));
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  cluster_arrive_relaxed();
  cluster_wait();  // neither CTA leaves while the other's MMAs read its terms
  if (tid == 0) gave_up = *reinterpret_cast<volatile int*>(g.err) != 0;
  __syncthreads();
  if (warp == kSplitWarps) {
    if (gave_up) {
      // a wait gave up: let MMAs that are still in flight drain before the memory is released
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 2000000ull) __nanosleep(1000);
    }
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
  if (gave_up) return;
  for (int t = tile0, number = 0; t < g.tiles; t += tile_step, ++number) {
    if (!((again[(number >> 5) & 31] >> (number & 31)) & 1u)) continue;
    const int tn = t / g.tiles_m, m0 = (t - tn * g.tiles_m) * (2 * kBM) + rank * kBM;
    float* sm = reinterpret_cast<float*>(gen);
#pragma unroll 1
    for (int side = 0; side < 2; ++side)  // (inlined: a call does not go with registers divided anew)
      sum_again_here<BN, KN, false, 8, kThreads / 32>(g, sm, m0, tn * (2 * BN) + side * BN, tid);
  }
}

template <typename Kernel>
int prepare(std::atomic<unsigned long long>& done, Kernel kernel, int smem) {  // done: one bit per device; threads may race to set it
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64 || !((done.load(std::memory_order_acquire) >> dev) & 1ull)) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (dev < 64) done.fetch_or(1ull << dev, std::memory_order_release);
  }
  return 0;
}
template <int BN, bool KN, bool FILL>
int prepare_tc() {
  static std::atomic<unsigned long long> done{0};
  return prepare(done, gemm_f32_tc_kernel<BN, KN, FILL>, Cfg<BN>::kSmem);
}
template <bool KN>
int prepare_pair() {
  static std::atomic<unsigned long long> done{0};
  return prepare(done, gemm_f32_pair_kernel<KN>, Cfg<128>::kSmem);
}

// rows of an operand whose second index is contiguous, as boxes of 32 numbers by `box` rows
bool mappable(const float* p, long long ld, int inner) {
  return !(reinterpret_cast<uintptr_t>(p) & 15) && ld % 4 == 0 && ld >= inner && ld < (1ll << 37);
}
int map_rows(CUtensorMap* map, const float* p, long long ld, int inner, int outer, int box) {
  const uint64_t dims[2] = {static_cast<uint64_t>(inner), static_cast<uint64_t>(outer)}, strides[1] = {static_cast<uint64_t>(ld) * 4};
  const uint32_t boxes[2] = {32, static_cast<uint32_t>(box)};
  return encode_tensor_map_f32(map, p, 2, dims, strides, boxes);
}

template <int BN, bool KN>
int launch_tc(const F32Args& g, bool mapped, int grid, cudaStream_t st) {
  CUtensorMap ma{}, mb{};
  int rc = 0;
  if (mapped && ((rc = map_rows(&ma, g.a, g.lda, g.K, g.M, kBM)) ||
                 (rc = map_rows(&mb, g.b, g.ldb, KN ? g.N : g.K, KN ? g.K : g.N, KN ? kBK : BN))))
    return rc;
  if ((rc = mapped ? prepare_tc<BN, KN, false>() : prepare_tc<BN, KN, true>())) return rc;
  return launch_kernel(mapped ? gemm_f32_tc_kernel<BN, KN, false> : gemm_f32_tc_kernel<BN, KN, true>, dim3(grid), dim3(kThreads), Cfg<BN>::kSmem, st,
                       g.split, ma, mb, g);
}

template <bool KN>
int launch_pair(const F32Args& g, int grid, cudaStream_t st) {
  CUtensorMap ma{}, mb{};
  int rc = 0;
  if ((rc = map_rows(&ma, g.a, g.lda, g.K, g.M, kBM)) || (rc = map_rows(&mb, g.b, g.ldb, KN ? g.N : g.K, KN ? g.K : g.N, KN ? kBK : 128)) ||
      (rc = prepare_pair<KN>()))
    return rc;
  return launch_kernel(gemm_f32_pair_kernel<KN>, dim3(grid), dim3(kThreads), Cfg<128>::kSmem, st, 2, ma, mb, g);
}

// Tile width (256: pairs of CTAs), K split and the clocks they are estimated to take: of 64 k of a tile, of a launch's start and end, and of the
// parts of a split K to meet.  Fitted to 23 shapes with every choice (at 1.85 GHz; 512^3, [K][N], 64-wide tiles with K in one, two, four parts 13.1,
// 10.3, 8.8 us; 51 x 268 x 3852 256, 128, 64, 32 wide 115, 94, 61, 56 us, 32 wide in eight parts 11.8; 1000 x 4096 x 1024 38, 55, 70, 103 us).  Where rows come
// by copies of four bytes these are the bound.  One CTA fills an SM, and 74, 33 and 15 clusters of two, four and eight such CTAs find place at once
// (594 x 800 x 2352, 35 tiles in four parts: 41 us; in two 33).
struct Choice { int bn, split, per; double clocks; };
Choice choose(int M, int N, int K, bool kn, bool mapped, int sms) {
  Choice best{};
  const int chunks = (K + kBK - 1) / kBK;
  const long long tiles_m = (M + kBM - 1) / kBM;
  for (int bn = 128; bn >= (kn ? 64 : 32); bn >>= 1) {
    const long long tiles = tiles_m * ((N + bn - 1) / bn);
    const double chunk = bn == 128 ? (mapped ? 2680.0 : 8200.0) : (bn == 64 ? (mapped ? 1670.0 : 6100.0) : (mapped ? 1560.0 : 5100.0));
    const double ends = bn == 32 ? 8700.0 : 10300.0, meet = bn == 128 ? 3700.0 : (bn == 64 ? 2200.0 : 900.0);
    for (int split = 1; split <= 8; split <<= 1) {
      const int per = (chunks + split - 1) / split, room = split == 8 ? sms * 5 / 6 : (split == 4 ? sms * 9 / 10 : sms);
      if (split > 1 && (tiles * split > room || per * (split - 1) >= chunks)) break;
      const double t = static_cast<double>((tiles + sms - 1) / sms) * per * chunk + ends + (split > 1 ? meet : 0.0);
      if (!best.bn || t < best.clocks) best = Choice{bn, split, per, t};
    }
  }
  if (mapped) {
    const long long tiles = (tiles_m + 1) / 2 * ((N + 255) / 256);
    const int pairs = sms / 2;
    const double t = static_cast<double>((tiles + pairs - 1) / pairs) * chunks * 3260.0 + 13800.0;
    if (t < best.clocks) best = Choice{256, 1, chunks, t};
  }
  return best;
}

}  // namespace

// A [M][K] with k contiguous and B as [N][K] or [K][N] with its second index contiguous, any alignment, stride and length of rows: rows that a tensor
// map cannot describe (mappable) are copied four bytes at a time.
bool gemm_f32_tc_takes(long long sak, long long sbk, long long sbn, int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0) return false;
  if (sak != 1) return false;
  if (static_cast<long long>((M + kBM - 1) / kBM) * ((N + 31) / 32) > 0x7fffffffLL) return false;
  return sbk == 1 || sbn == 1;
}

int gemm_f32_tc_prepare() {
  int rc = 0;
  if ((rc = prepare_tc<128, false, false>()) || (rc = prepare_tc<64, false, false>()) || (rc = prepare_tc<32, false, false>()) ||
      (rc = prepare_tc<128, true, false>()) || (rc = prepare_tc<64, true, false>()) || (rc = prepare_tc<128, false, true>()) ||
      (rc = prepare_tc<64, false, true>()) || (rc = prepare_tc<32, false, true>()) || (rc = prepare_tc<128, true, true>()) ||
      (rc = prepare_tc<64, true, true>()) || (rc = prepare_pair<false>()) || (rc = prepare_pair<true>()))
    return rc;
  return 0;
}

double gemm_f32_tc_clocks(const float* a, long long sam, const float* b, long long sbk, long long sbn, const float* c, long long scm, long long scn, int M,
                          int N, int K) {
  const bool kn = sbk != 1, mapped = mappable(a, sam, K) && mappable(b, kn ? sbk : sbn, kn ? N : K);
  const uintptr_t rows = reinterpret_cast<uintptr_t>(c) | static_cast<uintptr_t>(scm) * 4;
  // Results that are not stored in whole sectors: 867 x 2919 x 96 23.1 us, 1253 x 2612 x 96 16.4 (estimated without: 11.0 both).  What operands that
  // no map describes take was measured with such results.
  const double store = !mapped || (scn == 1 && !(rows & 31)) ? 0.0 : (scn == 1 && !(rows & 15) ? 0.003 : 0.0088);
  return choose(M, N, K, kn, mapped, sm_count()).clocks + store * M * N;
}

int gemm_f32_tc(const float* a, long long sam, const float* b, long long sbk, long long sbn, const float* bias, float* c, long long scm,
                long long scn, int M, int N, int K, cudaStream_t st) {
  if (!a || !b || !c || !gemm_f32_tc_takes(1, sbk, sbn, M, N, K)) return TEENY_ERR_BAD_ARG;
  F32Args g{};
  const bool kn = sbk != 1;
  g.a = a; g.b = b; g.bias = bias; g.c = c;
  g.lda = sam; g.ldb = kn ? sbk : sbn;
  g.scm = scm; g.scn = scn;
  g.M = M; g.N = N; g.K = K;
  g.err = device_error_word();
  if (!g.err) return TEENY_ERR_DRIVER;
  const int sms = sm_count();
  const bool mapped = mappable(a, g.lda, K) && mappable(b, g.ldb, kn ? N : K);
  const Choice x = choose(M, N, K, kn, mapped, sms);
  const int bm = x.bn == 256 ? 2 * kBM : kBM;
  g.tiles_m = (M + bm - 1) / bm;
  g.tiles = g.tiles_m * ((N + x.bn - 1) / x.bn);
  g.split = x.split;
  g.per = x.per;
  if (x.bn == 256) {
    const int grid = 2 * (g.tiles < sms / 2 ? g.tiles : sms / 2);
    return kn ? launch_pair<true>(g, grid, st) : launch_pair<false>(g, grid, st);
  }
  const int grid = x.split > 1 ? g.tiles * x.split : (g.tiles < sms ? g.tiles : sms);
  if (kn) return x.bn == 128 ? launch_tc<128, true>(g, mapped, grid, st) : launch_tc<64, true>(g, mapped, grid, st);
  if (x.bn == 128) return launch_tc<128, false>(g, mapped, grid, st);
  return x.bn == 64 ? launch_tc<64, false>(g, mapped, grid, st) : launch_tc<32, false>(g, mapped, grid, st);
}

}  // namespace teeny
