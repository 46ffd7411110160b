// f32 GEMM on the tensor cores with the accuracy of f32 multiply-adds: C[M, N] = A[M, K] B (+ bias), B as [N, K] or [K, N].
//
// An f32 number is the sum of three bf16 numbers, x = hi + mid + lo (8 + 8 + 8 bits, each the rounded rest of the one before), so a
// product is nine bf16 products, all exact in f32; the six largest are taken, the other three are below 2^-24 of the product.  What
// would lose accuracy is the tensor core's accumulator, which cuts off instead of rounding: after 1024 k the result would be off by
// 1e-6.  So the sum stays in it for 64 k only (smallest products first) and is then added to f32 registers, rounded.
//
// Bound: shared memory.  For 64 k of a 128 x 128 tile its 128 bytes a clock carry the f32 numbers in and out of L1 (1000 clocks), the
// stores of the terms (770) and the reads of 24 MMAs (1540), 3300 in all against 770 of the tensor pipe; 3100 were measured (by the counters L1 is 57 % busy and
// the tensor pipe 47 %: the stages' hand-overs keep it from the rest).  A pass
// that splits the operands beforehand would bring 6 bytes per number through L2 for every tile instead of 4.  So the split runs
// beside the products: warps 0-7 load f32 rows, split them and store the three terms of each operand as swizzled tiles (two stages
// of 96 KB), warps 8-15 move finished 64-k sums from tensor memory (two accumulators) into registers; a lane of warp 8 issues
// the MMAs of a chunk before it turns to the sums of the chunk before.  (16 splitting warps with the registers divided anew: no
// faster, 427 against 418 us for 2048 x 4096 x 4096.)
// Measured against f32 multiply-adds on the CUDA cores: 1000 x 4096 x 1024 198 -> 69 us, error against 64 bits 5.7e-7 -> 1.1e-7;
// 2048 x 4096 x 4096 1447 -> 478 us, 1.2e-6 -> 1.7e-7; 300 x 700 x 2000 46 -> 17 us; 512^3 14.1 -> 9.6 us.
//
// bf16 has the exponents of f32 but only eight bits, so the terms of a small number would run out of exponent: the third below 2^-110, all
// three below 2^-134.  Both operands are therefore taken times 2^24, with which every term of every f32 number, the smallest subnormal
// included, is a normal bf16 number or zero, and the sums leave tensor memory times 2^-48.  What that costs is at the other end: from
// 2^104 on an operand, and from 2^80 on a sum, may overflow, infinities and NaNs split into NaNs, and the sums of a tile with results that
// are not finite are made again for these, with f32 multiply-adds (every result infinite: 2048 x 4096 x 4096 2.9 ms, 512^3 34 us).  The scale costs
// up to 8 % with B as [N][K] (2048 x 4096 x 4096: 439 us without) and nothing with [K][N].
#include <atomic>

#include "common.cuh"
#include "kernels.h"

namespace teeny {

namespace {

constexpr int kBM = 128, kBK = 64;
constexpr int kSplitWarps = 8, kSumWarps = 8;
constexpr int kThreads = 32 * (kSplitWarps + kSumWarps);  // 16 warps: 128 registers each, the most with two warps of either kind per scheduler
constexpr float kUp = 0x1p24f, kDown = 0x1p-48f;  // of the operands, of the sums
constexpr int kTileA = kBM * 128;  // one bf16 term of 64 k of A: 128 bytes per row
template <int BN> struct Cfg {
  static constexpr int kTileB = BN * 128;
  static constexpr int kStage = 3 * (kTileA + kTileB);
  static constexpr int kSmem = 2 * kStage + 1024 + 128;
  static_assert(kBM * (BN + 4) * 4 <= 2 * kStage, "sums fit in the place of the terms");
  static constexpr int kParts = BN == 128 ? 1 : 2;  // of an accumulator, see issue()
  static constexpr int kAcc = kParts * BN;          // tensor memory columns of an accumulator
  static constexpr int kCols = 2 * kAcc;
  static constexpr int kPitch = BN + 4;             // floats of a row of sums in shared memory (split K)
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

// two numbers -> the three bf16 terms of kUp times them, packed
__device__ __forceinline__ void split3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  const f32x2 minus = pack2(-1.0f, -1.0f), v = mul2(pack2(x, y), pack2(kUp, kUp));
  const float2 u = unpack2(v);
  hi = pack_bf16x2(u.x, u.y);
  const f32x2 r = fma2(pack2(bf16_lo(hi), bf16_hi(hi)), minus, v);
  const float2 f = unpack2(r);
  mid = pack_bf16x2(f.x, f.y);
  const float2 q = unpack2(fma2(pack2(bf16_lo(mid), bf16_hi(mid)), minus, r));
  lo = pack_bf16x2(q.x, q.y);
}

__device__ __forceinline__ float4 ld_cluster4(uint32_t local, uint32_t rank) {
  float4 v;
  asm volatile("{\n\t.reg .u32 a;\n\tmapa.shared::cluster.u32 a, %4, %5;\n\tld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [a];\n\t}"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(local), "r"(rank) : "memory");
  return v;
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

__device__ __forceinline__ void copy16(uint32_t dst, const float* src, bool there) {  // zeros where nothing is
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(there ? 16 : 0) : "memory");
}

// The results of rows m0 .. m0 + 16 TM - 1 and columns n0 .. n0 + BN - 1 that are not finite, in f32 multiply-adds in the order of k, by all
// threads of the CTA: a warp has TM rows, a lane BN / 32 columns.  32 k at a time in two buffers; the next are on their way while one is
// multiplied.  The whole tile is summed whatever the number of such results, at about the rate of the CUDA-core kernel, and the finite
// ones keep what the tensor cores gave.
template <int BN, bool KN, int TM>
__device__ __noinline__ void sum_again(const F32Args& g, float* sm, int m0, int n0) {
  constexpr int kK = 32, kLd = kK + 4, kRows = 16 * TM, kA = kRows * kLd, kBuffer = kA + (KN ? kK * BN : BN * kLd), TN = BN / 32;
  static_assert(2 * kBuffer * 4 <= 2 * Cfg<BN>::kStage, "in the place of the terms");
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t base = smem_u32(sm);
  auto request = [&](int k0, int buf) {
    const uint32_t d = base + buf * kBuffer * 4;
    for (int i = tid; i < kRows * (kK / 4); i += kThreads) {
      const int r = i / (kK / 4), k = k0 + i % (kK / 4) * 4;
      const bool there = m0 + r < g.M && k < g.K;
      copy16(d + (r * kLd + i % (kK / 4) * 4) * 4, there ? g.a + (m0 + r) * g.lda + k : g.a, there);
    }
    for (int i = tid; i < BN * (kK / 4); i += kThreads) {
      if constexpr (KN) {
        const int r = i / (BN / 4), n = i % (BN / 4) * 4;
        const bool there = k0 + r < g.K && n0 + n < g.N;
        copy16(d + (kA + r * BN + n) * 4, there ? g.b + (k0 + r) * g.ldb + n0 + n : g.b, there);
      } else {
        const int r = i / (kK / 4), k = k0 + i % (kK / 4) * 4;
        const bool there = n0 + r < g.N && k < g.K;
        copy16(d + (kA + r * kLd + i % (kK / 4) * 4) * 4, there ? g.b + (n0 + r) * g.ldb + k : g.b, there);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;
  __syncthreads();  // the buffers are free
  request(0, 0);
  for (int k0 = 0, buf = 0; k0 < g.K; k0 += kK, buf ^= 1) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
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

template <int BN, bool KN>
__global__ void __launch_bounds__(kThreads, 1) gemm_f32_tc_kernel(const __grid_constant__ F32Args g) {
  using C = Cfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bars = base + 2 * C::kStage;
  auto full = [&](int s) { return bars + 8u * s; };           // a stage's terms are in place
  auto empty = [&](int s) { return bars + 16u + 8u * s; };    // the MMAs have read them
  auto acc_full = [&](int s) { return bars + 32u + 8u * s; };
  auto acc_empty = [&](int s) { return bars + 48u + 8u * s; };
  const uint32_t tmem_slot = bars + 64u;
  // bit i: a result of this CTA's tile number i (modulo the bits) is not finite and its sums are made again
  __shared__ unsigned again[32], gave_up;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = blockIdx.x % g.split, chunk0 = rank * g.per, chunks = min(g.per, (g.K + kBK - 1) / kBK - chunk0);
  const int tile0 = blockIdx.x / g.split, tile_step = gridDim.x / g.split;
  if (tid < 32) again[tid] = 0;
  if (tid == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(full(s), kSplitWarps);
      mbar_init(empty(s), 1);
      mbar_init(acc_full(s), 1);
      mbar_init(acc_empty(s), kSumWarps);
    }
    mbar_fence_init();
  }
  if (warp == kSplitWarps) {
    tmem_alloc(tmem_slot, C::kCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(gen + 2 * C::kStage + 64);
  pdl_wait();

  if (warp < kSplitWarps) {
    // ---- split: pieces of four neighbours, a warp's 32 side by side in memory (two K-major rows), 16 rows at a time ----
    constexpr int kPiecesA = kBM / 16, kPieces = (kBM + BN) / 16;
    constexpr int kRowN = BN / 4;  // pieces of a row of an N-major tile
    float4 v[kPieces];
    // What is requested next.  Rows behind the last one are read from the last one (they only reach results that are not stored), and
    // so are k behind K, whose products are made zero on the side of A.
    int tile = tile0, chunk = 0, m0 = 0, n0 = 0;
    const int row = tid >> 4, kp = (tid & 15) * 4, kb = tid / kRowN, nb = tid % kRowN * 4;
    const float *pa = g.a, *pb = g.b;
    auto place = [&]() {  // pointers of this thread's pieces in row 0
      const int k = min((chunk0 + chunk) * kBK + kp, g.K - 4);
      pa = g.a + k;
      pb = KN ? g.b + min(n0 + nb, g.N - 4) : g.b + k;
    };
    auto start_tile = [&]() {
      const int tn = tile / g.tiles_m;
      m0 = (tile - tn * g.tiles_m) * kBM + row;
      n0 = tn * BN + (KN ? 0 : row);
    };
    start_tile();
    place();
    auto request = [&](int j) {
      const int jj = j < kPiecesA ? j : j - kPiecesA;
      const float* p = j < kPiecesA ? pa + min(m0 + jj * 16, g.M - 1) * g.lda
                       : (!KN ? pb + min(n0 + jj * 16, g.N - 1) * g.ldb : pb + min((chunk0 + chunk) * kBK + kb + jj * (256 / kRowN), g.K - 1) * g.ldb);
      if (tile < g.tiles) v[j] = __ldg(reinterpret_cast<const float4*>(p));
    };
    auto advance = [&]() {
      if (++chunk == chunks) {
        chunk = 0;
        tile += tile_step;
        start_tile();
      }
      place();
    };
#pragma unroll
    for (int j = 0; j < kPieces; ++j) request(j);
    advance();
    int it = 0;
    bool ok = true;
    for (int t = tile0; ok && t < g.tiles; t += tile_step)
      for (int i = 0; i < chunks; ++i, ++it) {
        const int s = it & 1;
        if (!mbar_wait(empty(s), ((it >> 1) & 1) ^ 1, g.err, DEVERR_GEMM_PRODUCER)) { ok = false; break; }
        uint8_t* stage = gen + s * C::kStage;
        if ((chunk0 + i) * kBK + kp >= g.K) {
#pragma unroll
          for (int j = 0; j < kPiecesA; ++j) v[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
#pragma unroll
        for (int j = 0; j < kPieces; ++j) {
          uint2 hi, mid, lo;
          split3(v[j].x, v[j].y, hi.x, mid.x, lo.x);
          split3(v[j].z, v[j].w, hi.y, mid.y, lo.y);
          request(j);  // the same piece of the next chunk
          // 128-byte swizzle: 16 bytes (two pieces) number q of row r at q ^ (r & 7)
          int off;
          if (j < kPiecesA || !KN) {
            const int r = (j < kPiecesA ? j : j - kPiecesA) * 16 + row;
            off = r * 128 + (((kp >> 3) ^ (r & 7)) << 4) + (kp & 4) * 2;
          } else {
            const int k = kb + (j - kPiecesA) * (256 / kRowN);
            off = (nb >> 6) * (kBK * 128) + k * 128 + ((((nb >> 3) & 7) ^ (k & 7)) << 4) + (nb & 4) * 2;
          }
          uint8_t* d = stage + (j < kPiecesA ? 0 : 3 * kTileA) + off;
          constexpr int kB = C::kTileB;
          const int step = j < kPiecesA ? kTileA : kB;
          *reinterpret_cast<uint2*>(d) = hi;
          *reinterpret_cast<uint2*>(d + step) = mid;
          *reinterpret_cast<uint2*>(d + 2 * step) = lo;
        }
        advance();
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(full(s));
      }
  } else {
    // ---- sums: a warp owns 32 rows (TMEM lanes of its quarter) and half of the columns ----
    constexpr int kCols = BN / 2, kStep = kCols < 32 ? 16 : 32;
    const int w = warp - kSplitWarps, quarter = warp & 3, col0 = (w >> 2) * kCols;
    // Products of chunk number n of this CTA, the largest last: what is cut off is relative to the sum so far.  Narrow tiles are bound by
    // the number of MMAs (one in 90 clocks at best into the same accumulator), so there the terms of B, which lie side by side, are
    // taken two at a time: mid x (hi, mid), lo x hi, hi x lo, hi x (hi, mid) are 16 MMAs instead of 24, into two parts that are
    // added in the registers (64 x 4096 x 4096, K not split: 85 -> 72 us; 128 wide the second part costs more than it saves, 418 -> 449 us
    // for 2048 x 4096 x 4096).
    const int total = (g.tiles - tile0 + tile_step - 1) / tile_step * chunks;
    auto issue = [&](int n) -> bool {
      const int s = n & 1;
      const uint32_t ph = (n >> 1) & 1;
      if (!mbar_wait(acc_empty(s), ph ^ 1, g.err, DEVERR_GEMM_MMA) || !mbar_wait(full(s), ph, g.err, DEVERR_GEMM_MMA)) return false;
      tc_fence_after();
      const uint32_t sa = base + s * C::kStage, sb = sa + 3 * kTileA, d = tmem + s * C::kAcc;
      // (term of A, first term of B, how many terms of B side by side, part of the accumulator)
      constexpr int kSteps[2][6][4] = {{{0, 2, 1, 0}, {2, 0, 1, 0}, {1, 1, 1, 0}, {1, 0, 1, 0}, {0, 1, 1, 0}, {0, 0, 1, 0}},
                                       {{1, 0, 2, 0}, {2, 0, 1, 0}, {0, 2, 1, 1}, {0, 0, 2, 0}}};
#pragma unroll
      for (int q = 0; q < (C::kParts == 1 ? 6 : 4); ++q) {
        const int* p = kSteps[C::kParts - 1][q];
        const uint32_t idesc = make_idesc_bf16(kBM, BN * p[2], false, KN);
        const uint64_t da = make_smem_desc_sw128(sa + p[0] * kTileA, 16, 1024);
        const uint64_t db = make_smem_desc_sw128(sb + p[1] * C::kTileB, KN ? kBK * 128 : 16, 1024);
#pragma unroll
        for (int k = 0; k < 4; ++k)  // 16 k: 32 bytes of a K-major row, 16 rows of an N-major tile
          umma_bf16_ss(d + p[3] * BN, da + 2 * k, db + (KN ? 128 : 2) * k, idesc, q + k > 0 ? 1u : 0u);
      }
      umma_commit(empty(s));
      umma_commit(acc_full(s));
      return true;
    };
    const f32x2 down = pack2(kDown, kDown);
    const bool issuer = w == 0 && lane == 0;
    if (issuer && total > 0) issue(0);
    __syncwarp();
    int it = 0, number = 0;
    bool ok = true;
    for (int t = tile0; ok && t < g.tiles; t += tile_step, ++number) {
      f32x2 acc[kCols / 2];
#pragma unroll
      for (int e = 0; e < kCols / 2; ++e) acc[e] = pack2(0.0f, 0.0f);
      for (int i = 0; i < chunks; ++i, ++it) {
        const int s = it & 1;
        if (issuer && it + 1 < total) issue(it + 1);
        __syncwarp();
        if (!mbar_wait(acc_full(s), (it >> 1) & 1, g.err, DEVERR_GEMM_EPILOGUE)) { ok = false; break; }
        tc_fence_after();
        const uint32_t addr = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + s * C::kAcc + col0;
#pragma unroll
        for (int c = 0; c < kCols; c += kStep) {
#pragma unroll
          for (int p = C::kParts - 1; p >= 0; --p) {
            uint32_t r[kStep];
            if constexpr (kStep == 32) tmem_ld_32x32(addr + p * BN + c, r); else tmem_ld_32x16(addr + p * BN + c, r);
            tmem_wait_ld();
#pragma unroll
            for (int e = 0; e < kStep; e += 2) acc[(c + e) / 2] = fma2(pack2(__uint_as_float(r[e]), __uint_as_float(r[e + 1])), down, acc[(c + e) / 2]);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty(s));
      }
      if (!ok) break;
      if (g.split > 1) {  // (one tile) the terms' place takes the sums: every MMA that read it is done
        float* dst = reinterpret_cast<float*>(gen) + (quarter * 32 + lane) * C::kPitch + col0;
#pragma unroll
        for (int e = 0; e < kCols; e += 4) {
          const float2 x = unpack2(acc[e / 2]), y = unpack2(acc[e / 2 + 1]);
          *reinterpret_cast<float4*>(dst + e) = make_float4(x.x, x.y, y.x, y.y);
        }
        continue;
      }
      const int tn = t / g.tiles_m, m = (t - tn * g.tiles_m) * kBM + quarter * 32 + lane, n0 = tn * BN + col0;
      bool bad = false;
#pragma unroll
      for (int e = 0; e < kCols; e += 4) {
        const float2 x = unpack2(acc[e / 2]), y = unpack2(acc[e / 2 + 1]);
        bad |= store4(g, m, n0 + e, make_float4(x.x, x.y, y.x, y.y));
      }
      if (bad) atomicOr(&again[(number >> 5) & 31], 1u << (number & 31));
    }
  }
  if (g.split > 1) {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    // this CTA finishes kBM / split rows of the tile: the parts added in the order of k
    const int rows = kBM / g.split, tn = tile0 / g.tiles_m, m0 = (tile0 - tn * g.tiles_m) * kBM;
    for (int u = tid; u < rows * (BN / 4); u += kThreads) {
      const int r = rank * rows + u / (BN / 4), n = u % (BN / 4) * 4;
      const uint32_t at = base + static_cast<uint32_t>(r * C::kPitch + n) * 4;
      float4 v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (q < g.split) v[q] = ld_cluster4(at, q);
      float4 x = v[0];
#pragma unroll
      for (int q = 1; q < 8; ++q)
        if (q < g.split) x = make_float4(x.x + v[q].x, x.y + v[q].y, x.z + v[q].z, x.w + v[q].w);
      if (store4(g, m0 + r, tn * BN + n, x)) atomicOr(&again[0], 1u);
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  __syncwarp();
  if (tid == 0) gave_up = *reinterpret_cast<volatile int*>(g.err) != 0;
  tc_fence_before();
  __syncthreads();
  if (warp == kSplitWarps) {
    if (gave_up) {
      // a wait gave up: let MMAs that are still in flight drain before the memory is released
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 2000000ull) __nanosleep(1000);
    }
    tc_fence_after();
    tmem_dealloc(tmem, C::kCols);
  }
  if (gave_up) return;
  // (the barrier above: every result is stored, every MMA and every CTA of the cluster is done with this shared memory)
  for (int t = tile0, number = 0; t < g.tiles; t += tile_step, ++number) {
    if (!((again[(number >> 5) & 31] >> (number & 31)) & 1u)) continue;
    const int tn = t / g.tiles_m, m0 = (t - tn * g.tiles_m) * kBM + rank * (kBM / g.split), n0 = tn * BN;
    float* sm = reinterpret_cast<float*>(gen);
    switch (g.split) {
      case 1: sum_again<BN, KN, 8>(g, sm, m0, n0); break;
      case 2: sum_again<BN, KN, 4>(g, sm, m0, n0); break;
      case 4: sum_again<BN, KN, 2>(g, sm, m0, n0); break;
      default: sum_again<BN, KN, 1>(g, sm, m0, n0); break;
    }
  }
}

template <int BN, bool KN>
int prepare_tc() {
  static std::atomic<unsigned long long> done{0};  // one bit per device; threads may race to set it
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64 || !((done.load(std::memory_order_acquire) >> dev) & 1ull)) {
    const cudaError_t e = cudaFuncSetAttribute(gemm_f32_tc_kernel<BN, KN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<BN>::kSmem);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (dev < 64) done.fetch_or(1ull << dev, std::memory_order_release);
  }
  return 0;
}

template <int BN, bool KN>
int launch_tc(const F32Args& g, int grid, cudaStream_t st) {
  const int rc = prepare_tc<BN, KN>();
  if (rc) return rc;
  return launch_kernel(gemm_f32_tc_kernel<BN, KN>, dim3(grid), dim3(kThreads), Cfg<BN>::kSmem, st, g.split, g);
}

// Tile width, K split and the clocks they are estimated to take.  Measured: 3100, 2250 and 1980 clocks for 64 k of a tile 128, 64 and 32
// wide, 8000 to start and to finish, 2000 for the parts of a split K to meet (512^3, [K][N]: 15.8, 11.9, 9.8 us with one, two and
// four parts of 64-wide tiles).  One CTA fills an SM, and clusters of eight such CTAs find place on about half of the SMs only
// (8 x 64 CTAs one after the other: 7.7 us; 8 x 128: 12.5).
struct Choice { int bn, split, per; double clocks; };
Choice choose(int M, int N, int K, bool kn, int sms) {
  Choice best{};
  const int chunks = (K + kBK - 1) / kBK;
  const long long tiles_m = (M + kBM - 1) / kBM;
  for (int bn = 128; bn >= (kn ? 64 : 32); bn >>= 1) {
    const long long tiles = tiles_m * ((N + bn - 1) / bn);
    for (int split = 1; split <= 8; split <<= 1) {
      const int per = (chunks + split - 1) / split;
      if (split > 1 && (tiles * split > (split == 8 ? sms / 2 : sms) || per * (split - 1) >= chunks)) break;
      const double t = static_cast<double>((tiles + sms - 1) / sms) * per * (bn == 128 ? 3100.0 : (bn == 64 ? 2250.0 : 1980.0)) +
                       8000.0 + (split > 1 ? 2000.0 : 0.0);
      if (!best.bn || t < best.clocks) best = Choice{bn, split, per, t};
    }
  }
  return best;
}

}  // namespace

// A [M][K] with k contiguous and B as [N][K] or [K][N] with its second index contiguous, rows of whole 16-byte vectors.
bool gemm_f32_tc_takes(const float* a, long long sam, long long sak, const float* b, long long sbk, long long sbn, int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0) return false;
  if (((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15) || sak != 1 || sam % 4 || K % 4) return false;
  if (static_cast<long long>((M + kBM - 1) / kBM) * ((N + 31) / 32) > 0x7fffffffLL) return false;
  return (sbk == 1 && sbn % 4 == 0) || (sbn == 1 && sbk % 4 == 0 && N % 4 == 0);
}

int gemm_f32_tc_prepare() {
  int rc = 0;
  if ((rc = prepare_tc<128, false>()) || (rc = prepare_tc<64, false>()) || (rc = prepare_tc<32, false>()) || (rc = prepare_tc<128, true>()) ||
      (rc = prepare_tc<64, true>()))
    return rc;
  return 0;
}

double gemm_f32_tc_clocks(long long sbk, int M, int N, int K) { return choose(M, N, K, sbk != 1, sm_count()).clocks; }

int gemm_f32_tc(const float* a, long long sam, const float* b, long long sbk, long long sbn, const float* bias, float* c, long long scm,
                long long scn, int M, int N, int K, cudaStream_t st) {
  if (!a || !b || !c || !gemm_f32_tc_takes(a, sam, 1, b, sbk, sbn, M, N, K)) return TEENY_ERR_BAD_ARG;
  F32Args g{};
  const bool kn = sbk != 1;
  g.a = a; g.b = b; g.bias = bias; g.c = c;
  g.lda = sam; g.ldb = kn ? sbk : sbn;
  g.scm = scm; g.scn = scn;
  g.M = M; g.N = N; g.K = K;
  g.err = device_error_word();
  if (!g.err) return TEENY_ERR_DRIVER;
  const int sms = sm_count();
  const Choice x = choose(M, N, K, kn, sms);
  g.tiles_m = (M + kBM - 1) / kBM;
  g.tiles = g.tiles_m * ((N + x.bn - 1) / x.bn);
  g.split = x.split;
  g.per = x.per;
  const int grid = x.split > 1 ? g.tiles * x.split : (g.tiles < sms ? g.tiles : sms);
  if (kn) return x.bn == 128 ? launch_tc<128, true>(g, grid, st) : launch_tc<64, true>(g, grid, st);
  return x.bn == 128 ? launch_tc<128, false>(g, grid, st) : (x.bn == 64 ? launch_tc<64, false>(g, grid, st) : launch_tc<32, false>(g, grid, st));
}

}  // namespace teeny
