// Attention with f32 scores, probabilities and sums on the tensor cores: f32 operands, and bf16 operands whose head size the bf16 kernel
// (attention_prefill.cu) does not take.  Head sizes up to 128 in multiples of 8, grouped-query, optionally causal.
//
// Numbers are taken as in gemm_f32_tc.cu: an f32 number is the sum of three bf16 numbers, hi + mid + lo, and a product the six largest of
// the nine products of such terms (bf16 operands are one term, their probabilities three).  The tensor cores' accumulator cuts off instead
// of rounding, so it holds short sums only: a score (at most 128 products), and the values of one tile of keys, which are
// then added to f32 registers, rounded.
//
// A CTA has 128 query rows of a head and walks the keys in tiles of 8192 / D.  Roles: 8 warps load K and V, split them and store the
// swizzled terms (48 KB a tile and operand; the others do so for Q meanwhile); one lane issues the scores' MMAs and one the values'; 8 warps hold the rows, two threads
// a row with half of the tile's keys and half of the head's dimensions each: scores from tensor memory, one exponential per
// score, probabilities as three terms back to tensor memory, where the MMA reads them as its A operand.  They do so in two
// chunks with a barrier of their own, so that the next tile's first chunk is written while the products of the second one run.
// With a head size of 64, terms of V lie side by side and are taken by one MMA of 128 columns into two accumulators: an MMA of 64 columns
// takes no less time to issue.
//
// Both operands are taken times 2^24 and so are the probabilities, for the terms of small numbers to stay normal bf16 numbers.  At the
// other end, operands from 2^104 on, scores from 2^79 on, infinities and NaNs give rows that are not finite; these are made again by the
// same CTA with the CUDA-core tile.  So is a row of a causal tile in which a key that it must not see has such a value (0 times it is not 0).
//
// Bound: the issue slots.  A tile of 128 keys (D = 64) is 3100 clocks of the tensor pipe at its best and about 3400 issue slots of each scheduler, half of them
// the split of K and V, which every CTA of a head repeats; 5200 are taken, the chain being the split of a key tile, its 24 MMAs, and the next split into
// the same place (both operands of one tile twice do not fit beside Q).  With two places for K and one for V a tile took 7000 clocks.
// Measured on B200 back to back against the CUDA-core kernel, f32, 32 heads x 1000 x 1000: D = 64 278 -> 59.5 us (called alone 288 -> 66.7), error against 64 bits
// 6.0e-7 -> 1.9e-7, D = 128 560 -> 131 us, 6.0e-7 -> 1.9e-7; 8 heads x 300 x 300, D = 64 37 -> 15.8 us, 3.6e-7 -> 1.7e-7; bf16, 32 heads x 1000 x 1000, D = 64 312 ->
// 41 us.  Tensor pipe 42 % active (D = 128 39 %).  f32 with D = 128 spills 36 bytes a thread (stored; 88 loaded), the others none.
#include <atomic>
#include <cmath>
#include <type_traits>
#include <utility>

#include "attention_simt.cuh"
#include "mma.cuh"

namespace teeny {

namespace {

constexpr int kRows = 128;
constexpr int kRowWarps = 8, kSplitWarps = 8;
constexpr int kThreads = 32 * (kRowWarps + kSplitWarps + 4);  // the last four: two issue, two fill the warpgroup
constexpr int kRowRegs = 152, kSplitRegs = 64, kIssueRegs = 48;  // of 5 x 96: 2 x 152 + 2 x 64 + 48
constexpr float kUp = 0x1p24f;

// NT: terms of an operand.  D: head size, padded.
template <int NT, int D> struct Cfg {
  static constexpr int kKeys = 8192 / D;
  static constexpr int kChunks = D / 64;                         // 64 dimensions: rows of 128 bytes
  static constexpr int kTermQ = kRows * 128, kTermK = kKeys * 128;  // one term of 64 dimensions
  static constexpr int kQ = NT * kChunks * kTermQ, kTile = NT * kChunks * kTermK;
  static constexpr int kStagesK = NT == 3 ? 1 : 2, kStagesV = NT == 3 && D == 128 ? 1 : 2;
  static constexpr int kTerms = kQ + (kStagesK + kStagesV) * kTile;
  static constexpr bool kPairV = NT == 3 && D == 64;
  // Accumulators of a value: the products of the hi terms have one of their own, for every MMA into it costs a cut at its size
  static constexpr int kSumsV = NT == 1 ? 1 : (kPairV ? 3 : 2);
  static constexpr int kColS = kChunks * kKeys, kColP = 3 * kKeys / 2, kColO = kSumsV * D;  // a score has one for 64 dimensions
  static constexpr int kAtP = kColS, kAtO = kAtP + kColP;
  static_assert(kAtO + kColO <= 512, "tensor memory");
  // CUDA-core tiles of 32 rows by 128 threads each, in the place of the terms
  using Again = attn_simt::TileCfg<2, D / 64>;
  static constexpr int kGroups = 2 * Again::kSmemBytes <= kTerms ? 2 : 1;
  static_assert(Again::kSmemBytes <= kTerms, "fits");
  static constexpr int kBars = kTerms, kXch = kBars + 256, kSmem = kXch + 4 * kRows * 4 + 1024;
};

struct Args {
  const void *q, *k, *v;
  void* o;
  float* lse;
  AttnShape s;
  float to_log2;  // scale, log2(e) and the operands' factors: from a score in tensor memory to an exponent
  float from_o;   // the factors of the values' sums taken back
  int row_tiles;
  bool vec_out;
  int* err;
};

template <typename F, int... I>
__device__ __forceinline__ void each(std::integer_sequence<int, I...>, F f) { (f(std::integral_constant<int, I>{}), ...); }

// A tile of ROWS rows of one operand: loaded (`request`) in 16-byte pieces, a warp's side by side in memory, and stored as terms.
// Rows behind the last one are read from the last one (their scores are masked, their query rows not stored), dimensions behind D are zeros.
template <typename T, int NT, int D, int ROWS>
struct Operand {
  static constexpr int kPiece = 16 / sizeof(T), kPerRow = D / kPiece, kPieces = ROWS * kPerRow / (32 * kSplitWarps);
  static constexpr int kTerm = ROWS * 128;
  static __device__ __forceinline__ uint4 load(const T* base, long long stride, int row0, int rows, int dims, int tid, int j) {
    const int p = j * 32 * kSplitWarps + tid, row = p / kPerRow, d = p % kPerRow * kPiece;
    if (d >= dims) return make_uint4(0u, 0u, 0u, 0u);
    return __ldg(reinterpret_cast<const uint4*>(base + static_cast<long long>(min(row0 + row, rows - 1)) * stride + d));
  }
  static __device__ __forceinline__ void store(uint8_t* dst, const uint4 x, int tid, int j) {
    const int p = j * 32 * kSplitWarps + tid, row = p / kPerRow, d = p % kPerRow * kPiece;
    // [64 dimensions][term][row][128 bytes], 16-byte units swizzled
    uint8_t* to = dst + (d >> 6) * (NT * kTerm) + row * 128 + ((((d & 63) >> 3) ^ (row & 7)) << 4);
    if constexpr (NT == 1) {
      *reinterpret_cast<uint4*>(to) = x;
    } else {
      const f32x2 up = pack2(kUp, kUp);
      uint2 hi, mid, lo;
      bf16_terms3(mul2(pack2(__uint_as_float(x.x), __uint_as_float(x.y)), up), hi.x, mid.x, lo.x);
      bf16_terms3(mul2(pack2(__uint_as_float(x.z), __uint_as_float(x.w)), up), hi.y, mid.y, lo.y);
      to += (d & 4) * 2;
      *reinterpret_cast<uint2*>(to) = hi;
      *reinterpret_cast<uint2*>(to + kTerm) = mid;
      *reinterpret_cast<uint2*>(to + 2 * kTerm) = lo;
    }
  }
};

// Products, the smallest first (what is cut off is relative to the sum so far): term of A, first term of B, terms of B side by side, which
// accumulator they go to (the second term of a pair to the one behind it).
struct Product { int a, b, n, sum; };
__host__ __device__ constexpr int products(int na, int nb, int sums) { return sums == 3 ? 4 : (na == 3 && nb == 3 ? 6 : na * nb); }
__host__ __device__ constexpr Product product(int na, int nb, int sums, int i) {
  constexpr Product six[6] = {{0, 2, 1, 1}, {2, 0, 1, 1}, {1, 1, 1, 1}, {1, 0, 1, 1}, {0, 1, 1, 1}, {0, 0, 1, 0}};
  constexpr Product four[4] = {{1, 0, 2, 1}, {0, 1, 2, 1}, {2, 0, 1, 2}, {0, 0, 1, 0}};
  if (sums == 3) return four[i];
  Product p = nb == 3 ? six[i] : Product{na - 1 - i, 0, 1, 0};
  if (sums == 1) p.sum = 0;
  return p;
}
// whether product i is the first one into its accumulator
__host__ __device__ constexpr bool opens(int na, int nb, int sums, int i) {
  const Product p = product(na, nb, sums, i);
  for (int e = 0; e < i; ++e) {
    const Product o = product(na, nb, sums, e);
    if (p.sum >= o.sum && p.sum < o.sum + o.n) return false;
  }
  return true;
}

template <typename T, int NT, int D>
__global__ void __launch_bounds__(kThreads, 1) attention_f32_tc_kernel(const __grid_constant__ Args g) {
  using C = Cfg<NT, D>;
  using OpQ = Operand<T, NT, D, kRows>;
  using OpK = Operand<T, NT, D, C::kKeys>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  auto bar = [&](int i) { return base + C::kBars + 8u * i; };
  constexpr int Q_FULL = 0, K_FULL = 1, K_EMPTY = K_FULL + 2, V_FULL = K_EMPTY + 2, V_EMPTY = V_FULL + 2, S_FULL = V_EMPTY + 2,
                S_EMPTY = S_FULL + 1, P_FULL = S_EMPTY + 1, P_EMPTY = P_FULL + 2, O_FULL = P_EMPTY + 1, O_EMPTY = O_FULL + 1, kNumBars = O_EMPTY + 1;
  static_assert(8 * kNumBars + 8 <= 256, "barrier block");
  float* xch = reinterpret_cast<float*>(gen + C::kXch);  // [2 (tile parity)][2 halves][kRows]
  __shared__ unsigned again[4], failed, gave_up;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const AttnShape& s = g.s;
  const int tile = g.row_tiles - 1 - static_cast<int>(blockIdx.x % g.row_tiles);  // the longest rows (causal) start first
  const int h = static_cast<int>(blockIdx.x / g.row_tiles) % s.Hq, b = static_cast<int>(blockIdx.x / g.row_tiles) / s.Hq;
  const int hk = h / (s.Hq / s.Hkv), row0 = tile * kRows, shift = s.Skv - s.Sq;
  const int keys = s.causal ? min(s.Skv, min(row0 + kRows, s.Sq) + shift) : s.Skv;
  const int n = (keys + C::kKeys - 1) / C::kKeys;

  if (tid < 4) again[tid] = 0;
  if (tid == 4) failed = 0;
  if (tid == 0) {
    for (int i = 0; i < kNumBars; ++i) {
      uint32_t count = 1;
      if ((i >= K_FULL && i < K_EMPTY) || (i >= V_FULL && i < V_EMPTY)) count = kSplitWarps;
      else if (i == Q_FULL || i == S_EMPTY || i == P_FULL || i == P_FULL + 1 || i == O_EMPTY) count = kRowWarps;
      mbar_init(bar(i), count);
    }
    mbar_fence_init();
  }
  const uint32_t tmem_slot = base + C::kBars + 8u * kNumBars;
  if (warp == kRowWarps + kSplitWarps) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(gen + C::kBars + 8 * kNumBars);
  const uint32_t sm_q = base, sm_k = base + C::kQ, sm_v = sm_k + C::kStagesK * C::kTile;
  pdl_wait();

  if (warp >= kRowWarps + kSplitWarps) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kIssueRegs));
    const int role = warp - kRowWarps - kSplitWarps;
    if (role == 0 && lane == 0) {
      // ---- scores: S = Q K^T ----
      constexpr int kProducts = products(NT, NT, 1);
      bool ok = mbar_wait(bar(Q_FULL), 0, g.err, DEVERR_ATTN_MMA);
      for (int j = 0; ok && j < n; ++j) {
        const int st = j % C::kStagesK;
        if (!mbar_wait(bar(K_FULL + st), (j / C::kStagesK) & 1, g.err, DEVERR_ATTN_MMA) ||
            !mbar_wait(bar(S_EMPTY), (j & 1) ^ 1, g.err, DEVERR_ATTN_MMA)) break;
        tc_fence_after();
        const uint64_t dq = make_smem_desc_sw128(sm_q, 16, 1024), dk = make_smem_desc_sw128(sm_k + st * C::kTile, 16, 1024);
        each(std::make_integer_sequence<int, kProducts * C::kChunks * 4>{}, [&](auto number) {
          constexpr int i = number / (4 * C::kChunks), c = number / 4 % C::kChunks, k = number % 4;  // k: 16 dimensions, 32 bytes of a row
          constexpr Product of = product(NT, NT, 1, i);
          umma_ss_at<(c * NT + of.a) * C::kTermQ / 16 + 2 * k, (c * NT + of.b) * C::kTermK / 16 + 2 * k>(
              tmem + c * C::kKeys, dq, dk, make_idesc_bf16(kRows, C::kKeys * of.n, false, false), i + k > 0 ? 1u : 0u);
        });
        umma_commit(bar(K_EMPTY + st));
        umma_commit(bar(S_FULL));
      }
    } else if (role == 1 && lane == 0) {
      // ---- values: O = P V, the tile's keys in two chunks (a quarter of the keys from each half) ----
      constexpr int kProducts = products(3, NT, C::kSumsV);
      constexpr int kSteps = C::kKeys / 64;  // of 16 keys, per chunk and half
      for (int j = 0; j < n; ++j) {
        const int st = j % C::kStagesV;
        bool ok = mbar_wait(bar(V_FULL + st), (j / C::kStagesV) & 1, g.err, DEVERR_ATTN_MMA) &&
                  mbar_wait(bar(O_EMPTY), (j & 1) ^ 1, g.err, DEVERR_ATTN_MMA);
        const uint64_t dv = make_smem_desc_sw128(sm_v + st * C::kTile, C::kPairV ? C::kTermK : NT * C::kTermK, 1024);
        each(std::make_integer_sequence<int, 2>{}, [&](auto c) {
          ok = ok && mbar_wait(bar(P_FULL + c), j & 1, g.err, DEVERR_ATTN_MMA);
          if (!ok) return;
          tc_fence_after();
          each(std::make_integer_sequence<int, kProducts * 2 * kSteps>{}, [&](auto number) {
            constexpr int i = number / (2 * kSteps), k = number % (2 * kSteps);
            constexpr int key = (k / kSteps) * (C::kKeys / 2) + c * (C::kKeys / 4) + k % kSteps * 16;
            constexpr Product of = product(3, NT, C::kSumsV, i);
            umma_ts_at<of.a * (C::kKeys / 2) + key / 2, (of.b * C::kTermK + key * 128) / 16>(
                tmem + C::kAtO + of.sum * D, tmem + C::kAtP, dv, make_idesc_bf16(kRows, D * of.n, false, true), c + k > 0 || !opens(3, NT, C::kSumsV, i) ? 1u : 0u);
          });
          if (c == 0) umma_commit(bar(P_EMPTY));
        });
        if (!ok) break;
        umma_commit(bar(V_EMPTY + st));
        umma_commit(bar(O_FULL));
      }
    }
  } else if (warp >= kRowWarps) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kSplitRegs));
    // ---- loads and terms of K and V, tile by tile ----
    const int t = tid - 32 * kRowWarps;
    const T* kv[2] = {static_cast<const T*>(g.k) + b * s.k_sb + hk * s.k_sh, static_cast<const T*>(g.v) + b * s.v_sb + hk * s.v_sh};
    const long long stride[2] = {s.k_ss, s.v_ss};
    constexpr int kN = OpK::kPieces;
    uint4 x[kN];
#pragma unroll
    for (int i = 0; i < kN; ++i) x[i] = OpK::load(kv[0], stride[0], 0, s.Skv, s.D, t, i);
    bool ok = true;
    for (int j = 0; ok && j < n; ++j) {
#pragma unroll
      for (int op = 0; op < 2; ++op) {
        const int stages = op ? C::kStagesV : C::kStagesK, st = j % stages;
        if (!mbar_wait(bar((op ? V_EMPTY : K_EMPTY) + st), ((j / stages) & 1) ^ 1, g.err, DEVERR_ATTN_PRODUCER)) { ok = false; break; }
        uint8_t* dst = gen + C::kQ + (op ? C::kStagesK * C::kTile : 0) + st * C::kTile;
        const bool more = !op || j + 1 < n;
#pragma unroll
        for (int i = 0; i < kN; ++i) {
          OpK::store(dst, x[i], t, i);
          if (more) x[i] = OpK::load(kv[op ^ 1], stride[op ^ 1], (j + op) * C::kKeys, s.Skv, s.D, t, i);  // V of this tile or K of the next
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar((op ? V_FULL : K_FULL) + st));
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRowRegs));
    {  // the terms of Q, beside the first keys
      const T* q = static_cast<const T*>(g.q) + b * s.q_sb + h * s.q_sh;
      constexpr int kN = 8;
#pragma unroll
      for (int part = 0; part < OpQ::kPieces; part += kN) {
        uint4 x[kN];
#pragma unroll
        for (int i = 0; i < kN; ++i)
          if (part + i < OpQ::kPieces) x[i] = OpQ::load(q, s.q_ss, row0, s.Sq, s.D, tid, part + i);
#pragma unroll
        for (int i = 0; i < kN; ++i)
          if (part + i < OpQ::kPieces) OpQ::store(gen, x[i], tid, part + i);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(Q_FULL));
    }
    // ---- rows: thread = (row, half of the keys and of the dimensions) ----
    constexpr int kHalf = C::kKeys / 2, kDims = D / 2;
    const int quarter = warp & 3, half = warp >> 2, r = quarter * 32 + lane;
    const uint32_t lanes = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
    const int last = s.causal ? min(s.Skv - 1, row0 + r + shift) : s.Skv - 1;
    f32x2 acc[kDims / 2];
#pragma unroll
    for (int e = 0; e < kDims / 2; ++e) acc[e] = pack2(0.0f, 0.0f);
    float m = -INFINITY, neg = INFINITY, l = 0.0f;
    f32x2 check = pack2(0.0f, 0.0f);  // the sum of all scores: a sum of products that overflowed on the way may end as a probability of zero
    bool ok = true;
    // After a wait that gave up a warp goes on without waiting (nothing is stored then), for it meets the others at barriers.
    auto wait = [&](int i, uint32_t parity) { if (ok) ok = __all_sync(0xffffffffu, mbar_wait(bar(i), parity, g.err, DEVERR_ATTN_SOFTMAX)); };
    // the sums of a tile of keys, at the scale of the maximum so far, join the registers, which go on at `corr` times that scale
    auto take_sums = [&](float corr) {
      constexpr int kStep = D == 64 ? 32 : 16;  // (as many as the registers hold)
      tc_fence_after();
      const bool same = __all_sync(0xffffffffu, corr == 1.0f);
      const f32x2 one = pack2(1.0f, 1.0f), cc = pack2(corr, corr);
#pragma unroll
      for (int c = 0; c < kDims; c += kStep) {
#pragma unroll
        for (int i = C::kSumsV - 1; i >= 0; --i) {
          uint32_t x[kStep];
          if constexpr (kStep == 32) tmem_ld_32x32(lanes + C::kAtO + i * D + half * kDims + c, x);
          else tmem_ld_32x16(lanes + C::kAtO + i * D + half * kDims + c, x);
          tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < kStep; e += 2)
            acc[(c + e) / 2] = fma2(pack2(__uint_as_float(x[e]), __uint_as_float(x[e + 1])), one, acc[(c + e) / 2]);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(O_EMPTY));
      if (!same) {
#pragma unroll
        for (int e = 0; e < kDims / 2; ++e) acc[e] = mul2(acc[e], cc);
      }
    };
    for (int j = 0; j < n; ++j) {
      wait(S_FULL, j & 1);
      tc_fence_after();
      float x[kHalf];
#pragma unroll
      for (int c = 0; c < kHalf; c += 32) {
        uint32_t y[32];
        tmem_ld_32x32(lanes + half * kHalf + c, y);
        tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < 32; ++e) x[c + e] = __uint_as_float(y[e]);
        if constexpr (C::kChunks == 2) {
          tmem_ld_32x32(lanes + C::kKeys + half * kHalf + c, y);
          tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 32; ++e) x[c + e] += __uint_as_float(y[e]);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(S_EMPTY));
#pragma unroll
      for (int e = 0; e < kHalf; e += 2) check = fma2(pack2(x[e], x[e + 1]), pack2(1.0f, 1.0f), check);
      const int k0 = j * C::kKeys;
      if (k0 + C::kKeys > s.Skv || (s.causal && k0 + C::kKeys - 1 > row0 + shift)) {
#pragma unroll
        for (int e = 0; e < kHalf; ++e)
          if (k0 + half * kHalf + e > last) x[e] = -INFINITY;
      }
      float top[4] = {x[0], x[1], x[2], x[3]};
#pragma unroll
      for (int e = 4; e < kHalf; e += 4)
#pragma unroll
        for (int i = 0; i < 4; ++i) top[i] = fmaxf(top[i], x[e + i]);
      const float mine = fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3]));
      float* at = xch + (j & 1) * 2 * kRows + r;
      at[half * kRows] = mine;
      named_barrier_sync(1 + quarter, 64);
      m = fmaxf(m, fmaxf(mine, at[(half ^ 1) * kRows]));
      const float neg_now = -(m * g.to_log2);
      const float corr = ex2(neg_now - neg);
      neg = neg_now;
      l *= corr;
      const f32x2 cc = pack2(g.to_log2, g.to_log2), nn = pack2(neg, neg), up = pack2(kUp, kUp);
      f32x2 sum = pack2(0.0f, 0.0f);
      const f32x2 one = pack2(1.0f, 1.0f);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
#pragma unroll
        for (int e0 = c * (kHalf / 2); e0 < (c + 1) * (kHalf / 2); e0 += 16) {
          uint32_t hi[8], mid[8], lo[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const float2 z = unpack2(fma2(pack2(x[e0 + 2 * e], x[e0 + 2 * e + 1]), cc, nn));
            const f32x2 p = pack2(ex2(z.x), ex2(z.y));
            sum = fma2(p, one, sum);
            bf16_terms3(mul2(p, up), hi[e], mid[e], lo[e]);
          }
          if (c == 0 && e0 == 0 && j > 0) {
            wait(P_EMPTY, (j & 1) ^ 1);
            tc_fence_after();
          }
          const uint32_t to = lanes + C::kAtP + (half * kHalf + e0) / 2;
          tmem_st_32x8(to, hi);
          tmem_st_32x8(to + C::kKeys / 2, mid);
          tmem_st_32x8(to + C::kKeys, lo);
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(P_FULL + c));
        if (c == 0 && j > 0) {  // the second chunk's place is free once the sums are there
          wait(O_FULL, (j & 1) ^ 1);
          take_sums(corr);
        }
      }
      const float2 two = unpack2(sum);
      l += two.x + two.y;
    }
    wait(O_FULL, (n & 1) ^ 1);
    take_sums(1.0f);
    if (!ok) failed = 1;
    // both halves' sums of probabilities
    xch[half * kRows + r] = l;  // (the buffer of an even tile number: the last tile's other one is read no more behind this barrier)
    named_barrier_sync(5, 32 * kRowWarps);
    const int i = row0 + r;
    const float sum = xch[r] + xch[kRows + r];
    if (!failed) {
      const float2 seen = unpack2(check);
      bool bad = !(sum > 0.0f && sum < INFINITY) || !isfinite(seen.x + seen.y);
      // Quotients by one reciprocal and a correction: a division takes the long way around for the zeros of a padded head
      const float inv = 1.0f / sum;
      const f32x2 from = pack2(g.from_o, g.from_o), by = pack2(inv, inv), minus = pack2(-sum, -sum);
      auto quotient = [&](f32x2 a) {
        const f32x2 x = mul2(a, from), y = mul2(x, by);
        return unpack2(fma2(fma2(minus, y, x), by, y));
      };
      T* out = static_cast<T*>(g.o) + b * s.o_sb + h * s.o_sh + half * kDims;
      const int dims = s.D - half * kDims;
      // A row through the place of the terms (every MMA is done with them), so that a warp stores whole rows instead of 16 bytes of each of 32
      constexpr int kRowBytes = kDims * sizeof(T), kPitch = kRowBytes + 16, kPer = 16 / sizeof(T);
      uint8_t* box = gen + warp * 32 * kPitch;
#pragma unroll
      for (int e = 0; e < kDims / 2; e += kPer / 2) {
        float y[kPer];
#pragma unroll
        for (int q = 0; q < kPer; q += 2) {
          const float2 z = quotient(acc[e + q / 2]);
          y[q] = z.x;
          y[q + 1] = z.y;
        }
#pragma unroll
        for (int q = 0; q < kPer; ++q) bad |= !isfinite(y[q]) && 2 * e + q < dims;
        if (g.vec_out) {
          uint4 w;
          if constexpr (NT == 3) w = make_uint4(__float_as_uint(y[0]), __float_as_uint(y[1]), __float_as_uint(y[2]), __float_as_uint(y[3]));
          else w = make_uint4(pack_bf16x2(y[0], y[1]), pack_bf16x2(y[2], y[3]), pack_bf16x2(y[4], y[5]), pack_bf16x2(y[6], y[7]));
          *reinterpret_cast<uint4*>(box + lane * kPitch + e * 2 * sizeof(T)) = w;
        } else if (i < s.Sq) {
#pragma unroll
          for (int q = 0; q < kPer; ++q)
            if (2 * e + q < dims) attn_simt::store1(out + static_cast<long long>(i) * s.o_ss + 2 * e + q, y[q]);
        }
      }
      if (g.vec_out) {
        __syncwarp();
        constexpr int kLanes = kRowBytes / 16;
#pragma unroll 4
        for (int at = lane; at < 32 * kLanes; at += 32) {
          const int rr = at / kLanes, d = at % kLanes * kPer, row = row0 + quarter * 32 + rr;
          if (row < s.Sq && d < dims)
            *reinterpret_cast<uint4*>(out + static_cast<long long>(row) * s.o_ss + d) = *reinterpret_cast<const uint4*>(box + rr * kPitch + d * sizeof(T));
        }
      }
      if (g.lse && half == 0 && i < s.Sq) {  // maximum + log of the sum; the roundings of the product and of the sum join the result's own
        constexpr float kLn2 = 0.693147180559945309f, kRest = static_cast<float>(0.693147180559945309 - static_cast<double>(kLn2));
        const float top = -neg * kLn2, rest = fmaf(-neg, kRest, fmaf(-neg, kLn2, -top));
        const float lg = logf(sum), both = top + lg, part = both - top;
        const float y = both + (rest + ((top - (both - part)) + (lg - part)));
        g.lse[(static_cast<long long>(b) * s.Hq + h) * s.Sq + i] = y;
        bad |= !isfinite(y);
      }
      if (bad && i < s.Sq) atomicOr(&again[r >> 5], 1u << (r & 31));
    }
    named_barrier_sync(5, 32 * kRowWarps);  // every row is stored, every MMA is done with this shared memory
    const int group = warp >> 2;
    if (!failed && group < C::kGroups) {
      float* sm = reinterpret_cast<float*>(gen) + group * (C::Again::kSmemBytes / 4);
      for (int part = group; part < 4; part += C::kGroups) {
        if (!again[part]) continue;
        attn_simt::attention_tile<T, 2, D / 64, true>(static_cast<const T*>(g.q), static_cast<const T*>(g.k), static_cast<const T*>(g.v),
                                                      static_cast<T*>(g.o), g.lse, s, row0 + part * 32, h, b, true, tid & 127, sm, 6 + group, again[part]);
        named_barrier_sync(6 + group, 128);
      }
    }
  }
  __syncwarp();
  if (tid == 0) gave_up = *reinterpret_cast<volatile int*>(g.err) != 0;
  tc_fence_before();
  __syncthreads();
  if (warp == kRowWarps + kSplitWarps) {
    if (gave_up) {
      // a wait gave up: let MMAs that are still in flight drain before the memory is released
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 2000000ull) __nanosleep(1000);
    }
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

template <typename T, int NT, int D>
int launch(const Args& g, cudaStream_t st) {
  using C = Cfg<NT, D>;
  static std::atomic<unsigned long long> done{0};  // one bit per device; threads may race to set it
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64 || !((done.load(std::memory_order_acquire) >> dev) & 1ull)) {
    const cudaError_t e = cudaFuncSetAttribute(attention_f32_tc_kernel<T, NT, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmem);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (dev < 64) done.fetch_or(1ull << dev, std::memory_order_release);
  }
  const long long blocks = static_cast<long long>(g.row_tiles) * g.s.Hq * g.s.B;
  if (blocks > 0x7fffffffLL) return TEENY_ERR_BAD_ARG;
  return launch_kernel(attention_f32_tc_kernel<T, NT, D>, dim3(static_cast<unsigned>(blocks)), dim3(kThreads), C::kSmem, st, 1, g);
}

}  // namespace

template <typename T>
int attention_f32_tc(const T* q, const T* k, const T* v, T* o, float* lse, const AttnShape& s, cudaStream_t stream) {
  constexpr int kTerms = sizeof(T) == 4 ? 3 : 1;
  Args g{};
  g.q = q; g.k = k; g.v = v; g.o = o; g.lse = lse; g.s = s;
  // The accumulator cuts off at every MMA, which leaves a score short by part of a half-ulp on average.  What counts are the MMAs of the largest products, one
  // for 16 dimensions up to the four of an accumulator (zeros behind the head cut nothing off); two bf16 numbers' products are exact and the first sums of
  // them mostly so, the f32 operands' hi products meet a sum of the smaller ones from the first on.  Mean shortfall of logsumexp, 1000 keys, scores up to 4 sqrt(D),
  // the rounding of the scale taken off, D = 8, 16, 32, 64, 128: f32 4.2, 3.8, 5.2, 6.3, 6.5e-8, bf16 1.4, 1.8, 3.7, 5.5, - e-8.
  const int cuts = s.D >= 64 ? 4 : (s.D + 15) / 16;
  const double shortfall = kTerms == 3 ? 3.2e-8 + 0.8e-8 * cuts : 1.4e-8 * cuts;
  g.to_log2 = static_cast<float>(static_cast<double>(s.scale) * 1.4426950408889634 * (1.0 + shortfall) * (kTerms == 3 ? 0x1p-48 : 1.0));
  g.from_o = kTerms == 3 ? 0x1p-48f : 0x1p-24f;
  g.row_tiles = (s.Sq + kRows - 1) / kRows;
  g.vec_out = (s.o_sb | s.o_sh | s.o_ss) % static_cast<long long>(16 / sizeof(T)) == 0 && !(reinterpret_cast<uintptr_t>(o) & 15);
  g.err = device_error_word();
  if (!g.err) return TEENY_ERR_DRIVER;
  if (s.D <= 64) return launch<T, kTerms, 64>(g, stream);
  return launch<T, kTerms, 128>(g, stream);
}
template int attention_f32_tc<float>(const float*, const float*, const float*, float*, float*, const AttnShape&, cudaStream_t);
template int attention_f32_tc<bf16>(const bf16*, const bf16*, const bf16*, bf16*, float*, const AttnShape&, cudaStream_t);

// Waves of CTAs (one on an SM), each its start and its tiles of keys (measured: 16 to 640 keys, 1 to 6 waves).  The rule that compares it with the
// CUDA-core kernel's (attention_simt.cu) takes the slower of the two in 17 of 490 calls of random sizes, by 16 % on average.
double attention_f32_tc_us(bool f32, const AttnShape& s) {
  const bool wide = s.D > 64;
  const long long items = static_cast<long long>(s.B) * s.Hq * ((s.Sq + kRows - 1) / kRows), waves = (items + sm_count() - 1) / sm_count();
  const double tiles = std::ceil(attention_mean_keys(s) / (wide ? 64 : 128));
  return 0.8 + waves * (f32 ? (wide ? 7.5 + 4.0 * tiles : 5.6 + 3.35 * tiles) : (wide ? 6.0 + 1.4 * tiles : 5.0 + 1.75 * tiles));
}

// Head sizes, 16-byte rows, a positive scale that leaves the exponents room.
template <typename T>
bool attention_f32_tc_takes(const T* q, const T* k, const T* v, const AttnShape& s) {
  if (s.D < 8 || s.D > 128 || s.D % 8 || !(s.scale >= 0x1p-60f && s.scale <= 0x1p60f)) return false;
  const long long strides = s.q_sb | s.q_sh | s.q_ss | s.k_sb | s.k_sh | s.k_ss | s.v_sb | s.v_sh | s.v_ss;
  if (strides % static_cast<long long>(16 / sizeof(T))) return false;
  return !((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v)) & 15);
}
template bool attention_f32_tc_takes<float>(const float*, const float*, const float*, const AttnShape&);
template bool attention_f32_tc_takes<bf16>(const bf16*, const bf16*, const bf16*, const AttnShape&);

}  // namespace teeny
