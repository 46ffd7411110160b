// bf16 linear layers called as operators, Y[M, N] = X[M, K] W[N, K]^T (+ bias), with too few tiles to occupy the GPU: K of a tile over a cluster.
//
// The same assignment as gemm_bf16_skinny_kernel (gemm_bf16.cu): 128 weight rows fill the MMA's rows, BN tokens are its columns.  That kernel is
// built for decode steps: two CTAs an SM, so that the next kernel's find place beside it, and clusters of up to eight.  Called by itself its time
// is the way behind the last MMA: 128 x 4096 x 4096, clocks: first tile there 2000, last MMA done 8000, partial tile stored 9000, sums of the cluster
// done 15500, gone 18700; the two CTAs of an SM fetch 110 KB of partial sums from their clusters by 128 threads with 32 KB in flight.
// So here:
//   * a CTA has an SM to itself, and clusters are as wide as the tiles leave SMs;
//   * partial sums are sent, not fetched: bulk copies between the CTAs' shared memory, one for each other CTA, whose columns lie together.  Remote
//     loads brought 6 bytes a clock (32 KB of them: 8300 clocks; sent 2000);
//   * the cluster's barriers are relaxed arrivals, the first one behind the main loop: an arrival that releases took 1000 clocks;
//   * loops that issue are walked by the whole warp and one lane issues: descriptors stay in uniform registers (a 64-k block took
//     470 clocks to issue by a lone lane, now 255, which is what its four MMAs take);
//   * the ring is requested before tensor memory is there and the CTA meets; eight warps move the sums, by code for each cluster width.
// 128 x 4096 x 4096 now: last MMA done 6000, parted 6700, received 8700, stored 10100, gone 10500.
// Measured back to back on B200 (M x N x K, us, before -> now): 32 x 4096 x 4096 10.2 -> 6.5, 64 x 4096 x 4096 11.3 -> 7.7, 128 x 4096 x 4096 13.9 -> 8.6 (called alone 16.4 ->
// 12.3), 151 x 1944 x 704 11.2 -> 4.8, 512 x 1024 x 3072 12.7 -> 7.7.
#include <atomic>
#include <cmath>

#include "common.cuh"
#include "kernels.h"

namespace teeny {

namespace {

constexpr int kBM = 128, kBK = 64, kEpiWarps = 8, kThreads = 32 * (2 + kEpiWarps), kEpi = 32 * kEpiWarps;
constexpr int kMaxStages = 8, kSmem = 226 << 10, kSmemTwo = 112 << 10;

template <int BN> struct Cfg {
  static constexpr int kP = kBM * kBK * 2, kQ = BN * kBK * 2, kStage = kP + kQ;
  static constexpr int kPart = BN * kBM * 4;  // f32 partial tile [token][weight row], in the place of the ring
  static constexpr int kTmemCols = BN > 128 ? 256 : BN;
};

struct SplitArgs {
  int M, N, K, ldy;
  bf16* y;
  const bf16* bias;
  int k_blocks, per, stages;  // 64-k blocks, of a CTA; tiles in the ring
  int cw;                     // token columns that a CTA of the cluster finishes (the last ones: what is left)
  int ring;                   // bytes of the ring and of the partial tile that takes its place; behind them what the other CTAs send
  int vec;                    // Y takes 8-byte stores
  int glu;                    // kind (glu_f): W rows interleave 64 gate / 64 up channels, Y[M, N/2] = act(gate) * up
  int* err;
};

// Pieces of 4 weight rows of a token, the S parts added in the order of k.
template <int S>
__device__ __forceinline__ void finish(const SplitArgs& g, const float4* own, const float4* got, int rank, int m0, int tile, int columns) {
  const int t = threadIdx.x - 64, pieces = columns * (kBM / 4), row = tile * kBM + (t & 31) * 4;
  if (row >= g.N) return;
  float bias[4] = {};
  if (g.bias) {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (row + e < g.N) bias[e] = __bfloat162float(g.bias[row + e]);
  }
  const bool vec = g.vec && row + 4 <= g.N;
  const int end = min(pieces, (g.M - m0) * (kBM / 4));
  bf16* dst = g.y + static_cast<size_t>(m0 + (t >> 5)) * g.ldy + row;
  const float4* part[S];
#pragma unroll
  for (int q = 0; q < S; ++q) part[q] = (S == 1 || q == rank) ? own : got + (q - (q > rank)) * pieces;
#pragma unroll(S <= 2 ? 4 : 2)
  for (int u = t; u < end; u += kEpi, dst += static_cast<size_t>(kEpi / 32) * g.ldy) {
    float4 v[S];
#pragma unroll
    for (int q = 0; q < S; ++q) v[q] = part[q][u];
    float4 sum = v[0];
#pragma unroll
    for (int q = 1; q < S; ++q) sum = make_float4(sum.x + v[q].x, sum.y + v[q].y, sum.z + v[q].z, sum.w + v[q].w);
    const float o[4] = {sum.x + bias[0], sum.y + bias[1], sum.z + bias[2], sum.w + bias[3]};
    if (vec) {
      *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]));
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (row + e < g.N) dst[e] = __float2bfloat16_rn(o[e]);
    }
  }
}

// The same for a gated unit: a tile is 64 gate rows and the 64 up rows of the same channels; pieces of 4 channels of a token.
template <int S>
__device__ __forceinline__ void finish_glu(const SplitArgs& g, const float4* own, const float4* got, int rank, int m0, int tile, int columns) {
  const int t = threadIdx.x - 64, pieces = columns * (kBM / 4), at = tile * 64 + (t & 15) * 4;
  const float4* part[S];
#pragma unroll
  for (int q = 0; q < S; ++q) part[q] = (S == 1 || q == rank) ? own : got + (q - (q > rank)) * pieces;
  for (int u = t; u < columns * 16; u += kEpi) {
    const int m = m0 + (u >> 4), i = (u >> 4) * (kBM / 4) + (u & 15);
    float4 a = part[0][i], b = part[0][i + 16];
#pragma unroll
    for (int q = 1; q < S; ++q) {
      const float4 x = part[q][i], y = part[q][i + 16];
      a = make_float4(a.x + x.x, a.y + x.y, a.z + x.z, a.w + x.w);
      b = make_float4(b.x + y.x, b.y + y.y, b.z + y.z, b.w + y.w);
    }
    if (m >= g.M) continue;  // (N is a multiple of 128)
    const float o[4] = {glu_f(g.glu, a.x, b.x), glu_f(g.glu, a.y, b.y), glu_f(g.glu, a.z, b.z), glu_f(g.glu, a.w, b.w)};
    bf16* dst = g.y + static_cast<size_t>(m) * g.ldy + at;
    if (g.vec) {
      *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]));
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) dst[e] = __float2bfloat16_rn(o[e]);
    }
  }
}
template <int S>
__device__ __forceinline__ void finish_any(const SplitArgs& g, const float4* own, const float4* got, int rank, int m0, int tile, int columns) {
  if (g.glu) finish_glu<S>(g, own, got, rank, m0, tile, columns); else finish<S>(g, own, got, rank, m0, tile, columns);
}

// grid (S, weight tiles, token tiles), clusters of S along x
template <int BN>
__global__ void __launch_bounds__(kThreads, 1)
gemm_bf16_split_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const SplitArgs g) {
  using C = Cfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_mem[2 * kMaxStages + 2];
  __shared__ uint32_t tmem_at;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  float* part = reinterpret_cast<float*>(smem_raw + (base - smem_u32(smem_raw)));
  auto full = [&](int s) { return smem_u32(bar_mem) + 8u * s; };
  auto empty = [&](int s) { return smem_u32(bar_mem) + 8u * (kMaxStages + s); };
  const uint32_t acc_full = smem_u32(bar_mem) + 16u * kMaxStages, received = acc_full + 8u;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int S = static_cast<int>(cluster_size()), rank = static_cast<int>(cluster_rank());
  const int tile = blockIdx.y, m0 = blockIdx.z * BN;
  const int kb0 = rank * g.per, n = min(g.k_blocks, kb0 + g.per) - kb0;
  auto first_of = [&](int q) { return min(BN, q * g.cw); };  // token columns that CTA q finishes
  const int c0 = first_of(rank), columns = first_of(rank + 1) - c0;
  auto load = [&](int s, int kb) {
    const uint32_t sp = base + s * C::kStage;
    mbar_expect_tx(full(s), C::kStage);
    tma_load_2d(sp, &tmap_w, full(s), kb * kBK, tile * kBM);
    tma_load_2d(sp + C::kP, &tmap_x, full(s), kb * kBK, m0);
  };
  const bool one = elect_one();
  if (warp == 0) {
    if (one) {
      tma_prefetch_desc(&tmap_w);
      tma_prefetch_desc(&tmap_x);
      mbar_init(acc_full, 1);
      mbar_init(received, 1);
    }
    if (lane < g.stages) {
      mbar_init(full(lane), 1);
      mbar_init(empty(lane), 1);
    }
    mbar_fence_init();
    __syncwarp();
    pdl_wait();
    for (int i = 0; i < min(n, g.stages); ++i)
      if (one) load(i, kb0 + i);
  } else if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_at), C::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (S > 1) {
    if (tid == 0) mbar_expect_tx(received, (S - 1) * columns * (kBM * 4));
    __syncwarp();
    cluster_arrive_relaxed();  // this CTA's barriers exist
  }
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&tmem_at);
  if (warp != 0) pdl_wait();

  if (warp == 0) {
    for (int i = g.stages, s = 0, ph = 0; i < n; ++i) {
      if (!mbar_wait(empty(s), ph, g.err, DEVERR_GEMM_PRODUCER)) break;
      if (one) load(s, kb0 + i);
      if (++s == g.stages) { s = 0; ph ^= 1; }
    }
  } else if (warp == 1) {
    // The whole warp walks the loop, so that descriptors stay in uniform registers; one lane issues.
    const uint64_t dw = make_smem_desc_sw128(base, 16, 1024), dx = make_smem_desc_sw128(base + C::kP, 16, 1024);
    bool ok = true;
    int s = 0, ph = 0;
    uint32_t off = 0;
    bool ready = mbar_try_wait(full(0), 0);
    for (int i = 0; i < n; ++i) {
      if (!ready && !mbar_wait(full(s), ph, g.err, DEVERR_GEMM_MMA)) { ok = false; break; }
      tc_fence_after();
      if (one) umma_bf16_ss_x4<2, 2>(tmem, dw + off, dx + off, make_idesc_bf16(kBM, BN, false, false), i ? 1u : 0u);
      if (i + g.stages < n && one) umma_commit(empty(s));
      off += C::kStage / 16;
      if (++s == g.stages) { s = 0; ph ^= 1; off = 0; }
      ready = i + 1 < n && mbar_try_wait(full(s), ph);
    }
    if (ok && one) umma_commit(acc_full);
  } else if (mbar_wait(acc_full, 0, g.err, DEVERR_GEMM_EPILOGUE)) {
    // accumulator -> partial tile: a warp its 32 rows of half the columns
    tc_fence_after();
    const int quarter = warp & 3, c0 = ((warp - 2) >> 2) * (BN / 2);
    const uint32_t from = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + c0;
    float* to = part + c0 * kBM + quarter * 32 + lane;
    constexpr int kStep = BN / 2 >= 32 ? 32 : 16;
#pragma unroll
    for (int c = 0; c < BN / 2; c += kStep) {
      uint32_t r[kStep];
      if constexpr (kStep == 32) tmem_ld_32x32(from + c, r); else tmem_ld_32x16(from + c, r);
      tmem_wait_ld();
#pragma unroll
      for (int e = 0; e < kStep; ++e) to[(c + e) * kBM] = __uint_as_float(r[e]);
    }
    tc_fence_before();
    fence_proxy_async_smem();
  }
  __syncwarp();
  pdl_trigger();
  if (S > 1) cluster_wait();  // (of the arrival at the start)
  __syncthreads();
  if (warp >= 2) {
    const int gave_up = *reinterpret_cast<volatile int*>(g.err);
    if (S > 1 && warp == 2 && lane < S && lane != rank && !gave_up) {  // each other CTA gets the columns that it finishes
      const int q = lane, from = first_of(q), bytes = (first_of(q + 1) - from) * (kBM * 4);
      if (bytes > 0)
        send_bulk(map_rank(base + g.ring + (rank - (rank > q)) * bytes, q), base + from * (kBM * 4), bytes, map_rank(received, q));
    }
    bool ok = true;
    if (S > 1 && columns > 0) ok = mbar_wait(received, 0, g.err, DEVERR_GEMM_EPILOGUE);
    __syncwarp();
    if (S > 1) cluster_arrive_relaxed();  // what was sent here has arrived
    if (ok) {
      const float4* own = reinterpret_cast<const float4*>(part + c0 * kBM);
      const float4* got = reinterpret_cast<const float4*>(reinterpret_cast<uint8_t*>(part) + g.ring);
      switch (S) {
        case 1: finish_any<1>(g, own, got, rank, m0 + c0, tile, columns); break;
        case 2: finish_any<2>(g, own, got, rank, m0 + c0, tile, columns); break;
        case 3: finish_any<3>(g, own, got, rank, m0 + c0, tile, columns); break;
        case 4: finish_any<4>(g, own, got, rank, m0 + c0, tile, columns); break;
        case 5: finish_any<5>(g, own, got, rank, m0 + c0, tile, columns); break;
        case 6: finish_any<6>(g, own, got, rank, m0 + c0, tile, columns); break;
        case 7: finish_any<7>(g, own, got, rank, m0 + c0, tile, columns); break;
        default: finish_any<8>(g, own, got, rank, m0 + c0, tile, columns); break;
      }
    }
  } else if (S > 1) {
    cluster_arrive_relaxed();
  }
  __syncwarp();
  if (warp == 1) {
    if (*reinterpret_cast<volatile int*>(g.err) != 0) {
      // a wait gave up: let copies / MMAs that are still in flight drain before the memory is released
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 2000000ull) __nanosleep(1000);
    }
    tc_fence_after();
    tmem_dealloc(tmem, C::kTmemCols);
  }
  if (S > 1) cluster_wait();  // nobody leaves while what it sent is being read, or on its way
}

template <int BN>
int prepare() {
  static std::atomic<unsigned long long> done{0};  // one bit per device; threads may race to set it
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && (done.load(std::memory_order_acquire) >> dev) & 1ull) return 0;
  const cudaError_t e = cudaFuncSetAttribute(gemm_bf16_split_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
  if (e != cudaSuccess) return static_cast<int>(e);
  if (dev < 64) done.fetch_or(1ull << dev, std::memory_order_release);
  return 0;
}

template <int BN>
int launch(const CUtensorMap& tw, const CUtensorMap& tx, SplitArgs g, int split, cudaStream_t st) {
  using C = Cfg<BN>;
  const int rc = prepare<BN>();
  if (rc) return rc;
  g.cw = (BN + split - 1) / split;
  const int sent = (split - 1) * g.cw * (kBM * 4);
  // more tiles than SMs: two CTAs on an SM
  const long long ctas = static_cast<long long>((g.N + kBM - 1) / kBM) * ((g.M + BN - 1) / BN) * split;
  const int most = split == 1 && ctas > sm_count() ? kSmemTwo : kSmem, room = (most - 1024 - sent) / C::kStage;
  g.stages = g.per < kMaxStages ? g.per : kMaxStages;
  if (g.stages > room) g.stages = room;
  g.ring = g.stages * C::kStage > C::kPart ? g.stages * C::kStage : C::kPart;
  if (g.stages < 1 || 1024 + g.ring + sent > most) return TEENY_ERR_BAD_ARG;
  return launch_kernel(gemm_bf16_split_kernel<BN>, dim3(split, (g.N + kBM - 1) / kBM, (g.M + BN - 1) / BN), dim3(kThreads), 1024 + g.ring + sent, st,
                       static_cast<unsigned>(split), tw, tx, g);
}

}  // namespace

// Microseconds of K over `split` CTAs of 128 x bn tiles, which are all resident at once (0: they would not be): a start and an end, and the blocks of a
// CTA, each what its MMAs take to issue, its bytes at the rate of one SM, or all CTAs' bytes at the rate of L2 -- which are lower where rows do not start on
// 128 bytes (`lines`): a row of a tile is then two lines.  Fitted to calls with 16 to 2000 tokens (12 % off in the mean; what is taken is 1.8 % slower than the best of
// a size's choices).
double gemm_bf16_split_us(int M, int N, int K, bool lines, int bn, int split, int sms) {
  // clusters of 1 to 8 CTAs, one on an SM, that a B200 holds at once (cudaOccupancyMaxActiveClusters); single CTAs also two on an SM
  constexpr int kResident[8] = {296, 74, 45, 33, 26, 22, 15, 15};
  const int blocks = (K + kBK - 1) / kBK, per = (blocks + split - 1) / split;
  const long long tiles = static_cast<long long>((N + kBM - 1) / kBM) * ((M + bn - 1) / bn);
  if (tiles * 148 > static_cast<long long>(kResident[split - 1]) * sms || per * (split - 1) >= blocks || (split > 1 && per < 2)) return 0.0;
  if (bn == 256 && (split > 2 || tiles * split > sms)) return 0.0;  // (shared memory for less than three blocks)
  const double kb = kBK * 2.0 * (kBM + bn), narrow = bn / 128.0, ctas = static_cast<double>(tiles) * split, per_sm = ctas > sms ? ctas / sms : 1.0;
  const double issue = bn <= 128 ? 0.09 : (bn == 192 ? 0.21 : 0.32), sm = kb * per_sm / (lines ? 196e3 : 97e3), all = kb * ctas / (lines ? 17.0e6 : 11.1e6);
  const double block = std::pow(std::pow(issue, 6) + std::pow(sm, 6) + std::pow(all, 6), 1.0 / 6);
  const double ends = 2.26 + 0.75 * narrow + (split > 1 ? 2.58 * narrow * (split - 1) / split : 0.0);
  const double hbm = 2.0 * (static_cast<double>(N) * K + static_cast<double>(M) * K + static_cast<double>(M) * N) / 7.8e6;
  return 0.9 + ends * (per_sm > 1.0 ? (bn > 128 ? 1.8 : 1.43) : 1.0) + std::cbrt(std::pow(per * block, 3) + std::pow(hbm, 3));
}

SplitChoice gemm_bf16_split_choose(int M, int N, int K, bool lines, int sms) {
  SplitChoice best{};
  for (int bn : {32, 64, 128, 192, 256}) {
    if (bn >= 192 && M <= 128) break;
    for (int split = 1; split <= (bn >= 192 ? 4 : 8); ++split) {
      const double us = gemm_bf16_split_us(M, N, K, lines, bn, split, sms);
      if (us > 0.0 && (!best.bn || us < best.us)) best = SplitChoice{bn, split, us};
    }
  }
  return best;
}

int gemm_bf16_split_prepare() {
  int rc = 0;
  if ((rc = prepare<32>()) || (rc = prepare<64>()) || (rc = prepare<128>()) || (rc = prepare<192>())) return rc;
  return prepare<256>();
}

int gemm_bf16_split(const bf16* x, int ldx, const bf16* w, int ldw, const bf16* bias, bf16* y, int ldy, int M, int N, int K, int bn, int split,
                    int glu, cudaStream_t st) {
  if (!x || !w || !y || M <= 0 || N <= 0 || K <= 0 || split < 1 || split > 8 || (bn != 32 && bn != 64 && bn != 128 && bn != 192 && bn != 256)) return TEENY_ERR_BAD_ARG;
  if (((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) || ldx % 8 || ldw % 8) return TEENY_ERR_ALIGNMENT;
  SplitArgs g{};
  g.M = M; g.N = N; g.K = K; g.ldy = ldy; g.y = y; g.bias = bias;
  g.k_blocks = (K + kBK - 1) / kBK;
  g.per = (g.k_blocks + split - 1) / split;
  if (g.per * (split - 1) >= g.k_blocks) return TEENY_ERR_BAD_ARG;  // a CTA without products
  if ((N + kBM - 1) / kBM > 65535 || (M + bn - 1) / bn > 65535) return TEENY_ERR_BAD_ARG;
  if (glu && (bias || N % 128)) return TEENY_ERR_BAD_ARG;
  g.glu = glu;
  g.vec = ldy % 4 == 0 && !(reinterpret_cast<uintptr_t>(y) & 7);
  g.err = device_error_word();
  if (!g.err) return TEENY_ERR_DRIVER;
  CUtensorMap tw, tx;
  auto map = [&](CUtensorMap* t, const bf16* p, int ld, int rows, int box_rows) {
    const uint64_t dims[2] = {static_cast<uint64_t>(K), static_cast<uint64_t>(rows)}, strides[1] = {static_cast<uint64_t>(ld) * 2};
    const uint32_t box[2] = {kBK, static_cast<uint32_t>(box_rows)};
    return encode_tensor_map_bf16(t, p, 2, dims, strides, box);
  };
  int rc = map(&tw, w, ldw, N, kBM);
  if (!rc) rc = map(&tx, x, ldx, M, bn);
  if (rc) return rc;
  if (bn == 32) return launch<32>(tw, tx, g, split, st);
  if (bn == 64) return launch<64>(tw, tx, g, split, st);
  if (bn == 128) return launch<128>(tw, tx, g, split, st);
  return bn == 192 ? launch<192>(tw, tx, g, split, st) : launch<256>(tw, tx, g, split, st);
}

}  // namespace teeny
