// CUDA-core GEMM with genuine f32 products and accumulation (FFMA): C[m,n] = sum_k A[m,k] * B[k,n] (+ bias[n]).
// It serves (a) the f32 entry points for small products and layouts that the tensor-core kernel (gemm_f32_tc.cu) does not take, and (b) bf16 problems whose pointers or strides the TMA path cannot describe.  All operands are
// addressed through element strides so [K,N], [N,K] and padded layouts share the kernel.
//
// Bound: the FP32 pipe for large products, the chain over K for small ones.  A thread keeps a TM x TN block of sums and reads
// TM + TN words of shared memory per k -- at 8 x 8 those loads take as long as the multiply-adds, hence 16 x 8 --; the multiply-adds
// are packed pairs of rows.  The next 16-deep slice of both operands is in registers while the current one is multiplied
// (two buffers, one barrier per slice).  An operand that is contiguous along k is transposed on its way into shared memory.
// Small products have too few tiles for the SMs and a chain of K / 16 slices whose loads nothing hides: they take smaller tiles
// and KG groups of threads on alternating slices, whose sums are added in group order.
#include "common.cuh"
#include "kernels.h"

namespace teeny {

namespace {

constexpr int kTK = 16;  // k per slice

template <typename T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<bf16>(bf16 v) { return __bfloat162float(v); }
template <typename T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ bf16 from_f<bf16>(float v) { return __float2bfloat16_rn(v); }
__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const bf16* p) {
  const uint2 v = *reinterpret_cast<const uint2*>(p);
  return make_float4(bf16_lo(v.x), bf16_hi(v.x), bf16_lo(v.y), bf16_hi(v.y));
}

// One operand as a matrix of `rows` (M or N) by K.  How four neighbours are fetched: along k, along the rows, or one by one.
enum { kAlongK, kAlongRows, kSingly, kSinglyAlongRows };
template <typename T>
struct Operand {
  const T* p;
  long long s_row, s_k;
  int rows, mode;
};

template <int BM, int BN, int TM, int TN, int KG>
struct Tile {
  static constexpr int kGroup = (BM / TM) * (BN / TN);  // threads per group
  static constexpr int kThreads = kGroup * KG;
  static constexpr int kLdA = BM + 4, kLdB = BN + 4;
  static constexpr int kBuffer = kTK * (kLdA + kLdB);   // floats
  static_assert(kGroup % 32 == 0 && (BN / TN) % 8 == 0 && KG <= 8, "warps of 4 x 8 threads");
  static_assert(2 * kBuffer >= BM * BN || KG == 1, "a group's sums fit in its own buffers");
};

// Four neighbours number `e` of a slice (rows x 16): along the rows when the memory is contiguous that way, else along k.
template <typename T, int ROWS>
__device__ __forceinline__ float4 fetch(const Operand<T>& op, int row0, int k0, int K, int e) {
  if (op.mode == kAlongRows || op.mode == kSinglyAlongRows) {
    const int r = row0 + (e % (ROWS / 4)) * 4, k = k0 + e / (ROWS / 4);
    const T* p = op.p + static_cast<long long>(r) * op.s_row + static_cast<long long>(k) * op.s_k;
    if (op.mode == kAlongRows) return (r < op.rows && k < K) ? load4(p) : make_float4(0.f, 0.f, 0.f, 0.f);
    float v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = (r + i < op.rows && k < K) ? to_f<T>(p[i * op.s_row]) : 0.0f;
    return make_float4(v[0], v[1], v[2], v[3]);
  }
  const int r = row0 + (e >> 2), k = k0 + (e & 3) * 4;
  const T* p = op.p + static_cast<long long>(r) * op.s_row + static_cast<long long>(k) * op.s_k;
  if (op.mode == kAlongK) return (r < op.rows && k < K) ? load4(p) : make_float4(0.f, 0.f, 0.f, 0.f);
  float v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = (r < op.rows && k + i < K) ? to_f<T>(p[i * op.s_k]) : 0.0f;
  return make_float4(v[0], v[1], v[2], v[3]);
}
// the same four into the slice in shared memory, [16][ld] with the row index fastest
template <int ROWS>
__device__ __forceinline__ void place(float* s, int mode, int e, float4 v) {
  constexpr int kLd = ROWS + 4;
  if (mode == kAlongRows || mode == kSinglyAlongRows) {
    *reinterpret_cast<float4*>(s + e / (ROWS / 4) * kLd + (e % (ROWS / 4)) * 4) = v;
  } else {
    float* d = s + (e & 3) * 4 * kLd + (e >> 2);
    d[0] = v.x; d[kLd] = v.y; d[2 * kLd] = v.z; d[3 * kLd] = v.w;
  }
}

template <typename T, int BM, int BN, int TM, int TN, int KG>
__global__ void __launch_bounds__((Tile<BM, BN, TM, TN, KG>::kThreads), 2)
gemm_simt_kernel(const Operand<T> a, const Operand<T> b, const T* __restrict__ bias, T* __restrict__ c, long long scm, long long scn,
                 int K, int tiles_n) {
  using C = Tile<BM, BN, TM, TN, KG>;
  pdl_wait();
  __shared__ __align__(16) float smem[KG * 2 * C::kBuffer];
  const int g = threadIdx.x / C::kGroup, t = threadIdx.x % C::kGroup;
  const int warp = t >> 5, lane = t & 31;
  constexpr int kWarpsN = BN / TN / 8;
  const int im = warp / kWarpsN * 4 + (lane >> 3), in = warp % kWarpsN * 8 + (lane & 7);
  const int m0 = static_cast<int>(blockIdx.x / tiles_n) * BM, n0 = static_cast<int>(blockIdx.x % tiles_n) * BN;
  float* stage = smem + g * 2 * C::kBuffer;
  constexpr int kFetchA = BM * 4 / C::kGroup, kFetchB = BN * 4 / C::kGroup;

  f32x2 acc[TM / 2][TN];  // pairs of rows
#pragma unroll
  for (int i = 0; i < TM / 2; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = pack2(0.0f, 0.0f);

  float4 ra[kFetchA], rb[kFetchB];
  auto fetch_slice = [&](int k0) {
#pragma unroll
    for (int i = 0; i < kFetchA; ++i) ra[i] = fetch<T, BM>(a, m0, k0, K, t + i * C::kGroup);
#pragma unroll
    for (int i = 0; i < kFetchB; ++i) rb[i] = fetch<T, BN>(b, n0, k0, K, t + i * C::kGroup);
  };
  auto place_slice = [&](float* s) {
#pragma unroll
    for (int i = 0; i < kFetchA; ++i) place<BM>(s, a.mode, t + i * C::kGroup, ra[i]);
#pragma unroll
    for (int i = 0; i < kFetchB; ++i) place<BN>(s + kTK * C::kLdA, b.mode, t + i * C::kGroup, rb[i]);
  };
  auto group_sync = [&] {
    if constexpr (KG == 1) __syncthreads(); else named_barrier_sync(1 + g, C::kGroup);
  };

  int k0 = g * kTK, buf = 0;
  if (k0 < K) {
    fetch_slice(k0);
    place_slice(stage);
  }
  group_sync();
  for (; k0 < K; k0 += KG * kTK) {
    const bool more = k0 + KG * kTK < K;
    if (more) fetch_slice(k0 + KG * kTK);
    const float* as = stage + buf * C::kBuffer;
    const float* bs = as + kTK * C::kLdA;
#pragma unroll
    for (int kk = 0; kk < kTK; ++kk) {
      f32x2 av[TM / 2];
      float bv[TN];
      if constexpr (TM == 2) {
        av[0] = *reinterpret_cast<const f32x2*>(as + kk * C::kLdA + im * 2);
      } else {
#pragma unroll
        for (int i = 0; i < TM; i += 4) {
          const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(as + kk * C::kLdA + i * (BM / TM) + im * 4);
          av[i / 2] = x.x; av[i / 2 + 1] = x.y;
        }
      }
#pragma unroll
      for (int j = 0; j < TN; j += 4) {
        const float4 x = *reinterpret_cast<const float4*>(bs + kk * C::kLdB + j * (BN / TN) + in * 4);
        bv[j] = x.x; bv[j + 1] = x.y; bv[j + 2] = x.z; bv[j + 3] = x.w;
      }
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const f32x2 bb = pack2(bv[j], bv[j]);
#pragma unroll
        for (int i = 0; i < TM / 2; ++i) acc[i][j] = fma2(av[i], bb, acc[i][j]);
      }
    }
    if (more) place_slice(stage + (buf ^ 1) * C::kBuffer);
    group_sync();
    buf ^= 1;
  }

  auto row_of = [&](int i) { return TM == 2 ? im * 2 + i : (i & ~3) * (BM / TM) + im * 4 + (i & 3); };
  auto col_of = [&](int j) { return (j & ~3) * (BN / TN) + in * 4 + (j & 3); };
  auto put = [&](int gm, int gn, float v) {
    if (gm >= a.rows || gn >= b.rows) return;
    if (bias) v += to_f<T>(bias[gn]);
    c[static_cast<long long>(gm) * scm + static_cast<long long>(gn) * scn] = from_f<T>(v);
  };
  if constexpr (KG == 1) {
#pragma unroll
    for (int i = 0; i < TM; i += 2)
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const float2 v = unpack2(acc[i / 2][j]);
        put(m0 + row_of(i), n0 + col_of(j), v.x);
        put(m0 + row_of(i + 1), n0 + col_of(j), v.y);
      }
  } else {
#pragma unroll
    for (int i = 0; i < TM; i += 2)
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const float2 v = unpack2(acc[i / 2][j]);
        stage[row_of(i) * BN + col_of(j)] = v.x;
        stage[row_of(i + 1) * BN + col_of(j)] = v.y;
      }
    __syncthreads();
    for (int e = threadIdx.x; e < BM * BN; e += C::kThreads) {
      float v = smem[e];
#pragma unroll
      for (int q = 1; q < KG; ++q) v += smem[q * 2 * C::kBuffer + e];
      put(m0 + e / BN, n0 + e % BN, v);
    }
  }
}

// Measured on B200 (M x N x K = 2048 x 4096 x 4096: 1446 / 1589 / 2174 / 3803 us; 17 x 1000 x 1000: 113 / 37 / 27 / 12.6 us): the
// multiply-adds per clock that a tile reaches on a full SM, and the clocks that one of its slices takes when a chain of slices is all
// there is.
struct Choice { int bm, bn, kg; double rate, slice; };
constexpr double kEndsChain = 2800.0, kEndsPipe = 5000.0;  // start and end of a launch that a chain, or rounds of tiles, bounds
constexpr Choice kChoices[] = {{128, 128, 1, 92.0, 3500.0}, {64, 64, 2, 75.0, 2060.0}, {32, 64, 3, 55.0, 2130.0}, {16, 32, 6, 31.0, 1650.0}};

// The tile that is estimated to end first: rounds of tiles over the SMs at the tile's rate, or the chain of slices if that is longer.  To `least`, which is
// compared with the tensor cores' estimate, comes what a launch takes besides.
// 1000 x 4096 x 1024: 128 x 128 at 199 us (64 x 64: 210); 512^3: 32 x 64 at 16.5 us (64 x 64: 23, 16 x 32: 23).  The one 64 x 64 tile
// with 4 x 4 sums per thread that served every size before took 308 us and 50 us.  (Call by call, as in the table above; back to back in a
// graph a call takes 2.4 us less: 14.1 for 512^3.)
// bf16 takes the three smaller ones (`first` = 1): its operands come two bytes at a time where they are not aligned, which 256 threads an SM that
// hold 128 sums each do not keep up with (1000 x 4096 x 1024, odd rows: 368 us with 128 x 128, 281 with 64 x 64; f32 216 and 242).
int choose(long long M, long long N, long long K, int sms, double& least, int first = 0) {
  int best = first;
  double ends = 0.0;
  least = 0.0;
  for (int i = first; i < 4; ++i) {
    const Choice& x = kChoices[i];
    const long long tiles = ((M + x.bm - 1) / x.bm) * ((N + x.bn - 1) / x.bn);
    const double pipe = static_cast<double>((tiles + sms - 1) / sms) * x.bm * x.bn * K / x.rate;
    const double chain = static_cast<double>((K + kTK * x.kg - 1) / (kTK * x.kg)) * x.slice;
    const double t = pipe > chain ? pipe : chain;
    if (i == first || t < least) { least = t; best = i; ends = pipe > chain ? kEndsPipe : kEndsChain; }
  }
  least += ends;
  return best;
}

template <typename T>
Operand<T> operand(const T* p, long long s_row, long long s_k, int rows, int K) {
  const bool aligned = (reinterpret_cast<uintptr_t>(p) & (4 * sizeof(T) - 1)) == 0;
  int mode = s_row == 1 && s_k != 1 ? kSinglyAlongRows : kSingly;
  if (aligned && s_k == 1 && s_row % 4 == 0 && K % 4 == 0) mode = kAlongK;
  else if (aligned && s_row == 1 && s_k % 4 == 0 && rows % 4 == 0) mode = kAlongRows;
  return Operand<T>{p, s_row, s_k, rows, mode};
}

template <typename T>
int launch(const T* a, long long sam, long long sak, const T* b, long long sbk, long long sbn, const T* bias, T* c,
           long long scm, long long scn, int M, int N, int K, cudaStream_t st) {
  if (!a || !b || !c || M <= 0 || N <= 0 || K <= 0) return TEENY_ERR_BAD_ARG;
  if ((static_cast<long long>(M) + 63) / 64 > 65535) return TEENY_ERR_BAD_ARG;
  const Operand<T> oa = operand(a, sam, sak, M, K), ob = operand(b, sbn, sbk, N, K);
  double clocks;
  const Choice x = kChoices[choose(M, N, K, sm_count(), clocks, sizeof(T) == 2 ? 1 : 0)];
  const long long tiles_n = (static_cast<long long>(N) + x.bn - 1) / x.bn, tiles = (static_cast<long long>(M) + x.bm - 1) / x.bm * tiles_n;
  if (tiles > 0x7fffffffLL) return TEENY_ERR_BAD_ARG;
#define TEENY_SIMT(BM, BN, TM, TN, KG)                                                                                              \
  launch_kernel(gemm_simt_kernel<T, BM, BN, TM, TN, KG>, dim3(static_cast<unsigned>(tiles)), dim3(Tile<BM, BN, TM, TN, KG>::kThreads), \
                0, st, 1, oa, ob, bias, c, scm, scn, K, static_cast<int>(tiles_n))
  switch (x.bm) {
    case 128:
      if constexpr (sizeof(T) == 4) TEENY_SIMT(128, 128, 16, 8, 1);
      break;
    case 64: TEENY_SIMT(64, 64, 8, 4, 2); break;
    case 32: TEENY_SIMT(32, 64, 4, 4, 3); break;
    default: TEENY_SIMT(16, 32, 2, 4, 6); break;
  }
#undef TEENY_SIMT
  return static_cast<int>(cudaGetLastError());
}

}  // namespace

double gemm_f32_clocks(const float* a, long long sam, long long sak, const float* b, long long sbk, long long sbn, const float* c, long long scm,
                       long long scn, int M, int N, int K) {
  double here;
  choose(M, N, K, sm_count(), here);
  if (!gemm_f32_tc_takes(sak, sbk, sbn, M, N, K)) return here;
  const double there = gemm_f32_tc_clocks(a, sam, b, sbk, sbn, c, scm, scn, M, N, K);
  return there < here ? there : here;
}

int gemm_f32(const float* a, long long sam, long long sak, const float* b, long long sbk, long long sbn,
             const float* bias, float* c, long long scm, long long scn, int M, int N, int K, cudaStream_t stream) {
  // On the tensor cores where that is estimated to end first, and always with a smaller error: from about 1 M multiply-adds per
  // SM on.  Back to back, [N][K]: 64 x 512 x 512 6.8 us here, 8.0 there; 34 x 288 x 536 7.2, 9.0; 512^3 14.1, 8.6; 64 x 4096 x 4096 93,
  // 33.5; 300 x 700 x 2000 45.7, 14.5; 1000 x 2048 x 2048 236, 54; [K][N]: 3490 x 136 x 136 11.9, 8.2; 1051 x 592 x 104 10.1, 7.3; rows
  // of C off 32 bytes: 1325 x 801 x 88 9.4, 11.3.  Of 434 calls of random sizes with 16-byte rows the slower kernel is taken by more than 5 % in 19 (42 without the ends of
  // a launch here and the stores of such rows there).
  if (a && b && c && gemm_f32_tc_takes(sak, sbk, sbn, M, N, K)) {
    double here;
    choose(M, N, K, sm_count(), here);
    if (gemm_f32_tc_clocks(a, sam, b, sbk, sbn, c, scm, scn, M, N, K) < here) return gemm_f32_tc(a, sam, b, sbk, sbn, bias, c, scm, scn, M, N, K, stream);
  }
  return launch<float>(a, sam, sak, b, sbk, sbn, bias, c, scm, scn, M, N, K, stream);
}
int gemm_bf16_generic(const bf16* a, long long sam, long long sak, const bf16* b, long long sbk, long long sbn,
                      const bf16* bias, bf16* c, long long scm, long long scn, int M, int N, int K,
                      cudaStream_t stream) {
  return launch<bf16>(a, sam, sak, b, sbk, sbn, bias, c, scm, scn, M, N, K, stream);
}

}  // namespace teeny
