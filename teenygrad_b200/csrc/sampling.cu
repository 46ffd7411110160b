// Token sampling after the LM head: temperature, top-k and top-p (nucleus) over one row of bf16 logits per CTA.
//
// The reference ships only the row softmax next to the logits (kernels/teeny-kernels/src/nn/activation/softmax.rs:39;
// Op::TopK is unlowered, kernels/teeny-kernels/src/graph/mod.rs:2784); this is the step a serving loop needs behind
// it.  Definition (oracle/sampling.py restates it on the CPU):
//   1. candidates = the top_k entries of the row by (logit descending, index ascending);
//   2. e_i = exp((l_i - l_0) / temperature) in f32 over the candidates in that order, c_i = e_0 + ... + e_i summed
//      sequentially in f32;
//   3. nucleus = the shortest prefix with c_{n-1} >= top_p * c_last (at least one candidate);
//   4. the sample is the first candidate i < n with c_i > u * c_{n-1}, u in [0, 1) given per row by the caller.
//
// Bound: latency; a row is 300 KB and its logits have just been written.  A row is cut over a thread-block cluster (up to four CTAs, see
// sample_parts), which read their slices with 16-byte loads that later passes find in L1.  Each thread takes the largest of its columns' keys
// (packed pairs), and each of the row's P CTAs finds the ceil(K / P)-th largest of its 1024, a bit at a time by barriers that count.  The smallest
// of these P bounds is reached by at least K entries of the row, so every one of the top K is among the entries not below it, of which there are
// little more than K: only the threads whose largest reaches it look at their columns again.  The entries go into a list per CTA; the first CTA sorts
// their union.  One thread does the running sums, so that the result does not depend on a reduction tree; the cut and the pick are searches over them.
//
// Where they do not fit the list (ties), or the threads are too few, histograms decide: bf16 logits have 65536 possible values, so two 256-bin
// histograms (high byte, then low byte inside the deciding bin), which the cluster adds through distributed shared memory, give the k-th
// largest value exactly; what is at or above it goes into the lists (a row with thousands of ties, such as a masked one, is collected in index order
// instead).  For every row they are slower: logits share a handful of exponents, and a warp's 32 increments of the high byte's bins mostly hit the same one or two.
// Measured on B200, before (histograms, bitonic sort) and now: 32 x 151936, top-k 50 17.0 -> 11.8 us, top-k 1000 36.4 -> 19.8; 8 x 151936 16.4 -> 11.5;
// 64 x 151936 22.8 -> 13.9; 64 x 32768 13.0 -> 8.7; 5 x 1000 8.4 -> 6.7.
#include <atomic>

#include "common.cuh"
#include "kernels.h"

namespace teeny {

namespace {

constexpr int kSampleThreads = 1024;
constexpr int kMaxTopK = 1024;
constexpr int kMaxParts = 4;  // CTAs of a row (sample_parts)

// bf16 bit pattern -> 16-bit key whose unsigned order is the float order (NaNs sort above +inf; not expected here)
__device__ __forceinline__ unsigned sort_key(unsigned short bits) {
  return (bits & 0x8000u) ? (~static_cast<unsigned>(bits) & 0xFFFFu) : (static_cast<unsigned>(bits) | 0x8000u);
}
__device__ __forceinline__ float key_to_float(unsigned key) {
  const unsigned bits = (key & 0x8000u) ? (key & 0x7FFFu) : (~key & 0xFFFFu);
  return __uint_as_float(bits << 16);
}

// Largest bin b with (number of entries in bins above b) < want <= (number in bins >= b); `above` gets the former.  By one warp.
__device__ __forceinline__ void pick_bin(const unsigned* hist, unsigned want, unsigned* bin_out, unsigned* above_out) {
  const int lane = threadIdx.x & 31, first = 8 * (31 - lane);  // lane 0 holds the highest bins
  unsigned n[8], sum = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) sum += n[i] = hist[first + i];
  unsigned upto = sum;  // entries in this lane's bins and all above
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned t = __shfl_up_sync(0xffffffffu, upto, o);
    if (lane >= o) upto += t;
  }
  if (upto >= want && upto - sum < want) {  // exactly one lane
    unsigned above = upto - sum;
    int i = 7;
    while (i > 0 && above + n[i] < want) above += n[i--];
    *bin_out = static_cast<unsigned>(first + i);
    *above_out = above;
  }
}

struct __align__(16) PickShared {
  float e[kMaxTopK], c[kMaxTopK];
  unsigned n, pick;
};

// Steps 2-4 of the definition over the K sorted candidates in cand[]: exponentials in parallel, running sums by one thread in
// candidate order, the cut and the pick as the first of them that pass.  A candidate is (key << 32) | (0xFFFFFFFF - index).
__device__ __forceinline__ void pick_from_sorted(const unsigned long long* cand, PickShared& sh, unsigned K, float inv_temperature,
                                                 float top_p, float u, int* out_idx, float* out_prob) {
  const unsigned tid = threadIdx.x;
  const float l0 = key_to_float(static_cast<unsigned>(cand[0] >> 32));
  sh.e[tid] = tid < K ? expf((key_to_float(static_cast<unsigned>(cand[tid] >> 32)) - l0) * inv_temperature) : 0.0f;
  if (tid == 0) { sh.n = K; sh.pick = K; }
  __syncthreads();
  if (tid == 0) {
    float c = 0.0f;
    float4 x = *reinterpret_cast<const float4*>(sh.e), y = *reinterpret_cast<const float4*>(sh.e + 4);
    for (unsigned i = 0; i < K; i += 8) {  // the sums behind K are not read
      const unsigned next = min(i + 8, static_cast<unsigned>(kMaxTopK) - 8u);  // on its way while these are added
      const float4 xn = *reinterpret_cast<const float4*>(sh.e + next), yn = *reinterpret_cast<const float4*>(sh.e + next + 4);
      float4 r, t;
      r.x = c + x.x; r.y = r.x + x.y; r.z = r.y + x.z; r.w = r.z + x.w;
      t.x = r.w + y.x; t.y = t.x + y.y; t.z = t.y + y.z; t.w = t.z + y.w;
      c = t.w;
      *reinterpret_cast<float4*>(sh.c + i) = r;
      *reinterpret_cast<float4*>(sh.c + i + 4) = t;
      x = xn;
      y = yn;
    }
  }
  __syncthreads();
  // nucleus: shortest prefix whose mass reaches top_p of the total
  if (tid < K && sh.c[tid] >= top_p * sh.c[K - 1]) atomicMin(&sh.n, tid + 1);
  __syncthreads();
  const unsigned n = sh.n;
  const float mass = sh.c[n - 1];
  if (tid < n && sh.c[tid] > u * mass) atomicMin(&sh.pick, tid);
  __syncthreads();
  if (tid == 0) {
    const unsigned pick = sh.pick < n ? sh.pick : n - 1;
    *out_idx = static_cast<int>(0xFFFFFFFFu - static_cast<unsigned>(cand[pick] & 0xFFFFFFFFull));
    if (out_prob) *out_prob = sh.e[pick] / mass;
  }
}

// address of `local` (an address in this CTA's shared memory) in the shared memory of CTA `rank` of the cluster
__device__ __forceinline__ uint32_t peer_smem(const void* local, uint32_t rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(local)), "r"(rank));
  return a;
}
__device__ __forceinline__ uint32_t ld_peer_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_peer_u64(uint32_t addr) {
  unsigned long long v;
  asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(addr) : "memory");
  return v;
}

// f(index, key) for the columns [begin, end) of a row, 16 bytes at a time where the row is aligned
template <typename F>
__device__ __forceinline__ void for_keys(const unsigned short* row, int begin, int end, F f) {
  const int tid = threadIdx.x;
  if ((reinterpret_cast<uintptr_t>(row) & 15) == 0) {  // begin is a multiple of 8
    const int vend = begin + ((end - begin) & ~7);
#pragma unroll 4
    for (int i = begin + tid * 8; i < vend; i += kSampleThreads * 8) {
      const uint4 v = *reinterpret_cast<const uint4*>(row + i);
      const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        f(i + 2 * j, sort_key(static_cast<unsigned short>(w[j] & 0xffffu)));
        f(i + 2 * j + 1, sort_key(static_cast<unsigned short>(w[j] >> 16)));
      }
    }
    begin = vend;
  }
#pragma unroll 4
  for (int i = begin + tid; i < end; i += kSampleThreads) f(i, sort_key(row[i]));
}

constexpr unsigned kSampleList = 2048;  // candidates with their ties at the threshold that are sorted at once

// Descending bitonic sort of the first `n` (a power of two) slots.
__device__ __forceinline__ void sort_descending(unsigned long long* cand, unsigned n) {
  for (unsigned size = 2; size <= n; size <<= 1) {
    for (unsigned stride = size >> 1; stride > 0; stride >>= 1) {
      for (unsigned i = threadIdx.x; i < n / 2; i += kSampleThreads) {
        const unsigned lo = 2 * i - (i & (stride - 1)), hi = lo + stride;
        const unsigned long long a = cand[lo], b = cand[hi];
        if ((a < b) == ((lo & size) == 0)) { cand[lo] = b; cand[hi] = a; }
      }
      __syncthreads();
    }
  }
}

// Keys of two bf16 numbers at once.
__device__ __forceinline__ unsigned sort_keys2(unsigned w) { return w ^ (((w >> 15) & 0x00010001u) * 0xffffu | 0x80008000u); }

// Sorts the first n <= 128 slots of `from` descending into `to` by counting, for each, the larger ones (the slots differ): 1024 / (n rounded
// up) threads per slot.
__device__ __forceinline__ void sort_by_rank(const unsigned long long* from, unsigned long long* to, unsigned n) {
  unsigned lg = 5;  // threads of a slot
  while ((static_cast<unsigned>(kSampleThreads) >> lg) < n) --lg;
  const unsigned at = threadIdx.x >> lg, sub = threadIdx.x & ((1u << lg) - 1u);
  const unsigned long long mine = at < n ? from[at] : 0ull;
  unsigned larger = 0;
  for (unsigned i = sub; i < n; i += 1u << lg) larger += from[i] > mine ? 1u : 0u;
  for (unsigned o = 1u << lg >> 1; o > 0; o >>= 1) larger += __shfl_xor_sync(0xffffffffu, larger, o);
  if (at < n && sub == 0) to[larger] = mine;
  __syncthreads();
}

// Sorts the first n <= 2048 slots of `from`, whose keys are not below `lowest`, descending into `from` again: into bins, one per key, in the
// order of the keys (`other` has them then), and each by counting within its bin.  Returns false, with `from` as it was, where the keys are too far apart (1024:
// 8 octaves) or a bin too full.  1100 slots: about 1 us, the bitonic sort 8.
__device__ __forceinline__ bool sort_by_key(unsigned long long* from, unsigned long long* other, unsigned n, unsigned lowest, unsigned* count,
                                            unsigned* base, unsigned* warp_tot) {
  constexpr unsigned kBins = kSampleThreads, kMost = 128;
  const unsigned tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned long long x[2];
  unsigned bin[2], place[2];
  bool far = false;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const unsigned i = tid + kSampleThreads * j;
    x[j] = i < n ? from[i] : 0ull;
    bin[j] = static_cast<unsigned>(x[j] >> 32) - lowest;
    far |= i < n && bin[j] >= kBins;
  }
  count[tid] = 0;
  if (__syncthreads_or(far)) return false;
#pragma unroll
  for (int j = 0; j < 2; ++j)
    if (tid + kSampleThreads * j < n) place[j] = atomicAdd(count + bin[j], 1u);
  __syncthreads();
  // slots in the bins above: thread t has bin 1023 - t
  const unsigned mine = count[kBins - 1 - tid];
  unsigned upto = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned t = __shfl_up_sync(0xffffffffu, upto, o);
    if (lane >= o) upto += t;
  }
  if (lane == 31) warp_tot[warp] = upto;
  if (__syncthreads_or(mine > kMost)) return false;
  unsigned before = warp_tot[lane];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned t = __shfl_up_sync(0xffffffffu, before, o);
    if (lane >= o) before += t;
  }
  before = __shfl_sync(0xffffffffu, before, (warp + 31) & 31);
  base[kBins - 1 - tid] = upto - mine + (warp ? before : 0u);
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 2; ++j)
    if (tid + kSampleThreads * j < n) other[base[bin[j]] + place[j]] = x[j];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    if (tid + kSampleThreads * j >= n) continue;
    const unsigned b = base[bin[j]], end = b + count[bin[j]];
    unsigned at = b;
    for (unsigned i = b; i < end; ++i) at += other[i] > x[j] ? 1u : 0u;
    from[at] = x[j];
  }
  __syncthreads();
  return true;
}

struct SampleShared {
  unsigned hist[2][256];                       // this CTA's histograms
  unsigned sum[256];                           // the row's
  unsigned long long list[kSampleList];        // this CTA's candidates
  unsigned long long cand[kSampleList];        // the row's (first CTA)
  PickShared pick;
  unsigned bin, above, count, eq_base, bound, warp_tot[32];
};

// cand_out != null: stop after step 1 and write the K sorted candidates of the row, indices shifted by idx_offset, to
// cand_out[row * cand_stride ...] (a vocabulary shard's contribution under tensor parallelism; sample_merge_kernel
// finishes the job over all shards' lists).  A cluster of `parts` CTAs per row.
__global__ void __launch_bounds__(kSampleThreads, 1)
sample_top_k_top_p_kernel(const bf16* __restrict__ logits, long long ld, int cols, float inv_temperature, int top_k,
                          float top_p, const float* __restrict__ u, int* __restrict__ out_idx,
                          float* __restrict__ out_prob, unsigned long long* __restrict__ cand_out, int cand_stride,
                          int idx_offset, int parts, int by_bound) {
  __shared__ __align__(16) SampleShared sh;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned rank = parts > 1 ? cluster_rank() : 0u;
  const int r = static_cast<int>(blockIdx.x) / parts;
  const unsigned short* row = reinterpret_cast<const unsigned short*>(logits) + static_cast<size_t>(r) * ld;
  const unsigned K = static_cast<unsigned>(min(top_k, cols));
  const int slice = ((cols + parts - 1) / parts + 7) & ~7;
  const int begin = min(cols, static_cast<int>(rank) * slice), end = min(cols, begin + slice);
  auto sync_row = [&] { if (parts > 1) cluster_sync_all(); else __syncthreads(); };
  // the row's histogram from all CTAs', then the bin that holds entry number `want` from the top
  auto decide = [&](int level, unsigned want) {
    sync_row();
    if (tid < 256) {
      unsigned n = 0;
      if (parts > 1) {
        unsigned v[kMaxParts];
#pragma unroll
        for (int p = 0; p < kMaxParts; ++p) v[p] = p < parts ? ld_peer_u32(peer_smem(&sh.hist[level][tid], p)) : 0u;
#pragma unroll
        for (int p = 0; p < kMaxParts; ++p) n += v[p];
      } else {
        n = sh.hist[level][tid];
      }
      sh.sum[tid] = n;
    }
    __syncthreads();
    if (warp == 0) pick_bin(sh.sum, want, &sh.bin, &sh.above);
    __syncthreads();
  };

  if (tid < 512) sh.hist[tid >> 8][tid & 255] = 0;
  if (tid == 0) sh.count = 0;
  __syncthreads();
  pdl_wait();
  unsigned entries = 0, lowest = 0;  // in cand[], unsorted; no key is below
  bool found = false;
  if (by_bound) {
    // The row as 16-byte vectors behind `head` columns; the first and last columns that fill none are a few threads' of the first CTA.
    const int head = min(cols, static_cast<int>((16 - (reinterpret_cast<uintptr_t>(row) & 15)) & 15) >> 1), vecs = (cols - head) >> 3;
    const int per = (vecs + parts - 1) / parts, v0 = min(vecs, static_cast<int>(rank) * per), v1 = min(vecs, v0 + per);
    const int tail0 = head + 8 * vecs, odd = rank == 0 ? (tid < head ? tid : (tid - head < cols - tail0 ? tail0 + tid - head : -1)) : -1;
    const uint4* vec = reinterpret_cast<const uint4*>(row + head);
    unsigned top2 = 0;
#pragma unroll 4
    for (int i = v0 + tid; i < v1; i += kSampleThreads) {
      const uint4 v = vec[i];
      top2 = __vmaxu2(top2, __vmaxu2(__vmaxu2(sort_keys2(v.x), sort_keys2(v.y)), __vmaxu2(sort_keys2(v.z), sort_keys2(v.w))));
    }
    unsigned top = max(top2 & 0xffffu, top2 >> 16);
    if (odd >= 0) top = max(top, sort_key(row[odd]));
    unsigned bound = 0;
    const int want = static_cast<int>((K + parts - 1) / parts);
    for (unsigned bit = 0x8000u; bit; bit >>= 1)
      if (__syncthreads_count(top >= (bound | bit)) >= want) bound |= bit;
    if (parts > 1) {
      if (tid == 0) sh.bound = bound;
      cluster_sync_all();
      unsigned v[kMaxParts];
#pragma unroll
      for (int p = 0; p < kMaxParts; ++p) v[p] = p < parts ? ld_peer_u32(peer_smem(&sh.bound, p)) : bound;
#pragma unroll
      for (int p = 0; p < kMaxParts; ++p) bound = min(bound, v[p]);
    }
    if (top >= bound) {
      auto list = [&](int i, unsigned k) {
        if (k < bound) return;
        const unsigned at = atomicAdd(&sh.count, 1u);
        if (at < kSampleList) sh.list[at] = (static_cast<unsigned long long>(k) << 32) | (0xFFFFFFFFu - static_cast<unsigned>(i));
      };
      if (odd >= 0) list(odd, sort_key(row[odd]));
#pragma unroll 4
      for (int i = v0 + tid; i < v1; i += kSampleThreads) {
        const uint4 v = vec[i];
        const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          list(head + 8 * i + 2 * j, sort_key(static_cast<unsigned short>(w[j] & 0xffffu)));
          list(head + 8 * i + 2 * j + 1, sort_key(static_cast<unsigned short>(w[j] >> 16)));
        }
      }
    }
    sync_row();
    unsigned n[kMaxParts], total = 0;  // (a list that ran over has a count beyond it)
#pragma unroll
    for (int p = 0; p < kMaxParts; ++p) n[p] = p < parts ? (parts > 1 ? ld_peer_u32(peer_smem(&sh.count, p)) : sh.count) : 0u;
#pragma unroll
    for (int p = 0; p < kMaxParts; ++p) total += n[p];
    found = total <= kSampleList;
    if (found) {
      if (rank == 0) {
        unsigned at = 0;
#pragma unroll
        for (int p = 0; p < kMaxParts; ++p) {
          if (p >= parts) break;
          for (unsigned i = tid; i < n[p]; i += kSampleThreads) sh.cand[at + i] = parts > 1 ? ld_peer_u64(peer_smem(&sh.list[i], p)) : sh.list[i];
          at += n[p];
        }
      }
      if (parts > 1) cluster_sync_all(); else __syncthreads();  // nobody leaves while its list is being read
      if (rank != 0) return;
      entries = total;
      lowest = bound;
    } else {
      sync_row();  // the counts are read
      if (tid == 0) sh.count = 0;
    }
  }
  if (!found) {
    // ---- pass 1: histogram of the key's high byte ----
    for_keys(row, begin, end, [&](int, unsigned k) { atomicAdd(&sh.hist[0][k >> 8], 1u); });
    decide(0, K);
    const unsigned hi_bin = sh.bin, above_hi = sh.above;
    // ---- pass 2: histogram of the low byte inside that bin ----
    for_keys(row, begin, end, [&](int, unsigned k) { if ((k >> 8) == hi_bin) atomicAdd(&sh.hist[1][k & 255u], 1u); });
    decide(1, K - above_hi);
    const unsigned thresh = (hi_bin << 8) | sh.bin;        // the K-th largest key
    const unsigned above = above_hi + sh.above;            // entries above it
    const unsigned total = above + sh.sum[sh.bin];         // and with all of its ties
    // ---- pass 3 ----
    lowest = thresh;
    if (total <= kSampleList) {
      for_keys(row, begin, end, [&](int i, unsigned k) {
        if (k >= thresh) sh.list[atomicAdd(&sh.count, 1u)] = (static_cast<unsigned long long>(k) << 32) | (0xFFFFFFFFu - static_cast<unsigned>(i));
      });
      sync_row();
      if (rank == 0) {
        unsigned at = 0;
        for (int p = 0; p < parts; ++p) {
          const unsigned n = parts > 1 ? ld_peer_u32(peer_smem(&sh.count, p)) : sh.count;
          for (unsigned i = tid; i < n; i += kSampleThreads) sh.cand[at + i] = parts > 1 ? ld_peer_u64(peer_smem(&sh.list[i], p)) : sh.list[i];
          at += n;
        }
      }
      entries = total;
      if (parts > 1) cluster_sync_all();  // nobody leaves while its list is being read
      if (rank != 0) return;
    } else {
      if (parts > 1) cluster_sync_all();  // nor while its histogram is
      if (rank != 0) return;
      // in index order: everything above the threshold, and the first need_eq entries equal to it
      const unsigned need_eq = K - above;
      entries = K;
      if (tid == 0) sh.eq_base = 0;
      __syncthreads();
      for (int base = 0; base < cols; base += kSampleThreads) {
        const int i = base + tid;
        const unsigned k = i < cols ? sort_key(row[i]) : 0u;
        const bool gt = i < cols && k > thresh, eq = i < cols && k == thresh;
        // rank of this thread's tie among the ties of the tile (block-wide exclusive count in index order)
        const unsigned eq_mask = __ballot_sync(0xffffffffu, eq);
        if (lane == 0) sh.warp_tot[warp] = __popc(eq_mask);
        __syncthreads();
        unsigned before = sh.eq_base;
        for (int w = 0; w < warp; ++w) before += sh.warp_tot[w];
        before += __popc(eq_mask & ((1u << lane) - 1u));
        if (gt || (eq && before < need_eq)) {
          const unsigned slot = atomicAdd(&sh.count, 1u);
          if (slot < static_cast<unsigned>(kMaxTopK))
            sh.cand[slot] = (static_cast<unsigned long long>(k) << 32) | (0xFFFFFFFFu - static_cast<unsigned>(i));
        }
        __syncthreads();
        if (tid == 0) {
          unsigned t = 0;
          for (int w = 0; w < 32; ++w) t += sh.warp_tot[w];
          sh.eq_base += t;
        }
        __syncthreads();
      }
    }
    __syncthreads();
  }
  const unsigned long long* sorted_list = sh.cand;
  if (entries <= 128) {
    sort_by_rank(sh.cand, sh.list, entries);
    sorted_list = sh.list;
  } else if (!sort_by_key(sh.cand, sh.list, entries, lowest, reinterpret_cast<unsigned*>(sh.pick.e), reinterpret_cast<unsigned*>(sh.pick.c), sh.warp_tot)) {
    unsigned slots = 256;
    while (slots < entries) slots <<= 1;
    for (unsigned i = entries + tid; i < slots; i += kSampleThreads) sh.cand[i] = 0ull;  // these end up last
    __syncthreads();
    sort_descending(sh.cand, slots);
  }
  if (cand_out) {
    // entries past K are zero (smaller than any real candidate); the shift keeps (value desc, index asc) order
    if (tid < cand_stride) {
      const unsigned long long c = static_cast<unsigned>(tid) < K ? sorted_list[tid] : 0ull;
      cand_out[static_cast<size_t>(r) * cand_stride + tid] =
          static_cast<unsigned>(tid) < K ? ((c & 0xFFFFFFFF00000000ull) | ((c & 0xFFFFFFFFull) - static_cast<unsigned>(idx_offset))) : 0ull;
    }
    return;
  }
  pick_from_sorted(sorted_list, sh.pick, K, inv_temperature, top_p, u[r], out_idx + r, out_prob ? out_prob + r : nullptr);
}

// Whether the threads' largest keys bound the candidates well: a bound that k of g largest keys reach is reached by about -g ln(1 - k / g)
// entries, 1.6 g at k = 0.8 g.
bool sample_by_bound(int cols, int top_k, int parts) {
  const int k = ((top_k < cols ? top_k : cols) + parts - 1) / parts, groups = (cols / 8 + parts - 1) / parts;
  return 10 * k <= 8 * (groups < kSampleThreads ? groups : kSampleThreads);
}

// CTAs per row: up to four, while all clusters are resident at once (one CTA per SM by its 1024 threads; the GPU's SMs hold 33 clusters of four of these)
// and slices are no less than what the meetings of the cluster cost, or as many as the bounds take.  Top-k 50, one, two, four, eight CTAs a row:
// 1 x 151936 17.5, 13.3, 11.2, 12.2 us; 32 x 151936 18.4, 14.5, 12.4; 36 rows 18.6, 14.5, 20.4; 37 x 70001 12.2, 11.5; 16 x 32768 9.1, 9.7, 9.8, 19.2 (16 clusters
// of eight do not find place).
int sample_parts(int rows, int cols, int top_k) {
  const int sms = sm_count();
  const bool two = 2LL * rows <= sms, four = 9LL * rows <= 2 * sms;
  int parts = !two || cols < 65536 ? 1 : (four && cols >= 98304 ? kMaxParts : 2);
  while ((parts == 1 ? two : parts == 2 && four) && !sample_by_bound(cols, top_k, parts) && sample_by_bound(cols, top_k, 2 * parts)) parts *= 2;
  return parts;
}

// Tensor-parallel finish: lists[p * list_stride + row * K + i] is candidate i (sorted descending) of vocabulary shard p
// for this row; the top K of their union are found by rank counting -- a candidate's place in the union is the number
// of candidates above it, a binary search per list, and the keys are distinct -- and steps 2-4 follow as on one GPU,
// so every rank, given the same u, picks the same token as the unsharded kernel would.
__global__ void __launch_bounds__(kSampleThreads, 1)
sample_merge_kernel(const unsigned long long* __restrict__ lists, int parts, size_t list_stride, int K_list, int top_k,
                    float inv_temperature, float top_p, const float* __restrict__ u, int* __restrict__ out_idx,
                    float* __restrict__ out_prob) {
  pdl_wait();
  extern __shared__ unsigned long long all[];      // [parts][K_list]
  __shared__ unsigned long long cand[kMaxTopK];
  __shared__ __align__(16) PickShared pick;
  const int tid = threadIdx.x;
  const int total = parts * K_list;
  for (int i = tid; i < total; i += kSampleThreads) {
    const int p = i / K_list, e = i - p * K_list;
    all[i] = lists[static_cast<size_t>(p) * list_stride + static_cast<size_t>(blockIdx.x) * K_list + e];
  }
  for (int i = tid; i < kMaxTopK; i += kSampleThreads) cand[i] = 0ull;
  __syncthreads();
  unsigned live = 0;  // real candidates in the union (empty slots are zero)
  for (int i = tid; i < total; i += kSampleThreads) {
    const unsigned long long c = all[i];
    if (c == 0ull) continue;
    unsigned above = 0;
    for (int p = 0; p < parts; ++p) {  // entries of list p greater than c: lists are sorted descending
      const unsigned long long* lp = all + p * K_list;
      int lo = 0, hi = K_list;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (lp[mid] > c) lo = mid + 1; else hi = mid;
      }
      above += static_cast<unsigned>(lo);
    }
    if (above < static_cast<unsigned>(kMaxTopK)) cand[above] = c;
    ++live;
  }
  __shared__ unsigned s_live;
  if (tid == 0) s_live = 0;
  __syncthreads();
  if (live) atomicAdd(&s_live, live);
  __syncthreads();
  const unsigned K = min(static_cast<unsigned>(top_k), s_live);
  pick_from_sorted(cand, pick, K, inv_temperature, top_p, u[blockIdx.x], out_idx + blockIdx.x,
                   out_prob ? out_prob + blockIdx.x : nullptr);
}

// u[row] in [0, 1) as a pure function of (seed, step, row): a splitmix64 finaliser over the three, top 24 bits.
// (oracle/sampling.py restates it, so a generation can be replayed on the CPU.)
__global__ void sampling_uniform_kernel(unsigned long long seed, int step, const int* __restrict__ step_dev,
                                        float* __restrict__ u, int rows) {
  pdl_wait();
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= rows) return;
  const unsigned long long t = static_cast<unsigned long long>(step_dev ? *step_dev : step);
  unsigned long long x = seed ^ (t * 0x9E3779B97F4A7C15ull) ^ (static_cast<unsigned long long>(r) * 0xBF58476D1CE4E5B9ull);
  x ^= x >> 30; x *= 0xBF58476D1CE4E5B9ull;
  x ^= x >> 27; x *= 0x94D049BB133111EBull;
  x ^= x >> 31;
  u[r] = static_cast<float>(x >> 40) * (1.0f / 16777216.0f);
}

}  // namespace

int sampling_uniform(unsigned long long seed, int step, const int* step_dev, float* u, int rows, cudaStream_t st) {
  if (!u || rows < 0) return TEENY_ERR_BAD_ARG;
  if (rows == 0) return TEENY_OK;
  launch_kernel(sampling_uniform_kernel, dim3((rows + 127) / 128), dim3(128), 0, st, 1, seed, step, step_dev, u, rows);
  return static_cast<int>(cudaGetLastError());
}

int sample_top_k_top_p_bf16(const bf16* logits, long long ld, int rows, int cols, float temperature, int top_k,
                            float top_p, const float* u, int* out_idx, float* out_prob, cudaStream_t st) {
  if (!logits || !u || !out_idx || rows < 0 || cols <= 0 || ld < cols) return TEENY_ERR_BAD_ARG;
  if (!(temperature > 0.0f) || top_k < 1 || top_k > kMaxTopK || !(top_p > 0.0f) || top_p > 1.0f) return TEENY_ERR_BAD_ARG;
  if (rows == 0) return TEENY_OK;
  const int parts = sample_parts(rows, cols, top_k);
  launch_kernel(sample_top_k_top_p_kernel, dim3(rows * parts), dim3(kSampleThreads), 0, st, static_cast<unsigned>(parts), logits, ld, cols,
                1.0f / temperature, top_k, top_p, u, out_idx, out_prob, static_cast<unsigned long long*>(nullptr), 0, 0, parts,
                static_cast<int>(sample_by_bound(cols, top_k, parts)));
  return static_cast<int>(cudaGetLastError());
}

int sample_candidates_bf16(const bf16* logits, long long ld, int rows, int cols, int top_k, int idx_offset,
                           unsigned long long* cand_out, cudaStream_t st) {
  if (!logits || !cand_out || rows < 0 || cols <= 0 || ld < cols || top_k < 1 || top_k > kMaxTopK || idx_offset < 0)
    return TEENY_ERR_BAD_ARG;
  if (rows == 0) return TEENY_OK;
  const int parts = sample_parts(rows, cols, top_k);
  launch_kernel(sample_top_k_top_p_kernel, dim3(rows * parts), dim3(kSampleThreads), 0, st, static_cast<unsigned>(parts), logits, ld, cols,
                1.0f, top_k, 1.0f, static_cast<const float*>(nullptr), static_cast<int*>(nullptr), static_cast<float*>(nullptr), cand_out,
                top_k, idx_offset, parts, static_cast<int>(sample_by_bound(cols, top_k, parts)));
  return static_cast<int>(cudaGetLastError());
}

int sample_merge_prepare() {
  static std::atomic<unsigned long long> done{0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && (done.load(std::memory_order_acquire) >> dev) & 1ull) return 0;
  cudaError_t e = cudaFuncSetAttribute(sample_merge_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 8 * kMaxTopK * 8);
  if (e != cudaSuccess) return static_cast<int>(e);
  if (dev < 64) done.fetch_or(1ull << dev, std::memory_order_release);
  return 0;
}

int sample_merge(const unsigned long long* lists, int parts, size_t list_stride, int rows, float temperature, int top_k,
                 float top_p, const float* u, int* out_idx, float* out_prob, cudaStream_t st) {
  if (!lists || !u || !out_idx || parts < 1 || parts > 8 || rows < 0 || list_stride < static_cast<size_t>(rows) * top_k)
    return TEENY_ERR_BAD_ARG;
  if (!(temperature > 0.0f) || top_k < 1 || top_k > kMaxTopK || !(top_p > 0.0f) || top_p > 1.0f) return TEENY_ERR_BAD_ARG;
  if (rows == 0) return TEENY_OK;
  const int prc = sample_merge_prepare();
  if (prc) return prc;
  launch_kernel(sample_merge_kernel, dim3(rows), dim3(kSampleThreads), static_cast<size_t>(parts) * top_k * 8, st, 1, lists,
                parts, list_stride, top_k, top_k, 1.0f / temperature, top_p, u, out_idx, out_prob);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace teeny
