// Temperature / top-k / top-p sampling.
//
//   1. candidates: a lower bound of the row's k-th largest value from maxima of interleaved subsets, then one streaming pass against
//      it.  One CTA per row takes 1024 maxima of the whole row (k <= 1024); slices of a row, one CTA or a cluster, take 512 of the
//      first eighth of each slice, or 2048 of all of it.  The m-th part of n elements has -512 ln(1 - k / 512) m elements or fewer above the
//      bound from 512 maxima of it: 8.4 k of a row at k = 50, so the bound from an eighth is for small k.  Candidates that do not
//      fit (masses of ties, a row whose head is unlike its tail) are found by an exact radix select on order-preserving 32-bit
//      keys (integer histograms in shared memory, 12-bit first digit);
//   2. slices cut what they have to their exact k-th key first where it is much more; the candidates are bitonic-sorted by (logit descending,
//      index ascending) -- a total order, so neither the gather order nor the split over CTAs matters -- and cut to the first k plus ties;
//   3. softmax with temperature over the candidates, inclusive scan in a fixed tree, top-p cut
//      "keep token i iff the mass strictly before it is <= p" (first token always kept);
//   4. inverse-CDF draw with a Philox4x32-10 uniform keyed by (seed, row, offset).
//
// The draw is a pure function of (logits row, k, p, T, seed, offset, row index).  The reference
// delegates this to FlashInfer (rl_engine/kernels/sampling.py:41-78: softmax -> top_k_renorm_probs
// -> top_p_sampling_from_probs) and has no kernel of its own.
#include "../common/ptx.cuh"
#include "kernels.h"

#include <cuda_fp16.h>

#include <type_traits>

namespace rlk {

namespace {

constexpr int kRowThreads = 1024;  // of the kernel that gives a row one CTA
constexpr int kThreads = 512;      // of the one that gives it slices
constexpr int kCap = 2048;       // candidates that are sorted (k <= 1024 plus ties)
constexpr int kGather = 10240;   // candidates that are gathered: 80 KB, two CTAs per SM
// Up to this k one maximum per thread of an eighth of a slice can give the bound (at 512 there would be none left above it).
constexpr int kFewLimit = 256;
constexpr int kSampleShare = 8;
constexpr int kMinSample = kThreads * 16;  // elements

template <typename T> __device__ __forceinline__ float ldv(const T* p, int i);
template <> __device__ __forceinline__ float ldv<float>(const float* p, int i) { return p[i]; }
template <> __device__ __forceinline__ float ldv<__nv_bfloat16>(const __nv_bfloat16* p, int i) { return __bfloat162float(p[i]); }
template <> __device__ __forceinline__ float ldv<__half>(const __half* p, int i) { return __half2float(p[i]); }

__device__ __forceinline__ uint32_t f2key(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);  // larger float -> larger key
}
__device__ __forceinline__ float key2f(uint32_t k) {
  const uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  return __uint_as_float(u);
}

__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint2 k) {
  const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint32_t hi0 = __umulhi(M0, c.x), lo0 = M0 * c.x;
    const uint32_t hi1 = __umulhi(M1, c.z), lo1 = M1 * c.z;
    c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
    k.x += W0;
    k.y += W1;
  }
  return c;
}

__device__ __forceinline__ uint32_t cluster_size_x() {
  uint32_t n;
  asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(n));
  return n;
}
__device__ __forceinline__ uint32_t cluster_max_u32(uint32_t addr, uint32_t v) {
  uint32_t old;
  asm volatile("atom.relaxed.cluster.shared::cluster.max.u32 %0, [%1], %2;" : "=r"(old) : "r"(addr), "r"(v) : "memory");
  return old;
}
__device__ __forceinline__ uint32_t cluster_add_u32(uint32_t addr, uint32_t v) {
  uint32_t old;
  asm volatile("atom.relaxed.cluster.shared::cluster.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(addr), "r"(v) : "memory");
  return old;
}
__device__ __forceinline__ void cluster_store_u64(uint32_t addr, unsigned long long v) {
  asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}

struct SelectScratch {
  unsigned int bins[256];
  unsigned int prefix, remaining;
};

// The k-th largest (1-based) of the keys visited by `each` (a callable that calls its argument with (key, valid) the
// same number of times in every lane of a warp), to DIGITS 8-bit digits from the top; the digits below are zero.  Every
// thread of the block calls it; at least k valid keys must exist.
template <int DIGITS, typename Each>
__device__ __forceinline__ uint32_t block_kth_key(SelectScratch& s, unsigned int k, Each&& each) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t prefix = 0u, mask = 0u;
  unsigned int remaining = k;
#pragma unroll 1
  for (int d = 0; d < DIGITS; ++d) {
    const int shift = 24 - 8 * d;
    if (tid < 256) s.bins[tid] = 0u;
    __syncthreads();
    each([&](uint32_t key, bool valid) {
      // warp-aggregated counting: large keys share their leading bits, so most lanes of a warp hit the same bin
      const bool active = valid && (key & mask) == prefix;
      const uint32_t digit = (key >> shift) & 0xffu;
      const unsigned int peers = __match_any_sync(0xffffffffu, active ? digit : 0xffffffffu);
      if (active && lane == __ffs(peers) - 1) atomicAdd(&s.bins[digit], static_cast<unsigned int>(__popc(peers)));
    });
    __syncthreads();
    if (warp == 0) {
      // lane l owns bins 255 - 8 l ... 248 - 8 l (highest first); inclusive scan of the lanes' sums
      unsigned int mine = 0u;
#pragma unroll
      for (int j = 0; j < 8; ++j) mine += s.bins[255 - (lane * 8 + j)];
      unsigned int incl = mine;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const unsigned int o = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += o;
      }
      const unsigned int before = incl - mine;
      if (before < remaining && remaining <= incl) {  // exactly one lane: the digit is one of its bins
        unsigned int acc = before;
        int bin = 255 - lane * 8;
        for (int j = 0; j < 8; ++j) {
          bin = 255 - (lane * 8 + j);
          if (acc + s.bins[bin] >= remaining) break;
          acc += s.bins[bin];
        }
        s.prefix = prefix | (static_cast<uint32_t>(bin) << shift);
        s.remaining = remaining - acc;
      }
    }
    __syncthreads();
    prefix = s.prefix;
    remaining = s.remaining;
    mask |= 0xffu << shift;
    __syncthreads();
  }
  return prefix;
}

__device__ __forceinline__ unsigned long long pack_candidate(uint32_t key, int i) {
  return (static_cast<unsigned long long>(key) << 32) | (0xffffffffu - static_cast<uint32_t>(i));
}

// What both kernels keep in shared memory.
struct SampleState {
  unsigned long long cand[kCap];
  float prob[kCap];
  float warp_tot[32];
  unsigned int warp_cnt[32];
  SelectScratch select;
  unsigned int prefix, remaining, above, pop, count, nkeep, total, bound, overflow;
  float mass;
};

// f(vector, index of the vector) for the 16-byte vectors [v0, v1) of `p`, dealt to the block's threads, the next four in flight while
// four are looked at; f's third argument is the vector's place among the four.
// AHEAD false: one load at a time, for twice the blocks per SM.
template <int THREADS, bool AHEAD = true, typename F>
__device__ __forceinline__ void sweep_vectors(const uint4* __restrict__ p, int v0, int v1, F&& f) {
  if constexpr (!AHEAD) {
#pragma unroll 4
    for (int v = v0 + static_cast<int>(threadIdx.x); v < v1; v += THREADS) f(__ldg(p + v), v, 0);
    return;
  }
  constexpr int kUnroll = 4;
  uint4 q[kUnroll];
  int v = v0 + static_cast<int>(threadIdx.x);
#pragma unroll
  for (int u = 0; u < kUnroll; ++u)
    if (v + u * THREADS < v1) q[u] = __ldg(p + v + u * THREADS);
  while (v < v1) {
    uint4 now[kUnroll];
    const int at = v;
    v += kUnroll * THREADS;
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      now[u] = q[u];
      if (v + u * THREADS < v1) q[u] = __ldg(p + v + u * THREADS);
    }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u)
      if (at + u * THREADS < v1) f(now[u], at + u * THREADS, u);
  }
}

// The candidates of a row by an exact radix select, digits of 12, 8, 8 and 4 bits from the top; after each the threshold bin is
// located by a parallel suffix scan, until what lies above the bin and the bin itself fit the buffer.  hist: [4096].
template <int THREADS, typename T>
__device__ __forceinline__ void radix_candidates(SampleState& s, unsigned int* hist, const T* __restrict__ z, int V, int k) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    s.prefix = 0;
    s.remaining = static_cast<unsigned int>(k);
    s.above = 0;
    s.pop = static_cast<unsigned int>(V);
  }
  __syncthreads();
  int shift = 32;
#pragma unroll 1
  for (int pass = 0; pass < 4; ++pass) {
    const int bits = pass == 0 ? 12 : (pass == 3 ? 4 : 8);
    if (s.above + s.pop <= static_cast<unsigned int>(kCap)) break;  // uniform: shared values behind a barrier
    const uint32_t himask = pass == 0 ? 0u : (0xffffffffu << shift);
    shift -= bits;
    const int nb = 1 << bits;
    for (int i = tid; i < nb; i += THREADS) hist[i] = 0;
    __syncthreads();
    const uint32_t prefix = s.prefix;
    for (int i = tid; i < V; i += THREADS) {
      const uint32_t key = f2key(ldv(z, i));
      if ((key & himask) == prefix) atomicAdd(&hist[(key >> shift) & static_cast<uint32_t>(nb - 1)], 1u);
    }
    __syncthreads();
    // thread t owns `per` consecutive bins, highest bins first; block-wide exclusive scan of the per-thread sums
    const int per = (nb + THREADS - 1) / THREADS;
    const int top = nb - 1 - tid * per;  // highest bin of this thread
    unsigned int mine = 0;
    for (int j = 0; j < per; ++j)
      if (top - j >= 0) mine += hist[top - j];
    unsigned int incl = mine;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned int o = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += o;
    }
    if (lane == 31) s.warp_cnt[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      unsigned int w = lane < THREADS / 32 ? s.warp_cnt[lane] : 0u;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const unsigned int o = __shfl_up_sync(0xffffffffu, w, off);
        if (lane >= off) w += o;
      }
      if (lane < THREADS / 32) s.warp_cnt[lane] = w;
    }
    __syncthreads();
    const unsigned int before = (warp == 0 ? 0u : s.warp_cnt[warp - 1]) + (incl - mine);  // count in higher bins
    const unsigned int need = s.remaining;
    __syncthreads();
    if (before < need && need <= before + mine) {  // exactly one thread: the threshold bin is one of its bins
      unsigned int acc = before;
      int bsel = top;
      for (int j = 0; j < per; ++j) {
        bsel = top - j;
        if (acc + hist[bsel] >= need) break;
        acc += hist[bsel];
      }
      s.prefix = prefix | (static_cast<uint32_t>(bsel) << shift);
      s.remaining = need - acc;
      s.above += acc;
      s.pop = hist[bsel];
    }
    __syncthreads();
  }
  const uint32_t from = s.prefix;  // everything above the threshold bin plus the bin itself
  if (tid == 0) s.count = 0;
  __syncthreads();
  for (int i = tid; i < V; i += THREADS) {
    const uint32_t key = f2key(ldv(z, i));
    if (key >= from) {
      const unsigned int slot = atomicAdd(&s.count, 1u);
      if (slot < kCap) s.cand[slot] = pack_candidate(key, i);
    }
  }
  __syncthreads();
}

// Sorts the s.count candidates, cuts them to the first k plus ties, and draws.  The sums are a fixed tree whatever the number of
// threads (pairs of candidates, groups of 32 pairs, the groups): the draw does not depend on which kernel found the candidates.
template <int THREADS>
__device__ __forceinline__ void sort_and_draw(SampleState& s, int k, float top_p, float inv_temp, unsigned long long seed,
                                              unsigned long long offset, int row, long long* __restrict__ out_ids,
                                              float* __restrict__ out_logprob) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int n = static_cast<int>(s.count < static_cast<unsigned int>(kCap) ? s.count : kCap);
  // sort only as many slots as the candidates need (a power of two >= n, at least 64): the usual few dozen
  // candidates take 21 compare-exchange rounds instead of the 66 of the full buffer
  int sort_n = 64;
  while (sort_n < n) sort_n <<= 1;
  for (int i = n + tid; i < sort_n; i += THREADS) s.cand[i] = 0ull;
  __syncthreads();
  // bitonic sort, descending, sort_n elements.  Pairs t = 32 w .. 32 w + 31 at strides up to 32 stay inside the 64 elements
  // [64 w, 64 w + 64), which one warp owns, so those rounds need no block barrier.
  for (int size = 2; size <= sort_n; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int t = tid; t < sort_n / 2; t += THREADS) {
        const int lo = 2 * t - (t & (stride - 1));
        const int hi = lo + stride;
        const bool desc = ((lo & size) == 0);
        const unsigned long long a = s.cand[lo], b = s.cand[hi];
        if ((a < b) == desc) {
          s.cand[lo] = b;
          s.cand[hi] = a;
        }
      }
      if (stride > 32 || (stride == 1 && size >= 64)) __syncthreads();  // the next round crosses the warps' blocks
      else __syncwarp();
    }
  }

  // the candidates may extend below the k-th largest value: keep the first k and everything tied with the k-th
  {
    const uint32_t kth_key = static_cast<uint32_t>(s.cand[(k < n ? k : n) - 1] >> 32);
    if (tid == 0) s.count = 0;
    __syncthreads();
    unsigned int local = 0;
    for (int i = tid; i < n; i += THREADS)
      if (static_cast<uint32_t>(s.cand[i] >> 32) >= kth_key) ++local;
    if (local) atomicAdd(&s.count, local);
    __syncthreads();
    n = static_cast<int>(s.count);
  }

  // softmax over the candidates + inclusive scan (fixed tree) + top-p cut
  const float zmax = key2f(static_cast<uint32_t>(s.cand[0] >> 32));
  constexpr int kPairs = kCap / 2 / THREADS;  // consecutive pairs of candidates per thread
  static_assert(kPairs == 1 || kPairs == 2, "512 or 1024 threads");
  float e[2 * kPairs], pair[kPairs], incl[kPairs];
#pragma unroll
  for (int j = 0; j < 2 * kPairs; ++j) {
    const int i = 2 * kPairs * tid + j;
    e[j] = i < n ? expf((key2f(static_cast<uint32_t>(s.cand[i] >> 32)) - zmax) * inv_temp) : 0.f;
  }
#pragma unroll
  for (int j = 0; j < kPairs; ++j) incl[j] = pair[j] = e[2 * j] + e[2 * j + 1];
  // inclusive scan of 32 pairs: a warp's, or half a warp's where a thread holds two of them
  const int group = tid * kPairs / 32;
  if constexpr (kPairs == 1) {
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const float o = __shfl_up_sync(0xffffffffu, incl[0], off);
      if (lane >= off) incl[0] += o;
    }
  } else {
    const int l = lane & 15;
    const float left = __shfl_up_sync(0xffffffffu, incl[1], 1, 16);
    incl[1] += incl[0];
    if (l >= 1) incl[0] += left;
#pragma unroll
    for (int off = 1; off < 16; off <<= 1) {
      const float o0 = __shfl_up_sync(0xffffffffu, incl[0], off, 16), o1 = __shfl_up_sync(0xffffffffu, incl[1], off, 16);
      if (l >= off) {
        incl[0] += o0;
        incl[1] += o1;
      }
    }
  }
  if ((tid * kPairs + kPairs) % 32 == 0) s.warp_tot[group] = incl[kPairs - 1];
  __syncthreads();
  if (warp == 0) {
    float w = s.warp_tot[lane];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const float o = __shfl_up_sync(0xffffffffu, w, off);
      if (lane >= off) w += o;
    }
    s.warp_tot[lane] = w;  // inclusive over groups
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kPairs; ++j) {
    const float base = (group == 0 ? 0.f : s.warp_tot[group - 1]) + (incl[j] - pair[j]);  // mass before the pair
    const int i = 2 * (kPairs * tid + j);
    s.prob[i] = base + e[2 * j];
    s.prob[i + 1] = base + e[2 * j] + e[2 * j + 1];
  }
  __syncthreads();
  const float total = s.warp_tot[31];
  if (tid == 0) s.nkeep = 0;
  __syncthreads();
  // keep i iff mass strictly before i <= p * total ; kept set is a prefix, so count it
  {
    const float lim = top_p * total;
    unsigned int local = 0;
#pragma unroll
    for (int j = 0; j < 2 * kPairs; ++j) {
      const int i = 2 * kPairs * tid + j;
      if (i < n && (i == 0 || s.prob[i - 1] <= lim)) ++local;
    }
    if (local) atomicAdd(&s.nkeep, local);
  }
  __syncthreads();
  if (tid != 0) return;
  // inverse-CDF draw
  const int nkeep = s.nkeep < 1u ? 1 : static_cast<int>(s.nkeep);
  const float mass = s.prob[nkeep - 1];
  const uint4 rnd = philox4x32_10(
      make_uint4(static_cast<uint32_t>(offset), static_cast<uint32_t>(offset >> 32), static_cast<uint32_t>(row), 0u),
      make_uint2(static_cast<uint32_t>(seed), static_cast<uint32_t>(seed >> 32)));
  const float u = (static_cast<float>(rnd.x >> 8) + 0.5f) * (1.0f / 16777216.0f);
  const float target = u * mass;
  int lo = 0, hi = nkeep - 1;  // first i with prob[i] > target
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (s.prob[mid] > target) hi = mid;
    else lo = mid + 1;
  }
  out_ids[row] = static_cast<long long>(0xffffffffu - static_cast<uint32_t>(s.cand[lo] & 0xffffffffu));
  if (out_logprob) out_logprob[row] = logf((s.prob[lo] - (lo ? s.prob[lo - 1] : 0.f)) / mass);
}

// One CTA per row, TWO of them to an SM or one that keeps more loads in flight.  The bound is the k-th largest of 1024 interleaved
// maxima of the whole row.
template <typename T, bool TWO>
__global__ void __launch_bounds__(kRowThreads, TWO ? 2 : 1)
sample_rows_kernel(const T* __restrict__ logits, long long ld, int V, int top_k, float top_p, float inv_temp, unsigned long long seed,
                   unsigned long long offset, long long* __restrict__ out_ids, float* __restrict__ out_logprob) {
  __shared__ unsigned int hist[4096];
  __shared__ SampleState s;
  const int row = static_cast<int>(blockIdx.x), tid = threadIdx.x;
  const T* z = logits + static_cast<long long>(row) * ld;
  const int k = top_k < 1 ? 1 : (top_k > V ? V : top_k);
  constexpr int kVec = 16 / sizeof(T);
  int head = static_cast<int>(((16 - (reinterpret_cast<uintptr_t>(z) & 15u)) & 15u) / sizeof(T));
  if (head > V) head = V;
  const int nvec = (V - head) / kVec, tail = head + nvec * kVec, rest = head + (V - tail);
  const uint4* p = reinterpret_cast<const uint4*>(z + head);
  auto rest_at = [&](int i) { return i < head ? i : tail + (i - head); };
  if (tid == 0) s.count = 0;
  uint32_t best = 0u;  // smaller than the key of any number
  sweep_vectors<kRowThreads, !TWO>(p, 0, nvec, [&](const uint4& q, int, int) {
    const T* e = reinterpret_cast<const T*>(&q);
#pragma unroll
    for (int j = 0; j < kVec; ++j) best = max(best, f2key(ldv(e, j)));
  });
  for (int i = tid; i < rest; i += kRowThreads) best = max(best, f2key(ldv(z, rest_at(i))));
  // two digits (sign, exponent, seven mantissa bits) are enough: a bound a little lower costs a few more candidates
  const uint32_t from = block_kth_key<2>(s.select, static_cast<unsigned int>(k), [&](auto&& f) { f(best, true); });
  auto keep = [&](uint32_t key, int i) {
    const unsigned int slot = atomicAdd(&s.count, 1u);
    if (slot < kCap) s.cand[slot] = pack_candidate(key, i);
  };
  sweep_vectors<kRowThreads, !TWO>(p, 0, nvec, [&](const uint4& q, int v, int) {
    const T* e = reinterpret_cast<const T*>(&q);
    uint32_t kk[kVec], top = 0u;
#pragma unroll
    for (int j = 0; j < kVec; ++j) {
      kk[j] = f2key(ldv(e, j));
      top = max(top, kk[j]);
    }
    if (top >= from) {
#pragma unroll
      for (int j = 0; j < kVec; ++j)
        if (kk[j] >= from) keep(kk[j], head + v * kVec + j);
    }
  });
  for (int i = tid; i < rest; i += kRowThreads) {
    const uint32_t key = f2key(ldv(z, rest_at(i)));
    if (key >= from) keep(key, rest_at(i));
  }
  __syncthreads();
  const bool fits = s.count <= static_cast<unsigned int>(kCap);  // uniform
  __syncthreads();
  if (!fits) radix_candidates<kRowThreads>(s, hist, z, V, k);
  sort_and_draw<kRowThreads>(s, k, top_p, inv_temp, seed, offset, row, out_ids, out_logprob);
}

// One CTA or a cluster of CTAs per row, each with a contiguous slice of its 16-byte vectors (the unaligned head and the tail of the row go
// to the first).  The bound is the k-th largest of 512 interleaved maxima of the first eighth of a slice (`few`), or of 2048 of
// all of it -- a bound for the row whichever part of it it comes from; the slice is then streamed against it (what the first
// sweep read comes from L2).
template <typename T>
__global__ void __launch_bounds__(kThreads, 2)
sample_slices_kernel(const T* __restrict__ logits, long long ld, int V, int top_k, float top_p, float inv_temp,
                     unsigned long long seed, unsigned long long offset, long long* __restrict__ out_ids,
                     float* __restrict__ out_logprob, bool few) {
  extern __shared__ unsigned long long gather_buf[];  // [kGather]
  unsigned int* hist = reinterpret_cast<unsigned int*>(gather_buf);  // [4096], the radix select over the row only
  __shared__ SampleState s;

  const int parts = static_cast<int>(cluster_size_x()), part = static_cast<int>(cluster_ctarank());
  const int row = static_cast<int>(blockIdx.x) / parts;
  const T* z = logits + static_cast<long long>(row) * ld;
  const int tid = threadIdx.x;
  const int k = top_k < 1 ? 1 : (top_k > V ? V : top_k);

  if (tid == 0) {
    s.count = 0;
    s.total = 0;
    s.bound = 0;
    s.overflow = 0;
  }
  __syncthreads();
  if (parts > 1) cluster_sync();  // the first CTA's counters are set before anyone adds to them
  {
    constexpr int kVec = 16 / sizeof(T);
    int head = static_cast<int>(((16 - (reinterpret_cast<uintptr_t>(z) & 15u)) & 15u) / sizeof(T));
    if (head > V) head = V;
    const int nvec = (V - head) / kVec;
    const int per = (nvec + parts - 1) / parts;
    const int v0 = min(nvec, part * per), v1 = min(nvec, v0 + per);
    const uint4* p = reinterpret_cast<const uint4*>(z + head);
    constexpr int kUnroll = 4;
    uint32_t best[kUnroll] = {0u, 0u, 0u, 0u};  // smaller than the key of any number
    const int sample = few ? min(v1 - v0, max((v1 - v0) / kSampleShare, kMinSample / kVec)) : v1 - v0;
    sweep_vectors<kThreads>(p, v0, v0 + sample, [&](const uint4& q, int, int u) {
      const T* e = reinterpret_cast<const T*>(&q);
#pragma unroll
      for (int j = 0; j < kVec; ++j) best[u] = max(best[u], f2key(ldv(e, j)));
    });
    // two digits, as above
    uint32_t from;
    if (few) {
      const uint32_t top = max(max(best[0], best[1]), max(best[2], best[3]));
      from = block_kth_key<2>(s.select, static_cast<unsigned int>(k), [&](auto&& f) { f(top, true); });
    } else {
      from = block_kth_key<2>(s.select, static_cast<unsigned int>(k), [&](auto&& f) {
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) f(best[u], true);
      });
    }
    auto keep = [&](uint32_t kk, int i) {
      const unsigned int slot = atomicAdd(&s.count, 1u);
      if (slot < kGather) gather_buf[slot] = pack_candidate(kk, i);
    };
    sweep_vectors<kThreads>(p, v0, v1, [&](const uint4& q, int v, int) {
      const T* e = reinterpret_cast<const T*>(&q);
      uint32_t kk[kVec], top = 0u;
#pragma unroll
      for (int j = 0; j < kVec; ++j) {
        kk[j] = f2key(ldv(e, j));
        top = max(top, kk[j]);
      }
      if (top >= from) {
#pragma unroll
        for (int j = 0; j < kVec; ++j)
          if (kk[j] >= from) keep(kk[j], head + v * kVec + j);
      }
    });
    if (part == 0) {
      const int tail = head + nvec * kVec;
      for (int i = tid; i < head + (V - tail); i += kThreads) {
        const int at = i < head ? i : tail + (i - head);
        const uint32_t kk = f2key(ldv(z, at));
        if (kk >= from) keep(kk, at);
      }
    }
    __syncthreads();
    // the exact k-th key of the candidates of a slice: fewer of them leave it, or are sorted
    const unsigned int have = s.count;
    uint32_t bound = from;
    if (have > static_cast<unsigned int>(kGather)) {
      if (tid == 0) {
        if (parts > 1) cluster_max_u32(mapa_u32(smem_u32(&s.overflow), 0), 1u);
        else s.overflow = 1u;
      }
    } else if (have > static_cast<unsigned int>(parts > 1 ? 2 * k : kCap)) {
      const int rounds = static_cast<int>((have + kThreads - 1) / kThreads);
      bound = block_kth_key<4>(s.select, static_cast<unsigned int>(k), [&](auto&& f) {
        for (int r = 0; r < rounds; ++r) {
          const unsigned int i = r * kThreads + tid;
          const bool in = i < have;
          f(in ? static_cast<uint32_t>(gather_buf[i] >> 32) : 0u, in);
        }
      });
    }
    const unsigned int mine = min(have, static_cast<unsigned int>(kGather));
    if (parts > 1) {
      // the highest bound of the cluster holds for the row; what reaches it goes to the first CTA's sort buffer
      const uint32_t bound0 = mapa_u32(smem_u32(&s.bound), 0), total0 = mapa_u32(smem_u32(&s.total), 0);
      const uint32_t cand0 = mapa_u32(smem_u32(s.cand), 0);
      if (tid == 0) cluster_max_u32(bound0, bound);
      cluster_sync();
      asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(bound) : "r"(bound0) : "memory");
      for (unsigned int i0 = 0; i0 < mine; i0 += kThreads) {  // slots are reserved once per warp
        const unsigned int i = i0 + tid;
        const unsigned long long c = i < mine ? gather_buf[i] : 0ull;
        const bool send = i < mine && static_cast<uint32_t>(c >> 32) >= bound;
        const unsigned int who = __ballot_sync(0xffffffffu, send);
        unsigned int slot = 0u;
        if ((tid & 31) == 0 && who != 0u) slot = cluster_add_u32(total0, static_cast<unsigned int>(__popc(who)));
        slot = __shfl_sync(0xffffffffu, slot, 0) + __popc(who & ((1u << (tid & 31)) - 1u));
        if (send && slot < kCap) cluster_store_u64(cand0 + slot * 8u, c);
      }
      cluster_sync();
      if (part != 0) return;  // nothing of this CTA is read any more
    } else {
      for (unsigned int i = tid; i < mine; i += kThreads) {
        const unsigned long long c = gather_buf[i];
        if (static_cast<uint32_t>(c >> 32) >= bound) {
          const unsigned int slot = atomicAdd(&s.total, 1u);
          if (slot < kCap) s.cand[slot] = c;
        }
      }
    }
    __syncthreads();
    if (tid == 0) s.count = s.total;
    __syncthreads();
  }
  const bool fits = s.overflow == 0u && s.count <= static_cast<unsigned int>(kCap);  // uniform
  __syncthreads();
  if (!fits) radix_candidates<kThreads>(s, hist, z, V, k);
  sort_and_draw<kThreads>(s, k, top_p, inv_temp, seed, offset, row, out_ids, out_logprob);
}

// ---------------------------------------------------------------------------------------------
// Full-vocabulary nucleus sampling (no top-k): temperature softmax over the whole row, keep the
// smallest set of highest-probability tokens whose mass reaches top_p (all tokens tied with the
// cut value are kept), draw by inverse CDF in INDEX order inside the kept set.
//
// Masses are 40-bit fixed point in 64-bit integers, so sums do not depend on their order and the result is
// deterministic: a pure function of (row, top_p, T, seed, offset, row index).
//
// Three sweeps over the row, 16 bytes per access: maximum; histogram of the mass over 256 equal steps of (max - x) / T up to
// 28, beyond which the mass is 0 (equal steps hold a percent of the tokens each, where the leading bits of the key put nearly
// all into four bins); then the tokens of the step that holds the cut are gathered and every warp sums what lies
// above it in its own stretch of the row.  The cut itself is a radix search among the gathered tokens in shared memory, and the draw rescans
// one warp's stretch.  The histogram has one copy per lane, so the 32-bit atomics of a warp (14 bits of the mass
// at a time) hit 32 banks.  If the step does not fit the buffer (flat logits), a 4-pass radix search over the row's keys follows.
// ---------------------------------------------------------------------------------------------
constexpr int kNucleusThreads = 1024;

__device__ __forceinline__ unsigned long long fixed_mass(float x, float row_max, float inv_temp) {
  // exp((x - max) / T) in [0, 1], scaled by 2^40 and rounded down; every token gets at least 0
  const float e = __expf((x - row_max) * inv_temp);
  return static_cast<unsigned long long>(e * 1099511627776.0f);
}

constexpr int kSteps = 256;
constexpr int kMassBits = 14;   // of the 41 bits per histogram word: 2^18 tokens per lane fit 32 bits
constexpr int kMassWords = 3;
constexpr int kNucleusBytes = kMassWords * kSteps * 32 * 4;
constexpr int kNucleusGather = kNucleusBytes / 8;  // the histogram's memory is reused for the gathered tokens

// Calls f(value, index) for the elements of one warp's stretch of the row (stretches follow one another in index order).
// The 16-byte vectors are dealt to the warps evenly; the unaligned head belongs to the first, the tail to the last.
template <typename T, typename F>
__device__ __forceinline__ void for_each_in_stretch(const T* __restrict__ z, int V, F&& f) {
  constexpr int kVec = 16 / sizeof(T);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int head = static_cast<int>(((16 - (reinterpret_cast<uintptr_t>(z) & 15u)) & 15u) / sizeof(T));
  if (head > V) head = V;
  const int nvec = (V - head) / kVec, warps = kNucleusThreads / 32, per = (nvec + warps - 1) / warps;
  const int v0 = min(nvec, warp * per), v1 = min(nvec, v0 + per);
  const uint4* p = reinterpret_cast<const uint4*>(z + head);
  if (warp == 0 && lane < head) f(ldv(z, lane), lane);
  constexpr int kAhead = 4;
  int v = v0 + lane;
  for (; v + 32 * (kAhead - 1) < v1; v += 32 * kAhead) {
    uint4 q[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) q[u] = __ldg(p + v + 32 * u);
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const T* e = reinterpret_cast<const T*>(&q[u]);
#pragma unroll
      for (int j = 0; j < kVec; ++j) f(ldv(e, j), head + (v + 32 * u) * kVec + j);
    }
  }
  for (; v < v1; v += 32) {
    const uint4 q = __ldg(p + v);
    const T* e = reinterpret_cast<const T*>(&q);
#pragma unroll
    for (int j = 0; j < kVec; ++j) f(ldv(e, j), head + v * kVec + j);
  }
  const int tail = head + nvec * kVec;
  if (warp == warps - 1 && tail + lane < V) f(ldv(z, tail + lane), tail + lane);
}
// [begin, end) of warp `warp`'s stretch
template <typename T>
__device__ __forceinline__ int2 stretch_of(const T* z, int V, int warp) {
  constexpr int kVec = 16 / sizeof(T);
  int head = static_cast<int>(((16 - (reinterpret_cast<uintptr_t>(z) & 15u)) & 15u) / sizeof(T));
  if (head > V) head = V;
  const int nvec = (V - head) / kVec, warps = kNucleusThreads / 32, per = (nvec + warps - 1) / warps;
  const int v0 = min(nvec, warp * per), v1 = min(nvec, v0 + per);
  return make_int2(warp == 0 ? 0 : head + v0 * kVec, warp == warps - 1 ? V : head + v1 * kVec);
}

template <typename T>
__global__ void __launch_bounds__(kNucleusThreads)
sample_nucleus_kernel(const T* __restrict__ logits, long long ld, int V, float top_p, float inv_temp,
                      unsigned long long seed, unsigned long long offset, long long* __restrict__ out_ids,
                      float* __restrict__ out_logprob) {
  extern __shared__ unsigned long long dyn[];
  unsigned int* lanes = reinterpret_cast<unsigned int*>(dyn);  // [kMassWords][kSteps][32]
  unsigned long long* gathered = dyn;                          // [kNucleusGather]: key << 32 | index
  __shared__ unsigned long long hist[256];
  __shared__ unsigned long long warp_part[kNucleusThreads / 32];
  __shared__ float warp_max[kNucleusThreads / 32];
  __shared__ unsigned long long s_total, s_above, s_target, s_base;
  __shared__ uint32_t s_prefix;
  __shared__ int s_pick, s_step, s_warp;
  __shared__ unsigned int s_count;
  __shared__ float s_max;
  const int row = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const T* z = logits + static_cast<long long>(row) * ld;

  // ---- row maximum
  float m = -INFINITY;
  for_each_in_stretch(z, V, [&](float x, int) { m = fmaxf(m, x); });
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) warp_max[warp] = m;
  for (int i = tid; i < kMassWords * kSteps * 32; i += kNucleusThreads) lanes[i] = 0u;
  __syncthreads();
  if (warp == 0) {
    float r = warp_max[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r = fmaxf(r, __shfl_xor_sync(0xffffffffu, r, o));
    if (lane == 0) {
      s_max = r;
      s_prefix = 0u;
      s_above = 0ull;
      s_count = 0u;
      s_step = kSteps - 1;
    }
  }
  __syncthreads();
  const float row_max = s_max;

  // ---- mass per step of (max - x) / T: monotone in x, so the steps are in the order of the keys
  auto step_of = [&](float x) {
    const int b = static_cast<int>((row_max - x) * inv_temp * (kSteps / 28.f));
    return b < 0 ? 0 : (b < kSteps ? b : kSteps - 1);
  };
  for_each_in_stretch(z, V, [&](float x, int) {
    const unsigned long long mass = fixed_mass(x, row_max, inv_temp);
    if (mass == 0ull) return;
    unsigned int* h = lanes + step_of(x) * 32 + lane;
#pragma unroll
    for (int w = 0; w < kMassWords; ++w) {
      const unsigned int part = static_cast<unsigned int>(mass >> (w * kMassBits)) & ((1u << kMassBits) - 1u);
      if (part) atomicAdd(h + w * kSteps * 32, part);
    }
  });
  __syncthreads();
  for (int b = warp; b < kSteps; b += kNucleusThreads / 32) {
    unsigned long long sum = 0ull;
#pragma unroll
    for (int w = 0; w < kMassWords; ++w) sum += static_cast<unsigned long long>(lanes[(w * kSteps + b) * 32 + lane]) << (w * kMassBits);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) hist[b] = sum;
  }
  __syncthreads();
  // mass that the kept set must reach (at least one unit so that the best token is always kept), and the step that holds it
  auto locate = [&](bool descending, unsigned long long above0) {
    // lane l owns bins 8 l .. 8 l + 7 of the order; returns through s_step / s_above
    if (warp == 0) {
      unsigned long long mine = 0ull;
#pragma unroll
      for (int j = 0; j < 8; ++j) mine += hist[descending ? 255 - (lane * 8 + j) : lane * 8 + j];
      unsigned long long incl = mine;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const unsigned long long o = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += o;
      }
      const unsigned long long before = above0 + incl - mine;
      if (before < s_target && s_target <= before + mine) {  // at most one lane
        unsigned long long acc = before;
        int j = 0;
        for (; j < 7; ++j) {
          const unsigned long long h = hist[descending ? 255 - (lane * 8 + j) : lane * 8 + j];
          if (acc + h >= s_target) break;
          acc += h;
        }
        s_step = descending ? 255 - (lane * 8 + j) : lane * 8 + j;
        s_above = acc;  // mass of the tokens before the chosen bin
      }
    }
    __syncthreads();
  };
  if (warp == 0) {
    unsigned long long total = 0ull;
#pragma unroll
    for (int j = 0; j < 8; ++j) total += hist[lane * 8 + j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    if (lane == 0) {
      s_total = total;
      const double want = static_cast<double>(top_p) * static_cast<double>(total);
      const unsigned long long t = want < 1.0 ? 1ull : static_cast<unsigned long long>(want);
      s_target = t;
    }
  }
  __syncthreads();
  locate(false, 0ull);
  const int cut_step = s_step;

  // ---- gather the tokens of that step; mass of the kept tokens above it per stretch
  unsigned long long part = 0ull;
  for_each_in_stretch(z, V, [&](float x, int i) {
    const int b = step_of(x);
    if (b < cut_step) {
      part += fixed_mass(x, row_max, inv_temp);
    } else if (b == cut_step) {
      const unsigned int slot = atomicAdd(&s_count, 1u);
      if (slot < kNucleusGather) gathered[slot] = (static_cast<unsigned long long>(f2key(x)) << 32) | static_cast<uint32_t>(i);
    }
  });
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if (lane == 0) warp_part[warp] = part;
  __syncthreads();
  const unsigned int have = s_count;
  const bool fits = have <= static_cast<unsigned int>(kNucleusGather);  // uniform

  // ---- radix search for the cut key: after pass r its top 8 (r + 1) bits are known
  if (!fits && tid == 0) s_above = 0ull;
  __syncthreads();
  for (int pass = 0; pass < 4; ++pass) {
    const int shift = 24 - 8 * pass;
    for (int b = tid; b < 256; b += kNucleusThreads) hist[b] = 0ull;
    __syncthreads();
    const uint32_t prefix = s_prefix;
    const uint32_t mask = pass == 0 ? 0u : (0xffffffffu << (shift + 8));
    const unsigned long long above = s_above;
    if (fits) {
      for (unsigned int i = tid; i < have; i += kNucleusThreads) {
        const uint32_t key = static_cast<uint32_t>(gathered[i] >> 32);
        if ((key & mask) == (prefix & mask)) atomicAdd(&hist[(key >> shift) & 0xffu], fixed_mass(key2f(key), row_max, inv_temp));
      }
    } else {
      for (int i = tid; i < V; i += kNucleusThreads) {
        const float x = ldv(z, i);
        const uint32_t key = f2key(x);
        if ((key & mask) == (prefix & mask)) atomicAdd(&hist[(key >> shift) & 0xffu], fixed_mass(x, row_max, inv_temp));
      }
    }
    if (tid == 0) s_step = 0;
    __syncthreads();
    locate(true, above);
    if (tid == 0) s_prefix = prefix | (static_cast<uint32_t>(s_step) << shift);
    __syncthreads();
  }
  const uint32_t cut = s_prefix;  // keep every token with key >= cut

  // ---- mass of the kept set per stretch, then the draw
  if (fits) {
    for (unsigned int i = tid; i < have; i += kNucleusThreads) {
      const unsigned long long g = gathered[i];
      const uint32_t key = static_cast<uint32_t>(g >> 32);
      if (key < cut) continue;
      const int at = static_cast<int>(g & 0xffffffffu);
      int w = 0;  // the stretch that holds index `at`
      while (at >= stretch_of(z, V, w).y) ++w;
      atomicAdd(&warp_part[w], fixed_mass(key2f(key), row_max, inv_temp));
    }
  } else {
    part = 0ull;
    for_each_in_stretch(z, V, [&](float x, int) {
      if (f2key(x) >= cut) part += fixed_mass(x, row_max, inv_temp);
    });
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if (lane == 0) warp_part[warp] = part;
  }
  __syncthreads();
  if (tid == 0) {
    unsigned long long kept = 0ull;
    for (int w = 0; w < kNucleusThreads / 32; ++w) kept += warp_part[w];
    const uint4 rnd = philox4x32_10(
        make_uint4(static_cast<uint32_t>(offset), static_cast<uint32_t>(offset >> 32), static_cast<uint32_t>(row), 0u),
        make_uint2(static_cast<uint32_t>(seed), static_cast<uint32_t>(seed >> 32)));
    const double u = (static_cast<double>(rnd.x >> 8) + 0.5) * (1.0 / 16777216.0);
    unsigned long long t = static_cast<unsigned long long>(u * static_cast<double>(kept));
    if (t >= kept) t = kept ? kept - 1 : 0ull;
    s_total = kept;
    s_target = t;  // pick the first kept token (index order) whose inclusive cumulative mass exceeds t
    s_base = 0ull;
    s_pick = -1;
    s_warp = kNucleusThreads / 32;  // the stretch that holds it (none if nothing is kept)
    unsigned long long before = 0ull;
    for (int w = 0; w < kNucleusThreads / 32; ++w) {
      if (t < before + warp_part[w]) {
        s_warp = w;
        s_base = before;
        break;
      }
      before += warp_part[w];
    }
  }
  __syncthreads();
  const int2 range = s_warp < kNucleusThreads / 32 ? stretch_of(z, V, s_warp) : make_int2(0, 0);

  // ---- index-order scan of that stretch in tiles of kNucleusThreads tokens
  for (int base = range.x; base < range.y && s_pick < 0; base += kNucleusThreads) {
    const int i = base + tid;
    unsigned long long mine = 0ull;
    float x = 0.f;
    if (i < range.y) {
      x = ldv(z, i);
      if (f2key(x) >= cut) mine = fixed_mass(x, row_max, inv_temp);
    }
    unsigned long long incl = mine;  // inclusive scan inside the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    if (lane == 31) warp_part[warp] = incl;
    __syncthreads();
    unsigned long long before = s_base;
    for (int w = 0; w < warp; ++w) before += warp_part[w];
    const unsigned long long lo = before + incl - mine, hi = before + incl;
    if (mine != 0ull && lo <= s_target && s_target < hi) {
      s_pick = i;  // exactly one thread satisfies this
      out_ids[row] = i;
      if (out_logprob) out_logprob[row] = logf(static_cast<float>(static_cast<double>(mine) / static_cast<double>(s_total)));
    }
    __syncthreads();
    if (tid == 0) {
      unsigned long long tile = 0ull;
      for (int w = 0; w < kNucleusThreads / 32; ++w) tile += warp_part[w];
      s_base += tile;
    }
    __syncthreads();
  }
  if (tid == 0 && s_pick < 0) {  // all masses rounded to zero except none kept: fall back to the arg-max
    int best = 0;
    float bv = ldv(z, 0);
    for (int i = 1; i < V; ++i) {
      const float x = ldv(z, i);
      if (x > bv) {
        bv = x;
        best = i;
      }
    }
    out_ids[row] = best;
    if (out_logprob) out_logprob[row] = 0.f;
  }
}

}  // namespace

void sample_nucleus(const void* logits, long long ld, int dtype, int rows, int V, float top_p, float temperature,
                    unsigned long long seed, unsigned long long offset, long long* out_ids, float* out_logprob,
                    cudaStream_t stream) {
  if (rows <= 0) return;
  const float inv_temp = 1.f / temperature;
  auto launch = [&](auto kernel, auto* typed) {
    using T = std::remove_const_t<std::remove_pointer_t<decltype(typed)>>;
    static PerDeviceOnce configured;  // one per element type
    if (configured.first()) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kNucleusBytes);
    kernel<<<rows, kNucleusThreads, kNucleusBytes, stream>>>(static_cast<const T*>(logits), ld, V, top_p, inv_temp, seed, offset,
                                                             out_ids, out_logprob);
  };
  if (dtype == 0) launch(sample_nucleus_kernel<float>, static_cast<const float*>(nullptr));
  else if (dtype == 1) launch(sample_nucleus_kernel<__nv_bfloat16>, static_cast<const __nv_bfloat16*>(nullptr));
  else launch(sample_nucleus_kernel<__half>, static_cast<const __half*>(nullptr));
}

namespace {

// CTAs per row: enough for two on every SM, at most eight (the portable cluster size), and slices of at least twice the
// smallest sample: below that the merge is not repaid.  No more than leave room for 3 / 2 k candidates of each in the first
// one's sort buffer.
int sample_parts(int rows, int V, int k, int sm_count) {
  int parts = 1;
  while (parts < 8 && static_cast<long long>(rows) * parts <= sm_count && V / (parts * 2) >= 2 * kMinSample) parts *= 2;
  while (parts > 1 && static_cast<long long>(parts) * k * 3 > 2 * kCap) parts /= 2;
  return parts;
}

// Which kernel, measured over k = 1 .. 1000, 1 .. 256 rows, 5000 .. 151936 columns, fp32 and bf16 (us on one GPU; the draws are the
// same bits).  Rows that leave SMs idle get a CTA each, with deep loads (37 x 128256 fp32, k = 50: 19 against 23 with one load at a
// time); slices only where few long rows and a small k repay the cluster (1 x 151936, k = 20: 13 against 19; k = 100: no gain; 37
// rows: 27 against 21), or where k is so large that the bound from 1024 maxima lets through more than can be sorted (1 x 151936, k =
// 1000: 48 against 77).  More rows than SMs: two CTAs per SM (256 x 61000 bf16, k = 100: 23, slices 37).  Slices for the smallest k,
// for long rows with a small one, which they read once and an eighth (256 x 151936 fp32, k = 50: 48 against 59; k = 100: 61 against 60),
// for short rows, which suit their 512 threads (256 x 16000, k = 20: 12 against 14), and for the largest (256 x 128256, k = 1000: 88
// against 145).
int sample_route(int rows, int V, int k, int elem, int sm_count) {
  if (rows <= sm_count) {
    if (k > 800 && V > kMinSample) return kSampleFull;
    return rows * 7 <= sm_count && V >= 9 * kMinSample && k * 3000 <= V ? kSampleFew : kSampleRows;
  }
  const bool long_rows = static_cast<long long>(V) * elem >= 384 << 10;
  if (k <= 10 || (k <= 64 && (long_rows || V <= 2 * kMinSample)) || (k <= kFewLimit && V <= kMinSample)) return kSampleFew;
  return k > (V > kMinSample ? 640 : 800) ? kSampleFull : kSampleRows;
}

template <typename T>
void launch_sample(const void* logits, long long ld, int rows, int V, int top_k, float top_p, float inv_temp,
                   unsigned long long seed, unsigned long long offset, long long* out_ids, float* out_logprob, int sm_count, int route,
                   cudaStream_t stream) {
  const int parts = sample_parts(rows, V, top_k, sm_count);
  if (route == kSampleAuto) route = sample_route(rows, V, top_k, sizeof(T), sm_count);
  if (route == kSampleRows) {
    auto kernel = rows > sm_count ? sample_rows_kernel<T, true> : sample_rows_kernel<T, false>;
    kernel<<<rows, kRowThreads, 0, stream>>>(static_cast<const T*>(logits), ld, V, top_k, top_p, inv_temp, seed, offset, out_ids, out_logprob);
    return;
  }
  auto kernel = sample_slices_kernel<T>;
  constexpr int kBytes = kGather * 8;
  static PerDeviceOnce configured;
  if (configured.first()) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(rows) * parts);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(parts);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const bool few = route == kSampleFew;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<const T*>(logits), ld, V, top_k, top_p, inv_temp, seed, offset, out_ids, out_logprob, few);
}

}  // namespace

void sample_topk_topp(const void* logits, long long ld, int dtype, int rows, int V, int top_k, float top_p,
                      float temperature, unsigned long long seed, unsigned long long offset, long long* out_ids,
                      float* out_logprob, int sm_count, int route, cudaStream_t stream) {
  if (rows <= 0) return;
  const float inv_temp = 1.f / temperature;
  auto launch = [&](auto* typed) {
    launch_sample<std::remove_pointer_t<decltype(typed)>>(logits, ld, rows, V, top_k, top_p, inv_temp, seed, offset, out_ids, out_logprob,
                                                          sm_count, route, stream);
  };
  if (dtype == 0) launch(static_cast<float*>(nullptr));
  else if (dtype == 1) launch(static_cast<__nv_bfloat16*>(nullptr));
  else launch(static_cast<__half*>(nullptr));
}

int sample_few_limit() { return kFewLimit; }

int sample_topk_limit() { return 1024; }

}  // namespace rlk
