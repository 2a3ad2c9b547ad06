// Fused linear -> selected-token log-prob (+ entropy) for sm_100a.
//
// Forward: one persistent kernel computes z = hidden * W_local^T tile by tile with tcgen05 (the
// [N, V] logits only ever exist as 128 x 256 fp32 tiles in tensor memory), folds every tile into a
// per-row online (max, sum-exp, sum-exp*z, target-logit) record and pushes the record of each finished
// (row-tile, vocab-split) item into the partial buffer (EVERY tensor-parallel peer's, with plain peer
// stores over NVLink).  Once a row tile has all world x splits records they are merged in fixed
// (rank, split) order: on one GPU by the CTA that delivered the last one, under tensor parallelism in a
// merge phase behind the products.  No NCCL call, no separate combine kernel, bitwise identical on all ranks.
// Batches of more than one row tile run on CTA pairs (256 x 256 tiles).
//
// Backward (recompute): per token chunk, a second persistent kernel recomputes the logits tile and
// writes dz = g * (onehot - exp(z - lse)) as bf16 into a chunk workspace; the two products
// dz * W and dz^T * X then run on the shared GEMM mainloop with MN-major operands.
//
// What the reference does instead: csrc/cuda/fused_linear_logp_sm90.cu:55-280 (mma.sync tiles
// spilled to shared memory, row-serial softmax, separate combine kernel) and, for tensor
// parallelism, three NCCL all-reduces (rl_engine/kernels/ops/cuda/loss/linear_logp.py:151-161).
#include "../common/gemm2_sm100.cuh"
#include "../common/gemm_sm100.cuh"
#include "../common/tensormap.h"
#include "kernels.h"

namespace rlk {

constexpr int kLogpBN = 256;
constexpr int kLogpStages = 4;
constexpr int kLogpPairStages = 6;    // CTA-pair engine, statistics epilogue (no staging)
constexpr int kLogpPairStagesDz = 5;  // CTA-pair engine with the 64 KB dz staging tile
constexpr int kMaxWorld = 8;
// Vocab tiles per record (8192 columns), which is also one work item: a constant, so that the order of a row's sums depends
// neither on the other rows of the batch nor on the engine.  It is part of the numbers that a training run sees: the last bit
// of a log-sum-exp moves the rounding of a bf16 gradient, and with it what a run of many steps arrives at.
constexpr int kTilesPerRecord = 32;

struct LogpFwdParams {
  const long long* target;  // [N] global vocab ids
  const float* bias;        // [V_local] or null
  long long vocab_start;    // global id of local column 0
  long long global_vocab;   // > 0: a target id outside [0, global_vocab) is reported in the error word
  int rank, world;
  int slot_base;            // first record slot of this rank (sum of the lower ranks' items_per_m)
  int total_records;        // records per row over all ranks
  int row_tiles;            // 128-row tiles of tokens
  int n_pad;                // row pitch of the partial buffers (row_tiles * 128)
  float4* peer_partials[kMaxWorld];   // each: [world * items_per_m, n_pad] records (m2, s, t, zt)
  unsigned int* peer_counters[kMaxWorld];  // each: [row_tiles] arrival counters of the current set
  unsigned int* next_counters;        // local counters of the other set, zeroed by this launch
  int counter_capacity;
  float* logp;     // [N]
  float* lse;      // [N] or null
  float* entropy;  // [N] or null
  uint32_t* err;
  unsigned long long wait_limit_ns;
};

__device__ __forceinline__ void epi_bar_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

struct EpiLogpStats {
  using Params = LogpFwdParams;
  static constexpr int kCommWarps = 0;
  static constexpr int kStagingBytes = 0;
  struct State {
    float m2, s, t, zt;
    int tgt;  // local target column or -1
  };

  __device__ static void begin_item(State& st, const Params& ep, const GemmProblem& p, const WorkItem&, int row) {
    st.m2 = -INFINITY;
    st.s = 0.f;
    st.t = 0.f;
    st.zt = 0.f;
    st.tgt = -1;
    if (row < p.M) {
      const long long local = ep.target[row] - ep.vocab_start;
      if (local >= 0 && local < p.N) st.tgt = static_cast<int>(local);
    }
  }

  template <int BN>
  __device__ static void tile(State& st, const Params& ep, const GemmProblem& p, uint32_t acc, int /*row*/, int n0) {
#pragma unroll 1
    for (int c = 0; c < BN; c += 32) {
      uint32_t r[32];
      tmem_ld_32x32b_x32(acc + c, r);
      tmem_ld_wait();
      const int col0 = n0 + c;
      if (col0 >= p.N) continue;
      float v[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
      if (ep.bias != nullptr) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (col0 + j < p.N) v[j] += __ldg(ep.bias + col0 + j);
      }
      if (col0 + 32 > p.N) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (col0 + j >= p.N) v[j] = -INFINITY;
      }
      float cmax = v[0];
#pragma unroll
      for (int j = 1; j < 32; ++j) cmax = fmaxf(cmax, v[j]);
      const float new_m2 = fmaxf(st.m2, cmax * kLog2e);
      // columns of -inf only (a masked stretch of the vocabulary): exponents are taken against 0, the sum stays 0
      const float base = new_m2 == -INFINITY ? 0.f : new_m2;
      const float rescale = fast_exp2(st.m2 - base);  // 0 on the first chunk (m2 = -inf)
      // The exponentials bound this loop at short contractions (K = 512: 2048 cycles of them per tile and as many of products), so
      // the entropy's sum is formed only where it is asked for; the other sums are the same either way.
      float sum = 0.f;
      if (ep.entropy != nullptr) {
        float tsum = 0.f;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const float e = fast_exp2(fmaf(v[j], kLog2e, -base));
          sum += e;
          tsum = fmaf(e, (col0 + j < p.N) ? v[j] : 0.f, tsum);
        }
        st.t = fmaf(st.t, rescale, tsum);
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) sum += fast_exp2(fmaf(v[j], kLog2e, -base));
      }
      st.s = fmaf(st.s, rescale, sum);
      st.m2 = new_m2;
      const int tl = st.tgt - col0;
      if (tl >= 0 && tl < 32) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (j == tl) st.zt = v[j];
      }
    }
  }

  // `row` >> 7 is this CTA's 128-row tile under both engines (the pair engine's M-tiles hold two of them).
  __device__ static void end_item(State& st, const Params& ep, const GemmProblem& p, const WorkItem& w, int row) {
    const int t128 = row >> 7;
    if (t128 >= ep.row_tiles) return;  // second half of the last pair: no rows (uniform over the CTA)
    const float4 rec = make_float4(st.m2, st.s, st.t, st.zt);
    const size_t slot = static_cast<size_t>(ep.slot_base + w.split) * ep.n_pad + row;
    for (int r = 0; r < ep.world; ++r) ep.peer_partials[r][slot] = rec;
    if (ep.world == 1) {
      // One GPU: whoever delivers the last record of a row tile merges it at once.  Nobody waits, so the kernel does
      // not depend on all its CTAs being resident together, and the merges overlap other tiles' products.
      __threadfence();
      epi_bar_sync();
      __shared__ unsigned int s_last;
      if (threadIdx.x == 64) {
        unsigned int old;
        asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;"
                     : "=r"(old)
                     : "l"(ep.peer_counters[0] + t128), "r"(1u)
                     : "memory");
        s_last = old + 1u == static_cast<unsigned int>(ep.total_records) ? 1u : 0u;
        if (s_last) ep.peer_counters[0][t128] = 0u;  // the same set may be counted in again (a replayed CUDA graph)
      }
      epi_bar_sync();
      if (s_last) merge_row(ep, p, row, kMergeKernelId);
      return;
    }
    __threadfence_system();
    epi_bar_sync();
    if (threadIdx.x == 64) {  // one epilogue thread publishes the arrival
      for (int r = 0; r < ep.world; ++r) {
        asm volatile("red.release.sys.global.add.u32 [%0], %1;" ::"l"(ep.peer_counters[r] + t128), "r"(1u)
                     : "memory");
      }
    }
  }

  static constexpr uint32_t kMergeKernelId = 101u;

  // Fixed (rank, split) order: the maximum of all records, then the sums one record after the other against it.  A row's
  // value depends on its records only, not on the engine or the other rows.  Eight records' loads are in flight together.
  __device__ static void merge_row(const Params& ep, const GemmProblem& p, int row, uint32_t kernel_id) {
    if (row >= p.M) return;
    const float4* parts = ep.peer_partials[ep.rank] + row;
    const int records = ep.total_records;
    float M2 = -INFINITY, S = 0.f, T = 0.f, ZT = 0.f;
    // not through the read-only cache: other SMs and peers wrote these during this launch
#pragma unroll 8
    for (int i = 0; i < records; ++i) M2 = fmaxf(M2, __ldcg(&parts[static_cast<size_t>(i) * ep.n_pad].x));
    const float base = M2 == -INFINITY ? 0.f : M2;
#pragma unroll 8
    for (int i = 0; i < records; ++i) {
      const float4 rec = __ldcg(parts + static_cast<size_t>(i) * ep.n_pad);
      const float w = fast_exp2(rec.x - base);
      S = fmaf(rec.y, w, S);
      T = fmaf(rec.z, w, T);
      ZT += rec.w;
    }
    const float lse = (M2 + log2f(S)) * kLn2;
    if (ep.global_vocab > 0) {
      // The range check of the target ids happens here, on the device, instead of a host read-back per call: the
      // row's log-prob becomes NaN and the error word tells the host at its next check.
      const long long id = ep.target[row];
      if (id < 0 || id >= ep.global_vocab) {
        report_error(ep.err, kErrBadArgument, kernel_id, 11);
        ZT = __int_as_float(0x7fc00000);
      }
    }
    ep.logp[row] = ZT - lse;
    if (ep.lse != nullptr) ep.lse[row] = lse;
    if (ep.entropy != nullptr) ep.entropy[row] = lse - T / S;
  }
};

// Tensor parallelism only: merge phase, run by the 128 epilogue threads of each CTA after its GEMM items, attached to
// the shared mainloop through the epilogue functor's `finish` hook.
__device__ void logp_merge_phase(const LogpFwdParams& ep, const GemmProblem& p, uint32_t kernel_id) {
  const int tid = threadIdx.x - 64;  // 0..127
  const unsigned int expect = static_cast<unsigned int>(ep.total_records);
  const unsigned int* counters = ep.peer_counters[ep.rank];
  for (int t = blockIdx.x; t < ep.row_tiles; t += gridDim.x) {
    // bounded wait for all records of row tile t
    unsigned int seen = 0;
    uint64_t deadline = 0;
    bool ok = true;
    for (;;) {
      asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(seen) : "l"(counters + t) : "memory");
      if (seen >= expect) break;
      const uint64_t now = global_timer_ns();
      if (deadline == 0) deadline = now + ep.wait_limit_ns;
      if (now > deadline) {
        ok = false;
        break;
      }
      __nanosleep(200);
    }
    if (!ok) {
      report_error(ep.err, kErrPeerTimeout, kernel_id, 10);
      continue;
    }
    EpiLogpStats::merge_row(ep, p, t * kBM + tid, kernel_id);
  }
}

struct EpiLogpStatsWithMerge : EpiLogpStats {
  // Zero the counter set of the NEXT launch before this CTA publishes its first arrival.  A peer can
  // only begin its next launch after it has seen every arrival of this one, so the zeroing is ordered
  // before any arrival that will ever be counted in that set (every CTA of the grid owns >= 1 item).
  __device__ static void start(const Params& ep, const GemmProblem&) {
    const int tid = threadIdx.x - 64;
    for (int t = blockIdx.x * 128 + tid; t < ep.counter_capacity; t += gridDim.x * 128) ep.next_counters[t] = 0u;
    __threadfence();
    epi_bar_sync();
  }
  __device__ static void finish(const Params& ep, const GemmProblem& p, uint32_t kernel_id) {
    if (ep.world > 1) logp_merge_phase(ep, p, kernel_id);
  }
};

// ---------------------------------------------------------------------------------------------
// Backward epilogue: dz = g * (onehot - exp(z - lse)) written as bf16.
// ---------------------------------------------------------------------------------------------
struct LogpDzParams {
  CUtensorMap tmap_dz;  // bf16 [M, V_local], box 64 x 128, 128B swizzle
  const long long* target;
  const float* bias;
  const float* lse;    // [N] global log-sum-exp
  const float* grad;   // [N] dL/dlogp
  long long vocab_start;
};

// The tile is staged COLS columns at a time in 128B-swizzled shared memory and leaves by TMA stores: full lines reach
// L2 (one row per thread would scatter 16-byte pieces over 32 rows per instruction), M and V tails are clipped by the
// tensor map.
template <int COLS>
struct EpiLogpDz {
  static constexpr int kCommWarps = 0;
  static constexpr int kStagingBytes = kBM * COLS * 2;
  using Params = LogpDzParams;
  struct State {
    uint8_t* staging;
    float g, lse2;
    int tgt;
  };
  __device__ static void begin_item(State& st, const Params& ep, const GemmProblem& p, const WorkItem&, int row) {
    st.g = 0.f;
    st.lse2 = 0.f;
    st.tgt = -1;
    if (row < p.M) {
      st.g = ep.grad[row];
      st.lse2 = ep.lse[row] * kLog2e;
      const long long local = ep.target[row] - ep.vocab_start;
      if (local >= 0 && local < p.N) st.tgt = static_cast<int>(local);
    }
  }
  template <int BN>
  __device__ static void tile(State& st, const Params& ep, const GemmProblem& p, uint32_t acc, int row, int n0) {
    static_assert(BN % COLS == 0 && COLS % 64 == 0, "staging width must divide the tile width");
    const int r = ((threadIdx.x >> 5) & 3) * 32 + (threadIdx.x & 31);  // row inside the tile
    const int m0 = row - r;
#pragma unroll 1
    for (int seg = 0; seg < BN; seg += COLS) {
      if (threadIdx.x == 64) tma_store_wait_read<0>();  // the previous stores have finished reading the staging tile
      epi_bar_sync();
#pragma unroll 1
      for (int c = 0; c < COLS; c += 32) {
        uint32_t t[32];
        tmem_ld_32x32b_x32(acc + seg + c, t);
        tmem_ld_wait();
        const int col0 = n0 + seg + c;
        float d[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          float z = __uint_as_float(t[j]);
          if (ep.bias != nullptr && col0 + j < p.N) z += __ldg(ep.bias + col0 + j);
          d[j] = -st.g * fast_exp2(fmaf(z, kLog2e, -st.lse2));
        }
        const int tl = st.tgt - col0;
        if (tl >= 0 && tl < 32) {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (j == tl) d[j] += st.g;
        }
        uint8_t* box = st.staging + (c >> 6) * (kBM * 128) + r * 128;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          uint32_t w[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            __nv_bfloat162 b = __floats2bfloat162_rn(d[v * 8 + 2 * j], d[v * 8 + 2 * j + 1]);
            w[j] = *reinterpret_cast<uint32_t*>(&b);
          }
          const int chunk = ((c & 63) >> 3) + v;
          *reinterpret_cast<uint4*>(box + ((chunk ^ (r & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
      fence_proxy_async_smem();
      epi_bar_sync();
      if (threadIdx.x == 64 && m0 < p.M) {
#pragma unroll
        for (int b = 0; b < COLS / 64; ++b) {
          if (n0 + seg + b * 64 < p.N) tma_store_2d(&ep.tmap_dz, st.staging + b * (kBM * 128), n0 + seg + b * 64, m0);
        }
        tma_store_commit();
      }
    }
  }
  __device__ static void end_item(State&, const Params&, const GemmProblem&, const WorkItem&, int) {}
  __device__ static void finish(const Params&, const GemmProblem&, uint32_t) {
    if (threadIdx.x == 64) tma_store_wait<0>();  // the stores must have drained before the CTA's smem goes away
  }
  __device__ static void start(const Params&, const GemmProblem&) {}
};

// Column sums of a bf16 matrix [rows, V] (the bias gradient), in two fixed-order steps: kSumRows rows per block into
// fp32 partials, then the partials in order.  Eight columns per thread, one 16-byte load per row; the pitch is a
// multiple of 8, so the load of a ragged last vector stays inside its row.
constexpr int kSumRows = 128;
constexpr int kSumThreads = 128;

__global__ void __launch_bounds__(kSumThreads)
dz_colsum_kernel(const __nv_bfloat16* __restrict__ dz, long long ld, int rows, int V, float* __restrict__ part, int v_pad) {
  const int c = (blockIdx.x * kSumThreads + threadIdx.x) * 8;
  if (c >= V) return;
  const int r0 = blockIdx.y * kSumRows, r1 = min(rows, r0 + kSumRows);
  float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
  for (int r = r0; r < r1; ++r) {
    const uint4 q = __ldg(reinterpret_cast<const uint4*>(dz + r * ld + c));
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __bfloat1622float2(h[j]);
      s[2 * j] += f.x;
      s[2 * j + 1] += f.y;
    }
  }
  float4* out = reinterpret_cast<float4*>(part + static_cast<long long>(blockIdx.y) * v_pad + c);
  out[0] = make_float4(s[0], s[1], s[2], s[3]);
  out[1] = make_float4(s[4], s[5], s[6], s[7]);
}

__global__ void dz_colsum_finish_kernel(const float* __restrict__ part, int chunks, int V, int v_pad, float* __restrict__ out,
                                        bool accumulate) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= V) return;
  float s = accumulate ? out[c] : 0.f;
  for (int i = 0; i < chunks; ++i) s += part[static_cast<long long>(i) * v_pad + c];
  out[c] = s;
}

// ---------------------------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------------------------
// Per kernel, not per signature: the two engines' kernels have the same type.
template <auto Kernel>
static void set_smem(int bytes) {
  static PerDeviceOnce done;
  if (done.first()) {
    cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  }
}

int linear_logp_vocab_tiles_per_split() { return kTilesPerRecord; }

void linear_logp_workspace_shape(int n_tokens, int v_local, int world, int* items_per_m, int* n_pad, int* tiles_m) {
  const GemmProblem p = make_gemm_problem(n_tokens, v_local, 64, kLogpBN, linear_logp_vocab_tiles_per_split(), 1);
  *items_per_m = p.items_per_m;
  *tiles_m = p.tiles_m;
  *n_pad = p.tiles_m * kBM;
  (void)world;
}

namespace {

GemmProblem pair_problem(int M, int N, int K, int tiles_per_item) {
  GemmProblem p = make_gemm_problem(M, N, K, kLogpBN, tiles_per_item, 1);
  p.tiles_m = (M + kPairBM - 1) / kPairBM;
  p.num_items = p.tiles_m * p.items_per_m;
  p.group_m = raster_group_m(p.tiles_m, 2 * K, 8);
  return p;
}

// A pair of SMs and two single SMs do the same products per round of items; the pair reads a third less operand data
// through L2, the single engine pads M to 128 instead of 256.  So: pairs unless the padding costs them a round.
bool pair_is_better(int M, int items_per_m, int sm_count) {
  if (M <= kBM || sm_count < 2) return false;
  const long long single = static_cast<long long>((M + kBM - 1) / kBM) * items_per_m;
  const long long pair = static_cast<long long>((M + kPairBM - 1) / kPairBM) * items_per_m;
  const long long pairs = sm_count / 2;
  return (pair + pairs - 1) / pairs <= (single + sm_count - 1) / sm_count;
}

}  // namespace

void linear_logp_forward(const LinearLogpFwdArgs& a, cudaStream_t stream) {
  const int row_tiles = (a.n_tokens + kBM - 1) / kBM;
  const int records = ((a.v_local + kLogpBN - 1) / kLogpBN + kTilesPerRecord - 1) / kTilesPerRecord;
  // keep as many token tiles per group as stay L2-resident, so the weight streams from DRAM once per group
  GemmProblem p = make_gemm_problem(a.n_tokens, a.v_local, a.hidden_dim, kLogpBN, kTilesPerRecord,
                                    raster_group_m(row_tiles, a.hidden_dim, 16, 64ll << 20));
  const CUtensorMap ta = make_tmap_2d_bf16(a.hidden, a.n_tokens, a.hidden_dim, a.ld_hidden, kBM, kBK);
  LogpFwdParams ep;
  ep.target = a.target;
  ep.bias = a.bias;
  ep.vocab_start = a.vocab_start;
  ep.global_vocab = a.global_vocab;
  ep.rank = a.rank;
  ep.world = a.world;
  ep.slot_base = a.slot_base;
  ep.total_records = a.total_records > 0 ? a.total_records : records * a.world;
  ep.row_tiles = row_tiles;
  ep.n_pad = row_tiles * kBM;
  for (int r = 0; r < kMaxWorld; ++r) {
    ep.peer_partials[r] = r < a.world ? reinterpret_cast<float4*>(a.peer_partials[r]) : nullptr;
    ep.peer_counters[r] = r < a.world ? a.peer_counters[r] : nullptr;
  }
  ep.next_counters = a.next_counters;
  ep.counter_capacity = a.counter_capacity;
  ep.logp = a.logp;
  ep.lse = a.lse;
  ep.entropy = a.entropy;
  ep.err = a.err;
  ep.wait_limit_ns = a.wait_limit_ns ? a.wait_limit_ns : kWaitLimitNs;
  // Tensor parallelism stays on single CTAs: its merge waits for other CTAs' records, so all must be resident.
  if (a.world == 1 && pair_is_better(a.n_tokens, p.items_per_m, a.sm_count)) {
    p = pair_problem(a.n_tokens, a.v_local, a.hidden_dim, kTilesPerRecord);
    const CUtensorMap tb = make_tmap_2d_bf16(a.weight, a.v_local, a.hidden_dim, a.ld_weight, kLogpBN / 2, kBK);
    constexpr auto kernel = gemm_pair_sm100_kernel<kLogpBN, false, false, kLogpPairStages, EpiLogpStatsWithMerge>;
    using L = PairSmem<kLogpBN, kLogpPairStages>;
    set_smem<kernel>(L::kDynamicBytes);
    const int pairs = p.num_items < a.sm_count / 2 ? p.num_items : a.sm_count / 2;
    kernel<<<2 * pairs, kGemmThreads, L::kDynamicBytes, stream>>>(ta, tb, p, ep, a.err, 103u);
    return;
  }
  const CUtensorMap tb = make_tmap_2d_bf16(a.weight, a.v_local, a.hidden_dim, a.ld_weight, kLogpBN, kBK);
  constexpr auto kernel = gemm_sm100_kernel<kLogpBN, false, false, kLogpStages, EpiLogpStatsWithMerge>;
  using L = GemmSmem<kLogpBN, kLogpStages>;
  set_smem<kernel>(L::kDynamicBytes);
  int grid = p.num_items < a.sm_count ? p.num_items : a.sm_count;
  if (grid < 1) grid = 1;
  kernel<<<grid, kGemmThreads, L::kDynamicBytes, stream>>>(ta, tb, p, ep, a.err, 101u);
}

void linear_logp_dz(const LinearLogpDzArgs& a, cudaStream_t stream) {
  const GemmProblem p = make_gemm_problem(a.n_tokens, a.v_local, a.hidden_dim, kLogpBN, 1,
                                          raster_group_m((a.n_tokens + kBM - 1) / kBM, a.hidden_dim, 16, 64ll << 20));
  const CUtensorMap ta = make_tmap_2d_bf16(a.hidden, a.n_tokens, a.hidden_dim, a.ld_hidden, kBM, kBK);
  LogpDzParams ep;
  ep.tmap_dz = make_tmap_2d_bf16(a.dz, a.n_tokens, a.v_local, a.ld_dz, kBM, 64);
  ep.target = a.target;
  ep.bias = a.bias;
  ep.lse = a.lse;
  ep.grad = a.grad;
  ep.vocab_start = a.vocab_start;
  if (pair_is_better(a.n_tokens, p.items_per_m, a.sm_count)) {
    const GemmProblem pp = pair_problem(a.n_tokens, a.v_local, a.hidden_dim, 1);
    const CUtensorMap tb = make_tmap_2d_bf16(a.weight, a.v_local, a.hidden_dim, a.ld_weight, kLogpBN / 2, kBK);
    using Epi = EpiLogpDz<256>;
    constexpr auto kernel = gemm_pair_sm100_kernel<kLogpBN, false, false, kLogpPairStagesDz, Epi>;
    using L = PairSmem<kLogpBN, kLogpPairStagesDz, Epi::kStagingBytes>;
    set_smem<kernel>(L::kDynamicBytes);
    const int pairs = pp.num_items < a.sm_count / 2 ? pp.num_items : a.sm_count / 2;
    kernel<<<2 * pairs, kGemmThreads, L::kDynamicBytes, stream>>>(ta, tb, pp, ep, a.err, 104u);
    return;
  }
  const CUtensorMap tb = make_tmap_2d_bf16(a.weight, a.v_local, a.hidden_dim, a.ld_weight, kLogpBN, kBK);
  using Epi = EpiLogpDz<128>;
  constexpr auto kernel = gemm_sm100_kernel<kLogpBN, false, false, kLogpStages, Epi>;
  using L = GemmSmem<kLogpBN, kLogpStages, Epi::kStagingBytes>;
  set_smem<kernel>(L::kDynamicBytes);
  int grid = p.num_items < a.sm_count ? p.num_items : a.sm_count;
  if (grid < 1) grid = 1;
  kernel<<<grid, kGemmThreads, L::kDynamicBytes, stream>>>(ta, tb, p, ep, a.err, 102u);
}

long long dz_colsum_workspace_floats(int rows, int V) {
  return static_cast<long long>((rows + kSumRows - 1) / kSumRows) * ((V + 7) / 8 * 8);
}

void dz_colsum(const __nv_bfloat16* dz, long long ld, int rows, int V, float* workspace, float* out, bool accumulate,
               cudaStream_t stream) {
  if (rows <= 0 || V <= 0) return;
  const int v_pad = (V + 7) / 8 * 8, chunks = (rows + kSumRows - 1) / kSumRows;
  const dim3 grid((v_pad / 8 + kSumThreads - 1) / kSumThreads, chunks);
  dz_colsum_kernel<<<grid, kSumThreads, 0, stream>>>(dz, ld, rows, V, workspace, v_pad);
  dz_colsum_finish_kernel<<<(V + 255) / 256, 256, 0, stream>>>(workspace, chunks, V, v_pad, out, accumulate);
}

}  // namespace rlk
