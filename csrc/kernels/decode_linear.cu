// Linear layers of a decoding step (a handful of tokens): y = x W^T with the weight streamed once, and the elementwise
// work that follows a projection done in its epilogue.
//
// What bounds it: the weight bytes.  A skinny GEMM that keeps the tokens on the M side pads them to 128 rows, loads 16 KB
// of mostly empty token tile beside every 8 KB of weight and gets its parallelism from N alone (64 CTAs for a
// 4096-wide output).  Here the WEIGHT is the 128-row operand and the tokens are the N side (16 .. 128 columns), so a stage
// is 16 KB of weight and at most as much of tokens, and the (output tile, k-block) units of the whole layer are dealt to the
// CTAs in equal contiguous ranges: every SM streams the same number of bytes whatever the shape.  A tile that is cut by a range border is
// summed from fp32 partials in range order by whoever delivers the last one (no spinning, bitwise reproducible, the cut
// depends on the layer and the machine only, never on the tokens).  The plain GEMMs (bf16 and fp8), whose rows have the
// same bits at any number of rows, deal whole tiles.
//
// The CTA needs less than half an SM's shared memory on purpose: with programmatic dependent launch the next layer's CTAs
// become resident beside this one's and fetch their first weight stages (weights do not depend on the previous
// kernel) while this layer's tail drains.
//
//   warp 0     : TMA producer     warp 1 : tcgen05.mma issuer (128 x NT x 16)     warps 2..5 : epilogue, lane = output feature
#include <algorithm>

#include "../common/gemm_sm100.cuh"
#include "../common/tensormap.h"
#include "kernels.h"

namespace rlk {
namespace {

constexpr int kChunk = 16;  // tokens per epilogue step
constexpr uint32_t kKernelId = 120u;

__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// DEEP: the whole SM for one CTA.
template <int NT, bool DEEP>
struct DecSmem {
  static constexpr int kWBytes = 128 * 128;
  static constexpr int kXBytes = NT * 128;
  static constexpr int kStageBytes = kWBytes + kXBytes;
  static constexpr int kStages = DEEP ? 200 * 1024 / kStageBytes : (NT <= 32 ? 5 : (NT == 64 ? 4 : 3));
  static constexpr int kXch = kStages * kStageBytes;            // float [kChunk][128]
  static constexpr int kBars = kXch + kChunk * 128 * 4;
  static constexpr int kBytes = kBars + (2 * kStages + 4) * 8 + 16;
  static constexpr int kDynamic = kBytes + 1024;
  static_assert(kDynamic <= (DEEP ? 227 : 113) * 1024, "two CTAs must fit an SM, or one deep one");
};

// The (tile, k-block) units of CTA c: [c T / G, (c + 1) T / G), in units of `step` (one k-block, or a whole tile).
__device__ __forceinline__ long long range_begin(long long total, int c, int grid, int step = 1) {
  return total / step * c / grid * step;
}
__device__ __forceinline__ int range_owner(long long total, long long unit, int grid) {
  return static_cast<int>(((unit + 1) * grid - 1) / total);
}

template <int NT, int ELT, int MODE, bool DEEP>
__global__ void __launch_bounds__(192)
decode_linear_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                     const __grid_constant__ DecodeLinearArgs p, const int tiles, const int k_blocks) {
  using L = DecSmem<NT, DEEP>;
  constexpr int kElems = 128 / ELT;  // elements of one 128-byte k-block
  constexpr uint32_t kTmemCols = 2 * NT;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::kBars);
  uint64_t* empty_bar = full_bar + L::kStages;
  uint64_t* tmem_full = empty_bar + L::kStages;
  uint64_t* tmem_empty = tmem_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  float* xch = reinterpret_cast<float*>(smem + L::kXch);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long total = static_cast<long long>(tiles) * k_blocks;
  const int grid = static_cast<int>(gridDim.x), cta = static_cast<int>(blockIdx.x);
  const int step = p.whole_tiles ? k_blocks : 1;
  const long long u0 = range_begin(total, cta, grid, step), u1 = range_begin(total, cta + 1, grid, step);

  if (threadIdx.x == 0) {
    for (int s = 0; s < L::kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tmem_full[b], 1);
      mbar_init(&tmem_empty[b], 128);
    }
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      auto load_w = [&](long long u, int stage) {
        const int tile = static_cast<int>(u / k_blocks), k0 = static_cast<int>(u - static_cast<long long>(tile) * k_blocks) * kElems;
        uint8_t* sw = smem + stage * L::kStageBytes;
        mbar_arrive_expect_tx(&full_bar[stage], L::kStageBytes);
        if constexpr (MODE == kDecodeSwiglu) {  // 64 gate rows above the 64 up rows of the same outputs
          tma_load_2d(sw, &tmap_w, &full_bar[stage], k0, tile * 64);
          tma_load_2d(sw + L::kWBytes / 2, &tmap_w, &full_bar[stage], k0, p.N / 2 + tile * 64);
        } else {
          tma_load_2d(sw, &tmap_w, &full_bar[stage], k0, tile * 128);
        }
      };
      auto load_x = [&](long long u, int stage) {
        const int k0 = static_cast<int>(u % k_blocks) * kElems;
        tma_load_2d(smem + stage * L::kStageBytes + L::kWBytes, &tmap_x, &full_bar[stage], k0, 0);
      };
      // the first stages' weights are requested before the previous kernel has finished, its outputs afterwards
      if (!p.early_weights) grid_dep_wait();
      const int ahead = static_cast<int>(min(u1 - u0, static_cast<long long>(L::kStages)));
      for (int s = 0; s < ahead; ++s) load_w(u0 + s, s);
      grid_dep_wait();
      grid_dep_launch();
      for (int s = 0; s < ahead; ++s) load_x(u0 + s, s);
      int stage = ahead == L::kStages ? 0 : ahead;
      uint32_t phase = ahead == L::kStages ? 1 : 0;
      for (long long u = u0 + ahead; u < u1 && !*abort_flag; ++u) {
        mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.err, kKernelId, 1);
        if (*abort_flag) break;
        load_w(u, stage);
        load_x(u, stage);
        if (++stage == L::kStages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = ELT == 1 ? umma_idesc_e4m3(128, NT) : umma_idesc_bf16(128, NT, false, false);
      int stage = 0, buf = 0;
      uint32_t phase = 0, buf_phase = 0;
      for (long long u = u0; u < u1 && !*abort_flag;) {
        const int tile = static_cast<int>(u / k_blocks);
        const long long end = min(u1, static_cast<long long>(tile + 1) * k_blocks);
        mbar_wait(&tmem_empty[buf], buf_phase ^ 1, abort_flag, p.err, kKernelId, 2);
        if (*abort_flag) break;
        tc_fence_after();
        const uint32_t d = tmem + buf * NT;
        bool first = true;
        for (; u < end; ++u) {
          mbar_wait(&full_bar[stage], phase, abort_flag, p.err, kKernelId, 3);
          if (*abort_flag) break;
          tc_fence_after();
          const uint32_t sw = smem_u32(smem + stage * L::kStageBytes), sx = sw + L::kWBytes;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint64_t da = umma_smem_desc_sw128(sw + k * 32, 16, 1024), db = umma_smem_desc_sw128(sx + k * 32, 16, 1024);
            if constexpr (ELT == 1) umma_f8(d, da, db, idesc, first && k == 0 ? 0u : 1u);
            else umma_bf16(d, da, db, idesc, first && k == 0 ? 0u : 1u);
          }
          first = false;
          umma_commit(&empty_bar[stage]);
          if (++stage == L::kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
        umma_commit(&tmem_full[buf]);
        if (++buf == 2) {
          buf = 0;
          buf_phase ^= 1;
        }
      }
    }
  } else {
    grid_dep_wait();  // everything below reads or overwrites what earlier kernels touch
    const int quad = warp & 3;
    const int f = quad * 32 + lane;  // feature within the tile = TMEM lane
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    __shared__ unsigned int s_last;
    __shared__ long long pos_s[MODE == kDecodeQkv ? NT : 1], slot_s[MODE == kDecodeQkv ? NT : 1];
    if constexpr (MODE == kDecodeQkv) {  // one round trip for all tokens; an index outside its table is reported and skipped
      for (int t = threadIdx.x - 64; t < p.n; t += 128) {
        const long long pos = __ldcg(p.positions + t), slot = __ldcg(p.slots + t);
        const bool pos_ok = pos >= 0 && pos < p.table_rows, slot_ok = slot >= 0 && slot < p.cache_rows;
        if (!pos_ok) report_error(p.err, kErrBadIndex, kKernelId, 10);
        if (!slot_ok) report_error(p.err, kErrBadIndex, kKernelId, 11);
        pos_s[t] = pos_ok ? pos : 0;
        slot_s[t] = slot_ok ? slot : -1;
      }
      epi_sync();
    }
    int buf = 0;
    uint32_t buf_phase = 0;
    for (long long u = u0; u < u1;) {
      const int tile = static_cast<int>(u / k_blocks);
      const long long t0 = static_cast<long long>(tile) * k_blocks, t1 = t0 + k_blocks;
      const long long end = min(u1, t1);
      const bool whole = u == t0 && end == t1;
      mbar_wait(&tmem_full[buf], buf_phase, abort_flag, p.err, kKernelId, 4);
      tc_fence_after();
      const uint32_t acc = tmem + buf * NT + lane_addr;
      const int c_first = range_owner(total, t0, grid), c_last = range_owner(total, t1 - 1, grid);
      // partial slots: 2 c for the tile a range begins in, 2 c + 1 for the one it ends in
      auto slot_of = [&](int c) {
        const bool begins = range_begin(total, c, grid) >= t0;
        return p.partials + static_cast<long long>(2 * c + (begins ? 0 : 1)) * 128 * NT + f * 4;
      };
      bool finish = whole;
      if (!whole) {
        float* mine = slot_of(cta);
#pragma unroll 1
        for (int c0 = 0; c0 < NT; c0 += kChunk) {
          uint32_t r[kChunk];
          tmem_ld_32x32b_x16(acc + c0, r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < kChunk; j += 4) {
            *reinterpret_cast<uint4*>(mine + (c0 + j) * 128) = make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
          }
        }
        __threadfence();
        epi_sync();
        if (threadIdx.x == 64) {
          unsigned int old;
          asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;" : "=r"(old) : "l"(p.counters + tile), "r"(1u) : "memory");
          s_last = old + 1u == static_cast<unsigned int>(c_last - c_first + 1) ? 1u : 0u;
        }
        epi_sync();
        finish = s_last != 0u;
      }
      if (finish) {
        // row of W that this lane holds, its scale and bias
        int w_row = tile * 128 + f;
        if constexpr (MODE == kDecodeSwiglu) w_row = (f < 64 ? 0 : p.N / 2) + tile * 64 + (f & 63);
        const bool live = w_row < p.N;
        float sw = 1.f, bias = 0.f;
        if constexpr (ELT == 1) sw = live ? p.scale_w[w_row] : 0.f;
        if constexpr (MODE == kDecodeQkv) bias = p.bias != nullptr ? __bfloat162float(p.bias[w_row]) : 0.f;
#pragma unroll 1
        for (int c0 = 0; c0 < NT; c0 += kChunk) {
          if (c0 >= p.n) break;
          // everything this step needs from memory is requested together
          float v[kChunk], sx[kChunk], res[kChunk];
          if constexpr (ELT == 1) {
#pragma unroll
            for (int j = 0; j < kChunk; ++j) sx[j] = c0 + j < p.n ? __ldcg(p.scale_x + c0 + j) : 0.f;
          }
          if constexpr (MODE == kDecodeStore) {
            if (p.residual != nullptr && live) {
#pragma unroll
              for (int j = 0; j < kChunk; ++j)
                res[j] = c0 + j < p.n ? __bfloat162float(__ldcg(p.residual + static_cast<long long>(c0 + j) * p.ld_residual + w_row)) : 0.f;
            }
          }
          if (whole) {
            uint32_t r[kChunk];
            tmem_ld_32x32b_x16(acc + c0, r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < kChunk; ++j) v[j] = __uint_as_float(r[j]);
          } else {
#pragma unroll
            for (int j = 0; j < kChunk; ++j) v[j] = 0.f;
            // four partials at a time, all their loads in flight together; added in range order
            constexpr int kAhead = 4;
#pragma unroll 1
            for (int c = c_first; c <= c_last; c += kAhead) {
              float4 q[kAhead][kChunk / 4];
#pragma unroll
              for (int a = 0; a < kAhead; ++a) {
                if (c + a <= c_last) {
                  const float* part = slot_of(c + a) + c0 * 128;
#pragma unroll
                  for (int j = 0; j < kChunk / 4; ++j) q[a][j] = __ldcg(reinterpret_cast<const float4*>(part + j * 512));
                }
              }
#pragma unroll
              for (int a = 0; a < kAhead; ++a) {
                if (c + a <= c_last) {
#pragma unroll
                  for (int j = 0; j < kChunk / 4; ++j) {
                    v[4 * j] += q[a][j].x;
                    v[4 * j + 1] += q[a][j].y;
                    v[4 * j + 2] += q[a][j].z;
                    v[4 * j + 3] += q[a][j].w;
                  }
                }
              }
            }
          }
          if constexpr (ELT == 1) {
#pragma unroll
            for (int j = 0; j < kChunk; ++j) v[j] = v[j] * sx[j] * sw;  // the order of the 256-wide engines: the same bits
          }
          if constexpr (MODE == kDecodeStore) {
            if (live) {
#pragma unroll
              for (int j = 0; j < kChunk; ++j) {
                const int t = c0 + j;
                if (t < p.n) {
                  float x = v[j];
                  if (p.residual != nullptr) x += res[j];
                  p.out[static_cast<long long>(t) * p.ldo + w_row] = __float2bfloat16_rn(x);
                }
              }
            }
          } else {
            // pairs of features 64 lanes apart (gate and up, the two halves of a rotation) meet through shared memory
            epi_sync();  // the previous step's readers are done
#pragma unroll
            for (int j = 0; j < kChunk; ++j) xch[j * 128 + f] = v[j] + bias;
            epi_sync();
            if constexpr (MODE == kDecodeSwiglu) {
              const int o = tile * 64 + (f & 63);
#pragma unroll
              for (int i = 0; i < kChunk / 2; ++i) {  // each half of the lanes takes every other token
                const int j = 2 * i + (f >> 6), t = c0 + j;
                const float g = xch[j * 128 + (f & 63)], up = xch[j * 128 + 64 + (f & 63)];
                if (t < p.n) p.out[static_cast<long long>(t) * p.ldo + o] = __float2bfloat16_rn(g / (1.f + __expf(-g)) * up);
              }
            } else {  // kDecodeQkv: one tile is one head
              const int half = f & 63, kv_heads = p.hkv;
              float cs[kChunk], sn[kChunk];
              if (tile < p.hq + kv_heads) {
#pragma unroll
                for (int j = 0; j < kChunk; ++j) {
                  const long long at = c0 + j < p.n ? pos_s[c0 + j] * 64 + half : half;
                  cs[j] = __ldg(p.cos + at);
                  sn[j] = __ldg(p.sin + at);
                }
              }
              const int rep = p.hq / kv_heads, kv = tile / rep;
#pragma unroll
              for (int j = 0; j < kChunk; ++j) {
                const int t = c0 + j;
                if (t < p.n) {
                  float x = xch[j * 128 + f];
                  if (tile < p.hq + kv_heads) {
                    const float y = xch[j * 128 + (f ^ 64)];
                    x = f < 64 ? x * cs[j] - y * sn[j] : x * cs[j] + y * sn[j];
                  }
                  const __nv_bfloat16 b = __float2bfloat16_rn(x);
                  if (tile < p.hq) {
                    p.q_rows[((static_cast<long long>(t) * rep + tile - kv * rep) * kv_heads + kv) * 128 + f] = b;
                  } else if (slot_s[t] >= 0) {
                    const bool is_v = tile >= p.hq + kv_heads;
                    const int head = tile - p.hq - (is_v ? kv_heads : 0);
                    (is_v ? p.cache_v : p.cache_k)[(slot_s[t] * kv_heads + head) * 128 + f] = b;
                  }
                }
              }
            }
          }
        }
      }
      tc_fence_before();
      mbar_arrive(&tmem_empty[buf]);
      if (++buf == 2) {
        buf = 0;
        buf_phase ^= 1;
      }
      u = end;
    }
  }

  if (*abort_flag) {
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmemCols);
  }
}

// CTAs of a launch.  A tile cut between CTAs costs the last of them a round trip through memory (fence, counter, partials:
// 5 us and more at the end of a 20 us layer), a CTA that holds two cut tiles pays it twice.  So:
//   - up to two tiles per SM and no fewer than one: a CTA per tile, two to an SM; they share the memory's bandwidth evenly
//     whether an SM holds one or two (gate / up projection of 32 tokens, 235 MB: 52 -> 45 us).
//   - fewer: the largest number of equal K splits per tile that the SMs hold, if that uses three quarters of them (each
//     CTA has one tile: 21 -> 19 and 20 -> 18 us for 50 and 34 MB); ranges that ignore the tile borders otherwise, because
//     SMs left out cost more than the cut.  A step of four 4096-wide layers and a 128256-row head: 839 -> 792 us.
int grid_of(int tiles, int k_blocks, bool whole_tiles, int sm_count) {
  if (whole_tiles) return tiles <= 2 * sm_count ? tiles : sm_count;
  if (tiles >= sm_count) return tiles <= 2 * sm_count ? tiles : sm_count;
  const int splits = std::min(sm_count / tiles, k_blocks);
  if (tiles * splits * 4 >= sm_count * 3 || splits == k_blocks) return tiles * splits;
  return static_cast<int>(std::min<long long>(static_cast<long long>(tiles) * k_blocks, sm_count));
}

template <int NT, int ELT, int MODE, bool DEEP>
void launch_as(const DecodeLinearArgs& a, int tiles, int k_blocks, int grid, cudaStream_t stream) {
  using L = DecSmem<NT, DEEP>;
  const uint32_t w_box = MODE == kDecodeSwiglu ? 64 : 128;
  const CUtensorMap tw = ELT == 1 ? make_tmap_2d_u8(a.w, a.N, a.K, a.ld_w, w_box, 128)
                                  : make_tmap_2d_bf16(a.w, a.N, a.K, a.ld_w, w_box, 64);
  const CUtensorMap tx = ELT == 1 ? make_tmap_2d_u8(a.x, a.n, a.K, a.ld_x, NT, 128) : make_tmap_2d_bf16(a.x, a.n, a.K, a.ld_x, NT, 64);
  auto kernel = decode_linear_kernel<NT, ELT, MODE, DEEP>;
  static PerDeviceOnce configured;
  if (configured.first()) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kDynamic);
  launch_dependent(kernel, dim3(static_cast<unsigned>(grid)), dim3(192), L::kDynamic, stream, tw, tx, a, tiles, k_blocks);
}

template <int NT, int ELT, int MODE>
void launch(const DecodeLinearArgs& a, cudaStream_t stream) {
  const int tiles = MODE == kDecodeSwiglu ? a.N / 128 : (a.N + 127) / 128;
  const int k_blocks = (a.K * ELT + 127) / 128;
  const int grid = grid_of(tiles, k_blocks, a.whole_tiles, a.sm_count);
  if constexpr (ELT == 1) {
    // Whole tiles of an 8-bit weight that leave SMs idle: each CTA keeps twice the bytes in flight, with the shared memory of
    // the second CTA that its SM will not get (with three tokens, 16 projections 425 -> 400 us).
    if (grid <= a.sm_count / 2) return launch_as<NT, ELT, MODE, true>(a, tiles, k_blocks, grid, stream);
  }
  launch_as<NT, ELT, MODE, false>(a, tiles, k_blocks, grid, stream);
}

template <int NT>
void by_mode(const DecodeLinearArgs& a, cudaStream_t stream) {
  if (a.fp8) launch<NT, 1, kDecodeStore>(a, stream);
  else if (a.mode == kDecodeSwiglu) launch<NT, 2, kDecodeSwiglu>(a, stream);
  else if (a.mode == kDecodeQkv) launch<NT, 2, kDecodeQkv>(a, stream);
  else launch<NT, 2, kDecodeStore>(a, stream);
}

int padded_tokens(int n) { return n <= 16 ? 16 : (n <= 32 ? 32 : (n <= 64 ? 64 : 128)); }

}  // namespace

long long decode_linear_partial_floats(int n, int sm_count) { return 2ll * sm_count * 128 * padded_tokens(n); }

void decode_linear(const DecodeLinearArgs& a, cudaStream_t stream) {
  if (a.n <= 0 || a.N <= 0) return;
  const int nt = padded_tokens(a.n);
  if (nt == 16) by_mode<16>(a, stream);
  else if (nt == 32) by_mode<32>(a, stream);
  else if (nt == 64) by_mode<64>(a, stream);
  else by_mode<128>(a, stream);
}

}  // namespace rlk
