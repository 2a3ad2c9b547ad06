// Linear layers of a decoding step (a handful of tokens): y = x W^T with the weight streamed once, and the elementwise
// work that follows a projection done in its epilogue.
//
// What bounds it: the weight bytes.  A skinny GEMM that keeps the tokens on the M side pads them to 128 rows, loads 16 KB
// of mostly empty token tile beside every 8 KB of weight.  Here the WEIGHT is the row operand and the tokens are the N side
// (16 .. 128 columns), and a tile holds 64 or 128 rows of the weight (tile_rows_of).  The tensor core always multiplies 128
// rows: of a tile of 64 it reads whatever lies behind it in shared memory, and those lanes of the accumulator are never looked at.
//
// K is summed in one piece and every intermediate result is rounded where the separate kernels round it (the product to bf16,
// then bias, rotation, residual or SwiGLU): a row has the bits of those kernels, with any number of rows, and which kernel a
// projection runs on is a matter of speed alone.  What that costs: 16 columns or 128, an accumulation into the same columns
// takes 90 ns a step of 16, so 4096 of K are 22 us and 14336 are 72 us whatever the tile.  Splits of K over CTAs avoid it
// (50 MB for 32 tokens 19 us), but then a row's bits depend on the route, and the sum of the partials by one CTA made a step of
// four 1024-wide layers with 128 tokens 845 us instead of 383.
//
// A CTA needs less than half an SM's shared memory on purpose: with programmatic dependent launch the next layer's CTAs
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

constexpr uint32_t kKernelId = 120u;

template <int NT, int WR>
struct DecSmem {
  static constexpr int kChunk = 16;  // tokens per epilogue step
  static constexpr int kWBytes = WR * 128;
  static constexpr int kXBytes = NT * 128;
  static constexpr int kStageBytes = kWBytes + kXBytes;
  static constexpr int kXchBytes = kChunk * WR * 4;  // float [kChunk][WR]
  static constexpr int kLimit = 110 * 1024;          // two CTAs, their static shared memory and the reserved kilobytes fit an SM
  // the tensor core reads 128 rows from the start of every stage, the last one too
  static constexpr int kFitRead = (kLimit - 1024 - 128 * 128) / kStageBytes + 1;
  static constexpr int kFitUsed = (kLimit - 2048 - kXchBytes) / kStageBytes;
  static constexpr int kFit = kFitRead < kFitUsed ? kFitRead : kFitUsed;
  static constexpr int kStages = kFit < 16 ? kFit : 16;
  static constexpr int kXch = kStages * kStageBytes;
  static constexpr int kBars = kXch + kXchBytes;
  static constexpr int kUsed = kBars + (2 * kStages + 4) * 8 + 16;
  static constexpr int kRead = (kStages - 1) * kStageBytes + 128 * 128;
  static constexpr int kDynamic = (kUsed > kRead ? kUsed : kRead) + 1024;
  static_assert(kStages >= 2 && kDynamic <= kLimit, "two CTAs must fit an SM");
};

// The tiles of CTA c: [c T / G, (c + 1) T / G).
__device__ __forceinline__ int first_tile(int tiles, int c, int grid) {
  return static_cast<int>(static_cast<long long>(tiles) * c / grid);
}

__device__ __forceinline__ float round_bf16(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

template <int NT, int WR, int ELT, int MODE>
__global__ void __launch_bounds__(192, 2)
decode_linear_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                     const __grid_constant__ DecodeLinearArgs p, const int tiles, const int k_blocks) {
  using L = DecSmem<NT, WR>;
  constexpr int kChunk = L::kChunk;
  constexpr int kHalf = WR / 2;
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
  const int grid = static_cast<int>(gridDim.x), cta = static_cast<int>(blockIdx.x);
  const int t_begin = first_tile(tiles, cta, grid), t_end = first_tile(tiles, cta + 1, grid);

  if (threadIdx.x == 0) {
    for (int s = 0; s < L::kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tmem_full[b], 1);
      mbar_init(&tmem_empty[b], WR);
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
      auto load_w = [&](int tile, int kb, int stage) {
        const int k0 = kb * kElems;
        uint8_t* sw = smem + stage * L::kStageBytes;
        mbar_arrive_expect_tx(&full_bar[stage], L::kStageBytes);
        if constexpr (MODE == kDecodeSwiglu) {  // the gate rows above the up rows of the same outputs
          tma_load_2d(sw, &tmap_w, &full_bar[stage], k0, tile * kHalf);
          tma_load_2d(sw + L::kWBytes / 2, &tmap_w, &full_bar[stage], k0, p.N / 2 + tile * kHalf);
        } else if constexpr (MODE == kDecodeQkv) {  // rows of the first half of a head above their partners in the rotation
          constexpr int kPerHead = 128 / WR;
          const int row = tile / kPerHead * 128 + tile % kPerHead * kHalf;
          tma_load_2d(sw, &tmap_w, &full_bar[stage], k0, row);
          tma_load_2d(sw + L::kWBytes / 2, &tmap_w, &full_bar[stage], k0, row + 64);
        } else {
          tma_load_2d(sw, &tmap_w, &full_bar[stage], k0, tile * WR);
        }
      };
      auto load_x = [&](int kb, int stage) {
        tma_load_2d(smem + stage * L::kStageBytes + L::kWBytes, &tmap_x, &full_bar[stage], kb * kElems, 0);
      };
      // the first stages' weights are requested before the previous kernel has finished, its outputs afterwards
      if (!p.early_weights) grid_dep_wait();
      const int ahead = t_begin < t_end ? min(k_blocks, L::kStages) : 0;
      for (int s = 0; s < ahead; ++s) load_w(t_begin, s, s);
      grid_dep_wait();
      grid_dep_launch();
      for (int s = 0; s < ahead; ++s) load_x(s, s);
      int stage = ahead == L::kStages ? 0 : ahead, kb = ahead;
      uint32_t phase = ahead == L::kStages ? 1 : 0;
      for (int tile = t_begin; tile < t_end && !*abort_flag; ++tile, kb = 0) {
        for (; kb < k_blocks; ++kb) {
          mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.err, kKernelId, 1);
          if (*abort_flag) break;
          load_w(tile, kb, stage);
          load_x(kb, stage);
          if (++stage == L::kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = ELT == 1 ? umma_idesc_e4m3(128, NT) : umma_idesc_bf16(128, NT, false, false);
      int stage = 0, buf = 0;
      uint32_t phase = 0, buf_phase = 0;
      for (int tile = t_begin; tile < t_end && !*abort_flag; ++tile) {
        mbar_wait(&tmem_empty[buf], buf_phase ^ 1, abort_flag, p.err, kKernelId, 2);
        if (*abort_flag) break;
        tc_fence_after();
        const uint32_t d = tmem + buf * NT;
        for (int kb = 0; kb < k_blocks; ++kb) {
          mbar_wait(&full_bar[stage], phase, abort_flag, p.err, kKernelId, 3);
          if (*abort_flag) break;
          tc_fence_after();
          const uint32_t sw = smem_u32(smem + stage * L::kStageBytes), sx = sw + L::kWBytes;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint64_t da = umma_smem_desc_sw128(sw + k * 32, 16, 1024), db = umma_smem_desc_sw128(sx + k * 32, 16, 1024);
            if constexpr (ELT == 1) umma_f8(d, da, db, idesc, (kb | k) != 0 ? 1u : 0u);
            else umma_bf16(d, da, db, idesc, (kb | k) != 0 ? 1u : 0u);
          }
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
  } else if ((warp & 3) * 32 < WR) {  // the warps whose lanes of the accumulator hold rows of the tile
    grid_dep_wait();  // everything below reads or overwrites what earlier kernels touch
    auto sync = [] { asm volatile("bar.sync 1, %0;" ::"n"(WR) : "memory"); };
    const int quad = warp & 3;
    const int f = quad * 32 + lane;  // row of the tile = TMEM lane
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    __shared__ long long pos_s[MODE == kDecodeQkv ? NT : 1], slot_s[MODE == kDecodeQkv ? NT : 1];
    if constexpr (MODE == kDecodeQkv) {  // one round trip for all tokens; an index outside its table is reported and skipped
      for (int t = f; t < p.n; t += WR) {
        const long long pos = __ldcg(p.positions + t), slot = __ldcg(p.slots + t);
        const bool pos_ok = pos >= 0 && pos < p.table_rows, slot_ok = slot >= 0 && slot < p.cache_rows;
        if (!pos_ok) report_error(p.err, kErrBadIndex, kKernelId, 10);
        if (!slot_ok) report_error(p.err, kErrBadIndex, kKernelId, 11);
        pos_s[t] = pos_ok ? pos : 0;
        slot_s[t] = slot_ok ? slot : -1;
      }
      sync();
    }
    int buf = 0;
    uint32_t buf_phase = 0;
    for (int tile = t_begin; tile < t_end; ++tile) {
      // row of W that this lane holds, its scale and bias
      constexpr int kPerHead = 128 / WR;
      int w_row = tile * WR + f;
      if constexpr (MODE == kDecodeSwiglu) w_row = (f < kHalf ? 0 : p.N / 2) + tile * kHalf + (f & (kHalf - 1));
      if constexpr (MODE == kDecodeQkv)
        w_row = tile / kPerHead * 128 + tile % kPerHead * kHalf + (f & (kHalf - 1)) + (f < kHalf ? 0 : 64);
      const bool live = w_row < p.N;
      float sw = 1.f, bias = 0.f;
      if constexpr (ELT == 1) sw = live ? p.scale_w[w_row] : 0.f;
      if constexpr (MODE == kDecodeQkv) bias = p.bias != nullptr ? __bfloat162float(p.bias[w_row]) : 0.f;
      // the residual of the first tokens is requested while the products are formed, that of later ones a step ahead
      __nv_bfloat16 res[MODE == kDecodeStore ? kChunk : 1];
      auto load_residual = [&](int c0) {
        if constexpr (MODE == kDecodeStore) {
          if (p.residual != nullptr && live) {
#pragma unroll
            for (int j = 0; j < kChunk; ++j)
              if (c0 + j < p.n) res[j] = __ldcg(p.residual + static_cast<long long>(c0 + j) * p.ld_residual + w_row);
          }
        }
      };
      load_residual(0);
      mbar_wait(&tmem_full[buf], buf_phase, abort_flag, p.err, kKernelId, 4);
      tc_fence_after();
      const uint32_t acc = tmem + buf * NT + lane_addr;
#pragma unroll 1
      for (int c0 = 0; c0 < NT; c0 += kChunk) {
        if (c0 >= p.n) break;
        float v[kChunk], sx[kChunk];
        if constexpr (ELT == 1) {
#pragma unroll
          for (int j = 0; j < kChunk; ++j) sx[j] = c0 + j < p.n ? __ldcg(p.scale_x + c0 + j) : 0.f;
        }
        uint32_t r[kChunk];
        tmem_ld_32x32b_x16(acc + c0, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < kChunk; ++j) v[j] = __uint_as_float(r[j]);
        if constexpr (ELT == 1) {
#pragma unroll
          for (int j = 0; j < kChunk; ++j) v[j] = v[j] * sx[j] * sw;  // the order of the 256-wide engines: the same bits
        }
        if constexpr (MODE == kDecodeStore) {
          if (p.residual != nullptr) {
#pragma unroll
            for (int j = 0; j < kChunk; ++j) v[j] = round_bf16(v[j]) + __bfloat162float(res[j]);
            load_residual(c0 + kChunk);
          }
          if (live) {
#pragma unroll
            for (int j = 0; j < kChunk; ++j) {
              const int t = c0 + j;
              if (t < p.n) p.out[static_cast<long long>(t) * p.ldo + w_row] = __float2bfloat16_rn(v[j]);
            }
          }
        } else {
          // pairs of rows half a tile apart (gate and up, the two halves of a rotation) meet through shared memory
          sync();  // the previous step's readers are done
#pragma unroll
          for (int j = 0; j < kChunk; ++j) {
            float x = round_bf16(v[j]);
            if constexpr (MODE == kDecodeQkv) {
              if (p.bias != nullptr) x = round_bf16(x + bias);
            }
            xch[j * WR + f] = x;
          }
          sync();
          if constexpr (MODE == kDecodeSwiglu) {
            const int at = f & (kHalf - 1), o = tile * kHalf + at;
#pragma unroll
            for (int i = 0; i < kChunk / 2; ++i) {  // each half of the lanes takes every other token
              const int j = 2 * i + (f < kHalf ? 0 : 1), t = c0 + j;
              const float g = xch[j * WR + at], up = xch[j * WR + kHalf + at];
              if (t < p.n) p.out[static_cast<long long>(t) * p.ldo + o] = __float2bfloat16_rn(g / (1.f + __expf(-g)) * up);
            }
          } else {  // kDecodeQkv
            const int head = tile / kPerHead, half = tile % kPerHead * kHalf + (f & (kHalf - 1)), kv_heads = p.hkv;
            const int at = half + (f < kHalf ? 0 : 64);  // feature of the head
            float cs[kChunk], sn[kChunk];
            if (head < p.hq + kv_heads) {
#pragma unroll
              for (int j = 0; j < kChunk; ++j) {
                const long long i = c0 + j < p.n ? pos_s[c0 + j] * 64 + half : half;
                cs[j] = __ldg(p.cos + i);
                sn[j] = __ldg(p.sin + i);
              }
            }
            const int rep = p.hq / kv_heads, kv = head / rep;
#pragma unroll
            for (int j = 0; j < kChunk; ++j) {
              const int t = c0 + j;
              if (t < p.n) {
                float x = xch[j * WR + f];
                if (head < p.hq + kv_heads) {
                  const float y = xch[j * WR + (f ^ kHalf)];
                  x = f < kHalf ? x * cs[j] - y * sn[j] : x * cs[j] + y * sn[j];
                }
                const __nv_bfloat16 b = __float2bfloat16_rn(x);
                if (head < p.hq) {
                  p.q_rows[((static_cast<long long>(t) * rep + head - kv * rep) * kv_heads + kv) * 128 + at] = b;
                } else if (slot_s[t] >= 0) {
                  const bool is_v = head >= p.hq + kv_heads;
                  const int h = head - p.hq - (is_v ? kv_heads : 0);
                  (is_v ? p.cache_v : p.cache_k)[(slot_s[t] * kv_heads + h) * 128 + at] = b;
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

// Rows of the weight in a tile.  64 while every tile gets a CTA of its own with two to an SM, 128 beyond, where a CTA walks several:
// the tiles of 64 end a fifth sooner at 100 tokens (4096 x 4096: 35 against 43 us) and are equal at one, but a CTA's chain of
// accumulations is as long for 64 rows as for 128 (28672 x 4096: 82 against 37 us).
int tile_rows_of(int N, int sm_count) { return (N + 63) / 64 <= 2 * sm_count ? 64 : 128; }

template <int NT, int WR, int ELT, int MODE>
void launch(const DecodeLinearArgs& a, cudaStream_t stream) {
  using L = DecSmem<NT, WR>;
  const int tiles = (a.N + WR - 1) / WR;
  const int k_blocks = (a.K * ELT + 127) / 128;
  // a CTA per tile while two fit every SM (they share the memory's bandwidth evenly whether an SM holds one or two), contiguous
  // ranges of tiles for one CTA per SM beyond
  const int grid = tiles <= 2 * a.sm_count ? tiles : a.sm_count;
  constexpr uint32_t w_box = MODE == kDecodeStore ? WR : WR / 2;
  const CUtensorMap tw = ELT == 1 ? make_tmap_2d_u8(a.w, a.N, a.K, a.ld_w, w_box, 128)
                                  : make_tmap_2d_bf16(a.w, a.N, a.K, a.ld_w, w_box, 64);
  const CUtensorMap tx = ELT == 1 ? make_tmap_2d_u8(a.x, a.n, a.K, a.ld_x, NT, 128) : make_tmap_2d_bf16(a.x, a.n, a.K, a.ld_x, NT, 64);
  auto kernel = decode_linear_kernel<NT, WR, ELT, MODE>;
  static PerDeviceOnce configured;
  if (configured.first()) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kDynamic);
  launch_dependent(kernel, dim3(static_cast<unsigned>(grid)), dim3(192), L::kDynamic, stream, tw, tx, a, tiles, k_blocks);
}

template <int NT, int WR>
void by_mode(const DecodeLinearArgs& a, cudaStream_t stream) {
  if (a.fp8) launch<NT, WR, 1, kDecodeStore>(a, stream);
  else if (a.mode == kDecodeSwiglu) launch<NT, WR, 2, kDecodeSwiglu>(a, stream);
  else if (a.mode == kDecodeQkv) launch<NT, WR, 2, kDecodeQkv>(a, stream);
  else launch<NT, WR, 2, kDecodeStore>(a, stream);
}

template <int NT>
void by_rows(const DecodeLinearArgs& a, cudaStream_t stream) {
  const int rows = a.tile_rows > 0 ? a.tile_rows : tile_rows_of(a.N, a.sm_count);
  if (rows == 64) by_mode<NT, 64>(a, stream);
  else by_mode<NT, 128>(a, stream);
}

}  // namespace

void decode_linear(const DecodeLinearArgs& a, cudaStream_t stream) {
  if (a.n <= 0 || a.N <= 0) return;
  if (a.n <= 16) by_rows<16>(a, stream);
  else if (a.n <= 32) by_rows<32>(a, stream);
  else if (a.n <= 64) by_rows<64>(a, stream);
  else by_rows<128>(a, stream);
}

}  // namespace rlk
