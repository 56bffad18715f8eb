// Softmax top-k sparse MoE MLP of a block of rows (prefill chunk): the tokens are sorted by expert, so an expert's
// matrices are read once for all tokens that chose it instead of once per token.
//
//   moe_block_route_kernel    RMSNorm of every row in fp32, router logits, softmax, top-k; the normalised row also as
//                             a bf16 rounding and its remainder (the B operands of the projections)
//   moe_block_group_kernel    one block: the (row, rank) pairs sorted by expert into slots
//   moe_block_gather_kernel   the slots' activation rows
//   moe_block_gemm_kernel     grouped projections on tcgen05: gate/up with SwiGLU, then down times the routing weight;
//                             a shared expert runs through the same kernel as a group of all rows
//   moe_block_combine_kernel  residual + the row's slots in rank order + the shared expert
//
// Arithmetic is that of the decode step (moe.cu) up to roundings: fp32 normalised rows and fp32 SwiGLU outputs enter the
// projections as two bf16 parts (2^-17 of an element is lost), two MMAs into one fp32 accumulator.  Sums run in another
// order than there: a router logit is added by the lanes of a warp (there by a block of 256 threads), a row's contributions
// in rank order with the shared expert last (there per lane before the lanes are added).
//
// What bounds the projections: the expert weights out of HBM while an expert has up to about 128 tokens, the tensor
// pipe beyond.  A block therefore takes a pair of 128-row weight tiles (gate and up rows of the same index, or 256 rows
// of down) against all tokens of an expert, up to 128 at a time: 32 KB of weights per 64-wide slice and 16 MMAs of
// 128 x N x 16, which at N = 128 take as long as HBM needs for the weights.  Gate and up have an accumulator each, so
// SwiGLU needs no exchange between threads.
//
// Measured (whole prefill of 6 layers of 64 experts, hidden 2048; token by token before): 8 of 64 experts of 768, 300
// tokens 1.77 ms (122), 1000 tokens 2.5 ms (409); 6 of 64 of 1408 and a shared expert behind latent attention
// (mla_block.cu), 1000 tokens 5.0 ms (514).  Even two tokens are no slower than two steps (0.84 and 0.93 ms).
#include <algorithm>

#include "gemm_device.cuh"
#include "mma_bf16.cuh"
#include "moe_route.cuh"

namespace nb {
namespace {

// ---------------------------------------------------------------- routing ----
constexpr uint32_t kRouteWarps = 8;
constexpr uint32_t kRouteRows = 8;       // rows of a block, a warp per row in the norm and the routing
constexpr uint32_t kRouteExperts = 4;    // experts a warp takes at a time: a row's activations are read once for all

// Shared memory: rows_per_block x hidden fp32 (per row two planes: the first four of every eight elements, the last
// four), then rows x experts logits.
__global__ void __launch_bounds__(kRouteWarps * 32) moe_block_route_kernel(MoeBlockParams p, uint32_t rows_per_block) {
  extern __shared__ __align__(16) float route_smem[];
  pdl_trigger();
  pdl_wait();
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t row0 = blockIdx.x * rows_per_block;
  const uint32_t rows = p.rows - row0 < rows_per_block ? p.rows - row0 : rows_per_block;
  const uint32_t pieces = p.hidden / 8u;
  float *logits = route_smem + static_cast<uint64_t>(rows_per_block) * p.hidden;

  for (uint32_t r = warp; r < rows; r += kRouteWarps) {
    const uint64_t at = static_cast<uint64_t>(row0 + r) * p.hidden;
    const float4 *src = reinterpret_cast<const float4 *>(p.h + at);
    float4 *xa = reinterpret_cast<float4 *>(route_smem + static_cast<uint64_t>(r) * p.hidden), *xb = xa + pieces;
    float sumsq = 0.0f;
    for (uint32_t i = lane; i < pieces; i += 32u) {
      const float4 a = __ldcg(src + 2u * i), b = __ldcg(src + 2u * i + 1u);
      xa[i] = a;
      xb[i] = b;
      sumsq += a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w + b.x * b.x + b.y * b.y + b.z * b.z + b.w * b.w;
    }
    const float scale = rsqrtf(warp_sum(sumsq) / static_cast<float>(p.hidden) + p.eps);
    float shared_dot = 0.0f;
    for (uint32_t i = lane; i < pieces; i += 32u) {
      const uint4 w = *reinterpret_cast<const uint4 *>(p.norm_weight + 8u * i);
      float4 a = xa[i], b = xb[i];
      a.x = a.x * scale * bf16x2_lo(w.x), a.y = a.y * scale * bf16x2_hi(w.x);
      a.z = a.z * scale * bf16x2_lo(w.y), a.w = a.w * scale * bf16x2_hi(w.y);
      b.x = b.x * scale * bf16x2_lo(w.z), b.y = b.y * scale * bf16x2_hi(w.z);
      b.z = b.z * scale * bf16x2_lo(w.w), b.w = b.w * scale * bf16x2_hi(w.w);
      xa[i] = a;
      xb[i] = b;
      *reinterpret_cast<uint4 *>(p.x_hi + at + 8u * i) =
          make_uint4(pack_bf16_hi(a.x, a.y), pack_bf16_hi(a.z, a.w), pack_bf16_hi(b.x, b.y), pack_bf16_hi(b.z, b.w));
      *reinterpret_cast<uint4 *>(p.x_lo + at + 8u * i) =
          make_uint4(pack_bf16_lo(a.x, a.y), pack_bf16_lo(a.z, a.w), pack_bf16_lo(b.x, b.y), pack_bf16_lo(b.z, b.w));
      if (p.w_shared_router != nullptr) {
        const uint16_t *s = p.w_shared_router + 8u * i;
        shared_dot += bf16_bits_to_f32(s[0]) * a.x + bf16_bits_to_f32(s[1]) * a.y + bf16_bits_to_f32(s[2]) * a.z +
                      bf16_bits_to_f32(s[3]) * a.w + bf16_bits_to_f32(s[4]) * b.x + bf16_bits_to_f32(s[5]) * b.y +
                      bf16_bits_to_f32(s[6]) * b.z + bf16_bits_to_f32(s[7]) * b.w;
      }
    }
    if (p.shared_intermediate != 0) {
      shared_dot = warp_sum(shared_dot);
      if (lane == 0) p.shared_gate[row0 + r] = p.w_shared_router != nullptr ? sigmoid(shared_dot) : 1.0f;
    }
  }
  __syncthreads();

  for (uint32_t e0 = warp * kRouteExperts; e0 < p.num_experts; e0 += kRouteWarps * kRouteExperts) {
    float acc[kRouteExperts][kRouteRows];
#pragma unroll
    for (uint32_t k = 0; k < kRouteExperts; ++k)
#pragma unroll
      for (uint32_t r = 0; r < kRouteRows; ++r) acc[k][r] = 0.0f;
    for (uint32_t i = lane; i < pieces; i += 32u) {
      uint4 w[kRouteExperts];
#pragma unroll
      for (uint32_t k = 0; k < kRouteExperts; ++k) {
        const uint32_t e = e0 + k < p.num_experts ? e0 + k : p.num_experts - 1u;
        w[k] = __ldg(reinterpret_cast<const uint4 *>(p.w_router + static_cast<uint64_t>(e) * p.hidden) + i);
      }
#pragma unroll
      for (uint32_t r = 0; r < kRouteRows; ++r) {
        if (r >= rows) break;
        const float4 *xa = reinterpret_cast<const float4 *>(route_smem + static_cast<uint64_t>(r) * p.hidden);
        const float4 a = xa[i], b = xa[pieces + i];
#pragma unroll
        for (uint32_t k = 0; k < kRouteExperts; ++k) {
          float t = acc[k][r];
          t = fmaf(bf16x2_lo(w[k].x), a.x, t), t = fmaf(bf16x2_hi(w[k].x), a.y, t);
          t = fmaf(bf16x2_lo(w[k].y), a.z, t), t = fmaf(bf16x2_hi(w[k].y), a.w, t);
          t = fmaf(bf16x2_lo(w[k].z), b.x, t), t = fmaf(bf16x2_hi(w[k].z), b.y, t);
          t = fmaf(bf16x2_lo(w[k].w), b.z, t), t = fmaf(bf16x2_hi(w[k].w), b.w, t);
          acc[k][r] = t;
        }
      }
    }
#pragma unroll
    for (uint32_t k = 0; k < kRouteExperts; ++k)
#pragma unroll
      for (uint32_t r = 0; r < kRouteRows; ++r) {
        const float total = warp_sum(acc[k][r]);
        if (lane == 0 && r < rows && e0 + k < p.num_experts) logits[r * p.num_experts + e0 + k] = total;
      }
  }
  __syncthreads();

  for (uint32_t r = warp; r < rows; r += kRouteWarps) {
    const uint64_t at = static_cast<uint64_t>(row0 + r) * p.top_k;
    moe_route_warp(logits + r * p.num_experts, p.num_experts, p.top_k, p.norm_topk_prob, p.ids + at, p.weights + at);
  }
}

// ---------------------------------------------------------------- grouping ----
constexpr uint32_t kGroupThreads = 1024;

// Slots of an expert's tokens follow each other; the order inside an expert does not enter any result.
__global__ void __launch_bounds__(kGroupThreads) moe_block_group_kernel(MoeBlockParams p) {
  __shared__ uint32_t count[kMoeMaxExperts], next[kMoeMaxExperts];
  pdl_trigger();
  pdl_wait();
  const uint32_t pairs = p.rows * p.top_k;
  for (uint32_t e = threadIdx.x; e < kMoeMaxExperts; e += blockDim.x) count[e] = 0;
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < pairs; i += blockDim.x) atomicAdd(&count[__ldcg(p.ids + i)], 1u);
  __syncthreads();
  if (threadIdx.x < 32u) {
    uint32_t base = 0;
    for (uint32_t e0 = 0; e0 < p.num_experts; e0 += 32u) {
      const uint32_t e = e0 + threadIdx.x;
      const uint32_t c = e < p.num_experts ? count[e] : 0u;
      uint32_t before = c;
      for (uint32_t offset = 1; offset < 32u; offset <<= 1) {
        const uint32_t other = __shfl_up_sync(0xffffffffu, before, offset);
        if (threadIdx.x >= offset) before += other;
      }
      if (e < p.num_experts) {
        next[e] = base + before - c;
        p.offsets[e] = base + before - c;
      }
      base += __shfl_sync(0xffffffffu, before, 31);
    }
    if (threadIdx.x == 0) p.offsets[p.num_experts] = base;
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < pairs; i += blockDim.x) {
    const uint32_t slot = atomicAdd(&next[__ldcg(p.ids + i)], 1u);
    p.slot_of[i] = slot;
    p.row_of[slot] = i / p.top_k;
    p.slot_weight[slot] = __ldcg(p.weights + i);
  }
}

__global__ void __launch_bounds__(256) moe_block_gather_kernel(MoeBlockParams p) {
  pdl_trigger();
  pdl_wait();
  const uint64_t from = static_cast<uint64_t>(__ldcg(p.row_of + blockIdx.x)) * p.hidden;
  const uint64_t to = static_cast<uint64_t>(blockIdx.x) * p.hidden;
  for (uint32_t i = threadIdx.x; i < p.hidden / 8u; i += blockDim.x) {
    const uint4 hi = __ldcg(reinterpret_cast<const uint4 *>(p.x_hi + from) + i);
    const uint4 lo = __ldcg(reinterpret_cast<const uint4 *>(p.x_lo + from) + i);
    reinterpret_cast<uint4 *>(p.slot_hi + to)[i] = hi;
    reinterpret_cast<uint4 *>(p.slot_lo + to)[i] = lo;
  }
}

// out[row] = (contributions in rank order, then the shared expert's) + h[row]
__global__ void __launch_bounds__(256) moe_block_combine_kernel(MoeBlockParams p) {
  pdl_trigger();
  pdl_wait();
  const uint32_t row = blockIdx.x;
  __shared__ uint32_t slots[kMoeMaxTopK];
  if (threadIdx.x < p.top_k) slots[threadIdx.x] = __ldcg(p.slot_of + static_cast<uint64_t>(row) * p.top_k + threadIdx.x);
  __syncthreads();
  const uint64_t at = static_cast<uint64_t>(row) * p.hidden;
  for (uint32_t i = threadIdx.x; i < p.hidden / 4u; i += blockDim.x) {
    const float4 h = __ldcg(reinterpret_cast<const float4 *>(p.h + at) + i);
    float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
    for (uint32_t k = 0; k < p.top_k; ++k) {
      const float4 v = __ldcg(reinterpret_cast<const float4 *>(p.y + static_cast<uint64_t>(slots[k]) * p.hidden) + i);
      sum.x += v.x, sum.y += v.y, sum.z += v.z, sum.w += v.w;
    }
    if (p.shared_intermediate != 0) {
      const float4 v = __ldcg(reinterpret_cast<const float4 *>(p.y_shared + at) + i);
      sum.x += v.x, sum.y += v.y, sum.z += v.z, sum.w += v.w;
    }
    reinterpret_cast<float4 *>(p.out + at)[i] = make_float4(sum.x + h.x, sum.y + h.y, sum.z + h.z, sum.w + h.w);
  }
}

// ---------------------------------------------------------------- projections ----
constexpr uint32_t kThreads = 192;       // warp 0 TMA, warp 1 MMA, warps 2..5 epilogue, as in gemm_tc.cu
constexpr uint32_t kEpilogueThreads = 128;
constexpr uint32_t kMaxStages = 5;
constexpr uint32_t kMaxTokens = 128;     // of a tile

struct ExpertGemm {
  const uint32_t *offsets;   // [groups + 1] first slot of every group; null: one group of `tokens` rows
  uint32_t groups, tokens;
  uint32_t rows;             // output rows of a group: intermediate size (gate/up), hidden (down)
  uint32_t group_rows;       // rows of the weight maps from one group to the next
  uint32_t second_row;       // where the second weight tile of a pair lies behind the first in map_b
  uint32_t step;             // output rows a tile covers: 128 (gate/up), 256 (down)
  uint32_t slices;           // 64-wide slices of the inner dimension, the last maybe partial (zeros)
  uint32_t tile_tokens, stages;
  uint32_t gate_up;
  uint16_t *act_hi, *act_lo;  // gate/up: [slot][rows] silu(gate) * up as two bf16 parts
  float *y;                   // down: [slot][rows]
  const float *slot_weight;   // down: factor of a slot
  uint32_t *error_word;
};

struct ExpertShared {
  uint64_t full[kMaxStages], empty[kMaxStages];
  uint64_t acc_full[2], acc_empty[2];
  uint64_t drained;
  uint32_t tmem_base, abort;
  uint32_t first_tile[kMoeMaxExperts + 1];
};

struct ExpertTile {
  uint32_t group, row, slot, count;  // first output row; first slot, tokens
};

// Token tiles of a weight tile follow each other: its second reader finds it in the L2.
__device__ __forceinline__ ExpertTile expert_tile(const ExpertGemm &g, const ExpertShared &sh, uint32_t index) {
  uint32_t lo = 0, hi = g.groups;  // the last group whose first tile is not behind index
  while (hi - lo > 1u) {
    const uint32_t mid = (lo + hi) / 2u;
    if (sh.first_tile[mid] <= index)
      lo = mid;
    else
      hi = mid;
  }
  const uint32_t begin = g.offsets != nullptr ? __ldcg(g.offsets + lo) : 0u;
  const uint32_t end = g.offsets != nullptr ? __ldcg(g.offsets + lo + 1u) : g.tokens;
  const uint32_t token_tiles = (end - begin + g.tile_tokens - 1u) / g.tile_tokens;
  const uint32_t local = index - sh.first_tile[lo];
  ExpertTile t;
  t.group = lo;
  t.row = local / token_tiles * g.step;
  t.slot = begin + local % token_tiles * g.tile_tokens;
  t.count = end - t.slot < g.tile_tokens ? end - t.slot : g.tile_tokens;
  return t;
}

__host__ __device__ constexpr uint32_t expert_columns(uint32_t tile_tokens) { return 4u * tile_tokens; }  // two buffers of two accumulators

__global__ void __launch_bounds__(kThreads, 1)
moe_block_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                      const __grid_constant__ CUtensorMap map_hi, const __grid_constant__ CUtensorMap map_lo, ExpertGemm g) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *ring = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~uintptr_t{1023});
  const uint32_t x_bytes = g.tile_tokens * kSliceK * 2u;
  const uint32_t stage_bytes = 2u * kATileBytes + 2u * x_bytes;
  ExpertShared &sh = *reinterpret_cast<ExpertShared *>(ring + g.stages * stage_bytes);
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  volatile uint32_t *abort = &sh.abort;
  const uint32_t tmem_columns = expert_columns(g.tile_tokens);

  pdl_trigger();
  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < g.stages; ++s) {
      mbar_init(&sh.full[s], 1);
      mbar_init(&sh.empty[s], 1);
    }
    for (uint32_t a = 0; a < 2; ++a) {
      mbar_init(&sh.acc_full[a], 1);
      mbar_init(&sh.acc_empty[a], kEpilogueThreads);
    }
    mbar_init(&sh.drained, 1);
    sh.abort = 0;
    mbar_init_fence();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&sh.tmem_base)),
                 "r"(tmem_columns)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  pdl_wait();
  if (warp == 2) {  // first tile of every group
    const uint32_t row_tiles = (g.rows + g.step - 1u) / g.step;
    uint32_t base = 0;
    for (uint32_t e0 = 0; e0 < g.groups; e0 += 32u) {
      const uint32_t e = e0 + lane;
      uint32_t tiles = 0;
      if (e < g.groups) {
        const uint32_t tokens = g.offsets != nullptr ? __ldcg(g.offsets + e + 1u) - __ldcg(g.offsets + e) : g.tokens;
        tiles = (tokens + g.tile_tokens - 1u) / g.tile_tokens * row_tiles;
      }
      uint32_t before = tiles;
      for (uint32_t offset = 1; offset < 32u; offset <<= 1) {
        const uint32_t other = __shfl_up_sync(0xffffffffu, before, offset);
        if (lane >= offset) before += other;
      }
      if (e < g.groups) sh.first_tile[e] = base + before - tiles;
      base += __shfl_sync(0xffffffffu, before, 31);
    }
    if (lane == 0) sh.first_tile[g.groups] = base;
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = sh.tmem_base;
  const uint32_t tiles = sh.first_tile[g.groups];

  if (warp == 0) {
    if (elected()) {
      const uint64_t w_policy = l2_evict_first_policy(), x_policy = l2_evict_last_policy();
      uint32_t issued = 0;
      bool ok = true;
      for (uint32_t tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x) {
        const ExpertTile t = expert_tile(g, sh, tile);
        const uint32_t w_row = t.group * g.group_rows + t.row;
        for (uint32_t c = 0; c < g.slices; ++c, ++issued) {
          const uint32_t s = issued % g.stages;
          if (!abortable_wait(&sh.empty[s], ((issued / g.stages) & 1u) ^ 1u, abort, g.error_word)) {
            ok = false;
            break;
          }
          uint8_t *stage = ring + s * stage_bytes;
          mbar_arrive_expect_tx(&sh.full[s], stage_bytes);
          tma_load_2d(stage, &map_a, c * kSliceK, w_row, &sh.full[s], w_policy);
          tma_load_2d(stage + kATileBytes, &map_b, c * kSliceK, w_row + g.second_row, &sh.full[s], w_policy);
          tma_load_2d(stage + 2u * kATileBytes, &map_hi, c * kSliceK, t.slot, &sh.full[s], x_policy);
          tma_load_2d(stage + 2u * kATileBytes + x_bytes, &map_lo, c * kSliceK, t.slot, &sh.full[s], x_policy);
        }
      }
    }
  } else if (warp == 1) {
    if (elected()) {
      uint32_t consumed = 0, index = 0;
      bool ok = true;
      for (uint32_t tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x, ++index) {
        const ExpertTile t = expert_tile(g, sh, tile);
        const uint32_t idesc = instr_desc_bf16((t.count + 15u) & ~15u);
        const uint32_t acc = index & 1u;
        if (!abortable_wait(&sh.acc_empty[acc], ((index >> 1) & 1u) ^ 1u, abort, g.error_word)) break;
        tcgen05_fence_after();
        const uint32_t d0 = tmem_base + acc * 2u * g.tile_tokens, d1 = d0 + g.tile_tokens;
        for (uint32_t c = 0; c < g.slices; ++c, ++consumed) {
          const uint32_t s = consumed % g.stages;
          if (!abortable_wait(&sh.full[s], (consumed / g.stages) & 1u, abort, g.error_word)) {
            ok = false;
            break;
          }
          tcgen05_fence_after();
          const uint8_t *stage = ring + s * stage_bytes;
          const uint64_t a0 = kmajor_sw128_desc(stage), a1 = kmajor_sw128_desc(stage + kATileBytes);
          const uint64_t hi = kmajor_sw128_desc(stage + 2u * kATileBytes);
          const uint64_t lo = kmajor_sw128_desc(stage + 2u * kATileBytes + x_bytes);
#pragma unroll
          for (uint32_t k = 0; k < kSliceK / kUmmaK; ++k) {
            const uint32_t more = (c != 0 || k != 0) ? 1u : 0u;
            tcgen05_mma_f16(d0, a0 + 2ull * k, hi + 2ull * k, idesc, more);
            tcgen05_mma_f16(d0, a0 + 2ull * k, lo + 2ull * k, idesc, 1u);
            tcgen05_mma_f16(d1, a1 + 2ull * k, hi + 2ull * k, idesc, more);
            tcgen05_mma_f16(d1, a1 + 2ull * k, lo + 2ull * k, idesc, 1u);
          }
          tcgen05_commit(&sh.empty[s]);
        }
        if (ok) tcgen05_commit(&sh.acc_full[acc]);
      }
    }
  } else {
    const uint32_t quarter = warp & 3u;
    uint32_t index = 0;
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++index) {
      const uint32_t acc = index & 1u;
      const ExpertTile t = expert_tile(g, sh, tile);
      if (!warp_wait(&sh.acc_full[acc], (index >> 1) & 1u, abort, g.error_word)) break;
      tcgen05_fence_after();
      const uint32_t d0 = tmem_base + acc * 2u * g.tile_tokens + ((quarter * 32u) << 16), d1 = d0 + g.tile_tokens;
      const uint32_t row = t.row + quarter * 32u + lane;
      for (uint32_t m = 0; m < t.count; m += kGroup) {
        float a[kGroup], b[kGroup];
        tmem_load16(d0 + m, a);
        tmem_load16(d1 + m, b);
        if (g.gate_up != 0) {
          if (row < g.rows) {
            const uint64_t at = static_cast<uint64_t>(t.slot + m) * g.rows + row;
#pragma unroll
            for (uint32_t j = 0; j < kGroup; ++j) {
              if (m + j < t.count) {
                const float v = silu(a[j]) * b[j];
                const uint16_t hi = f32_to_bf16_bits(v);
                g.act_hi[at + static_cast<uint64_t>(j) * g.rows] = hi;
                g.act_lo[at + static_cast<uint64_t>(j) * g.rows] = f32_to_bf16_bits(v - bf16_bits_to_f32(hi));
              }
            }
          }
        } else {
#pragma unroll
          for (uint32_t j = 0; j < kGroup; ++j) {
            if (m + j < t.count) {
              const float w = __ldg(g.slot_weight + t.slot + m + j);
              float *dst = g.y + static_cast<uint64_t>(t.slot + m + j) * g.rows + row;
              if (row < g.rows) dst[0] = w * a[j];
              if (row + kTileRows < g.rows) dst[kTileRows] = w * b[j];
            }
          }
        }
      }
      tcgen05_fence_before();
      mbar_arrive(&sh.acc_empty[acc]);
    }
  }
  // ---- teardown: nothing stays in flight ----
  tcgen05_fence_before();
  __syncthreads();
  if (sh.abort != 0u) {
    if (threadIdx.x == 0) drain_copies(sh.full, g.stages);
    if (warp == 1 && elected()) drain_mmas(&sh.drained);
  }
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_columns) : "memory");
  }
}

// Tokens per tile: the expected load of an expert and some room, so that most experts are one tile; the tile is loaded
// whole whatever its expert's count, so it is no larger than it has to be.  The sizes make the accumulators a power of
// two of tensor-memory columns.
uint32_t expert_tile_tokens(uint32_t tokens, uint32_t groups) {
  const uint32_t room = groups == 1u ? tokens : tokens / groups + tokens / groups / 4u + 8u;
  return room <= 32u ? 32u : room <= 64u ? 64u : kMaxTokens;
}

uint32_t expert_stage_bytes(uint32_t tile_tokens) { return 2u * kATileBytes + 2u * tile_tokens * kSliceK * 2u; }
uint32_t expert_stages(uint32_t tile_tokens) { return std::min(kMaxStages, 216u * 1024u / expert_stage_bytes(tile_tokens)); }
uint32_t expert_smem_bytes(uint32_t tile_tokens) {
  return tensor_memory_smem(expert_columns(tile_tokens), 1024u + expert_stages(tile_tokens) * expert_stage_bytes(tile_tokens) +
                                                             static_cast<uint32_t>(sizeof(ExpertShared)) + 64u);
}

struct ExpertOperands {
  const uint16_t *a, *b;      // weights: first and second tile of a pair
  uint64_t map_rows_a, map_rows_b;
  uint32_t cols;
  const uint16_t *hi, *lo;    // activations [x_rows][cols]
  uint32_t x_rows;
};

cudaError_t launch_expert_gemm(cudaStream_t stream, ExpertGemm g, const ExpertOperands &o, uint32_t sm_count, bool pdl) {
  g.tile_tokens = expert_tile_tokens(o.x_rows, g.groups);
  g.slices = (o.cols + kSliceK - 1u) / kSliceK;
  g.stages = expert_stages(g.tile_tokens);
  CUtensorMap map_a, map_b, map_hi, map_lo;
  if (!encode_bf16_map_2d(&map_a, o.a, o.cols, o.map_rows_a, kSliceK, kTileRows) ||
      !encode_bf16_map_2d(&map_b, o.b, o.cols, o.map_rows_b, kSliceK, kTileRows) ||
      !encode_bf16_map_2d(&map_hi, o.hi, o.cols, o.x_rows, kSliceK, g.tile_tokens) ||
      !encode_bf16_map_2d(&map_lo, o.lo, o.cols, o.x_rows, kSliceK, g.tile_tokens))
    return cudaErrorNotSupported;
  // upper bound of the tiles: every group may have one that is not full
  const uint64_t row_tiles = (g.rows + g.step - 1u) / g.step;
  const uint64_t most = row_tiles * (o.x_rows / g.tile_tokens + std::min(g.groups, o.x_rows));
  const uint32_t blocks = static_cast<uint32_t>(std::min<uint64_t>(most, sm_count));
  return launch_with_pdl(moe_block_gemm_kernel, dim3(blocks), dim3(kThreads), expert_smem_bytes(g.tile_tokens), stream, pdl, map_a,
                         map_b, map_hi, map_lo, g);
}

uint32_t route_rows(uint32_t hidden, uint32_t experts) {
  const uint32_t fit = 200u * 1024u / (4u * (hidden + experts));
  return fit < kRouteRows ? fit : kRouteRows;
}

}  // namespace

bool moe_block_supported(const MoeBlockParams &p) {
  auto aligned = [](const void *ptr) { return reinterpret_cast<uintptr_t>(ptr) % 16u == 0; };
  return p.num_experts != 0 && p.num_experts <= kMoeMaxExperts && p.top_k != 0 && p.top_k <= kMoeMaxTopK &&
         p.top_k <= p.num_experts && p.hidden % 64u == 0 && p.moe_intermediate % 8u == 0 && p.shared_intermediate % 8u == 0 &&
         route_rows(p.hidden, p.num_experts) != 0 && p.expert_stride % p.hidden == 0 && p.expert_up_offset % p.hidden == 0 &&
         aligned(p.norm_weight) && aligned(p.w_router) && aligned(p.w_expert_gate_up) && aligned(p.w_expert_down) &&
         (p.shared_intermediate == 0 || (aligned(p.w_shared_gate) && aligned(p.w_shared_up) && aligned(p.w_shared_down)));
}

cudaError_t configure_moe_block() {
  cudaError_t err = cudaFuncSetAttribute(moe_block_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  if (err == cudaSuccess)
    err = cudaFuncSetAttribute(moe_block_route_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 208 * 1024);
  return err;
}

void moe_block_launches(std::vector<TensorMemoryLaunch> *out) {
  for (uint32_t tokens : {32u, 64u, kMaxTokens}) out->push_back({expert_smem_bytes(tokens), expert_columns(tokens)});
}

cudaError_t launch_moe_block(cudaStream_t stream, const MoeBlockParams &p, uint32_t sm_count, bool pdl, uint64_t *launches) {
  if (p.rows == 0 || !moe_block_supported(p)) return cudaErrorInvalidValue;
  const uint32_t slots = p.rows * p.top_k;
  const uint32_t per = route_rows(p.hidden, p.num_experts);
  const uint32_t route_smem = per * (p.hidden + p.num_experts) * 4u;
  cudaError_t err = launch_with_pdl(moe_block_route_kernel, dim3((p.rows + per - 1u) / per), dim3(kRouteWarps * 32), route_smem,
                                    stream, pdl, p, per);
  if (err == cudaSuccess) err = launch_with_pdl(moe_block_group_kernel, dim3(1), dim3(kGroupThreads), 0, stream, pdl, p);
  if (err == cudaSuccess) err = launch_with_pdl(moe_block_gather_kernel, dim3(slots), dim3(256), 0, stream, pdl, p);
  uint64_t n = 3;

  ExpertGemm g{};
  g.offsets = p.offsets;
  g.groups = p.num_experts;
  g.error_word = p.error_word;
  g.rows = p.moe_intermediate;
  g.group_rows = static_cast<uint32_t>(p.expert_stride / p.hidden);
  g.step = kTileRows;
  g.gate_up = 1;
  g.act_hi = p.act_hi;
  g.act_lo = p.act_lo;
  ExpertOperands o{};
  o.a = p.w_expert_gate_up;
  o.b = p.w_expert_gate_up + p.expert_up_offset;
  o.map_rows_a = o.map_rows_b = static_cast<uint64_t>(p.num_experts - 1u) * g.group_rows + p.moe_intermediate;
  o.cols = p.hidden;
  o.hi = p.slot_hi;
  o.lo = p.slot_lo;
  o.x_rows = slots;
  if (err == cudaSuccess) err = launch_expert_gemm(stream, g, o, sm_count, pdl);
  ExpertGemm d = g;
  d.rows = p.hidden;
  d.group_rows = p.hidden;
  d.second_row = kTileRows;
  d.step = 2u * kTileRows;
  d.gate_up = 0;
  d.y = p.y;
  d.slot_weight = p.slot_weight;
  ExpertOperands od{};
  od.a = od.b = p.w_expert_down;
  od.map_rows_a = od.map_rows_b = static_cast<uint64_t>(p.num_experts) * p.hidden;
  od.cols = p.moe_intermediate;
  od.hi = p.act_hi;
  od.lo = p.act_lo;
  od.x_rows = slots;
  if (err == cudaSuccess) err = launch_expert_gemm(stream, d, od, sm_count, pdl);
  n += 2;
  if (p.shared_intermediate != 0) {
    g.offsets = d.offsets = nullptr;
    g.groups = d.groups = 1;
    g.tokens = d.tokens = p.rows;
    g.rows = p.shared_intermediate;
    g.group_rows = 0;
    g.act_hi = p.shared_act_hi;
    g.act_lo = p.shared_act_lo;
    o.a = p.w_shared_gate;
    o.b = p.w_shared_up;
    o.map_rows_a = o.map_rows_b = p.shared_intermediate;
    o.hi = p.x_hi;
    o.lo = p.x_lo;
    o.x_rows = p.rows;
    if (err == cudaSuccess) err = launch_expert_gemm(stream, g, o, sm_count, pdl);
    d.group_rows = 0;
    d.y = p.y_shared;
    d.slot_weight = p.shared_gate;
    od.a = od.b = p.w_shared_down;
    od.map_rows_a = od.map_rows_b = p.hidden;
    od.cols = p.shared_intermediate;
    od.hi = p.shared_act_hi;
    od.lo = p.shared_act_lo;
    od.x_rows = p.rows;
    if (err == cudaSuccess) err = launch_expert_gemm(stream, d, od, sm_count, pdl);
    n += 2;
  }
  if (err == cudaSuccess) err = launch_with_pdl(moe_block_combine_kernel, dim3(p.rows), dim3(256), 0, stream, pdl, p);
  if (launches != nullptr) *launches += n + 1u;
  return err;
}

}  // namespace nb
