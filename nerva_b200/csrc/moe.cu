// Softmax top-k sparse MoE MLP of the resident decode step (Qwen3-MoE / Mixtral
// style).  The reference runs the whole MLP of a layer in ONE thread block
// (run_sparse_moe_mlp, hf_decode_sequence/device_ops.cuh:183-315); here it is three launches:
//   moe_router_kernel   a block per expert: residual add + RMSNorm (every block for itself, in registers), the
//                       expert's router logit; the blocks share the writing of the normalised row
//   moe_gate_up_kernel  softmax and top-k by (weight descending, index ascending), by a warp of every block, then
//                       the gate and up projections of the chosen experts (+ the shared expert) and SwiGLU
//   moe_down_kernel     the experts' down projections, added with the routing weights
// Arithmetic follows the reference kernel: the mat-vecs read the UNROUNDED fp32
// normalised hidden state and the unrounded fp32 SwiGLU output (unlike the dense
// path, which rounds both to bf16), accumulate in fp32, and the expert outputs
// are added as down += weight * y in rank order (per lane of a warp, the lanes last), the shared expert scaled by
// sigmoid(shared_router . x).
//
// What bounds it: the experts' weights out of HBM (8 experts of 768 x 2048: 75 MB, 11 us a layer), and in front of
// them the chain that has to know the routing.  So the router matrix is read once by the grid instead of by every
// block, what does not depend on the routing (barriers, the shared expert's weights) is set going before the
// dependency wait, and both projections deal their work so that no block waits for another: gate and up rows of a pair
// go to the same block, and a block of the down launch owns a range of output rows through all experts.
//
// Measured (a step's time per layer, by leaving a launch out; 8 of 64 experts of 768, hidden 2048): 49 -> 28 us.  In
// it the routing chain is 3 us, the gate/up stream 7.4 us (6.8 TB/s).  The step of 6 layers and head: 516 -> 390 us;
// 6 of 64 experts of 1408 and a shared one behind latent attention: 613 -> 498 us.
#include <algorithm>

#include "kernels.cuh"
#include "moe_route.cuh"
#include "row_stream.cuh"
#include "step_device.cuh"

namespace nb {
namespace {

__host__ __device__ inline uint32_t round128u(uint32_t v) { return (v + 127u) & ~127u; }

// ---- norm and router logits ----
constexpr uint32_t kRouterThreads = 256;
constexpr uint32_t kRouterKeep = 2;  // pieces of 8 elements a thread keeps in registers: rows of up to 4096

// Grid: a block per expert, and one for the shared expert's gate where that has a router.
__global__ void __launch_bounds__(kRouterThreads) moe_router_kernel(MoeExpertParams p) {
  __shared__ float scratch[40];
  pdl_trigger();
  const uint32_t pieces = p.hidden / 8u;
  const bool shared = blockIdx.x == p.num_experts;
  const uint4 *router = reinterpret_cast<const uint4 *>(shared ? p.w_shared_router : p.w_router + static_cast<uint64_t>(blockIdx.x) * p.hidden);
  const uint4 *norm = reinterpret_cast<const uint4 *>(p.norm_weight);
  uint4 w[kRouterKeep], n[kRouterKeep];
#pragma unroll
  for (uint32_t u = 0; u < kRouterKeep; ++u) {
    const uint32_t i = threadIdx.x + u * kRouterThreads;
    w[u] = i < pieces ? __ldg(router + i) : make_uint4(0u, 0u, 0u, 0u);
    n[u] = i < pieces ? __ldg(norm + i) : make_uint4(0u, 0u, 0u, 0u);
  }
  pdl_wait();
  // the order of the sum: (b or a) + bias, then + a when there are two addends
  auto load = [&p](uint32_t piece, float (&r)[8]) {
    const float4 *a = reinterpret_cast<const float4 *>(p.add_a) + 2u * piece;
    const float4 a0 = __ldcg(a), a1 = __ldcg(a + 1);
    const float va[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
    if (p.add_b != nullptr) {
      const float4 *b = reinterpret_cast<const float4 *>(p.add_b) + 2u * piece;
      const float4 b0 = __ldcg(b), b1 = __ldcg(b + 1);
      const float vb[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
      for (uint32_t j = 0; j < 8u; ++j) r[j] = vb[j];
    } else {
#pragma unroll
      for (uint32_t j = 0; j < 8u; ++j) r[j] = va[j];
    }
    if (p.add_bias != nullptr) {
#pragma unroll
      for (uint32_t j = 0; j < 8u; ++j) r[j] += bf16_bits_to_f32(p.add_bias[8u * piece + j]);
    }
    if (p.add_b != nullptr) {
#pragma unroll
      for (uint32_t j = 0; j < 8u; ++j) r[j] += va[j];
    }
  };
  float r[kRouterKeep][8], sumsq = 0.0f;
#pragma unroll
  for (uint32_t u = 0; u < kRouterKeep; ++u) {
    const uint32_t i = threadIdx.x + u * kRouterThreads;
#pragma unroll
    for (uint32_t j = 0; j < 8u; ++j) r[u][j] = 0.0f;
    if (i < pieces) load(i, r[u]);
#pragma unroll
    for (uint32_t j = 0; j < 8u; ++j) sumsq += r[u][j] * r[u][j];
  }
  for (uint32_t i = threadIdx.x + kRouterKeep * kRouterThreads; i < pieces; i += kRouterThreads) {
    float v[8];
    load(i, v);
#pragma unroll
    for (uint32_t j = 0; j < 8u; ++j) sumsq += v[j] * v[j];
  }
  const float scale = rsqrtf(block_sum(sumsq, scratch) / static_cast<float>(p.hidden) + p.eps);
  float dot = 0.0f;
  auto finish = [&](uint32_t i, const float (&v)[8], const uint4 &nw, const uint4 &rw) {
    const float wn[8] = {bf16x2_lo(nw.x), bf16x2_hi(nw.x), bf16x2_lo(nw.y), bf16x2_hi(nw.y),
                         bf16x2_lo(nw.z), bf16x2_hi(nw.z), bf16x2_lo(nw.w), bf16x2_hi(nw.w)};
    float x[8];
#pragma unroll
    for (uint32_t j = 0; j < 8u; ++j) x[j] = v[j] * scale * wn[j];
    const float4 xa = make_float4(x[0], x[1], x[2], x[3]), xb = make_float4(x[4], x[5], x[6], x[7]);
    dot = dot8_f32(rw, xa, xb, dot);
    if (i % gridDim.x != blockIdx.x) return;
    // this block's share of the row, in two planes (first and last four of every eight elements)
    reinterpret_cast<float4 *>(p.x_norm)[i] = xa;
    reinterpret_cast<float4 *>(p.x_norm)[pieces + i] = xb;
    if (p.resid_out != nullptr) {
      reinterpret_cast<float4 *>(p.resid_out)[2u * i] = make_float4(v[0], v[1], v[2], v[3]);
      reinterpret_cast<float4 *>(p.resid_out)[2u * i + 1u] = make_float4(v[4], v[5], v[6], v[7]);
    }
  };
#pragma unroll
  for (uint32_t u = 0; u < kRouterKeep; ++u) {
    const uint32_t i = threadIdx.x + u * kRouterThreads;
    if (i < pieces) finish(i, r[u], n[u], w[u]);
  }
  for (uint32_t i = threadIdx.x + kRouterKeep * kRouterThreads; i < pieces; i += kRouterThreads) {
    float v[8];
    load(i, v);
    finish(i, v, __ldg(norm + i), __ldg(router + i));
  }
  const float logit = block_sum(dot, scratch);
  if (threadIdx.x != 0) return;
  if (shared)
    *p.shared_gate = sigmoid(logit);
  else
    p.router_logits[blockIdx.x] = logit;
  // shared experts without a router are always on
  if (blockIdx.x == 0 && p.shared_intermediate != 0 && p.w_shared_router == nullptr) *p.shared_gate = 1.0f;
}

// The chosen experts held by this rank, in routing order: all of them, or under expert parallel those whose matrices
// are here.  By one warp; lane r holds chosen expert r.
__device__ __forceinline__ uint32_t held_experts(const MoeExpertParams &p, uint32_t id, float weight, uint32_t *ids, float *weights) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t local = id - p.expert_base;  // wraps to a large value below the base
  const bool here = lane < p.top_k && (p.expert_local == 0 || local < p.expert_local);
  const uint32_t mask = __ballot_sync(0xffffffffu, here);
  if (here) {
    const uint32_t at = __popc(mask & ((1u << lane) - 1u));
    ids[at] = local;
    weights[at] = weight;
  }
  return __popc(mask);
}

// ---- weight streams ----
// Each warp streams pieces of consecutive weights through a ring of its own in shared memory (1-D bulk copies, an
// mbarrier per slot) and is alone responsible for what it reads: no block barrier inside a stream.  Pieces are small
// (2 KB), so what a piece costs besides its multiply-adds counts: a warp's pieces follow each other by increments, and
// no index is divided.
constexpr uint32_t kMoeWarps = 16, kMoeThreads = kMoeWarps * 32u;
constexpr uint32_t kPieceCols = 1024, kPieceBytes = 2u * kPieceCols;  // of a weight row
constexpr uint32_t kMaxSlots = 8;

struct WarpRing {
  uint8_t *base;
  uint64_t *bars;
  uint32_t slots, slot_bytes;
  uint32_t issued = 0, issue_slot = 0;  // pieces, and the slot the next one goes to
  uint32_t consumed = 0, slot = 0, parity = 0;
  bool dead = false;
  __device__ __forceinline__ void init(uint8_t *ring, uint64_t *all_bars, uint32_t slot_count, uint32_t bytes) {
    const uint32_t warp = threadIdx.x >> 5;
    slots = slot_count;
    slot_bytes = bytes;
    base = ring + warp * slots * slot_bytes;
    bars = all_bars + warp * kMaxSlots;
    if (elected()) {
      for (uint32_t i = 0; i < slots; ++i) mbar_init(&bars[i], 1);
      mbar_init_fence();
    }
    __syncwarp();
  }
  __device__ __forceinline__ bool room() const { return !dead && issued - consumed < slots; }
  __device__ __forceinline__ void issued_one() {
    issued += 1;
    issue_slot = issue_slot + 1u == slots ? 0u : issue_slot + 1u;
  }
  // The oldest piece's slot, once it has landed.
  __device__ __forceinline__ const uint8_t *wait(uint32_t *error_word) {
    if (!dead && !warp_wait_bounded(&bars[slot], parity)) {
      dead = true;
      report_error(error_word, kErrTmaWaitTimeout);
    }
    return base + slot * slot_bytes;
  }
  __device__ __forceinline__ void release() {
    __syncwarp();
    consumed += 1;
    slot += 1;
    if (slot == slots) {
      slot = 0;
      parity ^= 1u;
    }
  }
  // After a timeout: copies still in flight get one more bounded chance to land before the shared memory is released.
  __device__ __forceinline__ void drain() {
    if (!dead) return;
    for (uint32_t c = issued > slots ? issued - slots : 0u; c < issued; ++c) mbar_wait_bounded(&bars[c % slots], (c / slots) & 1u);
  }
};

__device__ __forceinline__ float lane_sum(const float2 (&acc)[4]) {
  return ((acc[0].x + acc[0].y) + (acc[1].x + acc[1].y)) + ((acc[2].x + acc[2].y) + (acc[3].x + acc[3].y));
}

// ---- gate/up ----
// Work is dealt in pairs (row i of a gate matrix, row i of its up matrix), the shared expert's and the routed ones'
// each in equal shares to all blocks.  Inside a block the units are kPieceCols columns of a pair, in equal runs to
// the warps: the piece of the gate row and that of the up row share a slot and every activation they read.
struct GateUpShared {
  uint64_t bars[kMoeWarps * kMaxSlots];
  uint32_t ids[kMoeMaxTopK], route_ids[kMoeMaxTopK];
  float weights[kMoeMaxTopK], route_weights[kMoeMaxTopK];
  float logits[kMoeMaxExperts];
  uint32_t routed;
};

// A warp's run of units.
struct PairCursor {
  const uint16_t *gate;  // first element of the pair's gate row
  uint32_t row, col;     // of the matrix; first column of the unit
  uint32_t expert;       // index into ids
  uint32_t left;         // units
};

// Shared memory: ring | x (fp32, two planes) | GateUpShared | units' sums (gate, up).
__global__ void __launch_bounds__(kMoeThreads, 1) moe_gate_up_kernel(MoeExpertParams p) {
  extern __shared__ __align__(128) uint8_t smem[];
  const uint32_t ring_bytes = kMoeWarps * p.gate_up_slots * 2u * kPieceBytes;
  float *x = reinterpret_cast<float *>(smem + ring_bytes);
  GateUpShared &sh = *reinterpret_cast<GateUpShared *>(smem + ring_bytes + round128u(p.hidden * 4u));
  float2 *sums = reinterpret_cast<float2 *>(reinterpret_cast<uint8_t *>(&sh) + round128u(sizeof(GateUpShared)));
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t mi = p.moe_intermediate, hidden = p.hidden, parts = (hidden + kPieceCols - 1u) / kPieceCols;
  const uint64_t policy = l2_evict_first_policy();
  auto share = [](uint64_t total, uint32_t block) { return static_cast<uint32_t>(total * block / gridDim.x); };
  pdl_trigger();
  WarpRing ring;
  ring.init(smem, sh.bars, p.gate_up_slots, 2u * kPieceBytes);

  auto issue = [&](PairCursor &c, uint64_t up_offset) {
    const uint32_t bytes = hidden - c.col < kPieceCols ? (hidden - c.col) * 2u : kPieceBytes;
    if (elected()) {
      uint64_t *bar = &ring.bars[ring.issue_slot];
      uint8_t *dst = ring.base + ring.issue_slot * ring.slot_bytes;
      const uint16_t *src = c.gate + c.col;
      mbar_arrive_expect_tx(bar, 2u * bytes);
      tma_load_1d_hint(dst, src, bytes, bar, policy);
      tma_load_1d_hint(dst + kPieceBytes, src + up_offset, bytes, bar, policy);
    }
    ring.issued_one();
    c.left -= 1;
    c.col += kPieceCols;
    if (c.col >= hidden) {
      c.col = 0;
      c.row += 1;
      c.gate += hidden;
    }
  };
  // the shared expert's pieces do not depend on the routing: they come first in the streams
  const uint32_t shared_begin = share(p.shared_intermediate, blockIdx.x);
  const uint32_t shared_pairs = share(p.shared_intermediate, blockIdx.x + 1u) - shared_begin;
  const uint32_t shared_from = shared_pairs * parts * warp / kMoeWarps, shared_to = shared_pairs * parts * (warp + 1u) / kMoeWarps;
  PairCursor cs{p.w_shared_gate + static_cast<uint64_t>(shared_begin + shared_from / parts) * hidden, 0,
                shared_from % parts * kPieceCols, 0, shared_to - shared_from};
  const uint64_t shared_up = static_cast<uint64_t>(p.w_shared_up - p.w_shared_gate);
  while (cs.left != 0 && ring.room()) issue(cs, shared_up);
  pdl_wait();
  if (warp == 0) {
    for (uint32_t e = lane; e < p.num_experts; e += 32u) sh.logits[e] = __ldcg(p.router_logits + e);
    __syncwarp();
    moe_route_warp(sh.logits, p.num_experts, p.top_k, p.norm_topk_prob, sh.route_ids, sh.route_weights);
    __syncwarp();
    if (blockIdx.x == 0 && lane < p.top_k) {  // for the down launch
      p.expert_ids[lane] = sh.route_ids[lane];
      p.route_weights[lane] = sh.route_weights[lane];
    }
    const uint32_t chosen = lane < p.top_k ? lane : 0u;
    const uint32_t routed = held_experts(p, sh.route_ids[chosen], sh.route_weights[chosen], sh.ids, sh.weights);
    if (lane == 0) sh.routed = routed;
  } else {
    for (uint32_t i = threadIdx.x - 32u; i < hidden / 4u; i += kMoeThreads - 32u)
      reinterpret_cast<float4 *>(x)[i] = __ldcg(reinterpret_cast<const float4 *>(p.x_norm) + i);
  }
  __syncthreads();
  const uint32_t all_pairs = sh.routed * mi;
  const uint32_t begin = share(all_pairs, blockIdx.x), pairs = share(all_pairs, blockIdx.x + 1u) - begin;
  const uint32_t from = pairs * parts * warp / kMoeWarps, to = pairs * parts * (warp + 1u) / kMoeWarps;
  PairCursor c{nullptr, 0, from % parts * kPieceCols, 0, to - from};
  if (c.left != 0) {
    const uint32_t at = begin + from / parts;
    c.expert = at / mi;
    c.row = at % mi;
    c.gate = p.w_expert_gate_up + sh.ids[c.expert] * p.expert_stride + static_cast<uint64_t>(c.row) * hidden;
  }
  auto fill = [&]() {
    while (ring.room()) {
      if (cs.left != 0) {
        issue(cs, shared_up);
      } else if (c.left != 0) {
        if (c.row == mi) {
          c.row = 0;
          c.expert += 1;
          c.gate = p.w_expert_gate_up + sh.ids[c.expert] * p.expert_stride;
        }
        issue(c, p.expert_up_offset);
      } else {
        break;
      }
    }
  };
  const float4 *xa = reinterpret_cast<const float4 *>(x) + lane, *xb = xa + hidden / 8u;
  auto consume = [&](uint32_t first, uint32_t last, float2 *out) {
    uint32_t col = first % parts * kPieceCols;
    for (uint32_t u = first; u < last; ++u) {
      fill();
      const uint8_t *wp = ring.wait(p.error_word) + lane * 16u;
      const float4 *ca = xa + col / 8u, *cb = xb + col / 8u;
      float2 gate[4], up[4];
#pragma unroll
      for (uint32_t i = 0; i < 4u; ++i) gate[i] = up[i] = make_float2(0.0f, 0.0f);
      if (hidden - col >= kPieceCols) {
#pragma unroll
        for (uint32_t i = 0; i < 4u; ++i) {
          const float4 a = ca[32u * i], b = cb[32u * i];
          gate[i] = dot8_f32x2(lds128(wp + i * kSweepBytes), a, b, gate[i]);
          up[i] = dot8_f32x2(lds128(wp + kPieceBytes + i * kSweepBytes), a, b, up[i]);
        }
        col += kPieceCols;
      } else {
#pragma unroll
        for (uint32_t i = 0; i < 4u; ++i) {
          if (col + (32u * i + lane) * 8u >= hidden) continue;
          const float4 a = ca[32u * i], b = cb[32u * i];
          gate[i] = dot8_f32x2(lds128(wp + i * kSweepBytes), a, b, gate[i]);
          up[i] = dot8_f32x2(lds128(wp + kPieceBytes + i * kSweepBytes), a, b, up[i]);
        }
        col = hidden;
      }
      if (col >= hidden) col = 0;
      const float g = warp_sum(lane_sum(gate)), v = warp_sum(lane_sum(up));
      if (lane == 0) out[u] = make_float2(g, v);
      ring.release();
    }
  };
  consume(shared_from, shared_to, sums);
  consume(from, to, sums + shared_pairs * parts);
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < shared_pairs + pairs; i += kMoeThreads) {
    float gate = 0.0f, up = 0.0f;
    for (uint32_t k = 0; k < parts; ++k) {
      const float2 s = sums[i * parts + k];
      gate += s.x;
      up += s.y;
    }
    // activations: the routed experts' in routing order, then the shared expert's
    p.gate_up_out[i < shared_pairs ? all_pairs + shared_begin + i : begin + i - shared_pairs] = silu(gate) * up;
  }
  ring.drain();
}

// ---- down ----
// A block owns a range of output rows and reads them in every expert, a warp a row at a time: the lanes' partial sums
// of an expert are added times its weight, so that a row is reduced once.  The shared expert comes first in the
// stream (its weights do not wait for the routing) and last in the sum.
struct DownShared {
  uint64_t bars[kMoeWarps * kMaxSlots];
  uint32_t ids[kMoeMaxTopK];
  float weights[kMoeMaxTopK];
  float shared_gate;
  uint32_t routed;
};

// Shared memory: ring | activations (p.down_x_floats; fp32, two planes) | DownShared.  Where the activations
// of all experts do not fit together, the experts go in passes that do, and a row's sum goes on in out_f32.
__global__ void __launch_bounds__(kMoeThreads, 1) moe_down_kernel(MoeExpertParams p) {
  extern __shared__ __align__(128) uint8_t smem[];
  const uint32_t ring_bytes = kMoeWarps * p.down_slots * kPieceBytes;
  float *x = reinterpret_cast<float *>(smem + ring_bytes);
  DownShared &sh = *reinterpret_cast<DownShared *>(smem + ring_bytes + round128u(p.down_x_floats * 4u));
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t mi = p.moe_intermediate, si = p.shared_intermediate;
  const uint32_t row_begin = static_cast<uint32_t>(static_cast<uint64_t>(p.hidden) * blockIdx.x / gridDim.x);
  const uint32_t row_end = static_cast<uint32_t>(static_cast<uint64_t>(p.hidden) * (blockIdx.x + 1ull) / gridDim.x);
  const uint64_t policy = l2_evict_first_policy();
  pdl_trigger();
  WarpRing ring;
  ring.init(smem, sh.bars, p.down_slots, kPieceBytes);
  const uint32_t first = si != 0 ? 0u : 1u;  // matrix 0 is the shared expert's, matrix m > 0 routed expert m - 1

  uint32_t known = 1;                                   // matrices whose place is known: the shared one so far
  uint32_t pass_first = first, pass_end = 0xffffffffu;  // matrices of the issuing pass
  // the next piece: row, matrix, column
  uint32_t row = row_begin + warp, matrix = first, col = 0;
  auto fill = [&]() {
    while (ring.room() && row < row_end && matrix < known) {
      const uint32_t cols = matrix == 0 ? si : mi;
      const uint32_t bytes = cols - col < kPieceCols ? (cols - col) * 2u : kPieceBytes;
      if (elected()) {
        const uint16_t *src = matrix == 0 ? p.w_shared_down + static_cast<uint64_t>(row) * si
                                          : p.w_expert_down + (static_cast<uint64_t>(sh.ids[matrix - 1u]) * p.hidden + row) * mi;
        uint64_t *bar = &ring.bars[ring.issue_slot];
        mbar_arrive_expect_tx(bar, bytes);
        tma_load_1d_hint(ring.base + ring.issue_slot * kPieceBytes, src + col, bytes, bar, policy);
      }
      ring.issued_one();
      col += kPieceCols;
      if (col >= cols) {
        col = 0;
        matrix += 1;
        if (matrix == pass_end) {
          matrix = pass_first;
          row += kMoeWarps;
        }
      }
    }
  };
  fill();
  pdl_wait();
  if (warp == 0) {
    const uint32_t chosen = lane < p.top_k ? lane : 0u;
    const uint32_t routed = held_experts(p, __ldcg(p.expert_ids + chosen), __ldcg(p.route_weights + chosen), sh.ids, sh.weights);
    if (lane == 0) {
      sh.routed = routed;
      sh.shared_gate = si != 0 ? __ldcg(p.shared_gate) : 0.0f;
    }
  }
  __syncthreads();
  const uint32_t matrices = sh.routed + 1u;
  unsigned long long tag = 0;
  if (p.push.world > 1)
    tag = static_cast<unsigned long long>(static_cast<uint32_t>(*p.push.epoch) * p.push.per_epoch + p.push.offset) << 32;

  for (uint32_t m0 = first; m0 < matrices || m0 == first;) {
    // the matrices of this pass; pieces that are in flight already are those of the first pass's first matrix
    uint32_t m1 = m0, floats = 0;
    while (m1 < matrices && (m1 == m0 || floats + mi <= p.down_x_floats)) floats += m1++ == 0 ? si : mi;
    pass_end = m1;
    known = m1;
    if (m0 != first) {
      __syncthreads();  // the last pass's activations have been read
      pass_first = matrix = m0;
      row = row_begin + warp;
    } else if (matrix == m1 && m1 != m0) {  // a pass of one matrix whose first row is under way
      matrix = pass_first;
      row += kMoeWarps;
    }
    if (m1 != m0) fill();
    // their activations, the routed experts' and behind them the shared expert's, in two planes over all of them
    const uint32_t routed_from = m0 == 0 ? 0u : m0 - 1u, routed_floats = (m1 == 0 ? 0u : m1 - 1u - routed_from) * mi;
    const uint32_t quads = (routed_floats + (m0 == 0 ? si : 0u)) / 4u, plane = quads / 2u;
    const float4 *act = reinterpret_cast<const float4 *>(p.gate_up_out);
    const uint32_t routed_at = routed_from * mi / 4u, shared_at = (sh.routed * mi - routed_floats) / 4u;
    constexpr uint32_t kBatch = 4;  // loads in flight per thread
    for (uint32_t i0 = threadIdx.x; i0 < quads; i0 += kMoeThreads * kBatch) {
      float4 v[kBatch];
#pragma unroll
      for (uint32_t u = 0; u < kBatch; ++u) {
        const uint32_t i = i0 + u * kMoeThreads;
        if (i < quads) v[u] = __ldcg(act + i + (i < routed_floats / 4u ? routed_at : shared_at));
      }
#pragma unroll
      for (uint32_t u = 0; u < kBatch; ++u) {
        const uint32_t i = i0 + u * kMoeThreads;
        if (i < quads) reinterpret_cast<float4 *>(x)[(i & 1u) * plane + i / 2u] = v[u];
      }
    }
    __syncthreads();
    for (uint32_t r = row_begin + warp; r < row_end; r += kMoeWarps) {
      float sum = 0.0f, shared = 0.0f;  // of this lane
      const float resid = p.resid_in != nullptr && m1 == matrices && lane == 0 ? __ldcg(p.resid_in + r) : 0.0f;
      for (uint32_t m = m0; m < m1; ++m) {
        const uint32_t cols = m == 0 ? si : mi;
        const float4 *xa = reinterpret_cast<const float4 *>(x) + (m == 0 ? routed_floats : (m - 1u - routed_from) * mi) / 8u + lane;
        const float4 *xb = xa + plane;
        float2 acc[4];
#pragma unroll
        for (uint32_t i = 0; i < 4u; ++i) acc[i] = make_float2(0.0f, 0.0f);
        for (uint32_t left = cols; left != 0;) {
          fill();
          const uint8_t *wp = ring.wait(p.error_word) + lane * 16u;
          if (left >= kPieceCols) {
#pragma unroll
            for (uint32_t i = 0; i < 4u; ++i) acc[i] = dot8_f32x2(lds128(wp + i * kSweepBytes), xa[32u * i], xb[32u * i], acc[i]);
            left -= kPieceCols;
          } else {
#pragma unroll
            for (uint32_t i = 0; i < 4u; ++i) {
              if ((32u * i + lane) * 8u >= left) continue;
              acc[i] = dot8_f32x2(lds128(wp + i * kSweepBytes), xa[32u * i], xb[32u * i], acc[i]);
            }
            left = 0;
          }
          xa += kPieceCols / 8u;
          xb += kPieceCols / 8u;
          ring.release();
        }
        if (m == 0)
          shared = sh.shared_gate * lane_sum(acc);
        else
          sum += sh.weights[m - 1u] * lane_sum(acc);
      }
      sum = warp_sum(sum + shared);
      if (lane != 0) continue;
      if (m0 != first) sum += p.out_f32[r];  // earlier passes
      if (p.push.world > 1 && m1 == matrices) {
        // expert parallel: this rank's partial sum travels to every rank (projection.cu: the Store epilogue's push)
        const unsigned long long entry = tag | __float_as_uint(sum);
        const uint64_t at = static_cast<uint64_t>(p.push.rank) * p.hidden + r;
        for (uint32_t q = 0; q < p.push.world; ++q)
          asm volatile("st.volatile.global.u64 [%0], %1;" ::"l"(p.push.recv[q] + at), "l"(entry) : "memory");
      } else {
        p.out_f32[r] = p.resid_in != nullptr ? sum + resid : sum;
      }
    }
    if (m1 >= matrices) break;
    m0 = m1;
  }
  ring.drain();
}

// ---- launch shapes ----
struct MoePlan {
  uint32_t gate_up_blocks, gate_up_smem, down_blocks, down_smem;
};

// Dynamic shared memory a block may ask for.
constexpr uint32_t kMoeMaxDynamicSmem = 227u * 1024u;

// Fills p.gate_up_slots, p.down_slots and p.down_x_floats; false when a launch would not fit.
bool plan_moe(MoeExpertParams &p, uint32_t sm_count, MoePlan *plan) {
  const uint32_t mi = p.moe_intermediate, si = p.shared_intermediate;
  const uint32_t pairs = p.top_k * mi, parts = (p.hidden + kPieceCols - 1u) / kPieceCols;
  plan->gate_up_blocks = std::min(std::max(std::max(pairs, si), 1u), sm_count);
  const uint32_t units = (pairs / plan->gate_up_blocks + si / plan->gate_up_blocks + 2u) * parts;  // most of a block
  const uint32_t fixed_up = round128u(p.hidden * 4u) + round128u(sizeof(GateUpShared)) + round128u(units * 8u);
  // three slots of a warp keep 192 KB in flight; where the rest leaves no room for them, two or one
  for (p.gate_up_slots = 3u; p.gate_up_slots != 0; --p.gate_up_slots) {
    plan->gate_up_smem = kMoeWarps * p.gate_up_slots * 2u * kPieceBytes + fixed_up;
    if (plan->gate_up_smem <= kMoeMaxDynamicSmem) break;
  }
  if (p.gate_up_slots == 0) return false;
  plan->down_blocks = std::min(p.hidden, sm_count);
  const uint32_t fixed = round128u(sizeof(DownShared)) + 128u, all = pairs + si, longest = std::max(mi, si);
  // as many slots as fit beside all activations, or two slots and as many activations as fit
  for (p.down_slots = kMaxSlots; p.down_slots > 2u; --p.down_slots) {
    if (fixed + kMoeWarps * p.down_slots * kPieceBytes + all * 4u <= kMoeMaxDynamicSmem) break;
  }
  const uint32_t ring = kMoeWarps * p.down_slots * kPieceBytes;
  p.down_x_floats = std::min(all, (kMoeMaxDynamicSmem - fixed - ring) / 4u);
  if (p.down_x_floats < longest) return false;
  plan->down_smem = fixed + ring + round128u(p.down_x_floats * 4u);
  return plan->down_smem <= kMoeMaxDynamicSmem;
}

}  // namespace

bool moe_supported(uint32_t hidden, uint32_t moe_intermediate, uint32_t shared_intermediate,
                   uint32_t num_experts, uint32_t top_k, uint32_t sm_count) {
  if (num_experts == 0 || num_experts > kMoeMaxExperts || top_k == 0 || top_k > kMoeMaxTopK || top_k > num_experts) return false;
  if (hidden % 8u != 0 || moe_intermediate % 8u != 0 || shared_intermediate % 8u != 0) return false;
  MoeExpertParams p{};
  p.hidden = hidden;
  p.moe_intermediate = moe_intermediate;
  p.shared_intermediate = shared_intermediate;
  p.top_k = top_k;
  MoePlan plan{};
  return plan_moe(p, sm_count, &plan);
}

cudaError_t configure_moe_kernels() {
  cudaError_t err = cudaFuncSetAttribute(moe_gate_up_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMoeMaxDynamicSmem);
  if (err == cudaSuccess) err = cudaFuncSetAttribute(moe_down_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMoeMaxDynamicSmem);
  return err;
}

cudaError_t launch_moe_experts(cudaStream_t stream, const MoeExpertParams &params, uint32_t sm_count, bool pdl) {
  MoeExpertParams p = params;
  MoePlan plan{};
  if (p.x_norm == nullptr || p.router_logits == nullptr || p.w_router == nullptr ||
      !moe_supported(p.hidden, p.moe_intermediate, p.shared_intermediate, p.num_experts, p.top_k, sm_count) ||
      !plan_moe(p, sm_count, &plan))
    return cudaErrorNotSupported;
  const uint32_t router_blocks = p.num_experts + (p.shared_intermediate != 0 && p.w_shared_router != nullptr ? 1u : 0u);
  cudaError_t err = launch_with_pdl(moe_router_kernel, dim3(router_blocks), dim3(kRouterThreads), 0, stream, pdl, p);
  if (err == cudaSuccess)
    err = launch_with_pdl(moe_gate_up_kernel, dim3(plan.gate_up_blocks), dim3(kMoeThreads), plan.gate_up_smem, stream, pdl, p);
  if (err != cudaSuccess) return err;
  return launch_with_pdl(moe_down_kernel, dim3(plan.down_blocks), dim3(kMoeThreads), plan.down_smem, stream, pdl, p);
}

}  // namespace nb
