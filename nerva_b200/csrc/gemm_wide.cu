// Block projection of more than kGemmMaxTokens tokens (prefill chunks): Y[token][row] = W[row][:] . X[token][:],
// bf16 in, fp32 accumulate, on pairs of SMs.
//
// What bounds it: the tensor pipe.  With up to 256 tokens a weight byte is worth 512 flops and the projection is
// bound by HBM (gemm_tc.cu); from a few hundred tokens on it is arithmetic, and what the tensor pipe waits for is
// shared memory being filled from L2.  A lone SM with a 128 x 256 tile takes in 48 KB per 64-wide slice, which the
// L2 cannot deliver to 148 SMs at the MMA's rate; so two SMs of a cluster share one 256 x 256 tile
// (`tcgen05.mma.cta_group::2`): each loads its own 128 weight rows and HALF of the tokens, 32 KB per slice for the
// same arithmetic per SM, and holds the fp32 accumulator of its 128 rows in its own tensor memory.
//
// Decomposition: persistent pairs walk the tiles, tokens fastest, so that the pairs that run at one time share few
// weight tiles (each read from HBM once) and all token tiles (which stay in L2).  The inner dimension is never
// split: there is no workspace and no second launch.  Tokens per tile: choose_tile_tokens below.
//
// The epilogue runs under the MMAs of the next tile, but a tile's has to be shorter than a tile's MMAs (17 us at 4096
// columns), and the last one is not hidden: hence eight warps, values without branches and residuals a group ahead
// (row_epilogue, row_residual).
//
// Measured back to back, other weights each time, 2048 tokens, and in brackets with four epilogue warps, a branch per value and
// issuing threads chosen by lane: 24576 x 4096 with SwiGLU 260 us, 1586 TFLOP/s (394); 4096 x 12288 with residual 140 (178);
// 6144 x 4096 71 (96); 4096 x 4096 with residual 52 (85).
//
// Roles inside a block (320 threads), as in gemm_tc.cu: warp 0 issues the TMA copies into the block's own ring,
// warp 1 of the pair's first block issues the MMAs for both (its `full` barriers count the bytes of both blocks),
// warps 2..9 read the accumulator and run the epilogue, four of them every second group of tokens.  Commits of the MMAs
// are signalled to both blocks.  Two accumulator buffers of 256 columns let the epilogue of one tile run under the MMAs of the next.  Every wait is
// bounded; a wait that gives up sets the error word and the block's abort flag, the block drains and the pair
// leaves together.  No copy is multicast.
#include "gemm_device.cuh"

namespace nb {
namespace {

constexpr uint32_t kPairRows = 2u * kTileRows;  // MMA M over the pair
constexpr uint32_t kMinTileTokens = 64, kMaxTileTokens = 256;  // MMA N
constexpr uint32_t kTokenStep = 32;             // tile sizes: whole 8-row swizzle atoms in each half, N a multiple of 16
constexpr uint32_t kMaxStages = 8;
constexpr uint32_t kThreads = 320;
constexpr uint32_t kEpilogueWarps = 8;
constexpr uint32_t kTmemColumns = 512, kAccStride = 256;
constexpr uint32_t kLeaderMask = 0xfeffffffu;   // clears the bit of a shared::cluster address that names the pair's second block

struct WideShared {
  uint64_t full[kMaxStages], empty[kMaxStages];
  uint64_t acc_full[2], acc_empty[2];
  uint64_t drained;
  uint32_t tmem_base;
  uint32_t abort;
};

struct WideTiles {
  uint32_t row_tiles, token_tiles, tile_tokens;  // of kPairRows weight rows, of tile_tokens tokens
};

// Timeline stamp of the first or the last pair, by a thread of the block that issues its MMAs.
__device__ __forceinline__ void stamp_pair(unsigned long long *stamps, uint32_t slot, uint32_t pair, uint32_t pairs) {
  if (stamps == nullptr || (pair != 0 && pair + 1u != pairs)) return;
  unsigned long long now;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
  if (pair == 0) stamps[slot] = now;
  if (pair + 1u == pairs) stamps[4u + slot] = now;
}

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// A copy into this block's shared memory whose bytes are counted on the pair's first block.
__device__ __forceinline__ void tma_load_2d_pair(void *dst, const CUtensorMap *map, uint32_t x, uint32_t y, uint64_t *bar,
                                                 uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1, {%2, %3}], [%4], %5;" ::"r"(smem_addr(dst)),
      "l"(map), "r"(x), "r"(y), "r"(smem_addr(bar) & kLeaderMask), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void pair_mma(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives at the same barrier of the blocks in `mask` (bit 0: the pair's first) once the MMAs issued so far are done.
__device__ __forceinline__ void pair_commit(uint64_t *bar, uint16_t mask = 3) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_addr(bar)),
      "h"(mask)
      : "memory");
}
// Arrives at a barrier of the pair's first block.
__device__ __forceinline__ void leader_arrive(uint64_t *bar) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(remote) : "r"(smem_addr(bar)));
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote) : "memory");
}
// Instruction descriptor of the pair's MMA: fp32 accumulator, bf16 A and B, both K-major, N = n, M = 256.
__device__ __forceinline__ uint32_t pair_instr_desc(uint32_t n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((kPairRows >> 4) << 24);
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_wide_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, GemmKernelParams p,
                 WideTiles t) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *ring = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~uintptr_t{1023});
  const uint32_t half = t.tile_tokens / 2u;  // tokens of a tile that this block loads
  const uint32_t stage_bytes = kATileBytes + half * kSliceK * 2u;
  WideShared &sh = *reinterpret_cast<WideShared *>(ring + p.stages * stage_bytes);
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  volatile uint32_t *abort = &sh.abort;
  const uint32_t rank = cluster_rank();
  const uint32_t pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const uint32_t tiles = t.row_tiles * t.token_tiles, slices = p.cols / kSliceK;

  pdl_trigger();
  if (threadIdx.x == 0) {
    if (rank == 0) stamp_pair(p.stamps, kStampEntry, pair, pairs);
    for (uint32_t s = 0; s < p.stages; ++s) {
      mbar_init(&sh.full[s], 1);
      mbar_init(&sh.empty[s], 1);
    }
    for (uint32_t a = 0; a < 2; ++a) {
      mbar_init(&sh.acc_full[a], 1);
      mbar_init(&sh.acc_empty[a], 2u * kEpilogueWarps);  // the epilogue warps of both blocks
    }
    mbar_init(&sh.drained, 1);
    sh.abort = 0;
    mbar_init_fence();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&sh.tmem_base)),
                 "r"(kTmemColumns)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  cluster_sync();  // the barriers of both blocks exist
  tcgen05_fence_after();
  const uint32_t tmem_base = sh.tmem_base;

  if (warp == 0) {
    // ---------------- producer ----------------
    if (elected()) {
      const uint64_t w_policy = l2_evict_first_policy();  // a weight tile's readers run together
      const uint64_t x_policy = l2_evict_last_policy();
      bool ok = true, waited = false;
      uint32_t issued = 0;
      for (uint32_t tile = pair; ok && tile < tiles; tile += pairs) {
        const uint32_t w_row = (tile / t.token_tiles) * kPairRows + rank * kTileRows;
        const uint32_t x_row = (tile % t.token_tiles) * t.tile_tokens + rank * half;
        for (uint32_t c = 0; c < slices; ++c, ++issued) {
          const uint32_t s = issued % p.stages;
          if (!abortable_wait(&sh.empty[s], ((issued / p.stages) & 1u) ^ 1u, abort, p.error_word)) {
            ok = false;
            break;
          }
          uint8_t *stage = ring + s * stage_bytes;
          if (rank == 0) mbar_arrive_expect_tx(&sh.full[s], 2u * stage_bytes);  // both blocks' copies
          tma_load_2d_pair(stage, &map_w, c * kSliceK, w_row, &sh.full[s], w_policy);
          if (!waited) {  // the weights do not depend on the previous kernel, the tokens do
            pdl_wait();
            waited = true;
          }
          tma_load_2d_pair(stage + kATileBytes, &map_x, c * kSliceK, x_row, &sh.full[s], x_policy);
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer: the pair's first block ----------------
    if (rank == 0 && elected()) {
      const uint32_t idesc = pair_instr_desc(t.tile_tokens);
      // (in front of the loop: a test inside it took 3 % of a 512-token prefill)
      if (p.stamps != nullptr && abortable_wait(&sh.full[0], 0, abort, p.error_word)) stamp_pair(p.stamps, kStampAfterWait, pair, pairs);
      uint32_t consumed = 0, index = 0;
      bool ok = true;
      for (uint32_t tile = pair; ok && tile < tiles; tile += pairs, ++index) {
        const uint32_t acc = index & 1u;
        if (!abortable_wait(&sh.acc_empty[acc], ((index >> 1) & 1u) ^ 1u, abort, p.error_word)) break;
        tcgen05_fence_after();
        const uint32_t tmem_d = tmem_base + acc * kAccStride;
        for (uint32_t c = 0; c < slices; ++c, ++consumed) {
          const uint32_t s = consumed % p.stages;
          if (!abortable_wait(&sh.full[s], (consumed / p.stages) & 1u, abort, p.error_word)) {
            ok = false;
            break;
          }
          tcgen05_fence_after();
          const uint8_t *stage = ring + s * stage_bytes;
          const uint64_t desc_a = kmajor_sw128_desc(stage), desc_b = kmajor_sw128_desc(stage + kATileBytes);
#pragma unroll
          for (uint32_t k = 0; k < kSliceK / kUmmaK; ++k)
            pair_mma(tmem_d, desc_a + 2ull * k, desc_b + 2ull * k, idesc, (c != 0 || k != 0) ? 1u : 0u);
          pair_commit(&sh.empty[s]);
        }
        if (ok) pair_commit(&sh.acc_full[acc]);
      }
      stamp_pair(p.stamps, kStampAfterPrologue, pair, pairs);
    }
  } else {
    // ---------------- epilogue (warps 2..9) ----------------
    pdl_wait();
    const uint32_t quarter = warp & 3u, from = ((warp - 2u) >> 2) * kGroup;
    uint32_t index = 0;
    for (uint32_t tile = pair; tile < tiles; tile += pairs, ++index) {
      const uint32_t acc = index & 1u;
      const uint32_t taddr = tmem_base + acc * kAccStride + ((quarter * 32u) << 16);
      const uint32_t row = (tile / t.token_tiles) * kPairRows + rank * kTileRows + quarter * 32u + lane;
      const uint32_t m0 = (tile % t.token_tiles) * t.tile_tokens;
      const uint32_t count = p.tokens - m0 < t.tile_tokens ? p.tokens - m0 : t.tile_tokens;
      float resid[kGroup];
      row_residual<kGroup>(p, resid, row, m0 + from);
      if (!warp_wait(&sh.acc_full[acc], (index >> 1) & 1u, abort, p.error_word)) break;
      tcgen05_fence_after();
      for (uint32_t g = from; g < count; g += 2u * kGroup) {
        float v[kGroup], next[kGroup];
        tmem_load16(taddr + g, v);
        row_residual<kGroup>(p, next, row, m0 + g + 2u * kGroup);
        row_epilogue<kGroup>(p, v, resid, row, m0 + g, lane);
#pragma unroll
        for (uint32_t j = 0; j < kGroup; ++j) resid[j] = next[j];
      }
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) leader_arrive(&sh.acc_empty[acc]);
    }
  }
  // ---- teardown: the pair leaves together, with nothing in flight ----
  tcgen05_fence_before();
  __syncthreads();
  if (sh.abort != 0u && rank == 0) {  // the first block counts the copies of both and issues the MMAs
    if (threadIdx.x == 0) drain_copies(sh.full, p.stages);
    if (warp == 1 && elected()) {
      pair_commit(&sh.drained, 1);
      mbar_wait_bounded(&sh.drained, 0);
    }
  }
  __syncthreads();
  cluster_sync();
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemColumns) : "memory");
    if (rank == 0 && lane == 0) stamp_pair(p.stamps, kStampExit, pair, pairs);
  }
}

uint32_t wide_stage_bytes(uint32_t tile_tokens) { return kATileBytes + tile_tokens / 2u * kSliceK * 2u; }

uint32_t wide_stages(uint32_t tile_tokens) {
  const uint32_t stages = 222u * 1024u / wide_stage_bytes(tile_tokens);
  return stages < kMaxStages ? stages : kMaxStages;
}

uint32_t wide_smem_bytes(uint32_t tile_tokens) {
  return tensor_memory_smem(kTmemColumns, 1024u + wide_stages(tile_tokens) * wide_stage_bytes(tile_tokens) +
                                              static_cast<uint32_t>(sizeof(WideShared)) + 64u);
}

// Tokens per tile: the size with the shortest run of the slowest pair.  A slice costs a pair the larger of its MMA
// time (2 cycles per token) and the time its shared memory takes to fill (about 45 bytes per cycle and SM with all
// SMs loading and issuing threads chosen by lane; loads alone now take in 57, which changes the size for none of eight
// matrices of 2048 to 24576 rows at ten counts from 257 to 2048), so narrow tiles pay for the weight rows they re-read; wide ones may leave a last wave nearly empty.
uint32_t choose_tile_tokens(uint32_t rows, uint32_t tokens, uint32_t pairs) {
  const uint32_t row_tiles = (rows + kPairRows - 1u) / kPairRows;
  uint32_t best = kMaxTileTokens;
  uint64_t best_cost = ~0ull;
  for (uint32_t n = kMaxTileTokens; n >= kMinTileTokens; n -= kTokenStep) {
    const uint32_t tiles = row_tiles * ((tokens + n - 1u) / n);
    const uint64_t waves = (tiles + pairs - 1u) / pairs;
    const uint64_t fill = wide_stage_bytes(n) / 45u, mma = 2u * n;
    const uint64_t cost = waves * (fill > mma ? fill : mma);
    if (cost < best_cost) {
      best_cost = cost;
      best = n;
    }
  }
  return best;
}

}  // namespace

cudaError_t configure_gemm_wide_kernel() {
  return cudaFuncSetAttribute(gemm_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
}

void gemm_wide_launches(std::vector<TensorMemoryLaunch> *out) {
  for (uint32_t n = kMinTileTokens; n <= kMaxTileTokens; n += kTokenStep) out->push_back({wide_smem_bytes(n), kTmemColumns});
}

cudaError_t launch_gemm_wide(cudaStream_t stream, const GemmParams &g, uint32_t sm_count) {
  const uint32_t pairs = sm_count / 2u;
  WideTiles t{};
  t.tile_tokens = choose_tile_tokens(g.rows, g.tokens, pairs);
  t.row_tiles = (g.rows + kPairRows - 1u) / kPairRows;
  t.token_tiles = (g.tokens + t.tile_tokens - 1u) / t.tile_tokens;
  GemmKernelParams p = gemm_kernel_params(g);
  p.stages = wide_stages(t.tile_tokens);
  CUtensorMap map_w, map_x;
  if (!encode_bf16_map_2d(&map_w, g.weight, g.cols, g.rows, kSliceK, kTileRows) ||
      !encode_bf16_map_2d(&map_x, g.x, g.cols, g.tokens, kSliceK, t.tile_tokens / 2u))
    return cudaErrorNotSupported;
  const uint32_t tiles = t.row_tiles * t.token_tiles;
  return launch_with_pdl(gemm_wide_kernel, dim3(2u * (tiles < pairs ? tiles : pairs)), dim3(kThreads),
                         wide_smem_bytes(t.tile_tokens), stream, g.pdl != 0, map_w, map_x, p, t);
}

}  // namespace nb
