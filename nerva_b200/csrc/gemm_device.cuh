// Device-side pieces that the block projection kernels share (gemm_tc.cu: up to 256 tokens, gemm_wide.cu: more):
// TMA, tcgen05 and descriptor wrappers, bounded mbarrier waits, and the epilogue of one accumulator row.
#pragma once

#include <cuda.h>

#include "common.cuh"
#include "kernels.cuh"

namespace nb {

constexpr uint32_t kTileRows = 128;   // weight rows of one block's accumulator: the lanes of tensor memory
constexpr uint32_t kSliceK = 64;      // bf16 elements per ring stage along the inner dimension (128 bytes)
constexpr uint32_t kUmmaK = 16;       // inner elements per MMA instruction
constexpr uint32_t kATileBytes = kTileRows * kSliceK * 2u;
constexpr uint32_t kGroup = 16;       // tokens per tcgen05.ld

// The 512 columns of an SM's tensor memory are shared by the blocks that are resident together, and an allocation that does
// not fit waits until another block leaves.  With programmatic dependent launch the other block may be of a later launch
// that waits for this one's end, so blocks that can be resident together must never ask for more than there is.  Launches
// of up to kSharedColumns may share an SM (four of them fit); a launch that takes more asks for so much shared memory that
// no other block with tensor memory fits beside it, whatever registers and launch order would allow.
constexpr uint32_t kSharedColumns = 128;
constexpr uint32_t kSmemPerSm = 228u * 1024u, kSmemReserved = 1024u;  // per SM; by the system, per block
constexpr uint32_t kLeastTmemSmem = 88u * 1024u;                      // of every launch with tensor memory
constexpr uint32_t kAloneTmemSmem = kSmemPerSm - 2u * kSmemReserved - kLeastTmemSmem + 128u;
// Dynamic shared memory of a launch that takes `columns` of tensor memory and needs `bytes`.
__host__ __device__ constexpr uint32_t tensor_memory_smem(uint32_t columns, uint32_t bytes) {
  const uint32_t least = columns > kSharedColumns ? kAloneTmemSmem : kLeastTmemSmem;
  return bytes > least ? bytes : least;
}

struct GemmKernelParams {
  uint32_t rows, cols, tokens, n_pad;  // n_pad: tokens rounded up to 16 (the MMA N)
  uint32_t stages;
  uint32_t tmem_columns;  // allocation: two accumulator buffers of tmem_columns / 2 fp32 columns
  uint32_t epilogue;
  uint32_t split_row;         // kEpilogueStoreSwiglu: first row of the gate/up pairs (a multiple of 32)
  const float *resid_in;
  const uint16_t *row_scale;  // kEpilogueStore, optional: y is multiplied by row_scale[row] before the residual add
  const uint16_t *row_add;    // kEpilogueStore, optional: added to y
  uint32_t activation;        // of the gate in gate/up pairs
  float scale;                // kEpilogueStore: 0, or a factor on y
  float softcap;              // kEpilogueStore: 0, or y becomes softcap * tanh(y / softcap)
  float *out_f32;
  uint16_t *out_bf16;
  float *workspace;
  uint32_t *tickets;
  uint32_t *error_word;
  unsigned long long *stamps;
};

// The fields that a call's parameters give; the launchers fill the others.
inline GemmKernelParams gemm_kernel_params(const GemmParams &g) {
  GemmKernelParams p{};
  p.rows = g.rows;
  p.cols = g.cols;
  p.tokens = g.tokens;
  p.epilogue = g.epilogue;
  p.split_row = g.split_row;
  p.resid_in = g.resid_in;
  p.row_scale = g.row_scale;
  p.row_add = g.row_add;
  p.activation = g.activation;
  p.scale = g.scale;
  p.softcap = g.softcap;
  p.out_f32 = g.out_f32;
  p.out_bf16 = g.out_bf16;
  p.workspace = g.workspace;
  p.tickets = g.tickets;
  p.error_word = g.error_word;
  p.stamps = g.stamps;
  return p;
}

// ---- PTX wrappers ----
__device__ __forceinline__ bool abortable_wait(uint64_t *bar, uint32_t parity, volatile uint32_t *abort,
                                               uint32_t *error_word) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long start = clock64();
  for (;;) {
#pragma unroll 1
    for (uint32_t spin = 0; spin < 64; ++spin) {
      if (mbar_try_wait(bar, parity)) return true;
    }
    if (*abort != 0u) return false;
    if (clock64() - start > kWaitCycleLimit) {
      *abort = 1u;
      report_error(error_word, kErrTmaWaitTimeout);
      return false;
    }
  }
}
// All lanes of a warp wait; false for all of them when one gave up: what a wait in front of warp-wide tensor-memory accesses
// has to be, since each lane runs out of time, or sees the abort flag, by itself.
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity, volatile uint32_t *abort, uint32_t *error_word) {
  return __all_sync(0xffffffffu, abortable_wait(bar, parity, abort, error_word));
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, uint32_t x, uint32_t y, uint64_t *bar,
                                            uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1, {%2, %3}], [%4], %5;" ::"r"(smem_addr(dst)),
      "l"(map), "r"(x), "r"(y), "r"(smem_addr(bar)), "l"(policy)
      : "memory");
}
__device__ __forceinline__ uint64_t l2_evict_last_policy() {
  uint64_t policy;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(policy));
  return policy;
}
__device__ __forceinline__ void tcgen05_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tcgen05_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tcgen05_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
               : "memory");
}
__device__ __forceinline__ void tcgen05_mma_f16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                                uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_load16(uint32_t taddr, float *v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (uint32_t i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// A block that gives up a wait still owns what it has issued: its shared memory and its tensor memory go to the next block
// of the SM only when the copies into its rings have landed and its MMAs are done, or a bounded wait for them has run out.
__device__ __forceinline__ void drain_copies(uint64_t *full, uint32_t stages) {
  for (uint32_t s = 0; s < stages; ++s) {
    mbar_wait_bounded(&full[s], 0);
    mbar_wait_bounded(&full[s], 1);
  }
}
// By the thread that issued the MMAs; `bar` has one arrival and no other use.
__device__ __forceinline__ void drain_mmas(uint64_t *bar) {
  tcgen05_commit(bar);
  mbar_wait_bounded(bar, 0);
}

// Shared-memory matrix descriptor of a K-major tile whose rows are 128 bytes (one swizzle atom):
// start address, 8-row groups 1024 bytes apart, SWIZZLE_128B, descriptor version 1.
__device__ __forceinline__ uint64_t kmajor_sw128_desc(const void *tile) {
  const uint64_t addr = smem_addr(tile);
  return ((addr & 0x3ffffull) >> 4) | (1ull << 16) | (static_cast<uint64_t>(1024u >> 4) << 32) | (1ull << 46) |
         (2ull << 61);
}
// Instruction descriptor: fp32 accumulator, bf16 A and B, both K-major, N = n, M = 128.
__device__ __forceinline__ uint32_t instr_desc_bf16(uint32_t n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((kTileRows >> 4) << 24);
}

// True for accumulator rows that are gate/up pairs.
__device__ __forceinline__ bool epilogue_pairs(const GemmKernelParams &p, uint32_t row) {
  return p.epilogue == kEpilogueSwiglu || (p.epilogue == kEpilogueStoreSwiglu && row >= p.split_row);
}

// The residuals of N consecutive tokens m0 .. m0 + N - 1 of accumulator row `row`, zeros where there are none.  Apart from
// row_epilogue, so that a caller can ask for the next group's while it stores this one's, and all of them before the first
// store: the store might alias a later load (the stream is updated in place), so the compiler would wait for each in
// turn, a round trip to L2 per token.
template <uint32_t N>
__device__ __forceinline__ void row_residual(const GemmKernelParams &p, float (&resid)[N], uint32_t row, uint32_t m0) {
  const bool has = p.resid_in != nullptr && row < p.rows && !epilogue_pairs(p, row);
  const uint32_t width = p.epilogue == kEpilogueStoreSwiglu ? p.split_row : p.rows;
  const float *src = p.resid_in + static_cast<uint64_t>(m0) * width + row;
#pragma unroll
  for (uint32_t j = 0; j < N; ++j) resid[j] = has && m0 + j < p.tokens ? __ldcg(src + static_cast<uint64_t>(j) * width) : 0.0f;
}

// N consecutive tokens m0 .. m0 + N - 1 of accumulator row `row`, values in v, residuals from row_residual.  Called by all 32
// lanes of a warp whose lanes hold 32 consecutive rows (the first a multiple of 32).
template <uint32_t N>
__device__ __forceinline__ void row_epilogue(const GemmKernelParams &p, const float (&v)[N], const float (&resid)[N], uint32_t row,
                                             uint32_t m0, uint32_t lane) {
  static_assert(N % 2u == 0, "tokens are shared out between the lanes of a pair");
  if (epilogue_pairs(p, row)) {
    // rows interleaved (gate, up): of two tokens the gate's lane takes the first and the up's lane the second, and each
    // sends the other what it has of its token.  Values first, then the stores: with a branch around each value its
    // exponential and division ran one after the other (24576 x 4096, 2048 tokens: 394 us, 281 without any epilogue).  The
    // division itself is the one to nearest: an approximate one is no faster here (12011-token request 83.4 and 83.5 ms).
    const uint32_t base = p.epilogue == kEpilogueStoreSwiglu ? p.split_row : 0u;
    const uint32_t width = (p.rows - base) / 2u, odd = lane & 1u;
    const uint32_t column = (row - base) / 2u;
    const bool live = (row | 1u) < p.rows;
    auto store = [&](auto act) {  // one loop per activation
      uint16_t y[N / 2u];
#pragma unroll
      for (uint32_t j = 0; j < N; j += 2u) {
        const float theirs = __shfl_xor_sync(0xffffffffu, odd != 0 ? v[j] : v[j + 1u], 1);
        const float gate = odd != 0 ? theirs : v[j], up = odd != 0 ? v[j + 1u] : theirs;
        y[j / 2u] = f32_to_bf16_bits(act(gate) * up);
      }
      uint16_t *out = p.out_bf16 + static_cast<uint64_t>(m0 + odd) * width + column;
#pragma unroll
      for (uint32_t j = 0; j < N; j += 2u)
        if (live && m0 + odd + j < p.tokens) out[static_cast<uint64_t>(j) * width] = y[j / 2u];
    };
    if (p.activation == kActivationSilu)
      store([](float x) { return silu(x); });
    else
      store([](float x) { return activate(kActivationGeluTanh, x); });
  } else if (row < p.rows) {
    const uint32_t width = p.epilogue == kEpilogueStoreSwiglu ? p.split_row : p.rows;
    const float scale = (p.row_scale != nullptr ? bf16_bits_to_f32(p.row_scale[row]) : 1.0f) * (p.scale != 0.0f ? p.scale : 1.0f);
    const float add = p.row_add != nullptr ? bf16_bits_to_f32(p.row_add[row]) : 0.0f;
    float *out = p.out_f32 + static_cast<uint64_t>(m0) * width + row;
    float y[N];
#pragma unroll
    for (uint32_t j = 0; j < N; ++j) y[j] = fmaf(v[j], scale, add);
    if (p.softcap > 0.0f) {
#pragma unroll
      for (uint32_t j = 0; j < N; ++j) y[j] = p.softcap * tanhf(y[j] / p.softcap);
    }
#pragma unroll
    for (uint32_t j = 0; j < N; ++j) y[j] = p.resid_in != nullptr ? y[j] + resid[j] : y[j];
    if (m0 + N <= p.tokens) {
#pragma unroll
      for (uint32_t j = 0; j < N; ++j) out[static_cast<uint64_t>(j) * width] = y[j];
    } else {
#pragma unroll
      for (uint32_t j = 0; j < N; ++j)
        if (m0 + j < p.tokens) out[static_cast<uint64_t>(j) * width] = y[j];
    }
  }
}

}  // namespace nb
