// Attention of a block of one session's rows (prefill chunk) on the fifth-generation tensor pipe.
//
// A block of threads takes 128 (position, head) rows of one KV head, so the heads that share a KV head share its keys,
// and walks 128-key tiles up to the last row's own position:
//   S = Q K^T      tcgen05.mma, Q and K in shared memory, S (fp32) in tensor memory
//   P = exp2(S-m)  one thread per row: the row's 128 scores in registers, no exchange between threads
//   O += P V       tcgen05.mma, P in tensor memory in the place of S, V in shared memory as it is cached (token-major:
//                  the MMA takes it in the MN-major form), O (fp32) in tensor memory
// Queries and probabilities are fp32 values; each enters as a bf16 rounding and its remainder, two MMAs into the same
// accumulator, so a product loses only the rounding of the cached row (the contract of the other attention kernels).
//
// What bounds it: the MMAs, 4 x 512 cycles a tile (two parts of Q, two of P), and the hand-overs between them.  By clock stamps
// in a copy of this kernel a tile of a long walk takes 3500 cycles, 2090 of them issuing MMAs; the softmax warps wait 64 % of
// the time: a tile of theirs is 120 cycles of loads, 320 for the maximum, 1700 for 128 exponentials a thread, their sums and
// two packs.  S has two buffers: S(j+1) is computed while the softmax works on S(j), but S(j+2) goes where P(j) is and waits
// for its PV.  The output accumulator is rescaled only when a row's maximum has grown by more than 2^8 since the reference
// it uses (the probabilities stay below 2^8, the sums exact to fp32): after the first tiles that almost never happens.
// One 128-row tile per block (both parts of Q, 64 KB, and two stages of K and V, 128 KB, fill shared memory), and two
// groups of softmax warps, each with every second tile, a running maximum, a sum and an output accumulator of its own,
// added at the end.  The second group gives little: 2048 tokens, 32 heads, 117 us with one group, 114 with two when it was added.
//
// Measured (whole prefill, 8B shapes, 8 layers and head; row by row through the decode kernel before): 512 tokens 3.2 ms
// (5.5), 3001 tokens 13.2 (40.5), projections on pairs of SMs included; vuvolix 1.7b, window 1024, 2048 tokens 12.8 (38.4).
//
// Roles (320 threads): warps 0..3 and 4..7 softmax, rescaling and the output (warp w reads tensor-memory lanes
// 32 (w % 4) ..), warp 8 brings K and V (one 2-D TMA box per page and 64 columns, 128-byte swizzle), warp 9 issues the
// MMAs and cleans the values of tiles at an edge.  (cp.async by two warps instead of TMA: their 1800 instructions per
// tile took 10,700 cycles, five times the MMAs.)  Tiles outside every row's window are never loaded.
// Every wait is bounded; one that gives up sets the error word and the block's abort flag, and all roles leave.
#include "gemm_device.cuh"
#include "mma_bf16.cuh"
#include "window_device.cuh"

namespace nb {
namespace {

constexpr uint32_t kRows = 128;      // (position, head) rows: the MMA M and the lanes of tensor memory
constexpr uint32_t kKeys = 128;      // keys of a tile
constexpr uint32_t kStages = 2;      // of K and of V, each freed on its own
constexpr uint32_t kTilePages = kKeys / kPageTokens;
constexpr uint32_t kCopyWarp = 8, kMmaWarp = 9;  // in front of them two softmax groups of 128, a thread per row in each
constexpr uint32_t kAttentionThreads = 320;
constexpr uint32_t kBlockBytes = kRows * 128u;  // 128 rows of 64 bf16: one swizzled column block of a tile
constexpr uint32_t kTmemS = 0, kTmemO = 2u * kKeys, kTmemAll = 512;
constexpr float kRescaleAbove = 8.0f;

struct AttentionShared {
  uint64_t k_full[kStages], k_empty[kStages], v_full[kStages], v_empty[kStages];
  uint64_t s_full[2], p_full[2];
  uint64_t pv_done[2];  // PV of a group's tile
  uint64_t o_done;      // the last PV
  uint64_t drained;
  float m[2][kRows], l[2][kRows];  // the groups' softmax states
  uint32_t tmem_base;
  uint32_t abort;
  uint32_t taken_out;  // values that are not finite were taken out of a tile
};

// What the rows of a block see: 0 <= pos - key, and pos - key < window or key < keep_first.
struct Sight {
  uint32_t pos_first, pos_last, window, keep_first;
  __device__ __forceinline__ bool sees(uint32_t pos, uint32_t key) const {
    return key <= pos && (pos - key < window || key < keep_first);
  }
  __device__ __forceinline__ bool edge(uint32_t first) const {  // some row does not see some key of the tile
    return first + kKeys > pos_first + 1u || first < keep_first || pos_last - first >= window;
  }
};

// 16-byte piece `piece` of row `row` of a tile whose 64-element column blocks follow each other.
__device__ __forceinline__ uint32_t swizzled(uint32_t row, uint32_t piece) {
  return (piece >> 3) * kBlockBytes + row * 128u + (((piece & 7u) ^ (row & 7u)) << 4);
}
// Descriptor of V for one MMA: 16 keys x D values stored [key][64 values] per column block; the 8-key groups are 1024
// bytes apart, the column blocks kBlockBytes.
__device__ __forceinline__ uint64_t mn_major_sw128_desc(const void *tile) {
  const uint64_t addr = smem_addr(tile);
  return ((addr & 0x3ffffull) >> 4) | (static_cast<uint64_t>(kBlockBytes >> 4) << 16) |
         (static_cast<uint64_t>(1024u >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ uint32_t attention_instr_desc(uint32_t n, bool b_mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((b_mn_major ? 1u : 0u) << 16) | ((n >> 3) << 17) | ((kRows >> 4) << 24);
}
// A from tensor memory (two bf16 per 32-bit column, a row per lane), B from shared memory.
__device__ __forceinline__ void mma_tmem_a(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_load32(uint32_t taddr, float *v) {  // tmem_load_wait before the values are used
  uint32_t *r = reinterpret_cast<uint32_t *>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_load_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_store16(uint32_t taddr, const uint32_t *r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};" ::
          "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float exp2_ftz(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// A block's rows: (position, head) pairs f0 .. f_end - 1 of its KV head, and the tiles of keys that they walk.
template <bool EXTRAS>
struct Extent {
  uint32_t group, f0, f_end, base, kv_end, page_count;
  const uint32_t *page_table;
  uint32_t *error_word;
  Sight sight;
  TileWalk walk;
  bool inside;
  uint32_t tiles;
  __device__ __forceinline__ explicit Extent(const WindowAttentionParams &p) : walk(0u, 0u, kKeys) {
    const FusedAttentionRow &r0 = p.rows[0];
    group = p.s.heads / p.s.kv_heads;
    const uint32_t total_rows = p.row_count * group;
    f0 = (gridDim.y - 1u - blockIdx.y) * kRows;  // the longest walks first
    f_end = f0 + kRows < total_rows ? f0 + kRows : total_rows;
    base = r0.position;
    page_count = r0.page_count;
    page_table = r0.page_table;
    error_word = r0.error_word;
    sight.pos_first = base + f0 / group;
    sight.pos_last = base + (f_end - 1u) / group;
    sight.window = p.s.window != 0 ? p.s.window : 0xffffffffu;
    sight.keep_first = EXTRAS ? p.s.keep_first : 0u;
    inside = sight.pos_last < r0.max_context;
    const uint32_t window_lo = sight.pos_first + 1u > sight.window ? sight.pos_first + 1u - sight.window : 0u;  // of the first row
    kv_end = sight.pos_last + 1u;
    walk = TileWalk(sight.keep_first, window_lo, kKeys);
    tiles = inside ? walk.count(kv_end, kKeys) : 0u;
  }
};

// A probability of zero times a value that is not finite is not zero, and a tile at an edge holds values that some rows do
// not see.  Such values are set to zero in the tile, and the rows that do see them get them at the end (put_back).  The last
// page's rows behind the last query hold whatever the pool had: all zero.  By the MMA warp, which waits for the softmax of
// the tile anyway: as a part of the softmax, 16 rows' pieces a thread, the same looks cost 3 % of a 512-token prompt.
template <uint32_t D>
__device__ __forceinline__ void clean_values(uint8_t *tile, uint32_t used, uint32_t *taken_out) {
  constexpr uint32_t kPieces = D / 8u;
  const uint32_t lane = threadIdx.x & 31u;
  // all ones in the exponent carry into the sign's place, in both halves of a word
  auto marks = [](uint32_t v) { return (v & 0x7f807f80u) + 0x00800080u; };
  uint32_t any = 0;
#pragma unroll 8
  for (uint32_t i = lane; i < used * kPieces; i += 32u) {
    const uint4 w = lds128(tile + swizzled(i / kPieces, i % kPieces));
    any |= (marks(w.x) | marks(w.y)) | (marks(w.z) | marks(w.w));
  }
  const bool found = __any_sync(0xffffffffu, (any & 0x80008000u) != 0u);
  if (found) {
#pragma unroll 1
    for (uint32_t i = lane; i < used * kPieces; i += 32u) {
      uint4 *at = reinterpret_cast<uint4 *>(tile + swizzled(i / kPieces, i % kPieces));
      auto clean = [&](uint32_t v) { return v & ~(((marks(v) & 0x80008000u) >> 15) * 0xffffu); };
      const uint4 w = *at;
      *at = make_uint4(clean(w.x), clean(w.y), clean(w.z), clean(w.w));
    }
    if (lane == 0) *taken_out = 1;
  }
  const uint32_t page_end = (used + kPageTokens - 1u) / kPageTokens * kPageTokens;
  for (uint32_t i = used * kPieces + lane; i < page_end * kPieces; i += 32u)
    *reinterpret_cast<uint4 *>(tile + swizzled(i / kPieces, i % kPieces)) = make_uint4(0u, 0u, 0u, 0u);
  if (found || used < page_end) {
    fence_proxy_async();
    __syncwarp();
  }
}
// What clean_values took out of `columns` values of a row's KV head (`values`: those of the first cached row) and the row
// at `pos` sees: added to its output.
__device__ __noinline__ void put_back(uint16_t *out, const uint16_t *values, uint32_t columns, uint64_t row_stride,
                                      const uint32_t *page_table, uint32_t page_count, TileWalk walk, uint32_t tiles,
                                      Sight sight, uint32_t pos) {
  for (uint32_t c = 0; c < columns; ++c) {
    float sum = 0.0f;
    for (uint32_t j = 0; j < tiles; ++j) {
      const uint32_t first = walk.tile(j) * kKeys;
      if (!sight.edge(first)) continue;
      for (uint32_t key = first; key < first + kKeys && key <= pos; ++key) {
        const uint32_t page = page_table[key / kPageTokens];
        if (!sight.sees(pos, key) || page >= page_count) continue;
        const float v = bf16_bits_to_f32(values[(static_cast<uint64_t>(page) * kPageTokens + key % kPageTokens) * row_stride + c]);
        if (!isfinite(v)) sum += v;
      }
    }
    if (sum != 0.0f) out[c] = static_cast<uint16_t>(pack_bf16_hi(bf16_bits_to_f32(out[c]) + sum, 0.0f));
  }
}

template <uint32_t D, bool EXTRAS>
__global__ void __launch_bounds__(kAttentionThreads, 1) prefill_attention_kernel(const __grid_constant__ CUtensorMap map_k,
                                                                               const __grid_constant__ CUtensorMap map_v,
                                                                               WindowAttentionParams p) {
  constexpr uint32_t kColumnBlocks = D / 64u, kTileBytes = kColumnBlocks * kBlockBytes;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~uintptr_t{1023});
  uint8_t *q_hi = smem, *q_lo = smem + kTileBytes;
  uint8_t *k_ring = q_lo + kTileBytes, *v_ring = k_ring + kStages * kTileBytes;
  AttentionShared &sh = *reinterpret_cast<AttentionShared *>(v_ring + kStages * kTileBytes);
  volatile uint32_t *abort = &sh.abort;
  const WindowAttentionShape &s = p.s;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint64_t policy = l2_evict_last_policy();

  pdl_trigger();
  if (threadIdx.x == 0) {
    for (uint32_t i = 0; i < kStages; ++i) {
      mbar_init(&sh.k_full[i], 1);
      mbar_init(&sh.v_full[i], 1);
      mbar_init(&sh.k_empty[i], 1);
      mbar_init(&sh.v_empty[i], 1);
    }
    for (uint32_t i = 0; i < 2; ++i) {
      mbar_init(&sh.s_full[i], 1);
      mbar_init(&sh.p_full[i], kRows);
      mbar_init(&sh.pv_done[i], 1);
    }
    mbar_init(&sh.o_done, 1);
    mbar_init(&sh.drained, 1);
    sh.abort = 0;
    sh.taken_out = 0;
    mbar_init_fence();
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&sh.tmem_base)),
                 "r"(kTmemAll)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();  // barriers and tensor memory stand
  tcgen05_fence_after();
  const uint32_t tmem = sh.tmem_base;
  pdl_wait();
  const uint32_t kvh = blockIdx.x;
  const Extent<EXTRAS> e(p);
  const uint32_t group = e.group, f0 = e.f0, f_end = e.f_end, base = e.base, kv_end = e.kv_end;
  const uint32_t page_count = e.page_count;
  const uint32_t *page_table = e.page_table;
  uint32_t *error_word = e.error_word;
  const Sight sight = e.sight;
  const uint32_t pos_first = sight.pos_first, pos_last = sight.pos_last, window = sight.window, keep_first = sight.keep_first;
  const TileWalk walk = e.walk;
  const bool inside = e.inside;
  const uint32_t tiles = e.tiles;

  // Queries, scaled so that the softmax runs on exp2, as a bf16 rounding and its remainder.  By all warps but the one that
  // brings K and V, which begins at once, and three pieces of a thread in flight: one piece after the other, with K and V
  // held back until the queries stood, the start was much of a block with a short walk.  Prompts of 200 / 512 / 1500 tokens:
  // 2.57 -> 2.49 / 3.18 -> 3.10 / 5.45 -> 5.30 ms over 28 layers of 2048, 1.62 -> 1.59 / 2.05 -> 2.03 / 4.38 -> 4.33 ms over
  // 8 of 4096.  Four pieces are as fast but spill at a dimension of 64.
  if (warp != kCopyWarp) {
    constexpr uint32_t kWriters = kAttentionThreads - 32u, kPieces = kRows * (D / 8u), kBatch = 3;
    if (inside) {
      const float qscale = s.scale * kLog2e;
      const bool whole_pieces = s.qk_dim == D && p.qkv_stride % 4u == 0 && reinterpret_cast<uintptr_t>(p.qkv) % 16u == 0;
      for (uint32_t i0 = warp < kCopyWarp ? threadIdx.x : threadIdx.x - 32u; i0 < kPieces; i0 += kBatch * kWriters) {
        float x[kBatch][8];
#pragma unroll
        for (uint32_t u = 0; u < kBatch; ++u) {
          const uint32_t i = i0 + u * kWriters, row = i / (D / 8u), piece = i % (D / 8u), f = f0 + row;
#pragma unroll
          for (uint32_t j = 0; j < 8u; ++j) x[u][j] = 0.0f;
          if (i < kPieces && f < f_end) {
            const float *src = p.qkv + static_cast<uint64_t>(f / group) * p.qkv_stride + (kvh * group + f % group) * s.qk_dim;
            if (whole_pieces) {
              const float4 a = __ldcg(reinterpret_cast<const float4 *>(src + piece * 8u));
              const float4 b = __ldcg(reinterpret_cast<const float4 *>(src + piece * 8u + 4u));
              x[u][0] = a.x, x[u][1] = a.y, x[u][2] = a.z, x[u][3] = a.w, x[u][4] = b.x, x[u][5] = b.y, x[u][6] = b.z, x[u][7] = b.w;
            } else {
#pragma unroll
              for (uint32_t j = 0; j < 8u; ++j) x[u][j] = piece * 8u + j < s.qk_dim ? __ldcg(src + piece * 8u + j) : 0.0f;
            }
          }
        }
#pragma unroll
        for (uint32_t u = 0; u < kBatch; ++u) {
          const uint32_t i = i0 + u * kWriters;
          if (i >= kPieces) break;
#pragma unroll
          for (uint32_t j = 0; j < 8u; ++j) x[u][j] *= qscale;
          const uint32_t at = swizzled(i / (D / 8u), i % (D / 8u));
          *reinterpret_cast<uint4 *>(q_hi + at) = make_uint4(pack_bf16_hi(x[u][0], x[u][1]), pack_bf16_hi(x[u][2], x[u][3]),
                                                             pack_bf16_hi(x[u][4], x[u][5]), pack_bf16_hi(x[u][6], x[u][7]));
          *reinterpret_cast<uint4 *>(q_lo + at) = make_uint4(pack_bf16_lo(x[u][0], x[u][1]), pack_bf16_lo(x[u][2], x[u][3]),
                                                             pack_bf16_lo(x[u][4], x[u][5]), pack_bf16_lo(x[u][6], x[u][7]));
        }
      }
      fence_proxy_async();
    }
    asm volatile("barrier.sync 1, %0;" ::"n"(kWriters) : "memory");  // the writers and the MMA warp: the queries stand
  }

  if (warp == kMmaWarp) {
    // ---------------- MMA issuer: the warp waits together, an elected lane issues ----------------
    if (tiles != 0) {
      const uint32_t idesc_s = attention_instr_desc(kKeys, false), idesc_o = attention_instr_desc(D, true);
      auto scores = [&](uint32_t j) {  // S(j) = Q K(j)^T; its buffer held P(j - 2), which PV(j - 2) has read
        const uint32_t st = j % kStages;
        if (!warp_wait(&sh.k_full[st], (j / kStages) & 1u, abort, error_word)) return false;
        if (j >= 2u && !warp_wait(&sh.pv_done[j & 1u], ((j >> 1) & 1u) ^ 1u, abort, error_word)) return false;
        tcgen05_fence_after();
        if (!elected()) return true;
        const uint8_t *k = k_ring + st * kTileBytes;
#pragma unroll
        for (uint32_t part = 0; part < 2u; ++part) {
          const uint8_t *q = part == 0 ? q_hi : q_lo;
#pragma unroll
          for (uint32_t ks = 0; ks < D / kUmmaK; ++ks) {
            const uint64_t at = (ks & 3u) * 2ull;
            tcgen05_mma_f16(tmem + kTmemS + (j & 1u) * kKeys, kmajor_sw128_desc(q + (ks >> 2) * kBlockBytes) + at,
                            kmajor_sw128_desc(k + (ks >> 2) * kBlockBytes) + at, idesc_s, (part != 0 || ks != 0) ? 1u : 0u);
          }
        }
        tcgen05_commit(&sh.k_empty[st]);
        tcgen05_commit(&sh.s_full[j & 1u]);
        return true;
      };
      bool ok = scores(0) && (tiles < 2u || scores(1));
      for (uint32_t j = 0; ok && j < tiles; ++j) {
        const uint32_t st = j % kStages;
        if (!warp_wait(&sh.v_full[st], (j / kStages) & 1u, abort, error_word)) break;
        const uint32_t first = walk.tile(j) * kKeys;
        if (sight.edge(first))
          clean_values<D>(v_ring + st * kTileBytes, kv_end - first < kKeys ? kv_end - first : kKeys, &sh.taken_out);
        if (!warp_wait(&sh.p_full[j & 1u], (j >> 1) & 1u, abort, error_word)) break;
        tcgen05_fence_after();
        if (elected()) {
          const uint64_t v = mn_major_sw128_desc(v_ring + st * kTileBytes);
#pragma unroll
          for (uint32_t part = 0; part < 2u; ++part) {
#pragma unroll
            for (uint32_t ks = 0; ks < kKeys / kUmmaK; ++ks)
              mma_tmem_a(tmem + kTmemO + (j & 1u) * D, tmem + kTmemS + (j & 1u) * kKeys + part * (kKeys / 2u) + ks * (kUmmaK / 2u),
                         v + ks * ((kUmmaK * 128u) >> 4), idesc_o, (j >= 2u || part != 0 || ks != 0) ? 1u : 0u);
          }
          tcgen05_commit(&sh.v_empty[st]);
          tcgen05_commit(&sh.pv_done[j & 1u]);
          if (j + 1u == tiles) tcgen05_commit(&sh.o_done);
        }
        __syncwarp();
        if (j + 2u < tiles) ok = scores(j + 2u);
      }
    }
  } else if (warp == kCopyWarp) {
    // ---------------- K and V: lane i < 8 brings page i of the tile ----------------
    bool ok = true;
    for (uint32_t j = 0; ok && j < tiles; ++j) {
      const uint32_t first = walk.tile(j) * kKeys, st = j % kStages;
      uint32_t y = 0xffffffffu;  // a page behind the last query: rows outside the map, which read as zeros
      if (lane < kTilePages && first + lane * kPageTokens < kv_end) {
        const uint32_t page = page_table[first / kPageTokens + lane];
        if (page < page_count)
          y = page * kPageTokens;
        else
          report_error(error_word, kErrPageOutOfRange);
      }
      if (y == 0xffffffffu) y = page_count * kPageTokens;
#pragma unroll
      for (uint32_t what = 0; what < 2u; ++what) {
        uint64_t *full = what == 0 ? &sh.k_full[st] : &sh.v_full[st];
        if (ok && !warp_wait(what == 0 ? &sh.k_empty[st] : &sh.v_empty[st], ((j / kStages) & 1u) ^ 1u, abort, error_word)) ok = false;
        if (!ok) break;
        if (lane == 0) mbar_arrive_expect_tx(full, kTileBytes);
        __syncwarp();
        uint8_t *stage = (what == 0 ? k_ring : v_ring) + st * kTileBytes + lane * kPageTokens * 128u;
        if (lane < kTilePages) {
#pragma unroll
          for (uint32_t c = 0; c < kColumnBlocks; ++c)
            tma_load_2d(stage + c * kBlockBytes, what == 0 ? &map_k : &map_v, kvh * D + c * 64u, y, full, policy);
        }
      }
    }
  } else if (tiles != 0) {
    // ---------------- softmax ----------------
    const uint32_t half = warp >> 2, row = threadIdx.x & (kRows - 1u), f = f0 + row;
    const uint32_t pos = base + (f < f_end ? f : f_end - 1u) / group;
    const uint32_t lanes = ((warp & 3u) * 32u) << 16;
    const uint32_t s_addr = tmem + lanes + kTmemS + half * kKeys, o_addr = tmem + lanes + kTmemO + half * D;
    const float cap2 = s.softcap * kLog2e, inv_cap2 = cap2 > 0.0f ? 1.0f / cap2 : 0.0f;
    float m_ref = -INFINITY, l = 0.0f;
    bool ok = true;
    for (uint32_t j = half; j < tiles; j += 2u) {
      const uint32_t first = walk.tile(j) * kKeys;
      if (!warp_wait(&sh.s_full[half], (j >> 1) & 1u, abort, error_word)) {
        ok = false;
        break;
      }
      tcgen05_fence_after();
      float v[kKeys];
#pragma unroll
      for (uint32_t c = 0; c < kKeys; c += 32u) tmem_load32(s_addr + c, v + c);
      tmem_load_wait();
#pragma unroll
      for (uint32_t c = 0; c < kKeys; ++c) asm volatile("" : "+f"(v[c]));  // nothing that uses a score moves above the wait
      if (EXTRAS && cap2 > 0.0f) {
#pragma unroll
        for (uint32_t c = 0; c < kKeys; ++c) v[c] = cap_score_fast(v[c], cap2, inv_cap2);
      }
      // visible: 0 <= pos - key, and pos - key < window or key < keep_first; only tiles at an edge test it
      if (first + kKeys > pos_first + 1u || (EXTRAS && first < keep_first) || pos_last - first >= window) {
#pragma unroll
        for (uint32_t c = 0; c < kKeys; ++c) {
          const uint32_t key = first + c;
          if (!(key <= pos && (pos - key < window || (EXTRAS && key < keep_first)))) v[c] = -INFINITY;
        }
      }
      float top[4] = {v[0], v[1], v[2], v[3]};
#pragma unroll
      for (uint32_t c = 4; c < kKeys; ++c) top[c & 3u] = fmaxf(top[c & 3u], v[c]);
      const float m_tile = fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3]));
      // the accumulator keeps its reference until the maximum has left it far behind
      const bool grow = m_tile > m_ref + kRescaleAbove;  // also the first visible key: m_ref is -inf
      if (__any_sync(0xffffffffu, grow)) {
        const float m_new = grow ? m_tile : m_ref;
        const float corr = m_new == m_ref ? 1.0f : exp2_ftz(m_ref - m_new);  // 0 where nothing was seen before
        m_ref = m_new;
        l *= corr;
        if (j >= 2u) {  // the group's last PV is done: S(j) followed it
#pragma unroll 1
          for (uint32_t c = 0; c < D; c += 16u) {
            float o[16];
            tmem_load16(o_addr + c, o);
#pragma unroll
            for (uint32_t i = 0; i < 16u; ++i) o[i] *= corr;
            tmem_store16(o_addr + c, reinterpret_cast<const uint32_t *>(o));
          }
        }
      }
      const float ref = m_ref == -INFINITY ? 0.0f : m_ref;  // no key of the row seen yet: all probabilities are 0
      float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (uint32_t c = 0; c < kKeys; c += 32u) {
        uint32_t hi[16], lo[16];
#pragma unroll
        for (uint32_t i = 0; i < 16u; ++i) {
          const float a = exp2_ftz(v[c + 2u * i] - ref), b = exp2_ftz(v[c + 2u * i + 1u] - ref);
          sum[i & 1u] += a;
          sum[2u + (i & 1u)] += b;
          hi[i] = pack_bf16_hi(a, b);
          lo[i] = pack_bf16_hi(a - bf16x2_lo(hi[i]), b - bf16x2_hi(hi[i]));
        }
        tmem_store16(s_addr + c / 2u, hi);
        tmem_store16(s_addr + kKeys / 2u + c / 2u, lo);
      }
      l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
      tmem_store_wait();
      tcgen05_fence_before();
      mbar_arrive(&sh.p_full[half]);
    }
    sh.m[half][row] = m_ref;
    sh.l[half][row] = l;
    if (ok) ok = warp_wait(&sh.o_done, 0, abort, error_word);
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  if (warp < kCopyWarp && tiles != 0 && sh.abort == 0u) {
    // ---------------- output: half of a row's columns per thread, the two groups' parts added ----------------
    const uint32_t half = warp >> 2, row = threadIdx.x & (kRows - 1u), f = f0 + row;
    const uint32_t o_addr = tmem + (((warp & 3u) * 32u) << 16) + kTmemO;
    const bool live = f < f_end;
    const uint32_t h = kvh * group + f % group;
    const float m = fmaxf(sh.m[0][row], sh.m[1][row]);  // one of the groups has seen the row's own key: finite
    const float w0 = exp2_ftz(sh.m[0][row] - m), w1 = exp2_ftz(sh.m[1][row] - m);  // 0: nothing seen, maybe never written
    const float inv = live ? output_gate<EXTRAS>(p, f / group, h) / (sh.l[0][row] * w0 + sh.l[1][row] * w1) : 0.0f;
    uint16_t *dst = reinterpret_cast<uint16_t *>(p.out) + static_cast<uint64_t>(f / group) * p.out_stride + h * s.v_dim;
    const bool vector = s.v_dim == D && p.out_stride % 8u == 0 && reinterpret_cast<uintptr_t>(p.out) % 16u == 0;
#pragma unroll 1
    for (uint32_t c = half * (D / 2u); c < (half + 1u) * (D / 2u); c += 16u) {
      float o[16], o1[16];
      tmem_load16(o_addr + c, o);
      tmem_load16(o_addr + D + c, o1);
#pragma unroll
      for (uint32_t i = 0; i < 16u; ++i) o[i] = ((w0 > 0.0f ? o[i] * w0 : 0.0f) + (w1 > 0.0f ? o1[i] * w1 : 0.0f)) * inv;
      if (!live) {
        // nothing to store; the warp's next load wants all lanes
      } else if (vector) {
#pragma unroll
        for (uint32_t i = 0; i < 16u; i += 8u)
          *reinterpret_cast<uint4 *>(dst + c + i) = make_uint4(pack_bf16_hi(o[i], o[i + 1]), pack_bf16_hi(o[i + 2], o[i + 3]),
                                                               pack_bf16_hi(o[i + 4], o[i + 5]), pack_bf16_hi(o[i + 6], o[i + 7]));
      } else {
#pragma unroll
        for (uint32_t i = 0; i < 16u; ++i)
          if (c + i < s.v_dim) dst[c + i] = f32_to_bf16_bits(o[i]);
      }
      __syncwarp();
    }
    if (sh.taken_out != 0u && live && half * (D / 2u) < s.v_dim) {
      const Extent<EXTRAS> again(p);  // nothing of it stays in registers through the loops above
      const uint32_t c = half * (D / 2u), columns = s.v_dim - c < D / 2u ? s.v_dim - c : D / 2u;
      put_back(dst + c, static_cast<const uint16_t *>(p.values) + p.value_offset + kvh * D + c, columns,
               static_cast<uint64_t>(s.kv_heads) * D, again.page_table, again.page_count, again.walk, again.tiles, again.sight,
               again.base + f / group);
    }
  }
  // ---- teardown: nothing stays in flight ----
  tcgen05_fence_before();
  __syncthreads();
  if (sh.abort != 0u) {
    if (threadIdx.x == 0) drain_copies(sh.k_full, kStages);
    if (threadIdx.x == 32) drain_copies(sh.v_full, kStages);
    if (warp == kMmaWarp && elected()) drain_mmas(&sh.drained);
  }
  __syncthreads();
  if (warp == kMmaWarp) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemAll) : "memory");
  }
}

template <uint32_t D>
constexpr uint32_t attention_smem() {
  return tensor_memory_smem(kTmemAll, 1024u + (2u + 2u * kStages) * (D / 64u) * kBlockBytes +
                                          static_cast<uint32_t>(sizeof(AttentionShared)) + 64u);
}

}  // namespace

bool prefill_attention_supported(const WindowAttentionShape &s) {
  return s.heads % s.kv_heads == 0 && s.qk_pad == s.v_pad && (s.qk_pad == 64u || s.qk_pad == 128u);
}

cudaError_t configure_prefill_attention() {
  cudaError_t err = cudaSuccess;
  auto set = [&err](void (*kernel)(CUtensorMap, CUtensorMap, WindowAttentionParams), uint32_t bytes) {
    if (err == cudaSuccess) err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
  };
  set(prefill_attention_kernel<64, false>, attention_smem<64>());
  set(prefill_attention_kernel<64, true>, attention_smem<64>());
  set(prefill_attention_kernel<128, false>, attention_smem<128>());
  set(prefill_attention_kernel<128, true>, attention_smem<128>());
  return err;
}

void prefill_attention_launches(std::vector<TensorMemoryLaunch> *out) {
  out->push_back({attention_smem<64>(), kTmemAll});
  out->push_back({attention_smem<128>(), kTmemAll});
}

cudaError_t launch_prefill_attention(cudaStream_t stream, const WindowAttentionParams &p) {
  if (p.rows == nullptr || p.row_count == 0 || p.f32 != 0 || p.keys == nullptr || p.values == nullptr ||
      !prefill_attention_supported(p.s))
    return cudaErrorInvalidValue;
  const uint32_t rows = p.row_count * (p.s.heads / p.s.kv_heads), D = p.s.qk_pad;
  const uint64_t width = static_cast<uint64_t>(p.s.kv_heads) * D, tokens = static_cast<uint64_t>(p.page_count) * kPageTokens;
  CUtensorMap map_k, map_v;
  if (!encode_bf16_map_2d(&map_k, static_cast<const uint16_t *>(p.keys) + p.key_offset, width, tokens, 64, kPageTokens) ||
      !encode_bf16_map_2d(&map_v, static_cast<const uint16_t *>(p.values) + p.value_offset, width, tokens, 64, kPageTokens))
    return cudaErrorNotSupported;
  const dim3 grid(p.s.kv_heads, (rows + kRows - 1u) / kRows);
  const bool extras = has_extras(p.s);
  if (D == 64u)
    return launch_with_pdl(extras ? prefill_attention_kernel<64, true> : prefill_attention_kernel<64, false>, grid,
                           dim3(kAttentionThreads), attention_smem<64>(), stream, p.pdl != 0, map_k, map_v, p);
  return launch_with_pdl(extras ? prefill_attention_kernel<128, true> : prefill_attention_kernel<128, false>, grid,
                         dim3(kAttentionThreads), attention_smem<128>(), stream, p.pdl != 0, map_k, map_v, p);
}

}  // namespace nb
