// Weight-streaming matrix-vector core.
//
// A projection y[n] = sum_k W[n][k] * x[k] at one token is pure HBM streaming:
// every weight byte is read once and used once.  The rows of a projection are
// dealt to thread blocks as equal contiguous row ranges, and inside a block two rows
// are taken together: the sweeps (512 bytes of each row) of the block's row pairs are
// dealt to the warps in equal runs, cut anywhere in a row, so every warp of the
// grid streams the same amount of memory whatever the shape.  Each warp owns a
// private ring of shared-memory slots that it keeps filled with pieces ("chunks",
// at most kChunkBytes, never crossing the rows' ends) of its run through 1-D bulk
// TMA copies, one per row.  There is
// no block-level synchronisation in the loop: a warp waits only on the mbarrier
// of the slot it is about to read and refills that slot as soon as it has read it.
//
// The arithmetic is on the tensor pipe (mma.sync, see sweep_mma), not for its rate: a launch
// begins with a full ring, and what the stream loses is the time until the ring has been
// worked off.  With unpacking and FMAs a sweep of one row took 26 instructions and a block went through its ring
// at 25 bytes per cycle, hardly more than its share of HBM (22); with two MMAs and three loads for a sweep of two
// rows it is bound by shared memory, 85 bytes per cycle.  Steps before and after, us: vamidra 1.7b widths (28 layer
// runs) 1376 and 1249, vuvolix 1016 and 991, 8 layers of the 8B shapes 784 and 762, the 4-layer hidden-512 model 118 and 99.
//
// The chunk list runs ACROSS projections (a job list): weights do not depend on
// activations, so the issue side of a ring runs ahead into the next projection
// while the block is still normalising, attending or waiting at a grid barrier.
//
// A pair that lies inside one warp's range is reduced by that warp and its totals
// go to the block's row-total buffer in shared memory.  A pair cut by a range
// boundary leaves one partial per row and warp in that warp's two "edge" records.  After
// the block has synchronised, stream_row_total() adds the edge partials to the
// totals in ascending warp order, so results do not depend on timing and are
// bit-identical run to run.
#pragma once

#include "mma_bf16.cuh"

namespace nb {

constexpr uint32_t kStreamWarps = 8;
constexpr uint32_t kStreamThreads = kStreamWarps * 32;
constexpr uint32_t kStreamSlots = 3;
constexpr uint32_t kChunkBytes = 8192;               // of both rows of a pair
constexpr uint32_t kChunkRowBytes = kChunkBytes / 2u;
constexpr uint32_t kRingBytes = kStreamWarps * kStreamSlots * kChunkBytes;
constexpr uint32_t kSweepBytes = 512;  // 32 lanes x 16 bytes
static_assert(kChunkRowBytes % (4 * kSweepBytes) == 0, "a chunk is a whole number of 4-sweep steps");
constexpr uint32_t kNoRow = 0xffffffffu;

struct JobDesc {
  const uint16_t *weight;  // [rows][cols] bf16 row-major, 16-byte aligned, cols % 8 == 0
  uint32_t rows, cols;
  uint32_t unit;           // rows are dealt to blocks in multiples of `unit` (2 keeps gate/up pairs together)
  uint32_t whole;          // non-zero: the job belongs to this block alone (its list was built per block):
                           // all `rows` are this block's, nothing is dealt
};

// Rows [begin, end) of block `block` out of `blocks`, in units of `unit` rows.
__host__ __device__ inline void block_row_range(uint32_t rows, uint32_t unit, uint32_t block,
                                                uint32_t blocks, uint32_t *begin, uint32_t *end) {
  // units * block / blocks without 64-bit divisions, which a launch would wait for before its first copy
  const uint32_t units = rows / unit, each = units / blocks, rest = units % blocks;
  *begin = (each * block + rest * block / blocks) * unit;
  *end = (each * (block + 1u) + rest * (block + 1u) / blocks) * unit;
}
__host__ __device__ inline uint32_t max_rows_per_block(uint32_t rows, uint32_t unit, uint32_t blocks) {
  const uint32_t units = rows / unit;
  return ((units + blocks - 1) / blocks) * unit;
}

// One warp's share of one job.  Positions count the bytes of ONE row of each pair (pair p, column byte c: p * row_bytes
// + c); the range [begin, end) is the warp's.
struct WarpJob {
  const uint8_t *base;  // first byte of the block's first row
  uint32_t row_bytes;
  uint32_t rows;        // the block's; the last pair of an odd number has one
  uint32_t begin, end;
};

__device__ __forceinline__ WarpJob warp_job(const JobDesc &d) {
  uint32_t row_begin = 0, row_end = d.rows;
  if (d.whole == 0) block_row_range(d.rows, d.unit, blockIdx.x, gridDim.x, &row_begin, &row_end);
  WarpJob j;
  j.row_bytes = d.cols * 2u;
  j.base = reinterpret_cast<const uint8_t *>(d.weight) + static_cast<uint64_t>(row_begin) * j.row_bytes;
  j.rows = row_end - row_begin;
  const uint32_t warp = threadIdx.x >> 5, pairs = (j.rows + 1u) / 2u;
  if (j.row_bytes % kSweepBytes == 0) {
    // cut the block's pairs into equal runs of whole 512-byte lane sweeps
    const uint32_t sweeps = pairs * (j.row_bytes / kSweepBytes);
    j.begin = static_cast<uint32_t>(static_cast<uint64_t>(sweeps) * warp / kStreamWarps) * kSweepBytes;
    j.end = static_cast<uint32_t>(static_cast<uint64_t>(sweeps) * (warp + 1) / kStreamWarps) * kSweepBytes;
  } else {
    // rows that are not a whole number of sweeps are dealt in whole pairs
    j.begin = static_cast<uint32_t>(static_cast<uint64_t>(pairs) * warp / kStreamWarps) * j.row_bytes;
    j.end = static_cast<uint32_t>(static_cast<uint64_t>(pairs) * (warp + 1) / kStreamWarps) * j.row_bytes;
  }
  return j;
}

// A cursor walks a WarpJob chunk by chunk.
struct StreamCursor {
  uint32_t pos;      // position of the next chunk
  uint32_t row_end;  // end position of the pair that contains pos
  uint32_t pair;     // block-local index of that pair
};
__device__ __forceinline__ StreamCursor cursor_at_start(const WarpJob &j) {
  StreamCursor c;
  c.pos = j.begin;
  c.pair = j.begin / j.row_bytes;
  c.row_end = (c.pair + 1u) * j.row_bytes;
  return c;
}
// Length of the chunk at the cursor in each row, its position, the end of its pair and the pair's index;
// advances the cursor.
__device__ __forceinline__ uint32_t cursor_next(const WarpJob &j, StreamCursor &c, uint32_t *pos,
                                                uint32_t *row_end, uint32_t *pair) {
  uint32_t len = kChunkRowBytes;
  if (c.row_end - c.pos < len) len = c.row_end - c.pos;
  if (j.end - c.pos < len) len = j.end - c.pos;
  *pos = c.pos;
  *row_end = c.row_end;
  *pair = c.pair;
  c.pos += len;
  if (c.pos == c.row_end) {
    c.row_end += j.row_bytes;
    c.pair += 1u;
  }
  return len;
}

struct EdgeRecord {
  uint32_t pair;  // block-local pair, kNoRow when unused
  float value[2];
};

// Shared-memory bookkeeping of a block's streams.
struct StreamShared {
  uint64_t bars[kStreamWarps * kStreamSlots];
  EdgeRecord edge[kStreamWarps][2];
};

// Per-warp state.  Every field is warp-uniform.
struct RowStream {
  uint8_t *ring;
  uint64_t *bars;
  const JobDesc *jobs;
  uint32_t job_count;
  uint32_t issued, consumed;  // chunks
  bool dead;
  uint32_t drain_from, drain_to;
  uint32_t issue_job;
  WarpJob issue;
  StreamCursor issue_cursor;
  uint64_t policy;  // L2 evict-first: weights are read once per step
};

// SLOTS (at most kStreamSlots): ring slots per warp; a kernel that shares its SM with another takes fewer.
template <uint32_t SLOTS = kStreamSlots>
__device__ inline void stream_init(RowStream &rs, uint8_t *ring_base, StreamShared &sh,
                                   const JobDesc *jobs, uint32_t job_count) {
  const uint32_t warp = threadIdx.x >> 5;
  rs.ring = ring_base + warp * SLOTS * kChunkBytes;
  rs.bars = sh.bars + warp * SLOTS;
  rs.jobs = jobs;
  rs.job_count = job_count;
  rs.issued = rs.consumed = 0;
  rs.dead = false;
  rs.drain_from = rs.drain_to = 0;
  rs.policy = l2_evict_first_policy();
  rs.issue_job = 0;
  if (job_count != 0) {
    rs.issue = warp_job(jobs[0]);
    rs.issue_cursor = cursor_at_start(rs.issue);
  }
  if (elected()) {
    for (uint32_t s = 0; s < SLOTS; ++s) mbar_init(&rs.bars[s], 1);
    mbar_init_fence();
  }
  __syncwarp();
}

// Issues chunks, crossing into later jobs, while ring slots are free (at most `depth` in flight).
template <uint32_t SLOTS = kStreamSlots>
__device__ __forceinline__ void stream_fill(RowStream &rs, uint32_t depth = SLOTS) {
  if (rs.dead) return;
  while (rs.issue_job < rs.job_count && rs.issued - rs.consumed < depth) {
    if (rs.issue_cursor.pos >= rs.issue.end) {
      rs.issue_job += 1;
      if (rs.issue_job < rs.job_count) {
        rs.issue = warp_job(rs.jobs[rs.issue_job]);
        rs.issue_cursor = cursor_at_start(rs.issue);
      }
      continue;
    }
    uint32_t pos, row_end, pair;
    const uint32_t len = cursor_next(rs.issue, rs.issue_cursor, &pos, &row_end, &pair);
    const uint32_t slot = rs.issued % SLOTS;
    if (elected()) {
      const bool both = 2u * pair + 1u < rs.issue.rows;
      const uint8_t *src = rs.issue.base + pos + static_cast<uint64_t>(pair) * rs.issue.row_bytes;
      mbar_arrive_expect_tx(&rs.bars[slot], both ? 2u * len : len);
      tma_load_1d_hint(rs.ring + slot * kChunkBytes, src, len, &rs.bars[slot], rs.policy);
      if (both)
        tma_load_1d_hint(rs.ring + slot * kChunkBytes + kChunkRowBytes, src + rs.issue.row_bytes, len, &rs.bars[slot], rs.policy);
    }
    rs.issued += 1;
  }
}

// Asks L2 for the `bytes` that follow the chunks already issued, half of them in each row of the pair (the warp's own
// range of the current job only): the ring cannot hold more, but HBM can keep working while the block is busy with its
// prologue.
__device__ __forceinline__ void stream_prefetch_l2(const RowStream &rs, uint32_t bytes) {
  const uint32_t lane = threadIdx.x & 31u;
  if (rs.dead || bytes == 0 || rs.issue_job >= rs.job_count || lane > 1u) return;
  const StreamCursor &c = rs.issue_cursor;
  if (c.pos >= rs.issue.end || 2u * c.pair + lane >= rs.issue.rows) return;
  uint32_t size = (rs.issue.end < c.row_end ? rs.issue.end : c.row_end) - c.pos;
  if (size > bytes / 2u) size = bytes / 2u;
  size &= ~15u;
  if (size == 0) return;
  const uint8_t *src = rs.issue.base + c.pos + static_cast<uint64_t>(c.pair + lane) * rs.issue.row_bytes;
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(size) : "memory");
}

// Packed fp32 multiply-add (two lanes per instruction).
__device__ __forceinline__ float2 fma2(float a0, float a1, float b0, float b1, float2 c) {
  uint64_t a, b, cc, d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "f"(a0), "f"(a1));
  asm("mov.b64 %0, {%1, %2};" : "=l"(b) : "f"(b0), "f"(b1));
  asm("mov.b64 %0, {%1, %2};" : "=l"(cc) : "f"(c.x), "f"(c.y));
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(cc));
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(d));
  return r;
}
// dot of 8 bf16 weights with 8 fp32 activations, even elements into acc.x and odd ones into acc.y.
__device__ __forceinline__ float2 dot8_f32x2(const uint4 &w, const float4 &xa, const float4 &xb, float2 acc) {
  acc = fma2(bf16x2_lo(w.x), bf16x2_hi(w.x), xa.x, xa.y, acc);
  acc = fma2(bf16x2_lo(w.y), bf16x2_hi(w.y), xa.z, xa.w, acc);
  acc = fma2(bf16x2_lo(w.z), bf16x2_hi(w.z), xb.x, xb.y, acc);
  acc = fma2(bf16x2_lo(w.w), bf16x2_hi(w.w), xb.z, xb.w, acc);
  return acc;
}

// dot of 8 bf16 weights with 8 fp32 activations (the sparse-MoE path of the
// reference feeds unrounded activations to its mat-vec).
__device__ __forceinline__ float dot8_f32(const uint4 &w, const float4 &xa, const float4 &xb, float acc) {
  acc = fmaf(bf16x2_lo(w.x), xa.x, acc);
  acc = fmaf(bf16x2_hi(w.x), xa.y, acc);
  acc = fmaf(bf16x2_lo(w.y), xa.z, acc);
  acc = fmaf(bf16x2_hi(w.y), xa.w, acc);
  acc = fmaf(bf16x2_lo(w.z), xb.x, acc);
  acc = fmaf(bf16x2_hi(w.z), xb.y, acc);
  acc = fmaf(bf16x2_lo(w.w), xb.z, acc);
  acc = fmaf(bf16x2_hi(w.w), xb.w, acc);
  return acc;
}

// One lane sweep of a pair: 512 bytes of each row times the same 512 bytes of x.  A lane's 16 bytes are eight
// columns of 64-byte slab lane / 4; the fragments of the MMA take the slabs of the first row as rows 0..7 of A, those
// of the second as rows 8..15, and those of x as the columns of B, so the products of like slabs are the diagonals of
// the two halves of the accumulator.  What stands beside the diagonals is never read.
__device__ __forceinline__ void sweep_mma(float (&acc)[4], const uint4 &w0, const uint4 &w1, const uint4 &x) {
  mma_bf16(acc, {w0.x, w1.x, w0.y, w1.y}, x.x, x.y);
  mma_bf16(acc, {w0.z, w1.z, w0.w, w1.w}, x.z, x.w);
}

// Consumes job `index` (jobs are consumed in order, each exactly once, by every
// warp of the block).  `x` is the bf16 activation vector in shared memory;
// row_total[r] (shared, one float per block-local row, zeroed by the caller
// before the block's previous synchronisation) receives the totals of every pair
// that lies wholly inside this warp's range; partial sums go to sh.edge.
template <uint32_t SLOTS = kStreamSlots>
__device__ __forceinline__ void stream_consume(RowStream &rs, StreamShared &sh, uint32_t index,
                                               const void *x, float *row_total,
                                               uint32_t *error_word) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const WarpJob job = warp_job(rs.jobs[index]);
  StreamCursor cur = cursor_at_start(job);
  if (lane == 0) {
    sh.edge[warp][0].pair = kNoRow;
    sh.edge[warp][1].pair = kNoRow;
  }
  const bool odd_slab = (lane & 4u) != 0, diagonal = (lane & 3u) == lane >> 3;  // column lane / 4 is in c[odd_slab] of lane % 4 == lane / 8
  float sum0 = 0.0f, sum1 = 0.0f;
  uint32_t edges = 0;
  bool row_from_start = job.begin % job.row_bytes == 0;  // this warp has seen the current pair from its first column
  while (cur.pos < job.end) {
    uint32_t pos, row_end, pair;
    const uint32_t len = cursor_next(job, cur, &pos, &row_end, &pair);
    stream_fill<SLOTS>(rs);
    const uint32_t slot = rs.consumed % SLOTS;
    const uint32_t parity = (rs.consumed / SLOTS) & 1u;
    if (!rs.dead && !mbar_wait_bounded(&rs.bars[slot], parity)) {
      rs.dead = true;
      rs.drain_from = rs.consumed;
      rs.drain_to = rs.issued;
      report_error(error_word, kErrTmaWaitTimeout);
    }
    const uint8_t *wp = rs.ring + slot * kChunkBytes + lane * 16u;
    const uint32_t row_offset = pos - (row_end - job.row_bytes);  // bytes into the row
    const uint8_t *xp = reinterpret_cast<const uint8_t *>(x) + row_offset + lane * 16u;
    // four accumulators, zeroed per chunk: chains of four MMAs, whose sums meet in fp32 adds
    float acc[4][4];
#pragma unroll
    for (uint32_t i = 0; i < 4u; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.0f;
    if (len == kChunkRowBytes) {
#pragma unroll
      for (uint32_t i = 0; i < kChunkRowBytes / kSweepBytes; ++i)
        sweep_mma(acc[i & 3u], lds128(wp + i * kSweepBytes), lds128(wp + kChunkRowBytes + i * kSweepBytes), lds128(xp + i * kSweepBytes));
    } else {
      uint32_t off = 0;
      for (; off + 2u * kSweepBytes <= len; off += 2u * kSweepBytes) {
#pragma unroll
        for (uint32_t i = 0; i < 2u; ++i)
          sweep_mma(acc[i], lds128(wp + off + i * kSweepBytes), lds128(wp + kChunkRowBytes + off + i * kSweepBytes),
                    lds128(xp + off + i * kSweepBytes));
      }
      // a last sweep: whole, or (rows that are not a multiple of 512 bytes) of the lanes that still have data
      for (; off < len; off += kSweepBytes) {
        uint4 w0 = make_uint4(0u, 0u, 0u, 0u), w1 = w0, xv = w0;
        if (off + lane * 16u < len) {
          w0 = lds128(wp + off);
          w1 = lds128(wp + kChunkRowBytes + off);
          xv = lds128(xp + off);
        }
        __syncwarp();
        sweep_mma(acc[2], w0, w1, xv);
      }
    }
    if (odd_slab) {
      sum0 += (acc[0][1] + acc[1][1]) + (acc[2][1] + acc[3][1]);
      sum1 += (acc[0][3] + acc[1][3]) + (acc[2][3] + acc[3][3]);
    } else {
      sum0 += (acc[0][0] + acc[1][0]) + (acc[2][0] + acc[3][0]);
      sum1 += (acc[0][2] + acc[1][2]) + (acc[2][2] + acc[3][2]);
    }
    const bool row_done = pos + len == row_end;
    const bool range_done = pos + len == job.end;
    if (row_done || range_done) {
      // the first row's total to the lower half of the warp, the second's to the upper
      const float mine = diagonal ? (lane < 16u ? sum0 : sum1) : 0.0f, theirs = diagonal ? (lane < 16u ? sum1 : sum0) : 0.0f;
      float total = mine + __shfl_xor_sync(0xffffffffu, theirs, 16);
#pragma unroll
      for (int offset = 8; offset > 0; offset >>= 1) total += __shfl_xor_sync(0xffffffffu, total, offset);
      if ((lane & 15u) == 0) {
        const uint32_t row = 2u * pair + (lane >> 4);
        if (!(row_done && row_from_start)) {
          sh.edge[warp][edges].pair = pair;
          sh.edge[warp][edges].value[lane >> 4] = total;
        } else if (row < job.rows) {
          row_total[row] = total;
        }
      }
      if (!(row_done && row_from_start)) edges += 1;
      sum0 = sum1 = 0.0f;
      row_from_start = true;
    }
    __syncwarp();
    rs.consumed += 1;
  }
  // keep the ring full while the block goes on to its next phase
  stream_fill<SLOTS>(rs);
}

// After the block has synchronised behind stream_consume: row r's total with
// the partials of cut pairs added in ascending warp order.
__device__ __forceinline__ float stream_row_total(const StreamShared &sh, const float *row_total,
                                                  uint32_t r) {
  float total = row_total[r];
#pragma unroll
  for (uint32_t w = 0; w < kStreamWarps; ++w) {
    if (sh.edge[w][0].pair == r >> 1) total += sh.edge[w][0].value[r & 1u];
    if (sh.edge[w][1].pair == r >> 1) total += sh.edge[w][1].value[r & 1u];
  }
  return total;
}

// After a timeout: give copies still in flight one more bounded chance to land
// before the block's shared memory is released.
template <uint32_t SLOTS = kStreamSlots>
__device__ inline void stream_drain(RowStream &rs) {
  if (!rs.dead) return;
  for (uint32_t c = rs.drain_from; c < rs.drain_to; ++c) {
    mbar_wait_bounded(&rs.bars[c % SLOTS], (c / SLOTS) & 1u);
  }
}

}  // namespace nb
