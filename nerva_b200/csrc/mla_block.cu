// DeepSeek multi-head latent attention, absorbed form, for consecutive positions of one session (prefill chunk).
//
//   mla_block_cache_kernel   per row: rotary part of its queries in place, its cache row appended (the arithmetic, and
//                            so the cached bits, of the decode step: mla_session.cu)
//   mla_block_head_kernel    absorbed queries q_nope . W_UK, a small matrix product per head, and at the end the value
//                            projection lat . W_UV; fp32 rows as two bf16 parts on mma.sync
//   mla_block_attention_kernel  four positions x 16 heads are the 64 rows of a block's MMA tiles, which share every
//                            tile of 32 cached rows (a latent cache row serves all heads as key and as value)
//
// Queries, probabilities and latent outputs are fp32 values that enter a product as a bf16 rounding and its remainder;
// cached rows and weights are bf16 as stored; accumulation is fp32.
//
// What bounds the attention: shared memory.  Both parts of 64 query rows of 576 values fill 146 KB, so a block is
// alone on its SM and its phases (a tile from L2, 16 x 72 MMAs of scores, the softmax, 16 x 64 MMAs of values) follow
// each other; four positions per block are what fits, and each divides the tile loads and barriers per position.
// Measured: moe_block.cu has the prefill as a whole; 2 and 3 tokens take as long as that many steps (1.10 ms, 1.59 ms
// for 6 layers), 4 tokens 1.70 ms (steps 2.09), 64 tokens 2.6 ms (32.1).
#include <math.h>

#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"
#include "mma_bf16.cuh"

namespace nb {
namespace {

constexpr float kLog2e = 1.4426950408889634f;

// Interleaved rotary pair, as in mla_session.cu.
__device__ __forceinline__ void rope_pair(float &left, float &right, uint32_t pair, uint32_t dim, uint32_t position, float theta) {
  const float exponent = static_cast<float>(2u * pair) / static_cast<float>(dim);
  const float angle = static_cast<float>(position) * (1.0f / powf(theta, exponent));
  float s, c;
  sincosf(angle, &s, &c);
  const float l = left, r = right;
  left = l * c - r * s;
  right = r * c + l * s;
}

__global__ void __launch_bounds__(256) mla_block_cache_kernel(MlaBlockParams p) {
  __shared__ float scratch[40];
  pdl_trigger();
  pdl_wait();
  const uint32_t row_index = blockIdx.x, position = p.first_position + row_index;
  if (position >= p.max_context) return;
  const uint32_t qdim = p.nope + p.rope, width = p.rank + p.rope, pairs = p.rope / 2u;
  float *q = p.qkv + static_cast<uint64_t>(row_index) * p.qkv_stride;
  if (p.rope_theta > 0.0f) {
    for (uint32_t i = threadIdx.x; i < p.heads * pairs; i += blockDim.x) {
      float *at = q + i / pairs * qdim + p.nope + 2u * (i % pairs);
      rope_pair(at[0], at[1], i % pairs, p.rope, position, p.rope_theta);
    }
  }
  const float *kv = q + static_cast<uint64_t>(p.heads) * qdim;
  float sumsq = 0.0f;
  for (uint32_t i = threadIdx.x; i < p.rank; i += blockDim.x) sumsq += kv[i] * kv[i];
  const float scale = rsqrtf(block_sum(sumsq, scratch) / static_cast<float>(p.rank) + p.eps);
  const uint32_t page = p.page_table[position / NERVA_KV_CACHE_BLOCK_TOKENS];
  if (page >= p.page_count) {
    if (threadIdx.x == 0) report_error(p.error_word, kErrPageOutOfRange);
    return;
  }
  uint16_t *row = p.cache + (static_cast<uint64_t>(page) * NERVA_KV_CACHE_BLOCK_TOKENS + position % NERVA_KV_CACHE_BLOCK_TOKENS) * width;
  for (uint32_t i = threadIdx.x; i < p.rank; i += blockDim.x)
    row[i] = f32_to_bf16_bits(kv[i] * scale * bf16_bits_to_f32(p.kv_a_norm[i]));
  if (threadIdx.x < pairs) {
    float l = bf16_round(kv[p.rank + 2u * threadIdx.x]), r = bf16_round(kv[p.rank + 2u * threadIdx.x + 1u]);
    if (p.rope_theta > 0.0f) rope_pair(l, r, threadIdx.x, p.rope, position, p.rope_theta);
    row[p.rank + 2u * threadIdx.x] = f32_to_bf16_bits(l);
    row[p.rank + 2u * threadIdx.x + 1u] = f32_to_bf16_bits(r);
  }
}

// C[row][n] = sum_k A[row][k] B[k][n] of head blockIdx.y, on 64 x 64 tiles, 64 of k at a time.  B is bf16, stored
// [k][n] (W_UK: k the query's features, n the latent's) or [n][k] (W_UV).  A is fp32, in two bf16 parts.
struct HeadProduct {
  const float *a;
  uint64_t a_row, a_head;    // strides
  const uint16_t *b;
  uint64_t b_head;
  uint32_t b_stride;         // from one k (or n) to the next
  float *c_f32;              // one of the two
  uint16_t *c_bf16;
  uint64_t c_row, c_head;
  uint32_t rows, n, k;
};
constexpr uint32_t kHeadTile = 64, kHeadStride = kHeadTile + 8u;  // 144-byte rows: conflict-free fragment loads

template <bool K_MAJOR>  // B stored [n][k]
__global__ void __launch_bounds__(256) mla_block_head_kernel(HeadProduct p) {
  __shared__ __align__(16) uint16_t a_hi[kHeadTile * kHeadStride], a_lo[kHeadTile * kHeadStride], b_sh[kHeadTile * kHeadStride];
  pdl_trigger();
  pdl_wait();
  const uint32_t n0 = blockIdx.x * kHeadTile, h = blockIdx.y, r0 = blockIdx.z * kHeadTile;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t g = lane >> 2, t = lane & 3u;
  const uint32_t m_at = (warp & 3u) * 16u, n_at = (warp >> 2) * 32u;  // this warp's 16 x 32 of the tile
  const float *a = p.a + h * p.a_head;
  const uint16_t *b = p.b + h * p.b_head;
  float c[4][4] = {};
  for (uint32_t k0 = 0; k0 < p.k; k0 += kHeadTile) {
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kHeadTile * kHeadTile / 2u; i += 256u) {
      const uint32_t r = i / 32u, k = 2u * (i % 32u);
      float x = 0.0f, y = 0.0f;
      if (r0 + r < p.rows) {
        const float *src = a + (r0 + r) * p.a_row + k0 + k;
        if (k0 + k < p.k) x = __ldcg(src);
        if (k0 + k + 1u < p.k) y = __ldcg(src + 1);
      }
      *reinterpret_cast<uint32_t *>(a_hi + r * kHeadStride + k) = pack_bf16_hi(x, y);
      *reinterpret_cast<uint32_t *>(a_lo + r * kHeadStride + k) = pack_bf16_lo(x, y);
    }
    for (uint32_t i = threadIdx.x; i < kHeadTile * kHeadTile; i += 256u) {
      const uint32_t outer = i / kHeadTile, inner = i % kHeadTile;
      const uint32_t k = k0 + (K_MAJOR ? inner : outer), n = n0 + (K_MAJOR ? outer : inner);
      const uint64_t at = K_MAJOR ? static_cast<uint64_t>(n) * p.b_stride + k : static_cast<uint64_t>(k) * p.b_stride + n;
      b_sh[outer * kHeadStride + inner] = k < p.k && n < p.n ? __ldg(b + at) : static_cast<uint16_t>(0);
    }
    __syncthreads();
#pragma unroll
    for (uint32_t ks = 0; ks < kHeadTile; ks += 16u) {
      uint32_t hi[4], lo[4];
      const uint32_t a_at = (m_at + (lane & 15u)) * kHeadStride + ks + (lane >> 4) * 8u;
      ldmatrix_x4(hi, smem_addr(a_hi + a_at));
      ldmatrix_x4(lo, smem_addr(a_lo + a_at));
#pragma unroll
      for (uint32_t half = 0; half < 2u; ++half) {
        uint32_t w[4];  // two n-tiles of 8: k rows 0..7 and 8..15 of each
        const uint32_t n = n_at + half * 16u;
        if (K_MAJOR) {
          ldmatrix_x4(w, smem_addr(b_sh + (n + (lane >> 4) * 8u + (lane & 7u)) * kHeadStride + ks + ((lane >> 3) & 1u) * 8u));
        } else {
          ldmatrix_x4_trans(w, smem_addr(b_sh + (ks + ((lane >> 3) & 1u) * 8u + (lane & 7u)) * kHeadStride + n + (lane >> 4) * 8u));
        }
        mma_bf16(c[2u * half], hi, w[0], w[1]);
        mma_bf16(c[2u * half], lo, w[0], w[1]);
        mma_bf16(c[2u * half + 1u], hi, w[2], w[3]);
        mma_bf16(c[2u * half + 1u], lo, w[2], w[3]);
      }
    }
  }
#pragma unroll
  for (uint32_t i = 0; i < 4u; ++i) {
#pragma unroll
    for (uint32_t j = 0; j < 4u; ++j) {
      const uint32_t row = r0 + m_at + g + (j >> 1) * 8u, n = n0 + n_at + i * 8u + 2u * t + (j & 1u);
      if (row >= p.rows || n >= p.n) continue;
      const uint64_t at = row * p.c_row + h * p.c_head + n;
      if (p.c_f32 != nullptr)
        p.c_f32[at] = c[i][j];
      else
        p.c_bf16[at] = f32_to_bf16_bits(c[i][j]);
    }
  }
}

// ---- attention ----
constexpr uint32_t kTokens = 4, kHeadSlots = 16, kM = kTokens * kHeadSlots;  // rows of a block
constexpr uint32_t kKeys = 32;                                              // cached rows of a tile
constexpr uint32_t kPStride = kKeys + 8u;

__host__ __device__ inline uint32_t row_bytes_of(uint32_t rank, uint32_t rope) { return (rank + rope) * 2u + 16u; }
__host__ __device__ inline uint32_t attention_smem(uint32_t rank, uint32_t rope) {
  return (2u * kM + kKeys) * row_bytes_of(rank, rope) + 4u * kM * kKeys * 4u + 2u * kM * kPStride * 2u + 2u * kM * 4u;
}

template <uint32_t NT>  // n-tiles of 8 features per warp in the value product: rank / 128
__global__ void __launch_bounds__(512, 1) mla_block_attention_kernel(MlaBlockParams p) {
  constexpr uint32_t RANK = NT * 128u;
  extern __shared__ __align__(16) uint8_t smem[];
  pdl_trigger();
  pdl_wait();
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t g = lane >> 2, t = lane & 3u;
  const uint32_t width = RANK + p.rope, row_bytes = row_bytes_of(RANK, p.rope);
  const uint32_t k_steps = (width + 15u) / 16u;  // the row's padding is zero
  uint8_t *q_hi = smem, *q_lo = q_hi + kM * row_bytes, *tile = q_lo + kM * row_bytes;
  float *s_part = reinterpret_cast<float *>(tile + kKeys * row_bytes);  // [4 quarters][64 rows][32 keys]
  uint16_t *p_hi = reinterpret_cast<uint16_t *>(s_part + 4u * kM * kKeys), *p_lo = p_hi + kM * kPStride;
  float *rescale = reinterpret_cast<float *>(p_lo + kM * kPStride), *total = rescale + kM;

  const uint32_t first_row = (gridDim.x - 1u - blockIdx.x) * kTokens;  // the longest walks first
  const uint32_t rows = p.rows - first_row < kTokens ? p.rows - first_row : kTokens;
  const uint32_t pos0 = p.first_position + first_row, context = pos0 + rows;
  if (context > p.max_context) return;
  const uint32_t tiles = (context + kKeys - 1u) / kKeys;

  {
    const float qscale = kLog2e * rsqrtf(static_cast<float>(p.nope + p.rope));
    const uint32_t words = row_bytes / 4u;
    for (uint32_t i = threadIdx.x; i < kM * words; i += 512u) {
      const uint32_t m = i / words, k = 2u * (i % words);
      const uint32_t row = m / kHeadSlots, h = m % kHeadSlots;
      float2 v = make_float2(0.0f, 0.0f);
      if (row < rows && h < p.heads) {
        if (k < RANK)
          v = __ldcg(reinterpret_cast<const float2 *>(p.ql + (static_cast<uint64_t>(first_row + row) * p.heads + h) * RANK + k));
        else if (k < width) {
          const float *src = p.qkv + static_cast<uint64_t>(first_row + row) * p.qkv_stride + h * (p.nope + p.rope) + p.nope + (k - RANK);
          v = make_float2(__ldcg(src), __ldcg(src + 1));
        }
      }
      v.x *= qscale;
      v.y *= qscale;
      *reinterpret_cast<uint32_t *>(q_hi + m * row_bytes + 2u * k) = pack_bf16_hi(v.x, v.y);
      *reinterpret_cast<uint32_t *>(q_lo + m * row_bytes + 2u * k) = pack_bf16_lo(v.x, v.y);
    }
  }
  // warp w keeps the maximum and sum of rows 4 w .. 4 w + 3, and its features of all rows
  float m_run[4], l_run[4], acc[kTokens][NT][4];
#pragma unroll
  for (uint32_t i = 0; i < 4u; ++i) m_run[i] = -INFINITY, l_run[i] = 0.0f;
#pragma unroll
  for (uint32_t mt = 0; mt < kTokens; ++mt)
#pragma unroll
    for (uint32_t i = 0; i < NT; ++i) acc[mt][i][0] = acc[mt][i][1] = acc[mt][i][2] = acc[mt][i][3] = 0.0f;

  for (uint32_t tl = 0; tl < tiles; ++tl) {
    const uint32_t token0 = tl * kKeys;
    const uint32_t valid = context - token0 < kKeys ? context - token0 : kKeys;
    __syncthreads();
    const uint32_t pieces = row_bytes / 16u;
    constexpr uint32_t kBatch = 5;  // 32 rows of rank 512 + rope 64 are 4.6 pieces per thread
    for (uint32_t from = threadIdx.x; from < kKeys * pieces; from += 512u * kBatch) {
      uint4 v[kBatch];
#pragma unroll
      for (uint32_t u = 0; u < kBatch; ++u) {
        const uint32_t i = from + u * 512u, r = i / pieces, piece = i % pieces;
        v[u] = make_uint4(0u, 0u, 0u, 0u);
        if (i >= kKeys * pieces || r >= valid || piece >= width / 8u) continue;
        uint32_t page = p.page_table[(token0 + r) / NERVA_KV_CACHE_BLOCK_TOKENS];
        if (page >= p.page_count) {
          report_error(p.error_word, kErrPageOutOfRange);
          page = 0;
        }
        const uint16_t *src = p.cache + (static_cast<uint64_t>(page) * NERVA_KV_CACHE_BLOCK_TOKENS +
                                         (token0 + r) % NERVA_KV_CACHE_BLOCK_TOKENS) * width + piece * 8u;
        v[u] = __ldcg(reinterpret_cast<const uint4 *>(src));
      }
#pragma unroll
      for (uint32_t u = 0; u < kBatch; ++u) {
        const uint32_t i = from + u * 512u;
        if (i < kKeys * pieces) *reinterpret_cast<uint4 *>(tile + (i / pieces) * row_bytes + (i % pieces) * 16u) = v[u];
      }
    }
    __syncthreads();
    {
      // ---- scores: 32 rows x 16 keys over a quarter of the features ----
      const uint32_t m_at = (warp & 1u) * 32u, n_at = ((warp >> 1) & 1u) * 16u, quarter = warp >> 2;
      const uint32_t per = (k_steps + 3u) / 4u;
      const uint32_t ks_end = (quarter + 1u) * per < k_steps ? (quarter + 1u) * per : k_steps;
      float c[2][2][4] = {};
      const uint32_t a_off = (m_at + (lane & 15u)) * row_bytes + (lane >> 4) * 16u;
      const uint32_t b_addr = smem_addr(tile + (n_at + (lane >> 4) * 8u + (lane & 7u)) * row_bytes + ((lane >> 3) & 1u) * 16u);
      const uint32_t hi_addr = smem_addr(q_hi + a_off), lo_addr = smem_addr(q_lo + a_off);
      for (uint32_t ks = quarter * per; ks < ks_end; ++ks) {
        uint32_t b[4];
        ldmatrix_x4(b, b_addr + ks * 32u);
#pragma unroll
        for (uint32_t m = 0; m < 2u; ++m) {
          uint32_t hi[4], lo[4];
          ldmatrix_x4(hi, hi_addr + m * 16u * row_bytes + ks * 32u);
          ldmatrix_x4(lo, lo_addr + m * 16u * row_bytes + ks * 32u);
          mma_bf16(c[m][0], hi, b[0], b[1]);
          mma_bf16(c[m][1], hi, b[2], b[3]);
          mma_bf16(c[m][0], lo, b[0], b[1]);
          mma_bf16(c[m][1], lo, b[2], b[3]);
        }
      }
#pragma unroll
      for (uint32_t m = 0; m < 2u; ++m)
#pragma unroll
        for (uint32_t n = 0; n < 2u; ++n) {
          float *out = s_part + (quarter * kM + m_at + m * 16u + g) * kKeys + n_at + n * 8u + 2u * t;
          *reinterpret_cast<float2 *>(out) = make_float2(c[m][n][0], c[m][n][1]);
          *reinterpret_cast<float2 *>(out + 8u * kKeys) = make_float2(c[m][n][2], c[m][n][3]);
        }
    }
    __syncthreads();
#pragma unroll
    for (uint32_t i = 0; i < 4u; ++i) {
      // ---- softmax: lane = key; the four rows of a warp are four heads of one position ----
      const uint32_t m = warp * 4u + i;
      const float *sp = s_part + m * kKeys + lane;
      float s = ((sp[0] + sp[kM * kKeys]) + sp[2u * kM * kKeys]) + sp[3u * kM * kKeys];
      if (token0 + lane > pos0 + m / kHeadSlots) s = -INFINITY;
      const float m_new = fmaxf(m_run[i], warp_max(s));  // finite from the first tile on: position 0 is seen by all
      const float corr = exp2f(m_run[i] - m_new), pr = exp2f(s - m_new);
      l_run[i] = l_run[i] * corr + warp_sum(pr);
      m_run[i] = m_new;
      const uint16_t hi = f32_to_bf16_bits(pr);
      p_hi[m * kPStride + lane] = hi;
      p_lo[m * kPStride + lane] = f32_to_bf16_bits(pr - bf16_bits_to_f32(hi));
      if (lane == 0) rescale[m] = corr;
    }
    __syncthreads();
#pragma unroll
    for (uint32_t mt = 0; mt < kTokens; ++mt) {
      const float corr_a = rescale[mt * 16u + g], corr_b = rescale[mt * 16u + g + 8u];
#pragma unroll
      for (uint32_t i = 0; i < NT; ++i) {
        acc[mt][i][0] *= corr_a;
        acc[mt][i][1] *= corr_a;
        acc[mt][i][2] *= corr_b;
        acc[mt][i][3] *= corr_b;
      }
    }
    // A zero probability times a value that is not finite is not zero: where a position of the block does not see every row
    // of the tile, the rows it does not see are masked out of its product.
    auto value_product = [&](auto masked) {
#pragma unroll(masked ? 1 : kKeys / 16u)
    for (uint32_t ks = 0; ks < kKeys / 16u; ++ks) {
      const uint32_t row = ks * 16u + ((lane >> 3) & 1u) * 8u + (lane & 7u);
      uint32_t b[NT][2];
      if constexpr (NT >= 2) {
#pragma unroll
        for (uint32_t i = 0; i < NT; i += 2u) {
          uint32_t w[4];
          ldmatrix_x4_trans(w, smem_addr(tile + row * row_bytes + (warp * NT + i + (lane >> 4)) * 16u));
          b[i][0] = w[0], b[i][1] = w[1], b[i + 1u][0] = w[2], b[i + 1u][1] = w[3];
        }
      } else {
        uint32_t w[4];  // one n-tile per warp: lanes 16..31 repeat the addresses of lanes 0..15
        ldmatrix_x4_trans(w, smem_addr(tile + row * row_bytes + warp * 16u));
        b[0][0] = w[0], b[0][1] = w[1];
      }
#pragma unroll
      for (uint32_t mt = 0; mt < kTokens; ++mt) {
        uint32_t hi[4], lo[4];
        const uint32_t at = (mt * 16u + (lane & 15u)) * kPStride + ks * 16u + (lane >> 4) * 8u;
        ldmatrix_x4(hi, smem_addr(p_hi + at));
        ldmatrix_x4(lo, smem_addr(p_lo + at));
        uint32_t seen0 = 0xffffffffu, seen1 = 0xffffffffu;  // of rows 2 t, 2 t + 1 and of rows 2 t + 8, 2 t + 9
        if constexpr (masked) {
          const uint32_t key = token0 + ks * 16u + 2u * t, pos = pos0 + mt;
          seen0 = (key <= pos ? 0xffffu : 0u) | (key + 1u <= pos ? 0xffff0000u : 0u);
          seen1 = (key + 8u <= pos ? 0xffffu : 0u) | (key + 9u <= pos ? 0xffff0000u : 0u);
        }
#pragma unroll
        for (uint32_t i = 0; i < NT; ++i) {
          mma_bf16(acc[mt][i], hi, b[i][0] & seen0, b[i][1] & seen1);
          mma_bf16(acc[mt][i], lo, b[i][0] & seen0, b[i][1] & seen1);
        }
      }
    }
    };
    if (token0 + kKeys > pos0 + 1u)
      value_product(std::true_type{});
    else
      value_product(std::false_type{});
  }
  if (lane == 0) {
#pragma unroll
    for (uint32_t i = 0; i < 4u; ++i) total[warp * 4u + i] = l_run[i];
  }
  __syncthreads();
#pragma unroll
  for (uint32_t mt = 0; mt < kTokens; ++mt) {
    if (mt >= rows) break;
    float *out = p.latent + (static_cast<uint64_t>(first_row + mt) * p.heads) * RANK;
    const float inv_a = 1.0f / total[mt * 16u + g], inv_b = 1.0f / total[mt * 16u + g + 8u];
#pragma unroll
    for (uint32_t i = 0; i < NT; ++i) {
      const uint32_t feature = (warp * NT + i) * 8u + 2u * t;
      if (g < p.heads)
        *reinterpret_cast<float2 *>(out + static_cast<uint64_t>(g) * RANK + feature) = make_float2(acc[mt][i][0] * inv_a, acc[mt][i][1] * inv_a);
      if (g + 8u < p.heads)
        *reinterpret_cast<float2 *>(out + static_cast<uint64_t>(g + 8u) * RANK + feature) =
            make_float2(acc[mt][i][2] * inv_b, acc[mt][i][3] * inv_b);
    }
  }
}

}  // namespace

cudaError_t configure_mla_block() {
  const int bytes = static_cast<int>(attention_smem(512, 64));
  cudaError_t err = cudaFuncSetAttribute(mla_block_attention_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (err == cudaSuccess)
    err = cudaFuncSetAttribute(mla_block_attention_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (err == cudaSuccess)
    err = cudaFuncSetAttribute(mla_block_attention_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  return err;
}

cudaError_t launch_mla_block(cudaStream_t stream, const MlaBlockParams &p, bool pdl, uint64_t *launches) {
  if (p.rows == 0 || !mla_session_supported(p.heads, p.rank, p.nope, p.rope, p.v_dim)) return cudaErrorInvalidValue;
  cudaError_t err = launch_with_pdl(mla_block_cache_kernel, dim3(p.rows), dim3(256), 0, stream, pdl, p);
  HeadProduct q{};
  q.a = p.qkv;
  q.a_row = p.qkv_stride;
  q.a_head = p.nope + p.rope;
  q.b = p.w_kv_b;
  q.b_head = static_cast<uint64_t>(p.nope + p.v_dim) * p.rank;
  q.b_stride = p.rank;
  q.c_f32 = p.ql;
  q.c_row = static_cast<uint64_t>(p.heads) * p.rank;
  q.c_head = p.rank;
  q.rows = p.rows;
  q.n = p.rank;
  q.k = p.nope;
  const uint32_t row_tiles = (p.rows + kHeadTile - 1u) / kHeadTile;
  if (err == cudaSuccess)
    err = launch_with_pdl(mla_block_head_kernel<false>, dim3((p.rank + kHeadTile - 1u) / kHeadTile, p.heads, row_tiles), dim3(256), 0,
                          stream, pdl, q);
  const dim3 grid((p.rows + kTokens - 1u) / kTokens);
  const uint32_t smem = attention_smem(p.rank, p.rope);
  if (err == cudaSuccess) {
    auto kernel = p.rank == 128u ? mla_block_attention_kernel<1> : p.rank == 256u ? mla_block_attention_kernel<2> : mla_block_attention_kernel<4>;
    err = launch_with_pdl(kernel, grid, dim3(512), smem, stream, pdl, p);
  }
  HeadProduct v{};
  v.a = p.latent;
  v.a_row = q.c_row;
  v.a_head = p.rank;
  v.b = p.w_kv_b + static_cast<uint64_t>(p.nope) * p.rank;
  v.b_head = q.b_head;
  v.b_stride = p.rank;
  v.c_bf16 = p.out;
  v.c_row = static_cast<uint64_t>(p.heads) * p.v_dim;
  v.c_head = p.v_dim;
  v.rows = p.rows;
  v.n = p.v_dim;
  v.k = p.rank;
  if (err == cudaSuccess)
    err = launch_with_pdl(mla_block_head_kernel<true>, dim3((p.v_dim + kHeadTile - 1u) / kHeadTile, p.heads, row_tiles), dim3(256), 0,
                          stream, pdl, v);
  if (launches != nullptr) *launches += 4;
  return err;
}

}  // namespace nb
