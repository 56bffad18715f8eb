// Device-side pieces that the windowed attention kernels share (window_attention.cu, prefill_attention.cu).
#pragma once

#include "common.cuh"
#include "kernels.cuh"

namespace nb {

constexpr float kLog2e = 1.4426950408889634f;
constexpr uint32_t kPageTokens = NERVA_KV_CACHE_BLOCK_TOKENS;

template <uint32_t BYTES>
__device__ __forceinline__ void cp_async_zfill(void *dst, const void *src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(valid ? BYTES : 0u)
               : "memory");
}
__device__ __forceinline__ void cp_async_16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// The tiles of `size` tokens a query walks: those that hold kept first positions and lie in front of the
// window, then the window's.
struct TileWalk {
  uint32_t kept, first;  // tiles in front; first tile of the window
  __device__ __forceinline__ TileWalk(uint32_t keep_first, uint32_t lo, uint32_t size) {
    first = lo / size;
    kept = (keep_first + size - 1u) / size;
    if (kept > first) kept = first;
  }
  __device__ __forceinline__ uint32_t count(uint32_t end, uint32_t size) const {  // tiles, for a window that ends at `end`
    return kept + (end + size - 1u) / size - first;
  }
  __device__ __forceinline__ uint32_t tile(uint32_t i) const { return i < kept ? i : first + (i - kept); }
};

// EXTRAS of the kernels: kept first positions, score cap and output gates.  Without them the code
// is the plain window's.
__host__ __device__ inline bool has_extras(const WindowAttentionShape &s) {
  return s.keep_first != 0 || s.softcap > 0.0f || s.head_gate != 0;
}

// Soft cap of a score that carries a factor log2(e), through one exponential: absolute error a few 1e-7 of the cap.
__device__ __forceinline__ float cap_score_fast(float score, float cap2, float inv_cap2) {
  const float e = exp2f(score * inv_cap2 * (2.0f * kLog2e));
  return cap2 - __fdividef(2.0f * cap2, e + 1.0f);
}

// Factor of a head's output.
template <bool EXTRAS>
__device__ __forceinline__ float output_gate(const WindowAttentionParams &p, uint32_t row, uint32_t h) {
  const WindowAttentionShape &s = p.s;
  if (!EXTRAS || s.head_gate == 0) return 1.0f;
  const uint32_t at = (s.heads + s.kv_heads) * s.qk_dim + s.kv_heads * s.v_dim + h;
  return sigmoid(__ldcg(p.qkv + static_cast<uint64_t>(row) * p.qkv_stride + at));
}

// Cached row (page, slot) of a KV head, in elements of a row of `width` per head.
__device__ __forceinline__ uint64_t cache_row(uint32_t page, uint32_t token, uint32_t kv_heads, uint32_t kvh, uint32_t width) {
  return ((static_cast<uint64_t>(page) * kPageTokens + token % kPageTokens) * kv_heads + kvh) * width;
}

}  // namespace nb
