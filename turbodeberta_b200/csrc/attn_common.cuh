// What the two tensor-core attention kernels share: tile sizes, shared-memory accessors, tensor maps, and the rule that
// splits a long sequence's keys between them.
#pragma once
#include "tdb_internal.h"
#include "ptx_sm100.cuh"

namespace tdb {

constexpr int BQ = 128, BK = 128, HD = 64;

__device__ __forceinline__ float lds_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ void sts_f32(uint32_t addr, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ uint4 lds_128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void sts_128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// Makes this thread's earlier shared-memory writes visible to the asynchronous proxy (the tensor cores' operand fetch).
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Long sequences, both kernels at work: for a pair of query tiles (256 rows from q0p = q0 rounded down) the key tiles
// [0, near_first) and [near_end, ...) lie at or beyond the saturation distance for every row, on one side each; the kernel for
// band tiles takes the tiles in between and leaves its running softmax state, the far kernel carries it on.
__device__ __forceinline__ int near_first(int q0, int sat) {
  const int q0p = q0 & ~(2 * BQ - 1);
  return q0p >= sat + BK - 1 ? (q0p - sat - (BK - 1)) / BK + 1 : 0;
}
__device__ __forceinline__ int near_end(int q0, int sat) {
  const int q0p = q0 & ~(2 * BQ - 1);
  return (q0p + 2 * BQ - 1 + sat + BK - 1) / BK;
}

// The state handed over lies tile by tile (query tile, head): 64 x 128 outputs with the rows contiguous, since both kernels
// have a row per thread, and 128 (exponent, sum) pairs.  Packed form: sequence e's tiles start at e + (its first token) / 128,
// which leaves room for a partial last tile of every sequence before it.
__host__ __device__ __forceinline__ int64_t partial_tile(const AttnParams& p, int64_t tok0, int seq, int bcoord, int q0) {
  return p.varlen ? tok0 / BQ + seq + q0 / BQ : (int64_t)bcoord * ((p.L + BQ - 1) / BQ) + q0 / BQ;
}

// [tokens] x [heads] x 64 bf16 (and batch rows), boxes of 128 tokens of one head; 128-byte swizzle.
int token_map(CUtensorMap* m, const void* ptr, int64_t tokens, int H, int B, int64_t sb, int64_t st, int64_t sh, const char* what);
// [heads] x [rows] x 64 bf16, boxes of box_rows rows of one head; 128-byte swizzle.
int table_map(CUtensorMap* m, const void* ptr, int rows, int H, int box_rows, const char* what);
int launch_attn_far(const AttnParams& p, int64_t tiles, int sms, cudaStream_t s);

}  // namespace tdb
