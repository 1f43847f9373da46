// Warp-level tensor products on 64-row bf16 tiles in shared memory, for the kernels whose tiles are too few or whose operands
// are too scattered for tensor memory.
#pragma once
#include "tdb_internal.h"

namespace tdb {

constexpr int ST = 64, SP = 72, S_THREADS = 128;     // tile rows, row pitch in elements (144 bytes: conflict-free ldmatrix)

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// 64 rows of 64 bf16, by THREADS threads; rows at or beyond `rows` become zeros (the caller's padding may hold anything).
template <int THREADS = S_THREADS>
__device__ __forceinline__ void stage(__nv_bfloat16* dst, const __nv_bfloat16* src, int64_t pitch, int rows) {
#pragma unroll
  for (int i = 0; i < ST * 8 / THREADS; ++i) {
    const int e = threadIdx.x + i * THREADS, row = e >> 3, c = e & 7;
    const bool real = row < rows;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(saddr(dst + row * SP + c * 8)),
                 "l"(src + (real ? (int64_t)row * pitch + c * 8 : 0)), "r"(real ? 16 : 0) : "memory");
  }
}
__device__ __forceinline__ void ldsm4(uint32_t* r, const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(saddr(p)) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t* r, const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(saddr(p)) : "memory");
}
__device__ __forceinline__ void mma(float* d, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const __nv_bfloat162 t = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&t);
}

}  // namespace tdb
