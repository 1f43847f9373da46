// The encoder's kernels around its matrix products and the attention: the embeddings, residual + LayerNorm, GELU, and the passage between
// padded batches and the packed token stream.  All of them are bound by memory traffic (or, for a handful of tokens, by the
// launch): each reads its inputs once and writes its output once.
#include "tdb_internal.h"
#include "gelu.cuh"

namespace tdb {

namespace {

template <typename T> struct Vec;                    // 16 bytes of T as fp32
template <> struct Vec<float> {
  static constexpr int N = 4;
  static __device__ __forceinline__ void unpack(const uint4& v, float* f) {
    f[0] = __uint_as_float(v.x); f[1] = __uint_as_float(v.y); f[2] = __uint_as_float(v.z); f[3] = __uint_as_float(v.w);
  }
  static __device__ __forceinline__ uint4 pack(const float* f) {
    return make_uint4(__float_as_uint(f[0]), __float_as_uint(f[1]), __float_as_uint(f[2]), __float_as_uint(f[3]));
  }
};
template <> struct Vec<__nv_bfloat16> {
  static constexpr int N = 8;
  static __device__ __forceinline__ void unpack(const uint4& v, float* f) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { f[2 * i] = __uint_as_float(w[i] << 16); f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u); }
  }
  static __device__ __forceinline__ uint4 pack(const float* f) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __nv_bfloat162 t = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t*>(&t);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
  }
};

__device__ __forceinline__ float rounded(float x, float) { return x; }
__device__ __forceinline__ float rounded(float x, __nv_bfloat16) { return __bfloat162float(__float2bfloat16_rn(x)); }

__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
  return x;
}

// out may be x.  No __restrict__ on the activations: the kernel may have started beside the one that writes them, and the
// non-coherent loads that it allows are not part of what wait_for_stream() makes visible.
// out = LayerNorm(x + res) * w + b, one warp per row, the row held in registers (fp32 sum, mean and variance).  Per row three
// row-sized transfers; 9.2k x 1024 bf16 (57 MB): 24 + 8 us as an addition and a LayerNorm kernel, 11.4 us here.
// FEW: for a few rows the loads' latency is the kernel's time, so w and b come first; with many rows they are in the first-level
// cache and better left out of the registers (9.2k x 1024: 13.8 us with, 11.4 without).
template <typename T, int NV, bool FEW>
__global__ void __launch_bounds__(128) add_layernorm_kernel(const T* x, const T* res, const T* __restrict__ w,
                                                            const T* __restrict__ b, float eps, int64_t rows, int hidden, T* out) {
  constexpr int N = Vec<T>::N;
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  const int lane = threadIdx.x % 32, nv = hidden / N;
  if (row >= rows) return;
  const uint4* xr = reinterpret_cast<const uint4*>(x + row * hidden);
  const uint4* rr = reinterpret_cast<const uint4*>(res + row * hidden);
  float f[NV][N];
  float sum = 0.f;
  uint4 wv[FEW ? NV : 1], bv[FEW ? NV : 1];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = lane + 32 * i;
    if (FEW && c < nv) { wv[FEW ? i : 0] = __ldg(reinterpret_cast<const uint4*>(w) + c); bv[FEW ? i : 0] = __ldg(reinterpret_cast<const uint4*>(b) + c); }
  }
  wait_for_stream();                                 // the weights, above, are older than the kernel in front
  let_next_start();
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = lane + 32 * i;
    if (c < nv) {
      float g[N];
      Vec<T>::unpack(xr[c], f[i]);
      Vec<T>::unpack(rr[c], g);
#pragma unroll
      for (int e = 0; e < N; ++e) { f[i][e] += g[e]; sum += f[i][e]; }
    }
  }
  const float mean = warp_sum(sum) / (float)hidden;
  float sq = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i)
    if (lane + 32 * i < nv) {
#pragma unroll
      for (int e = 0; e < N; ++e) { const float d = f[i][e] - mean; sq = fmaf(d, d, sq); }
    }
  const float inv = rsqrtf(warp_sum(sq) / (float)hidden + eps);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = lane + 32 * i;
    if (c < nv) {
      float g[N], a[N];
      Vec<T>::unpack(FEW ? wv[FEW ? i : 0] : __ldg(reinterpret_cast<const uint4*>(w) + c), g);
      Vec<T>::unpack(FEW ? bv[FEW ? i : 0] : __ldg(reinterpret_cast<const uint4*>(b) + c), a);
#pragma unroll
      for (int e = 0; e < N; ++e) f[i][e] = fmaf((f[i][e] - mean) * inv, g[e], a[e]);
      reinterpret_cast<uint4*>(out + row * hidden)[c] = Vec<T>::pack(f[i]);
    }
  }
}

template <typename T>
int launch_add_layernorm_t(const void* x, const void* res, const void* w, const void* b, float eps, int64_t rows, int hidden, void* out,
                           bool early, cudaStream_t s) {
  constexpr int PER = 32 * Vec<T>::N;
  const int nv = (hidden + PER - 1) / PER;
  int sms = 0;
  if (const int rc = device_sms(&sms)) return rc;
  const int warps = rows >= 16 * sms ? 4 : 1;        // few rows: one per block, so that they spread over the SMs
  const unsigned blocks = (unsigned)((rows + warps - 1) / warps);
#define TDB_LN(NV)                                                                                                              \
  if (nv <= NV) {                                                                                                               \
    return cuda_fail(launch_stream(warps == 1 ? add_layernorm_kernel<T, NV, true> : add_layernorm_kernel<T, NV, false>, dim3(blocks), 32 * warps, 0, s, early, (const T*)x, (const T*)res,           \
                                  (const T*)w, (const T*)b, eps, rows, hidden, (T*)out), "add_layernorm launch");                  \
  }
  TDB_LN(1) TDB_LN(3) TDB_LN(4) TDB_LN(6) TDB_LN(8)
#undef TDB_LN
  set_error("add_layernorm: hidden size %d is not supported", hidden);
  return TDB_ERR_SHAPE;
}

// out = LayerNorm(table[ids]) * w + b, times the padding mask: a model's input, one warp per token.  Bound by the rows that come and go
// (32 x 512 tokens of 1024 bf16: 33 MB each way, the padding's row from L2); as a gather, a LayerNorm, the mask's conversion and a
// multiplication they took 96 us there, and for one short text some 60 us of launches.  The roundings are those of these four.
template <typename T, int NV, typename I>
__global__ void __launch_bounds__(128) embed_kernel(const I* __restrict__ ids, const T* __restrict__ table, int64_t vocabulary, const T* __restrict__ w,
                                                    const T* __restrict__ b, float eps, const void* __restrict__ mask, int mask_bytes,
                                                    int64_t rows, int hidden, T* __restrict__ out, int32_t* status) {
  constexpr int N = Vec<T>::N;
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  const int lane = threadIdx.x % 32, nv = hidden / N;
  if (row >= rows) return;
  int64_t id = ids[row];
  if (id < 0 || id >= vocabulary) {
    if (lane == 0) *reinterpret_cast<volatile int32_t*>(status + 3) = 1;
    id = 0;
  }
  const float keep = mask_bytes == 8 ? (float)static_cast<const int64_t*>(mask)[row] : (float)static_cast<const uint8_t*>(mask)[row];
  const uint4* src = reinterpret_cast<const uint4*>(table + id * hidden);
  float f[NV][N], sum = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i)
    if (lane + 32 * i < nv) {
      Vec<T>::unpack(__ldg(src + lane + 32 * i), f[i]);
#pragma unroll
      for (int e = 0; e < N; ++e) sum += f[i][e];
    }
  const float mean = warp_sum(sum) / (float)hidden;
  float sq = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i)
    if (lane + 32 * i < nv) {
#pragma unroll
      for (int e = 0; e < N; ++e) { const float d = f[i][e] - mean; sq = fmaf(d, d, sq); }
    }
  const float inv = rsqrtf(warp_sum(sq) / (float)hidden + eps);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = lane + 32 * i;
    if (c < nv) {
      float g[N], a[N];
      Vec<T>::unpack(__ldg(reinterpret_cast<const uint4*>(w) + c), g);
      Vec<T>::unpack(__ldg(reinterpret_cast<const uint4*>(b) + c), a);
#pragma unroll
      for (int e = 0; e < N; ++e) f[i][e] = rounded(fmaf((f[i][e] - mean) * inv, g[e], a[e]), T()) * rounded(keep, T());
      reinterpret_cast<uint4*>(out + row * hidden)[c] = Vec<T>::pack(f[i]);
    }
  }
}

template <typename T, typename I>
int launch_embed_t(const void* ids, const void* table, int64_t vocabulary, const void* w, const void* b, float eps, const void* mask, int mask_bytes,
                   int64_t rows, int hidden, void* out, int32_t* status, cudaStream_t s) {
  constexpr int PER = 32 * Vec<T>::N;
  const int nv = (hidden + PER - 1) / PER;
  int sms = 0;
  if (const int rc = device_sms(&sms)) return rc;
  const int warps = rows >= 16 * sms ? 4 : 1;        // few rows: one per block, so that they spread over the SMs
  const unsigned blocks = (unsigned)((rows + warps - 1) / warps);
#define TDB_EMBED(NV)                                                                                                           \
  if (nv <= NV) {                                                                                                               \
    embed_kernel<T, NV, I><<<blocks, 32 * warps, 0, s>>>((const I*)ids, (const T*)table, vocabulary, (const T*)w, (const T*)b, eps, mask, mask_bytes, rows, \
                                                         hidden, (T*)out, status);                                              \
    return cuda_fail(cudaGetLastError(), "embed launch");                                                                       \
  }
  TDB_EMBED(1) TDB_EMBED(3) TDB_EMBED(4) TDB_EMBED(6) TDB_EMBED(8)
#undef TDB_EMBED
  set_error("embed: hidden size %d is not supported", hidden);
  return TDB_ERR_SHAPE;
}

// x <- x * Phi(x) (the exact GELU), in place.  9.2k x 4096 bf16 (75 MB in, 75 MB out): 37 us with erff, 24 with the above.
template <typename T>
__global__ void __launch_bounds__(256) gelu_kernel(uint4* __restrict__ x, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  wait_for_stream();
  float f[Vec<T>::N];
  Vec<T>::unpack(x[i], f);
#pragma unroll
  for (int e = 0; e < Vec<T>::N; ++e) f[e] = gelu(f[e], T());
  x[i] = Vec<T>::pack(f);
}

// Padding mask [B, L] -> lengths, offsets and what the host has to know (out: all ones, right padded, tokens, longest),
// one block per row; the block that finishes last adds up the rows.  ticket[0]: zero before and after; ticket[1] likewise.
template <typename M>
__global__ void __launch_bounds__(256) mask_rows_kernel(const M* __restrict__ mask, int B, int L, int32_t* __restrict__ seqlens,
                                                        int32_t* __restrict__ cu, int32_t* ticket, volatile int32_t* out) {
  __shared__ int total, holes, last;
  const int t = threadIdx.x;
  if (t == 0) { total = 0; holes = 0; }
  __syncthreads();
  const M* row = mask + (int64_t)blockIdx.x * L;
  int n = 0, hole = 0;
  for (int i = t; i < L; i += 256) {
    const bool on = row[i] != 0;
    n += on;
    hole |= on && i > 0 && row[i - 1] == 0;          // a valid token behind a padded one
  }
  atomicAdd(&total, n);
  if (hole) holes = 1;
  __syncthreads();
  if (t == 0) {
    seqlens[blockIdx.x] = total;
    if (holes) atomicExch(ticket + 1, 1);
    __threadfence();
    last = atomicInc(reinterpret_cast<unsigned int*>(ticket), gridDim.x - 1) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last || t >= 32) return;
  __threadfence();
  int run = 0, longest = 0, full = 1;
  for (int b0 = 0; b0 < B; b0 += 32) {
    const int b = b0 + t;
    const int len = b < B ? *reinterpret_cast<volatile int32_t*>(seqlens + b) : 0;
    if (b < B) { longest = max(longest, len); full &= len == L; }
    int inc = len;
#pragma unroll
    for (int off = 1; off < 32; off *= 2) {
      const int o = __shfl_up_sync(0xffffffffu, inc, off);
      if (t >= off) inc += o;
    }
    if (b < B) cu[b + 1] = run + inc;
    run += __shfl_sync(0xffffffffu, inc, 31);
  }
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    longest = max(longest, __shfl_xor_sync(0xffffffffu, longest, off));
    full &= __shfl_xor_sync(0xffffffffu, full, off);
  }
  if (t == 0) {
    cu[0] = 0;
    out[0] = full; out[1] = atomicExch(ticket + 1, 0) == 0; out[2] = run; out[3] = longest;
  }
}

// pos[b * L + i] = place of the token in the packed stream, or -1.  One warp per row.
template <typename M>
__global__ void __launch_bounds__(32) mask_positions_kernel(const M* __restrict__ mask, const int32_t* __restrict__ cu, int L, int32_t* __restrict__ pos) {
  const int64_t base = (int64_t)blockIdx.x * L;
  const int lane = threadIdx.x;
  int at = cu[blockIdx.x];
  for (int i0 = 0; i0 < L; i0 += 32) {
    const int i = i0 + lane;
    const bool on = i < L && mask[base + i] != 0;
    const uint32_t m = __ballot_sync(0xffffffffu, on);
    if (i < L) pos[base + i] = on ? at + __popc(m & ((1u << lane) - 1u)) : -1;
    at += __popc(m);
  }
}

// One warp per padded row of `vecs` 16-byte pieces.  PACK: padded -> packed; otherwise packed -> padded, zeros where padding is.
template <bool PACK>
__global__ void __launch_bounds__(256) repack_kernel(const uint4* __restrict__ src, const int32_t* __restrict__ pos, int64_t rows, int vecs,
                                                     uint4* __restrict__ dst) {
  const int64_t row = (int64_t)blockIdx.x * 8 + threadIdx.x / 32;
  if (row >= rows) return;
  const int64_t at = pos[row];
  if (PACK && at < 0) return;
  for (int c = threadIdx.x % 32; c < vecs; c += 32) {
    if (PACK) dst[at * vecs + c] = src[row * vecs + c];
    else dst[row * vecs + c] = at < 0 ? make_uint4(0, 0, 0, 0) : src[at * vecs + c];
  }
}

}  // namespace
}  // namespace tdb

using namespace tdb;

extern "C" {

int tdb_add_layernorm(const void* x, const void* res, const void* w, const void* b, float eps, int64_t rows, int hidden, int dtype,
                      void* out, int early, void* stream) {
  if (rows == 0) return TDB_OK;
  return dtype == TDB_DTYPE_F32 ? launch_add_layernorm_t<float>(x, res, w, b, eps, rows, hidden, out, early, (cudaStream_t)stream)
                                : launch_add_layernorm_t<__nv_bfloat16>(x, res, w, b, eps, rows, hidden, out, early, (cudaStream_t)stream);
}

int tdb_embed(const void* ids, int id_bytes, const void* table, int64_t vocabulary, const void* w, const void* b, float eps, const void* mask,
              int mask_bytes, int64_t rows, int hidden, int dtype, void* out, int32_t* status, void* stream) {
  if (rows == 0) return TDB_OK;
  auto run = id_bytes == 8 ? (dtype == TDB_DTYPE_F32 ? launch_embed_t<float, int64_t> : launch_embed_t<__nv_bfloat16, int64_t>)
                           : (dtype == TDB_DTYPE_F32 ? launch_embed_t<float, int32_t> : launch_embed_t<__nv_bfloat16, int32_t>);
  return run(ids, table, vocabulary, w, b, eps, mask, mask_bytes, rows, hidden, out, status, (cudaStream_t)stream);
}

int tdb_gelu(void* x, int64_t elements, int dtype, void* stream) {
  const int64_t n = elements / (dtype == TDB_DTYPE_F32 ? 4 : 8);
  if (n == 0) return TDB_OK;
  const unsigned blocks = (unsigned)((n + 255) / 256);
  return cuda_fail(launch_early(dtype == TDB_DTYPE_F32 ? gelu_kernel<float> : gelu_kernel<__nv_bfloat16>, dim3(blocks), 256, 0,
                                (cudaStream_t)stream, (uint4*)x, n), "gelu launch");
}

int tdb_mask_rows(const void* mask, int elem_bytes, int B, int L, int32_t* seqlens, int32_t* cu, int32_t* ticket, int32_t* out, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (elem_bytes == 8) mask_rows_kernel<<<B, 256, 0, s>>>((const int64_t*)mask, B, L, seqlens, cu, ticket, out);
  else mask_rows_kernel<<<B, 256, 0, s>>>((const uint8_t*)mask, B, L, seqlens, cu, ticket, out);
  return cuda_fail(cudaGetLastError(), "mask_rows launch");
}

int tdb_mask_positions(const void* mask, int elem_bytes, const int32_t* cu, int B, int L, int32_t* pos, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (elem_bytes == 8) mask_positions_kernel<<<B, 32, 0, s>>>((const int64_t*)mask, cu, L, pos);
  else mask_positions_kernel<<<B, 32, 0, s>>>((const uint8_t*)mask, cu, L, pos);
  return cuda_fail(cudaGetLastError(), "mask_positions launch");
}

int tdb_repack(int pack, const void* src, const int32_t* pos, int64_t rows, int row_bytes, void* dst, void* stream) {
  const unsigned blocks = (unsigned)((rows + 7) / 8);
  if (pack) repack_kernel<true><<<blocks, 256, 0, (cudaStream_t)stream>>>((const uint4*)src, pos, rows, row_bytes / 16, (uint4*)dst);
  else repack_kernel<false><<<blocks, 256, 0, (cudaStream_t)stream>>>((const uint4*)src, pos, rows, row_bytes / 16, (uint4*)dst);
  return cuda_fail(cudaGetLastError(), "repack launch");
}

}  // extern "C"
