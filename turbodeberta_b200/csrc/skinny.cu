// y = x W^T + b (optionally through GELU) in bf16 for a handful of tokens: the projections of a short request.
//
// Bound by the latency of one trip to memory for the weights (1.2 to 9.4 MB per projection) and by the launch in front of it,
// so the weights do not wait for anything: a block owns 8 or 16 output features, its eight warps share the columns, and every
// thread has its part of W in registers before it waits for the kernel in front, which may still be running (the launcher
// says which launches may).  Then it reads x (L2), multiplies with the warp-level tensor instruction, and the warps' partial
// sums are added up through shared memory.
// The order of the columns inside a product is free as long as x and W share it, so a thread's fragments of two k16 steps are
// one 16-byte load: lane % 4 takes eight consecutive columns of every 32.
#include "attn_warp_mma.cuh"
#include "gelu.cuh"

namespace tdb {

namespace {

constexpr int WARPS = 8, KB = 32;                    // columns of one 16-byte load by four lanes

// MT: tiles of 16 tokens; NF: groups of 8 features; NB: blocks of 32 columns per warp.
template <int MT, int NF, int NB, bool GELU>
__global__ void __launch_bounds__(WARPS * 32) skinny_kernel(const __nv_bfloat16* x, const __nv_bfloat16* __restrict__ w,
                                                            const __nv_bfloat16* __restrict__ bias, int T, int K, int N,
                                                            __nv_bfloat16* y) {     // x, y: no __restrict__, see encoder.cu
  __shared__ float part[WARPS][MT * 16][NF * 8];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, g = lane / 4, t = lane % 4;
  const int n0 = blockIdx.x * NF * 8, blocks = K / KB;
  uint4 wf[NB][NF];
#pragma unroll
  for (int i = 0; i < NB; ++i)
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      const int b = warp + WARPS * i, n = n0 + 8 * f + g;
      wf[i][f] = make_uint4(0, 0, 0, 0);
      if (b < blocks && n < N) wf[i][f] = __ldg(reinterpret_cast<const uint4*>(w + (int64_t)n * K + b * KB) + t);
    }
  wait_for_stream();
  let_next_start();
  float acc[MT][NF][4];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int f = 0; f < NF; ++f)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[m][f][e] = 0.f;
#pragma unroll
  for (int i = 0; i < NB; ++i) {
    const int b = warp + WARPS * i;
    if (b >= blocks) break;
    uint4 a[MT][2];                                  // rows beyond T repeat the last one; their results are dropped
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int r = 0; r < 2; ++r)
        a[m][r] = *(reinterpret_cast<const uint4*>(x + (int64_t)min(16 * m + g + 8 * r, T - 1) * K + b * KB) + t);
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const uint32_t lo[4] = {a[m][0].x, a[m][1].x, a[m][0].y, a[m][1].y}, hi[4] = {a[m][0].z, a[m][1].z, a[m][0].w, a[m][1].w};
#pragma unroll
      for (int f = 0; f < NF; ++f) {
        mma(acc[m][f], lo, wf[i][f].x, wf[i][f].y);
        mma(acc[m][f], hi, wf[i][f].z, wf[i][f].w);
      }
    }
  }
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int f = 0; f < NF; ++f)
#pragma unroll
      for (int r = 0; r < 2; ++r)
        *reinterpret_cast<float2*>(&part[warp][16 * m + g + 8 * r][8 * f + 2 * t]) = make_float2(acc[m][f][2 * r], acc[m][f][2 * r + 1]);
  __syncthreads();
  constexpr int PAIRS = NF * 4;
  for (int e = threadIdx.x; e < MT * 16 * PAIRS; e += WARPS * 32) {
    const int row = e / PAIRS, c = 2 * (e % PAIRS);
    if (row >= T || n0 + c >= N) continue;
    const __nv_bfloat162 bb = *reinterpret_cast<const __nv_bfloat162*>(bias + n0 + c);
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int k = 0; k < WARPS; ++k) {
      const float2 v = *reinterpret_cast<const float2*>(&part[k][row][c]);
      s0 += v.x; s1 += v.y;
    }
    s0 += __low2float(bb); s1 += __high2float(bb);
    if (GELU) { s0 = gelu(s0, __nv_bfloat16()); s1 = gelu(s1, __nv_bfloat16()); }
    *reinterpret_cast<uint32_t*>(y + (int64_t)row * N + n0 + c) = pack2(s0, s1);
  }
}

template <int MT, int NF, int NB>
cudaError_t launch(const void* x, const void* w, const void* b, int T, int K, int N, bool gelu, bool early, void* y, cudaStream_t s) {
  const dim3 grid((N + 8 * NF - 1) / (8 * NF));
  using B = __nv_bfloat16;
  return launch_stream(gelu ? skinny_kernel<MT, NF, NB, true> : skinny_kernel<MT, NF, NB, false>, grid, WARPS * 32, 0, s, early,
                       (const B*)x, (const B*)w, (const B*)b, T, K, N, (B*)y);
}

template <int MT>
cudaError_t launch_rows(const void* x, const void* w, const void* b, int T, int K, int N, bool gelu, bool early, void* y, int sms, cudaStream_t s) {
  const int nb = (K / KB + WARPS - 1) / WARPS;
  // 16 features per block read x half as often, 8 make more blocks.  What decides is how many blocks of 8 an SM would get: up to 16
  // tokens three are no worse than two of 16, with two token tiles a second one already is.  us per projection, weights from memory,
  // 8 against 16 features: 16 tokens, K 768, N 2304 2.58 and 2.62, N 3072 3.44 and 3.44, N 4096 4.28 and 3.61; 32 tokens, K 768, N 1024
  // 2.68 and 2.63, N 1536 2.97 and 2.71, N 2560 4.30 and 3.54; K 1024, N 1024 2.85 and 2.93, N 3072 5.41 and 4.70.  More columns
  // leave no registers for 16.
  if (nb <= 4)
    return N > 8 * sms * (MT == 1 ? 3 : 1) ? launch<MT, 2, 4>(x, w, b, T, K, N, gelu, early, y, s) : launch<MT, 1, 4>(x, w, b, T, K, N, gelu, early, y, s);
  if (nb <= 8) return launch<MT, 1, 8>(x, w, b, T, K, N, gelu, early, y, s);
  if (nb <= 12) return launch<MT, 1, 12>(x, w, b, T, K, N, gelu, early, y, s);
  return launch<MT, 1, 16>(x, w, b, T, K, N, gelu, early, y, s);
}

}  // namespace

}  // namespace tdb

using namespace tdb;

extern "C" {

// Every block reads all of x, so the line lies where that costs more than the library's tiles do.  us per projection, weights from
// memory, this kernel against the library's.  32 tokens: K 768 and N 768 2.5 and 3.3, N 2304 3.0 and 3.9, N 3072 4.1 and 4.2, K 3072
// and N 768 5.8 and 6.6; K 1024 and N 3072 4.7 and 4.7, N 4096 5.5 and 5.0 (where GELU in the epilogue saves a launch).  With three token
// tiles the narrow projections would still gain and the wide ones lose, 48 tokens: 3.2 and 3.3, 4.0 and 4.1, 4.8 and 4.4, 6.5 and
// 6.7; K 1024 5.6 and 4.8, 5.9 and 5.1; with four all lose (64 tokens: 3.5 and 3.3, 4.2 and 4.0, 5.6 and 4.4, 7.0 and 6.8).  Larger weights
// than those lose too: a pass of twelve layers of hidden size 1280, 32 tokens, without a limit, with it, and with the library for all 603, 548,
// 544; of 1536 682, 601, 595; six layers of 2048, 8 tokens 467, 435, 437, 32 tokens 497, 408, 408.  Passes of 8, 16 and 32 tokens with this kernel, and with
// the library: twelve layers of hidden size 384 324, 314, 322 and 384, 361, 362; of 640 392, 399, 419 and 465, 440, 435; and where
// encoder_short.cu does not come in because every layer is returned, the base model 635, 644, 668 and 843, 790, 785, the large one 1095, 1119, 1214
// and 1404, 1415, 1379.  K up to what a warp's registers hold.
int tdb_skinny_applies(int64_t T, int64_t K, int64_t N) {
  return T <= SKINNY_TOKENS && K % KB == 0 && K <= KB * WARPS * 16 && N % 8 == 0 && K * N <= 4500000;
}

int tdb_skinny(const void* x, const void* w, const void* b, int T, int K, int N, int gelu, int early, void* y, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  int sms = 0;
  if (const int rc = device_sms(&sms)) return rc;
  const cudaError_t e = T <= 16 ? launch_rows<1>(x, w, b, T, K, N, gelu, early, y, sms, s)
                                : launch_rows<2>(x, w, b, T, K, N, gelu, early, y, sms, s);
  return cuda_fail(e, "skinny projection launch");
}

}  // extern "C"
