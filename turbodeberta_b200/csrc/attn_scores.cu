// Attention with materialised position scores (the legacy operator form), bf16: the two position products arrive as tensors
// c2p_scores[q, r] = Q[q].Kr[r] and p2c_scores[k, r] = K[k].Qr[r] and are gathered,
//
//   score[q,k] = (Q[q].K[k] + c2p_scores[q, idx(q-k)] + p2c_scores[k, idx(q-k)]) * sm_scale
//
// (p2c at idx(k-q) with TDB_FLAG_P2C_MIRRORED).  Bound by the score tensors: 8 x 256 tokens of 12 heads bring 50 MB of them,
// against 1.6 GFLOP; so the products run on the warp-level tensor instruction, and the work is in the gather.  The distances of
// a 64 x 64 tile reach at most 127 neighbouring columns, so each of its c2p and p2c rows is one short run: the runs are copied
// to shared memory in 16-byte pieces and gathered there (WINDOW); the next tile comes in behind the gather, beside the exponentials
// and P.V.  Rows that are not 16-byte aligned are gathered from global
// memory, where a fragment register's 32 lanes are 8 short runs of c2p rows, or 4 of p2c rows, which the first-level cache
// takes one line at a time.  One block of four warps owns 64 query rows and walks key tiles of 64; three blocks per SM cover
// each other's copies.  P keeps two bf16 terms (value and remainder) for P.V, so nothing but the output is rounded to bf16.
// 8 x 256 tokens, 12 heads: CUDA-core kernel 142 us per call, gathered from global memory 46, with windows 38 (kernel 22.9 us); the
// columns kept as byte offsets, copies by running pointers and masks in the last tile only took 40 % of the instructions out:
// 34.0 (kernel 19.0 us, 2.6 TB/s of scores).  Three blocks of four warps per SM are now what it waits for: a tile's chain from its
// windows to P.V.  Tiles of 32 keys, twice in shared memory, were slower (kernel 24.8 us: as many instructions again per key), and
// the index table read a tile ahead changed nothing.
#include "attn_blocks.cuh"
#include "attn_warp_mma.cuh"
#include "ptx_sm100.cuh"
#include <float.h>
#include <math_constants.h>

namespace tdb {

namespace {

constexpr int WCH = 17, WP = 136;                    // 16-byte pieces of a score row's window, its pitch in elements (conflict-free)

__device__ __forceinline__ float bf(unsigned short h) { return __uint_as_float((uint32_t)h << 16); }
__device__ __forceinline__ unsigned short at_byte(const unsigned short* p, int offset) {
  return *reinterpret_cast<const unsigned short*>(reinterpret_cast<const char*>(p) + offset);
}

// As stage(), along a running pointer: fewer instructions, where those are what a tile costs.
__device__ __forceinline__ void stage_along(__nv_bfloat16* dst, const __nv_bfloat16* src, int64_t pitch, int rows) {
  const int c = threadIdx.x & 7, row = threadIdx.x >> 3;
  constexpr int STEP = S_THREADS / 8;
  const __nv_bfloat16* from = src + row * pitch + c * 8;
  const uint32_t to = saddr(dst + row * SP + c * 8);
#pragma unroll
  for (int i = 0; i < ST / STEP; ++i, from += STEP * pitch) {
    const bool real = row + i * STEP < rows;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to + 2u * i * STEP * SP), "l"(real ? from : src), "r"(real ? 16 : 0) : "memory");
  }
}

// The columns [lo, lo + 8 * pieces) of 64 rows to shared memory: sixteen threads per row, and one piece that they leave.
__device__ __forceinline__ void stage_window(unsigned short* dst, const unsigned short* src, int64_t pitch, int rows, int lo, int pieces) {
  auto copy = [](uint32_t to, const unsigned short* from) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(from) : "memory");
  };
  const int c = threadIdx.x & 15, row = threadIdx.x >> 4;
  constexpr int STEP = S_THREADS / 16;
  const unsigned short* from = src + row * pitch + lo + c * 8;
  const uint32_t to = saddr(dst + row * WP + c * 8);
  const int real = c < pieces ? rows : 0;
#pragma unroll
  for (int i = 0; i < ST / STEP; ++i, from += STEP * pitch)
    if (row + i * STEP < real) copy(to + 2u * i * STEP * WP, from);
  if (pieces == WCH && (int)threadIdx.x < min(ST, rows))
    copy(saddr(dst + threadIdx.x * WP + 8 * (WCH - 1)), src + threadIdx.x * pitch + lo + 8 * (WCH - 1));
}

template <bool C2P, bool P2C, bool WINDOW>
__global__ void __launch_bounds__(S_THREADS, 3) attn_scores_kernel(const AttnParams p) {
  extern __shared__ __align__(16) unsigned char smem[];
  __nv_bfloat16* const sQ = reinterpret_cast<__nv_bfloat16*>(smem);
  __nv_bfloat16 *const sK = sQ + ST * SP, *const sV = sK + ST * SP;      // V twice: the next tile comes in beside P.V
  unsigned short* const wC = reinterpret_cast<unsigned short*>(sV + 2 * ST * SP);
  unsigned short* const wP = wC + (C2P ? ST * WP : 0);
  // column of distance q0 - k0 - 63 + x in the c2p and the p2c rows, in bytes from the window's (or the row's) beginning
  __shared__ int sAt[2][2 * ST];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int s = longest_first(p, blockIdx.z), h = blockIdx.y, q0 = blockIdx.x * ST;
  int len, rows;
  int64_t tok0;
  int b;
  if (!sequence_of(p, s, len, rows, tok0, b) || q0 >= rows) return;
  __nv_bfloat16* const ob = reinterpret_cast<__nv_bfloat16*>(p.o) + b * p.o_sb + tok0 * p.o_st + h * p.o_sh;
  float* const lse = p.lse ? p.lse + b * p.lse_sb + h * p.lse_sh + tok0 : nullptr;
  using bf16 = __nv_bfloat16;
  const bf16* const qb = reinterpret_cast<const bf16*>(p.q) + b * p.q_sb + tok0 * p.q_st + h * p.q_sh;
  const bf16* const kb = reinterpret_cast<const bf16*>(p.k) + b * p.k_sb + tok0 * p.k_st + h * p.k_sh;
  const bf16* const vb = reinterpret_cast<const bf16*>(p.v) + b * p.v_sb + tok0 * p.v_st + h * p.v_sh;
  const unsigned short* const c2p = C2P ? reinterpret_cast<const unsigned short*>(p.c2p_scores) + b * p.c2p_sb + tok0 * p.c2p_st + h * p.c2p_sh : nullptr;
  const unsigned short* const p2c = P2C ? reinterpret_cast<const unsigned short*>(p.p2c_scores) + b * p.p2c_sb + tok0 * p.p2c_st + h * p.p2c_sh : nullptr;
  const int dm = p.idx_delta_max;
  auto row_of = [&](int delta) { return p.idx[delta < -dm ? 0 : (delta > dm ? 2 * dm : delta + dm)]; };

  // this thread's rows r0 and r0 + 8 of the block, its keys 2 (lane % 4) + {0, 1} of every group of eight
  const int r0 = warp * 16 + lane / 4, kc = 2 * (lane % 4);
  float o[8][4], m[2] = {-FLT_MAX, -FLT_MAX}, l[2] = {0.f, 0.f};         // not -inf: see attn_simt.cu
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[i][e] = 0.f;
  const float sl2 = p.sm_scale * 1.4426950408889634f;

  if (q0 < len) {
    stage_along(sQ, qb + (int64_t)q0 * p.q_st, p.q_st, len - q0);
    const bool mirrored = p.flags & TDB_FLAG_P2C_MIRRORED;
    auto load_tile = [&](int k0, int buf) {
      stage_along(sK, kb + (int64_t)k0 * p.k_st, p.k_st, len - k0);
      stage_along(sV + buf * ST * SP, vb + (int64_t)k0 * p.v_st, p.v_st, len - k0);
      int lo_c = 0, lo_p = 0;
      if (WINDOW) {                                  // the index grows with the distance: the ends of its range are the window's
        if (C2P) {
          const int hi = row_of(q0 - k0 + ST - 1);
          lo_c = row_of(q0 - k0 - (ST - 1)) & ~7;
          stage_window(wC, c2p + (int64_t)q0 * p.c2p_st, p.c2p_st, len - q0, lo_c, (hi - lo_c) / 8 + 1);
        }
        if (P2C) {
          const int d = mirrored ? k0 - q0 : q0 - k0, hi = row_of(d + ST - 1);
          lo_p = row_of(d - (ST - 1)) & ~7;
          stage_window(wP, p2c + (int64_t)k0 * p.p2c_st, p.p2c_st, len - k0, lo_p, (hi - lo_p) / 8 + 1);
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      const int delta = q0 - k0 - (ST - 1) + (int)threadIdx.x;
      if (C2P) sAt[0][threadIdx.x] = 2 * (row_of(delta) - lo_c);
      if (P2C) sAt[1][threadIdx.x] = 2 * (row_of(mirrored ? -delta : delta) - lo_p);
    };
    load_tile(0, 0);
    uint32_t qf[4][4];
    // rows beyond the sequence read the last row's scores: in bounds, and their results are dropped
    const int qr[2] = {min(q0 + r0, len - 1), min(q0 + r0 + 8, len - 1)};
    for (int k0 = 0, buf = 0; k0 < len; k0 += ST, buf ^= 1) {
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
      const bool partial = k0 + ST > len;            // keys beyond the sequence
      if (k0 == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) ldsm4(qf[i], sQ + (warp * 16 + (lane & 15)) * SP + 16 * i + 8 * (lane >> 4));
      }
      float sc[8][4];
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        // gathers first: 32 loads in flight behind the products
        unsigned short gc[4][4], gp[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int kl = 8 * (4 * half + i) + kc + (e & 1), rl = r0 + 8 * (e >> 1);
            const int x = rl - kl + ST - 1;
            if (C2P) gc[i][e] = WINDOW ? at_byte(wC + rl * WP, sAt[0][x]) : __ldg(c2p + (int64_t)qr[e >> 1] * p.c2p_st + sAt[0][x] / 2);
            if (P2C) gp[i][e] = WINDOW ? at_byte(wP + kl * WP, sAt[1][x]) : __ldg(p2c + (int64_t)min(k0 + kl, len - 1) * p.p2c_st + sAt[1][x] / 2);
          }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) sc[4 * half + i][e] = 0.f;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            uint32_t kf[4];                          // keys 8j..8j+15, columns 16kk..+15
            const int j = 4 * half + 2 * i;
            ldsm4(kf, sK + (8 * j + (lane & 7) + 8 * (lane >> 4)) * SP + 16 * kk + 8 * ((lane >> 3) & 1));
            mma(sc[j], qf[kk], kf[0], kf[1]);
            mma(sc[j + 1], qf[kk], kf[2], kf[3]);
          }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            float x = sc[4 * half + i][e];
            if (C2P) x += bf(gc[i][e]);
            if (P2C) x += bf(gp[i][e]);
            sc[4 * half + i][e] = x * sl2;
          }
      }
      __syncthreads();                               // K and the windows have been read; V's other buffer, in the tile before
      if (k0 + ST < len) load_tile(k0 + ST, buf ^ 1);
      if (partial) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (k0 + 8 * i + kc + (e & 1) >= len) sc[i][e] = -CUDART_INF_F;
      }
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        float mx = m[r];
#pragma unroll
        for (int i = 0; i < 8; ++i) mx = fmaxf(mx, fmaxf(sc[i][2 * r], sc[i][2 * r + 1]));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const float corr = ptx::ex2(m[r] - mx);
        m[r] = mx;
        float sum = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int e = 2 * r; e < 2 * r + 2; ++e) { sc[i][e] = ptx::ex2(sc[i][e] - mx); sum += sc[i][e]; }
        l[r] = l[r] * corr + sum;
#pragma unroll
        for (int i = 0; i < 8; ++i) { o[i][2 * r] *= corr; o[i][2 * r + 1] *= corr; }
      }
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {               // keys 16kk..+15
        const float *a = sc[2 * kk], *c = sc[2 * kk + 1];
        uint32_t hi[4] = {pack2(a[0], a[1]), pack2(a[2], a[3]), pack2(c[0], c[1]), pack2(c[2], c[3])}, lo[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float* v = (e < 2 ? a : c) + 2 * (e & 1);
          lo[e] = pack2(v[0] - __uint_as_float(hi[e] << 16), v[1] - __uint_as_float(hi[e] & 0xffff0000u));
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint32_t vf[4];                            // keys 16kk..+15, columns 16i..+15
          ldsm4t(vf, sV + buf * ST * SP + (16 * kk + (lane & 15)) * SP + 16 * i + 8 * (lane >> 4));
          mma(o[2 * i], hi, vf[0], vf[1]);
          mma(o[2 * i + 1], hi, vf[2], vf[3]);
          mma(o[2 * i], lo, vf[0], vf[1]);
          mma(o[2 * i + 1], lo, vf[2], vf[3]);
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int row = q0 + r0 + 8 * r;
    float sum = l[r];
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    if (row >= rows) continue;
    const bool valid = row < len;                    // padded query rows of the padded form: zeros
    const float inv = valid ? 1.f / sum : 0.f;
    uint32_t* const dst = reinterpret_cast<uint32_t*>(ob + (int64_t)row * p.o_st + kc);
#pragma unroll
    for (int i = 0; i < 8; ++i) dst[4 * i] = valid ? pack2(o[i][2 * r] * inv, o[i][2 * r + 1] * inv) : 0u;
    if (lse && lane % 4 == 0) lse[row] = valid ? m[r] * 0.6931471805599453f + logf(sum) : 0.f;
  }
}

}  // namespace

template <bool C2P, bool P2C, bool WINDOW>
static int launch_scores(const AttnParams& p, dim3 grid, cudaStream_t s) {
  constexpr int SMEM = (ST * SP * 4 + (WINDOW ? ((C2P ? 1 : 0) + (P2C ? 1 : 0)) * ST * WP : 0)) * 2;
  auto kern = attn_scores_kernel<C2P, P2C, WINDOW>;
  const int rc = opt_in_smem(reinterpret_cast<const void*>(kern), SMEM);
  if (rc) return rc;
  kern<<<grid, S_THREADS, SMEM, s>>>(p);
  return cuda_fail(cudaGetLastError(), "attn_scores launch");
}

int launch_attn_scores(const AttnParams& p, cudaStream_t s) {
  dim3 grid((p.L + ST - 1) / ST, p.H, p.n_seqs);
  const bool c2p = p.flags & TDB_FLAG_C2P, p2c = p.flags & TDB_FLAG_P2C;
  // 16-byte pieces of every row: aligned bases, strides and row length
  auto pieces = [&](const void* x, int64_t sb, int64_t st, int64_t sh) {
    return (reinterpret_cast<uintptr_t>(x) & 15) == 0 && ((sb | st | sh | p.two_span) & 7) == 0;
  };
  const bool window = (!c2p || pieces(p.c2p_scores, p.c2p_sb, p.c2p_st, p.c2p_sh)) && (!p2c || pieces(p.p2c_scores, p.p2c_sb, p.p2c_st, p.p2c_sh));
  if (c2p && p2c) return window ? launch_scores<true, true, true>(p, grid, s) : launch_scores<true, true, false>(p, grid, s);
  if (c2p) return window ? launch_scores<true, false, true>(p, grid, s) : launch_scores<true, false, false>(p, grid, s);
  return window ? launch_scores<false, true, true>(p, grid, s) : launch_scores<false, true, false>(p, grid, s);
}

}  // namespace tdb
