// Sequences of at most 64 tokens, bf16, projected tables: one block of four warps per sequence and head.
//
// Such a call is bound by latency, not by any unit: one score tile per head.  The persistent tensor-memory kernel takes 7.3 us
// for it (scheduler ring, tensor-memory allocation and a chain of nine hand-offs between its roles); here the tile is four
// barriers long.  Both bands are formed by the warp-level tensor instruction, q.Kr for the 80 distances of a warp's 16 query
// rows and k.Qr for those of 16 key rows, kept in fp32 in shared memory and read back along the diagonal:
//
//   s[i][j] = (Q[i].K[j] + C[i][i - j] + P2[j][i - j]) * scale ;  P as bf16 ;  O = P . V
//
// 40 tokens, 12 heads: 4.2 us.
#include "attn_warp_mma.cuh"
#include <math_constants.h>

namespace tdb {

namespace {

constexpr int BP = 84;                               // pitch of a band row, in floats (80 distances)

template <bool C2P, bool P2C>
__global__ void __launch_bounds__(S_THREADS) attn_small_kernel(const AttnParams p) {
  using bf16 = __nv_bfloat16;
  extern __shared__ __align__(16) unsigned char smem[];
  bf16* const sQ = reinterpret_cast<bf16*>(smem);
  bf16 *const sK = sQ + ST * SP, *const sV = sK + ST * SP, *const sKr = sV + ST * SP;
  bf16* const sQr = sKr + (C2P ? 2 * ST * SP : 0);
  float* const bC = reinterpret_cast<float*>(sQr + (P2C ? 2 * ST * SP : 0));
  float* const bP = bC + (C2P ? ST * BP : 0);
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, h = blockIdx.x, b = blockIdx.y;
  wait_for_stream();
  let_next_start();
  int len, rows_out;                                 // valid tokens, rows that exist in the output
  int64_t tok0 = 0;
  int64_t seq = b;
  if (p.varlen) {
    tok0 = p.cu_seqlens[b]; seq = 0;
    rows_out = len = min(p.cu_seqlens[b + 1] - (int)tok0, ST);
  } else {
    len = p.seqlens ? p.seqlens[b] : p.L;
    len = len < 0 ? 0 : (len > p.L ? p.L : len);
    rows_out = p.L;
  }
  const bf16* const qb = reinterpret_cast<const bf16*>(p.q) + seq * p.q_sb + tok0 * p.q_st + h * p.q_sh;
  const bf16* const kb = reinterpret_cast<const bf16*>(p.k) + seq * p.k_sb + tok0 * p.k_st + h * p.k_sh;
  const bf16* const vb = reinterpret_cast<const bf16*>(p.v) + seq * p.v_sb + tok0 * p.v_st + h * p.v_sh;
  bf16* const ob = reinterpret_cast<bf16*>(p.o) + seq * p.o_sb + tok0 * p.o_st + h * p.o_sh;
  float* const lse = p.lse ? p.lse + seq * p.lse_sb + h * p.lse_sh + tok0 : nullptr;
  if (len <= 0) {                                    // nothing but padding: zeros
    for (int e = threadIdx.x; e < rows_out * 8; e += S_THREADS)
      *reinterpret_cast<uint4*>(ob + (e >> 3) * p.o_st + (e & 7) * 8) = make_uint4(0, 0, 0, 0);
    if (lse)
      for (int e = threadIdx.x; e < rows_out; e += S_THREADS) lse[e] = 0.f;
    return;
  }
  stage(sQ, qb, p.q_st, len);
  stage(sK, kb, p.k_st, len);
  const int64_t table = ((int64_t)h * p.exp_rows + p.exp_delta_max - (ST - 1)) * 64;       // row x: distance x - 63
  if (C2P) {
    const bf16* t = reinterpret_cast<const bf16*>(p.kr_exp) + table;
    stage(sKr, t, 64, ST);
    stage(sKr + ST * SP, t + ST * 64, 64, ST);
  }
  if (P2C) {
    const bf16* t = reinterpret_cast<const bf16*>(p.qr_exp) + table;
    stage(sQr, t, 64, ST);
    stage(sQr + ST * SP, t + ST * 64, 64, ST);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  stage(sV, vb, p.v_st, len);
  asm volatile("cp.async.commit_group;" ::: "memory");
  asm volatile("cp.async.wait_group 1;" ::: "memory");
  __syncthreads();

  const int r0 = lane / 4, kc = 2 * (lane % 4);      // rows r0, r0 + 8 of the warp's sixteen; columns kc, kc + 1 of every eight
  const bool rows = 16 * warp < len;                 // the warp has query (and key) rows at all
  uint32_t qf[4][4];
  float* const myC = bC + 16 * warp * BP;
  if (rows) {
#pragma unroll
    for (int i = 0; i < 4; ++i) ldsm4(qf[i], sQ + (16 * warp + (lane & 15)) * SP + 16 * i + 8 * (lane >> 4));
    // one band: 16 rows (fragments a) against the 80 table rows from x0
    auto band = [&](float* dst, const uint32_t (*a)[4], const bf16* tab, int x0) {
#pragma unroll
      for (int n = 0; n < 5; ++n) {
        float d[2][4] = {};
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          uint32_t kf[4];
          ldsm4(kf, tab + (x0 + 16 * n + (lane & 7) + 8 * (lane >> 4)) * SP + 16 * kk + 8 * ((lane >> 3) & 1));
          mma(d[0], a[kk], kf[0], kf[1]);
          mma(d[1], a[kk], kf[2], kf[3]);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int e = 0; e < 2; ++e)
            *reinterpret_cast<float2*>(dst + (r0 + 8 * e) * BP + 16 * n + 8 * i + kc) = make_float2(d[i][2 * e], d[i][2 * e + 1]);
      }
    };
    if (C2P) band(myC, qf, sKr, 16 * warp);          // C[i][x]: distance x + 16 warp - 63
    if (P2C) {
      uint32_t kf[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) ldsm4(kf[i], sK + (16 * warp + (lane & 15)) * SP + 16 * i + 8 * (lane >> 4));
      band(bP + 16 * warp * BP, kf, sQr, 48 - 16 * warp);      // P2[j][x]: distance x - 15 - 16 warp
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  if (rows) {
    float sc[8][4], o[8][4];
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) sc[j][e] = o[j][e] = 0.f;
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
#pragma unroll
      for (int j = 0; j < 8; j += 2) {
        uint32_t kf[4];
        ldsm4(kf, sK + (8 * j + (lane & 7) + 8 * (lane >> 4)) * SP + 16 * kk + 8 * ((lane >> 3) & 1));
        mma(sc[j], qf[kk], kf[0], kf[1]);
        mma(sc[j + 1], qf[kk], kf[2], kf[3]);
      }
    const float sl2 = p.sm_scale * 1.4426950408889634f;
    float m[2] = {-CUDART_INF_F, -CUDART_INF_F}, l[2] = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int il = r0 + 8 * (e >> 1), kl = 8 * j + kc + (e & 1);
        float x = sc[j][e];
        if (C2P) x += myC[il * BP + il - kl + ST - 1];
        if (P2C) x += bP[kl * BP + 16 * warp + il - (kl & 15) + 15];       // rows beyond the sequence are masked just below
        x = kl < len ? x * sl2 : -CUDART_INF_F;
        sc[j][e] = x;
        m[e >> 1] = fmaxf(m[e >> 1], x);
      }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      m[r] = fmaxf(m[r], __shfl_xor_sync(0xffffffffu, m[r], 1));
      m[r] = fmaxf(m[r], __shfl_xor_sync(0xffffffffu, m[r], 2));
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int e = 2 * r; e < 2 * r + 2; ++e) { sc[j][e] = exp2f(sc[j][e] - m[r]); l[r] += sc[j][e]; }
      l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
      l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
    }
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {                 // keys 16kk..+15
      const float *a = sc[2 * kk], *c = sc[2 * kk + 1];
      const uint32_t pf[4] = {pack2(a[0], a[1]), pack2(a[2], a[3]), pack2(c[0], c[1]), pack2(c[2], c[3])};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint32_t vf[4];
        ldsm4t(vf, sV + (16 * kk + (lane & 15)) * SP + 16 * i + 8 * (lane >> 4));
        mma(o[2 * i], pf, vf[0], vf[1]);
        mma(o[2 * i + 1], pf, vf[2], vf[3]);
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int row = 16 * warp + r0 + 8 * r;
      if (row >= len) continue;
      const float inv = 1.f / l[r];
      uint32_t* const dst = reinterpret_cast<uint32_t*>(ob + row * p.o_st + kc);
#pragma unroll
      for (int i = 0; i < 8; ++i) dst[4 * i] = pack2(o[i][2 * r] * inv, o[i][2 * r + 1] * inv);
      if (lse && lane % 4 == 0) lse[row] = m[r] * 0.6931471805599453f + logf(l[r]);
    }
  }
  // padded query rows: zeros
  for (int e = threadIdx.x + len * 8; e < rows_out * 8; e += S_THREADS)
    *reinterpret_cast<uint4*>(ob + (e >> 3) * p.o_st + (e & 7) * 8) = make_uint4(0, 0, 0, 0);
  if (lse)
    for (int e = threadIdx.x + len; e < rows_out; e += S_THREADS) lse[e] = 0.f;
}

template <bool C2P, bool P2C>
int launch_small(const AttnParams& p, cudaStream_t s) {
  constexpr int TERMS = (C2P ? 1 : 0) + (P2C ? 1 : 0), SMEM = ST * SP * 2 * (3 + 2 * TERMS) + ST * BP * 4 * TERMS;
  auto kern = attn_small_kernel<C2P, P2C>;
  if (SMEM > 48 * 1024) {
    const int rc = opt_in_smem(reinterpret_cast<const void*>(kern), SMEM);
    if (rc) return rc;
  }
  return cuda_fail(launch_early(kern, dim3(p.H, p.n_seqs), S_THREADS, SMEM, s, p), "attn_small launch");
}

}  // namespace

// The grid has one block per sequence and head.  Packed sequences only where the longest is known: with a caller's max_seqlen
// they go to the other kernel, which takes any lengths the offsets may turn out to have.
bool small_applicable(const AttnParams& p) { return (!p.varlen || p.lengths_known) && p.L <= ST && p.n_seqs <= 65535; }

int launch_attn_small(const AttnParams& p, cudaStream_t s) {
  const bool c2p = p.flags & TDB_FLAG_C2P, p2c = p.flags & TDB_FLAG_P2C;
  if (c2p && p2c) return launch_small<true, true>(p, s);
  if (c2p) return launch_small<true, false>(p, s);
  if (p2c) return launch_small<false, true>(p, s);
  return launch_small<false, false>(p, s);
}

}  // namespace tdb
