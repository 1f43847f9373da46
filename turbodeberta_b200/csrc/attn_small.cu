// Sequences of at most 128 tokens, bf16, projected tables: one block per sequence, head and 64 query rows.
//
// Such a call is bound by latency, not by any unit: one or two score tiles per block.  The persistent tensor-memory kernel takes 7.3 us
// for 64 tokens and 7.8 for 128 (scheduler ring, tensor-memory allocation and a chain of nine hand-offs between its roles); here one tile
// is two barriers long, and two are six.  Both bands are formed by the warp-level tensor instruction, q.Kr for the 80 distances of a warp's 16 query
// rows and k.Qr for those of 16 key rows, kept in fp32 in shared memory and read back along the diagonal:
//
//   s[i][j] = (Q[i].K[j] + C[i][i - j] + P2[j][i - j]) * scale ;  P as bf16 ;  O = P . V
//
// The second tile's operands come in beside the diagonal reads of the first.  Table rows are copied one by one, so that tables which
// belong to one call are taken as they are, by index (DIRECT), and not expanded first, which is a launch and 2.8 us.
#include "attn_warp_mma.cuh"
#include <math_constants.h>

namespace tdb {

namespace {

constexpr int BP = 84;                               // pitch of a band row, in floats (80 distances)
// Warps per 16 query rows.  Two share the bands' columns and take 32 keys of a tile each; with one tile that gains what meeting for
// maxima, sums and outputs costs (4 x 64 tokens: 16.1 us per call with one, 16.4 with two).
template <int TILES> constexpr int halves_of = TILES;
template <int TILES> constexpr int threads_of = 128 * halves_of<TILES>;
constexpr int OP = 68;                               // pitch of an output row on its way from one of the two to the other

template <bool C2P, bool P2C, int TILES, bool DIRECT>
__global__ void __launch_bounds__(threads_of<TILES>) attn_small_kernel(const AttnParams p) {
  constexpr int HALVES = halves_of<TILES>, THREADS = threads_of<TILES>, KEYS = ST / HALVES;
  using bf16 = __nv_bfloat16;
  extern __shared__ __align__(16) unsigned char smem[];
  bf16* const sQ = reinterpret_cast<bf16*>(smem);
  bf16 *const sK = sQ + ST * SP, *const sV = sK + ST * SP, *const sKr = sV + ST * SP;
  bf16* const sQr = sKr + (C2P ? 2 * ST * SP : 0);
  float* const bC = reinterpret_cast<float*>(sQr + (P2C ? 2 * ST * SP : 0));
  float* const bP = bC + (C2P ? ST * BP : 0);
  const int warp = threadIdx.x / 32 % 4, half = threadIdx.x / 128, lane = threadIdx.x % 32, h = blockIdx.x, b = blockIdx.y, q0 = TILES > 1 ? blockIdx.z * ST : 0;
  wait_for_stream();
  let_next_start();
  int len, rows_out;                                 // valid tokens, rows that exist in the output
  int64_t tok0 = 0;
  int64_t seq = b;
  if (p.varlen) {
    tok0 = p.cu_seqlens[b]; seq = 0;
    rows_out = len = min(p.cu_seqlens[b + 1] - (int)tok0, TILES * ST);
  } else {
    len = p.seqlens ? p.seqlens[b] : p.L;
    len = len < 0 ? 0 : (len > p.L ? p.L : len);
    rows_out = p.L;
  }
  const bf16* const qb = reinterpret_cast<const bf16*>(p.q) + seq * p.q_sb + (tok0 + q0) * p.q_st + h * p.q_sh;
  const bf16* const kb = reinterpret_cast<const bf16*>(p.k) + seq * p.k_sb + tok0 * p.k_st + h * p.k_sh;
  const bf16* const vb = reinterpret_cast<const bf16*>(p.v) + seq * p.v_sb + tok0 * p.v_st + h * p.v_sh;
  bf16* const ob = reinterpret_cast<bf16*>(p.o) + seq * p.o_sb + (tok0 + q0) * p.o_st + h * p.o_sh;
  float* const lse = p.lse ? p.lse + seq * p.lse_sb + h * p.lse_sh + tok0 + q0 : nullptr;
  const int own = min(len - q0, ST);                 // valid query rows of this block
  auto zero_padding = [&](int from) {                // query rows that exist in the output only
    for (int e = threadIdx.x + from * 8; e < min(rows_out - q0, ST) * 8; e += THREADS)
      *reinterpret_cast<uint4*>(ob + (e >> 3) * p.o_st + (e & 7) * 8) = make_uint4(0, 0, 0, 0);
    if (lse)
      for (int e = threadIdx.x + from; e < min(rows_out - q0, ST); e += THREADS) lse[e] = 0.f;
  };
  if (own <= 0) {
    zero_padding(0);
    return;
  }

  // The 128 rows of a head's table for the distances d0 .. d0 + 127.
  auto stage_table = [&](bf16* dst, const void* expanded, const void* table, int d0) {
    if constexpr (!DIRECT) {
      const bf16* t = reinterpret_cast<const bf16*>(expanded) + ((int64_t)h * p.exp_rows + p.exp_delta_max + d0) * 64;
      stage<THREADS>(dst, t, 64, ST);
      stage<THREADS>(dst + ST * SP, t + ST * 64, 64, ST);
    } else {
      constexpr int STEP = THREADS / 8, N = 2 * ST / STEP;
      const int dm = p.idx_delta_max, c = threadIdx.x & 7, row = threadIdx.x >> 3;
      const bf16* t = reinterpret_cast<const bf16*>(table) + (int64_t)h * p.two_span * 64 + c * 8;
      int at[N];
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const int d = d0 + row + i * STEP;
        at[i] = p.idx[d < -dm ? 0 : (d > dm ? 2 * dm : d + dm)];
      }
#pragma unroll
      for (int i = 0; i < N; ++i)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(saddr(dst + (row + i * STEP) * SP + c * 8)), "l"(t + at[i] * 64) : "memory");
    }
  };
  // K and the tables' windows (row x: distance q0 - k0 - 63 + x), then V; of the second tile V goes where Q was
  auto load_tile = [&](int t) {
    const int k0 = t * ST;
    stage<THREADS>(sK, kb + (int64_t)k0 * p.k_st, p.k_st, len - k0);
    if (C2P) stage_table(sKr, p.kr_exp, p.kr, q0 - k0 - (ST - 1));
    if (P2C) stage_table(sQr, p.qr_exp, p.qr, q0 - k0 - (ST - 1));
    asm volatile("cp.async.commit_group;" ::: "memory");
    stage<THREADS>(t ? sQ : sV, vb + (int64_t)k0 * p.v_st, p.v_st, len - k0);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  stage<THREADS>(sQ, qb, p.q_st, len - q0);
  load_tile(0);
  zero_padding(own);

  const int r0 = lane / 4, kc = 2 * (lane % 4);      // rows r0, r0 + 8 of the warp's sixteen; columns kc, kc + 1 of every eight
  const bool rows = 16 * warp < own;                 // the warp has query rows at all
  uint32_t qf[4][4];
  float* const myC = bC + 16 * warp * BP;
  float sc[TILES * KEYS / 8][4];                     // keys KEYS * half + 8 j + kc, + 1 of a tile
#pragma unroll
  for (int j = 0; j < TILES * KEYS / 8; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) sc[j][e] = 0.f;
  const float sl2 = p.sm_scale * 1.4426950408889634f;
  float m[2] = {-CUDART_INF_F, -CUDART_INF_F}, l[2] = {0.f, 0.f};
#pragma unroll
  for (int t = 0; t < TILES; ++t) {
    const int k0 = t * ST;
    if (t > 0 && k0 >= len) break;
    asm volatile("cp.async.wait_group 1;" ::: "memory");           // all but the last V
    __syncthreads();                                               // also: the bands of the tile before have been read
    // of one band, 16 rows (fragments a) against the 80 table rows from x0: the columns of pieces n0 .. n1 - 1 of sixteen
    auto band = [&](float* dst, const uint32_t (*a)[4], const bf16* tab, int x0, int n0, int n1) {
#pragma unroll
      for (int n = n0; n < n1; ++n) {
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
    auto scores = [&]() {
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
#pragma unroll
        for (int j = 0; j < KEYS / 8; j += 2) {
          uint32_t kf[4];
          ldsm4(kf, sK + (KEYS * half + 8 * j + (lane & 7) + 8 * (lane >> 4)) * SP + 16 * kk + 8 * ((lane >> 3) & 1));
          mma(sc[KEYS / 8 * t + j], qf[kk], kf[0], kf[1]);
          mma(sc[KEYS / 8 * t + j + 1], qf[kk], kf[2], kf[3]);
        }
    };
    if (rows) {
      if (t == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) ldsm4(qf[i], sQ + (16 * warp + (lane & 15)) * SP + 16 * i + 8 * (lane >> 4));
      }
      if (C2P) {                                     // C[i][x]: distance x + 16 warp - 63 (+ q0 - k0)
        if (half == 0) band(myC, qf, sKr, 16 * warp, 0, HALVES == 1 ? 5 : 3);
        else band(myC, qf, sKr, 16 * warp, 3, 5);
      }
      if (TILES > 1) scores();                       // K's place is taken below
    }
    if (P2C && k0 + 16 * warp < len) {
      uint32_t kf[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) ldsm4(kf[i], sK + (16 * warp + (lane & 15)) * SP + 16 * i + 8 * (lane >> 4));
      // P2[j][x]: distance x - 15 - 16 warp (+ q0 - k0)
      if (half == 0) band(bP + 16 * warp * BP, kf, sQr, 48 - 16 * warp, 0, HALVES == 1 ? 5 : 2);
      else band(bP + 16 * warp * BP, kf, sQr, 48 - 16 * warp, 2, 5);
    }
    if (TILES == 1) asm volatile("cp.async.wait_all;" ::: "memory");          // V, which nothing below waits for then
    __syncthreads();
    if (t + 1 < TILES && k0 + ST < len) load_tile(t + 1);
    if (rows) {
      if (TILES == 1) scores();
#pragma unroll
      for (int j = 0; j < KEYS / 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int il = r0 + 8 * (e >> 1), kl = KEYS * half + 8 * j + kc + (e & 1);
          float x = sc[KEYS / 8 * t + j][e];
          if (C2P) x += myC[il * BP + il - kl + ST - 1];
          if (P2C) x += bP[kl * BP + 16 * warp + il - (kl & 15) + 15];       // rows beyond the sequence are masked just below
          x = k0 + kl < len ? x * sl2 : -CUDART_INF_F;
          sc[KEYS / 8 * t + j][e] = x;
          m[e >> 1] = fmaxf(m[e >> 1], x);
        }
    }
  }
  // the two warps of a row agree on its maximum; the row's sums and outputs meet below
  float* const ex = reinterpret_cast<float*>(sK);    // [half][row]: K is not needed any more
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    m[r] = fmaxf(m[r], __shfl_xor_sync(0xffffffffu, m[r], 1));
    m[r] = fmaxf(m[r], __shfl_xor_sync(0xffffffffu, m[r], 2));
    if (HALVES == 2 && lane % 4 == 0) ex[half * ST + 16 * warp + r0 + 8 * r] = m[r];
  }
  if (TILES > 1) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();                                 // the maxima and V are there, and the bands have been read
  }
  float o[8][4] = {};
  if (rows) {
#pragma unroll
    for (int r = 0; r < 2; ++r)                      // finite: key 0 is valid
      if (HALVES == 2) m[r] = fmaxf(m[r], ex[(half ^ 1) * ST + 16 * warp + r0 + 8 * r]);
#pragma unroll
    for (int t = 0; t < TILES; ++t) {
      if (t * ST + KEYS * half >= len) break;
#pragma unroll
      for (int j = KEYS / 8 * t; j < KEYS / 8 * (t + 1); ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) { sc[j][e] = exp2f(sc[j][e] - m[e >> 1]); l[e >> 1] += sc[j][e]; }
      const bf16* const v = (t ? sQ : sV) + KEYS * half * SP;
#pragma unroll
      for (int kk = 0; kk < KEYS / 16; ++kk) {       // keys 16kk..+15 of the warp's
        const float *a = sc[KEYS / 8 * t + 2 * kk], *c = sc[KEYS / 8 * t + 2 * kk + 1];
        const uint32_t pf[4] = {pack2(a[0], a[1]), pack2(a[2], a[3]), pack2(c[0], c[1]), pack2(c[2], c[3])};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint32_t vf[4];
          ldsm4t(vf, v + (16 * kk + (lane & 15)) * SP + 16 * i + 8 * (lane >> 4));
          mma(o[2 * i], pf, vf[0], vf[1]);
          mma(o[2 * i + 1], pf, vf[2], vf[3]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
      l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
    }
  }
  // Of two warps each finishes 32 of the 64 columns, and hands the other its part of the others: in the tables' place.
  constexpr int MINE = 8 / HALVES;                   // groups of eight columns
  float *const xo = reinterpret_cast<float*>(sKr), *const xl = ex + 2 * ST;
  const int first = half * 32, other = 32 - first;
  if (HALVES == 2) {
    if (rows) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int row = 16 * warp + r0 + 8 * r;
        if (lane % 4 == 0) xl[half * ST + row] = l[r];
#pragma unroll
        for (int i = 0; i < MINE; ++i)
          *reinterpret_cast<float2*>(xo + row * OP + other + 8 * i + kc) =
              half ? make_float2(o[i][2 * r], o[i][2 * r + 1]) : make_float2(o[8 - MINE + i][2 * r], o[8 - MINE + i][2 * r + 1]);
      }
    }
    __syncthreads();
  }
  if (!rows) return;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int row = 16 * warp + r0 + 8 * r;
    if (row >= own) continue;
    const float sum = HALVES == 2 ? xl[row] + xl[ST + row] : l[r], inv = 1.f / sum;
    uint32_t* const dst = reinterpret_cast<uint32_t*>(ob + row * p.o_st + first + kc);
#pragma unroll
    for (int i = 0; i < MINE; ++i) {
      float2 v = half ? make_float2(o[8 - MINE + i][2 * r], o[8 - MINE + i][2 * r + 1]) : make_float2(o[i][2 * r], o[i][2 * r + 1]);
      if (HALVES == 2) {
        const float2 a = *reinterpret_cast<const float2*>(xo + row * OP + first + 8 * i + kc);
        v.x += a.x; v.y += a.y;
      }
      dst[4 * i] = pack2(v.x * inv, v.y * inv);
    }
    if (lse && half == 0 && lane % 4 == 0) lse[row] = m[r] * 0.6931471805599453f + logf(sum);
  }
}

template <bool C2P, bool P2C, int TILES, bool DIRECT>
int launch_variant(const AttnParams& p, cudaStream_t s) {
  constexpr int TERMS = (C2P ? 1 : 0) + (P2C ? 1 : 0), SMEM = ST * SP * 2 * (3 + 2 * TERMS) + ST * BP * 4 * TERMS + (TERMS ? 0 : ST * OP * 4);
  static_assert(ST * OP * 4 <= 2 * ST * SP * 2, "the outputs fit where a table was");
  auto kern = attn_small_kernel<C2P, P2C, TILES, DIRECT>;
  if (SMEM > 48 * 1024) {
    const int rc = opt_in_smem(reinterpret_cast<const void*>(kern), SMEM);
    if (rc) return rc;
  }
  return cuda_fail(launch_early(kern, dim3(p.H, p.n_seqs, TILES), threads_of<TILES>, SMEM, s, p), "attn_small launch");
}

template <bool C2P, bool P2C, int TILES>
int launch_small(const AttnParams& p, cudaStream_t s) {
  return (C2P || P2C) && p.direct_tables ? launch_variant<C2P, P2C, TILES, C2P || P2C>(p, s) : launch_variant<C2P, P2C, TILES, false>(p, s);
}

template <int TILES>
int launch_tiles(const AttnParams& p, cudaStream_t s) {
  const bool c2p = p.flags & TDB_FLAG_C2P, p2c = p.flags & TDB_FLAG_P2C;
  if (c2p && p2c) return launch_small<true, true, TILES>(p, s);
  if (c2p) return launch_small<true, false, TILES>(p, s);
  if (p2c) return launch_small<false, true, TILES>(p, s);
  return launch_small<false, false, TILES>(p, s);
}

}  // namespace

// Packed sequences only where the longest is known: with a caller's max_seqlen they go to the other kernel, which takes any lengths
// the offsets may turn out to have.  Up to 64 tokens always; up
// to 128 as long as the blocks have an SM each (12 heads, 128 tokens, us per call, this kernel and the other: 1 sequence 18.7 and 19.9, 4
// 18.8 and 20.2, 6 19.2 and 20.2; with two blocks on some SMs, 8 sequences, 23.1 and 21.1), or two, where it saves the other one's
// expanded tables (8 sequences 26.2 and 28.2, 12 26.6 and 28.7).
bool small_applicable(const AttnParams& p) {
  if ((p.varlen && !p.lengths_known) || p.L > 2 * ST || p.n_seqs > 65535) return false;
  if (p.L <= ST) return true;
  int sms = 0;
  return device_sms(&sms) == 0 && 2 * (int64_t)p.n_seqs * p.H <= (p.direct_tables ? 2 : 1) * (int64_t)sms;
}

int launch_attn_small(const AttnParams& p, cudaStream_t s) { return p.L <= ST ? launch_tiles<1>(p, s) : launch_tiles<2>(p, s); }

}  // namespace tdb
