// CUDA-core disentangled attention: exact fp32 arithmetic on f32 or bf16 inputs.
//
// This is the full-precision path (fp32 inputs must land within 1e-4 of the eager module, which the bf16 tensor-core
// pipeline cannot do), the path of materialised position scores in f32, and the cross-check for the tensor-core kernel.
//
//   score[q,k] = (Q[q].K[k] + Q[q].Kr[r] + K[k].Qr[r]) * sm_scale,  r = idx[clamp(q-k)]
//
// Legacy form, f32: the two position products arrive materialised (c2p_scores[q, r], p2c_scores[k, r]) and are only
// gathered (attn_scores.cu does so in bf16); with TDB_FLAG_P2C_MIRRORED the p2c term is read at idx[clamp(k-q)], the reference kernel's convention.
//
// Bound by the FMA pipes and, close behind, by shared-memory reads (256 fp32 multiply-adds per score with both terms).
// A block owns 8R query rows and walks the keys in tiles of 64.  A thread owns R x 8 scores at rows ti + 8r and
// keys tj + 8s, so that the distance of each of them is (ti - tj) + 8 (r - s): R + 7 table rows per term serve all 8R
// scores, every product that is formed is a score's own (a band of q.Kr products over all distances of a tile would be
// twice as many), and nothing has to be skewed or gathered afterwards.  Operand rows are staged fp32, 36-word pitch, half a
// head (32 columns) at a time: eight consecutive rows fall on different banks, and four pairs of warps fit on an SM, which cover
// each other's loads.  The rows of one query tile stay inside one warp, so the softmax needs shuffles only.
// One call of 8 x (48..387) fp32 tokens with 12 heads and both terms: 195 us, 28 TFLOP/s (one warp per query row, keys spread
// over its lanes, every operand read row by row through L1: 1902 us; with one multiply-add per instruction: 234 us).
//
// Sums are kept short, because the rounding error of a chain grows with the square root of its length: half a head's terms
// of a score have a sum of their own, P.V is summed over 16 keys, those sums over the tile, and the tiles' one by one.  Relative
// 2-norm of the error against float64: 1.7e-7 at 8 x 48..387, 1.8e-7 at 8 x 512, 2.0e-7 at 2 x 2048 (one chain over all terms of a
// score and over all keys: 3.6e-7, 4.5e-7, 8.3e-7, at the same speed; one warp per query row: 1.9e-7, 2.0e-7, 2.3e-7; without
// the sum per tile: 1.8e-7, 1.9e-7, 2.6e-7).
//
// A block is bound by its own chain of key tiles, some 6 to 9 us each, so two or four pairs of warps (GROUPS) take every second or fourth
// tile of the same query rows, and their states are added at the end (the rule of the launch has the times).  2 x 128: 35.0 us per
// call with one pair, 29.4; 8 x (48..387) 208 and 195.
#include "attn_blocks.cuh"
#include "ptx_sm100.cuh"
#include <float.h>
#include <math_constants.h>

namespace tdb {
using namespace ptx;

namespace {

constexpr int KT = 64, HALF = 32, HP = HALF + 4, DP = 64 + 4, THREADS = 64 /* of a group */, PV = 16;

__device__ __forceinline__ void cp_async16(float* dst, const void* src, bool real) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(real ? 16 : 0) : "memory");
}

// COLS columns of ROWS rows to shared memory as fp32; src(row) is the row's first element, or null for a row of zeros.
template <typename T, int COLS, int PITCH, typename F>
__device__ __forceinline__ void stage_rows(float* dst, int rows, const T* any, F src, int tid, int threads = THREADS) {
  constexpr int PER = 16 / sizeof(T), CH = COLS / PER;
  for (int e = tid; e < rows * CH; e += threads) {
    const int row = e / CH, c = e % CH;
    const T* s = src(row);
    float* d = dst + row * PITCH + c * PER;
    if constexpr (sizeof(T) == 4) {
      cp_async16(d, s ? s + c * PER : any, s != nullptr);
    } else {
      uint4 t = make_uint4(0, 0, 0, 0);
      if (s) t = __ldg(reinterpret_cast<const uint4*>(s) + c);
      const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
      for (int i = 0; i < 2; ++i)
        *reinterpret_cast<float4*>(d + 4 * i) =
            make_float4(__uint_as_float(w[2 * i] << 16), __uint_as_float(w[2 * i] & 0xffff0000u),
                        __uint_as_float(w[2 * i + 1] << 16), __uint_as_float(w[2 * i + 1] & 0xffff0000u));
    }
  }
}
// The threads of one group (a whole block where there is only one).
template <int GROUPS> __device__ __forceinline__ void group_sync(int group) {
  if (GROUPS == 1) __syncthreads();
  else asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(THREADS) : "memory");
}
template <int GROUPS> __device__ __forceinline__ void staged(int group) {
  asm volatile("cp.async.wait_all;" ::: "memory");
  group_sync<GROUPS>(group);
}

// A pair (f32x2) holds the sums over even and odd columns.
struct Four { f32x2 lo, hi; };                       // four columns
__device__ __forceinline__ Four load4(const float* p) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  return {v.x, v.y};
}
__device__ __forceinline__ void fma4(f32x2& acc, const Four& a, const Four& b) { fma2(acc, a.lo, b.lo); fma2(acc, a.hi, b.hi); }

__device__ __forceinline__ void store4(float* d, float a, float b, float c, float e) { *reinterpret_cast<float4*>(d) = make_float4(a, b, c, e); }
__device__ __forceinline__ void store4(__nv_bfloat16* d, float a, float b, float c, float e) {
  __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(c, e);
  uint2 v;
  v.x = *reinterpret_cast<uint32_t*>(&lo); v.y = *reinterpret_cast<uint32_t*>(&hi);
  *reinterpret_cast<uint2*>(d) = v;
}

// Of a group: P, and the operand rows of half a head, over which V comes.
template <int R, bool TABLES> constexpr int operand_floats = (KT + (TABLES ? 2 * (8 * R + KT) : 0)) * HP;
template <int R, bool TABLES> constexpr int group_floats = 8 * R * DP + (operand_floats<R, TABLES> > KT * DP ? operand_floats<R, TABLES> : KT * DP);
template <int R, bool TABLES, int GROUPS> constexpr int smem_floats = 8 * R * DP + GROUPS * group_floats<R, TABLES>;

// TABLES: position terms from the projected tables (either may be absent); otherwise none, or in f32 gathered scores.
// GROUPS: pairs of warps that share the query rows and take every GROUPS-th key tile each; the first adds the others' states up.
template <typename T, int R, bool TABLES, int GROUPS>
__global__ void __launch_bounds__(THREADS * GROUPS, 4 / GROUPS) attn_simt_kernel(const AttnParams p) {
  constexpr bool GATHER = !TABLES && sizeof(T) == 4;
  constexpr int QT = 8 * R, XR = QT + KT;           // XR: table rows a tile can touch (QT + KT - 1, padded)
  extern __shared__ __align__(16) float smem[];
  float* const sQ = smem;                            // [QT][DP]
  const int group = GROUPS == 1 ? 0 : (int)threadIdx.x / THREADS, tid = (int)threadIdx.x - group * THREADS;
  float* const sP = sQ + QT * DP + group * group_floats<R, TABLES>;        // [QT][DP]
  float* const sK = sP + QT * DP;                    // [KT][HP], half a head
  float* const sKr = sK + KT * HP;                   // [XR][HP]
  float* const sQr = sKr + XR * HP;                  // [XR][HP]
  float* const sV = sK;                              // [KT][DP], over the three above
  __shared__ int rows_of[GROUPS][XR];                // first element of the table row of distance q0 - k0 - 63 + x
  int* const sRow = rows_of[group];

  const int warp = tid / 32, lane = tid % 32;
  const int ti = warp * 4 + lane / 8, tj = lane % 8;
  const int s = longest_first(p, blockIdx.z), h = blockIdx.y, q0 = blockIdx.x * QT;
  int len, rows;
  int64_t tok0;
  int b;
  if (!sequence_of(p, s, len, rows, tok0, b) || q0 >= rows) return;
  T* const ob = reinterpret_cast<T*>(p.o) + b * p.o_sb + tok0 * p.o_st + h * p.o_sh;
  float* const lse = p.lse ? p.lse + b * p.lse_sb + h * p.lse_sh + tok0 : nullptr;

  const T* const qb = reinterpret_cast<const T*>(p.q) + b * p.q_sb + tok0 * p.q_st + h * p.q_sh;
  const T* const kb = reinterpret_cast<const T*>(p.k) + b * p.k_sb + tok0 * p.k_st + h * p.k_sh;
  const T* const vb = reinterpret_cast<const T*>(p.v) + b * p.v_sb + tok0 * p.v_st + h * p.v_sh;
  const T* const krh = (TABLES && (p.flags & TDB_FLAG_C2P)) ? reinterpret_cast<const T*>(p.kr) + (int64_t)h * p.two_span * 64 : nullptr;
  const T* const qrh = (TABLES && (p.flags & TDB_FLAG_P2C)) ? reinterpret_cast<const T*>(p.qr) + (int64_t)h * p.two_span * 64 : nullptr;
  // materialised scores: the base of this head's c2p rows (one per query) and p2c rows (one per key)
  const T* const c2p_base = (GATHER && (p.flags & TDB_FLAG_C2P))
      ? reinterpret_cast<const T*>(p.c2p_scores) + b * p.c2p_sb + tok0 * p.c2p_st + h * p.c2p_sh : nullptr;
  const T* const p2c_base = (GATHER && (p.flags & TDB_FLAG_P2C))
      ? reinterpret_cast<const T*>(p.p2c_scores) + b * p.p2c_sb + tok0 * p.p2c_st + h * p.p2c_sh : nullptr;
  const int dm = p.idx_delta_max;
  auto clamped = [&](int delta) { return delta < -dm ? 0 : (delta > dm ? 2 * dm : delta + dm); };

  f32x2 o[R][4];                                     // eight output columns
  // The maximum starts at the lowest finite value: a row whose scores so far are all -inf (score tensors that hide keys, or whose sum leaves
  // fp32's range) has a reference to take them against, and they get weight 0 instead of exp(-inf + inf).  A row with no other score ends as 0 / 0.
  float m[R], l[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    m[r] = -FLT_MAX; l[r] = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) o[r][c] = 0ull;
  }

  if (q0 < len) {
    stage_rows<T, 64, DP>(sQ, QT, qb, [&](int row) { return q0 + row < len ? qb + (int64_t)(q0 + row) * p.q_st : nullptr; }, threadIdx.x, THREADS * GROUPS);
    auto table_rows = [&](int k0) {
      if (TABLES)
        for (int x = tid; x < XR; x += THREADS) sRow[x] = p.idx[clamped(q0 - k0 - (KT - 1) + x)] * 64;
    };
    table_rows(group * KT);
    if (GROUPS > 1) asm volatile("cp.async.wait_all;" ::: "memory");        // Q is everybody's
    __syncthreads();
    for (int k0 = group * KT; k0 < len; k0 += GROUPS * KT) {
      float acc[R][8];
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[r][c] = 0.f;
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        const int d0 = half * HALF;
        f32x2 acc2[R][8];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int c = 0; c < 8; ++c) acc2[r][c] = 0ull;
        stage_rows<T, HALF, HP>(sK, KT, kb, [&](int row) { return k0 + row < len ? kb + (int64_t)(k0 + row) * p.k_st + d0 : nullptr; }, tid);
        if (TABLES) {
          auto table_row = [&](const T* t, int x) { return t + sRow[x] + d0; };
          if (krh) stage_rows<T, HALF, HP>(sKr, XR, krh, [&](int x) { return table_row(krh, x); }, tid);
          if (qrh) stage_rows<T, HALF, HP>(sQr, XR, qrh, [&](int x) { return table_row(qrh, x); }, tid);
        }
        staged<GROUPS>(group);
        const float* const kp = sK + tj * HP;
        const float* const qp = sQ + ti * DP + d0;
        const int x0 = ti - tj + (KT - 1) - 56;      // table row of (r, s) is x0 + 8 (r - s + 7)
#pragma unroll 1
        for (int d = 0; d < HALF; d += 4) {
          Four kf[8];
#pragma unroll
          for (int c = 0; c < 8; ++c) kf[c] = load4(kp + 8 * c * HP + d);
          if (TABLES && krh) {
            Four t[R + 7];
#pragma unroll
            for (int x = 0; x < R + 7; ++x) t[x] = load4(sKr + (x0 + 8 * x) * HP + d);
#pragma unroll
            for (int r = 0; r < R; ++r) {
              const Four qf = load4(qp + 8 * r * DP + d);
#pragma unroll
              for (int c = 0; c < 8; ++c) { fma4(acc2[r][c], qf, kf[c]); fma4(acc2[r][c], qf, t[r - c + 7]); }
            }
          } else {
#pragma unroll
            for (int r = 0; r < R; ++r) {
              const Four qf = load4(qp + 8 * r * DP + d);
#pragma unroll
              for (int c = 0; c < 8; ++c) fma4(acc2[r][c], qf, kf[c]);
            }
          }
          if (TABLES && qrh) {
            Four t[R + 7];
#pragma unroll
            for (int x = 0; x < R + 7; ++x) t[x] = load4(sQr + (x0 + 8 * x) * HP + d);
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
              for (int c = 0; c < 8; ++c) fma4(acc2[r][c], kf[c], t[r - c + 7]);
          }
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int c = 0; c < 8; ++c) { const float2 v = halves(acc2[r][c]); acc[r][c] += v.x + v.y; }
        group_sync<GROUPS>(group);
      }
      table_rows(k0 + GROUPS * KT);                  // for the next tile; V replaces the operand rows while the softmax runs
      stage_rows<T, 64, DP>(sV, KT, vb, [&](int row) { return k0 + row < len ? vb + (int64_t)(k0 + row) * p.v_st : nullptr; }, tid);
      float corr[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int qi = q0 + ti + 8 * r;
        float mx = -CUDART_INF_F;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const int kj = k0 + tj + 8 * c;
          float sc = acc[r][c];
          if (GATHER && kj < len && qi < len) {
            const int x = clamped(qi - kj);
            if (c2p_base) sc += (float)c2p_base[(int64_t)qi * p.c2p_st + p.idx[x]];
            if (p2c_base) sc += (float)p2c_base[(int64_t)kj * p.p2c_st + p.idx[(p.flags & TDB_FLAG_P2C_MIRRORED) ? 2 * dm - x : x]];
          }
          sc = kj < len ? sc * p.sm_scale : -CUDART_INF_F;
          acc[r][c] = sc;
          mx = fmaxf(mx, sc);
        }
#pragma unroll
        for (int off = 1; off < 8; off *= 2) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
        const float mn = fmaxf(m[r], mx);
        corr[r] = expf(m[r] - mn);
        m[r] = mn;
        float sum = 0.f;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float e = expf(acc[r][c] - mn);
          sum += e;
          sP[(ti + 8 * r) * DP + tj + 8 * c] = e;
        }
        l[r] = l[r] * corr[r] + sum;
      }
      staged<GROUPS>(group);                         // also makes the warp's own rows of P visible to its lanes
      f32x2 tile[R][4];
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) tile[r][c] = 0ull;
#pragma unroll 1
      for (int j0 = 0; j0 < KT; j0 += PV) {
        f32x2 part[R][4];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int c = 0; c < 4; ++c) part[r][c] = 0ull;
#pragma unroll
        for (int j = j0; j < j0 + PV; j += 4) {
          float4 pf[R];
#pragma unroll
          for (int r = 0; r < R; ++r) pf[r] = *reinterpret_cast<const float4*>(sP + (ti + 8 * r) * DP + j);
#pragma unroll
          for (int jj = 0; jj < 4; ++jj) {
            const Four a = load4(sV + (j + jj) * DP + 4 * tj), c = load4(sV + (j + jj) * DP + 32 + 4 * tj);
#pragma unroll
            for (int r = 0; r < R; ++r) {
              const float w = jj == 0 ? pf[r].x : jj == 1 ? pf[r].y : jj == 2 ? pf[r].z : pf[r].w;
              const f32x2 ww = pair(w, w);
              fma2(part[r][0], ww, a.lo); fma2(part[r][1], ww, a.hi); fma2(part[r][2], ww, c.lo); fma2(part[r][3], ww, c.hi);
            }
          }
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int c = 0; c < 4; ++c) add2(tile[r][c], part[r][c]);
      }
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          f32x2 sum = tile[r][c];
          fma2(sum, o[r][c], pair(corr[r], corr[r]));
          o[r][c] = sum;
        }
      group_sync<GROUPS>(group);                     // the next tile's operand rows go where V is
    }
  }
  if constexpr (GROUPS > 1) {
    // A group's state of a thread's rows: maximum, sum and eight outputs, to where its P was; a group without a key tile has none.
    constexpr int STATE = R * 10;
    static_assert(STATE * THREADS <= group_floats<R, TABLES>, "the state fits");
    if (group > 0) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float* const d = sP + r * 10 * THREADS + tid;
        d[0] = m[r]; d[THREADS] = l[r];
#pragma unroll
        for (int c = 0; c < 4; ++c) { const float2 v = halves(o[r][c]); d[(2 + 2 * c) * THREADS] = v.x; d[(3 + 2 * c) * THREADS] = v.y; }
      }
    }
    __syncthreads();
    if (group > 0) return;
    for (int g = 1; g < GROUPS && g * KT < len; ++g) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float* const d = sP + g * group_floats<R, TABLES> + r * 10 * THREADS + tid;
        const float mn = fmaxf(m[r], d[0]), mine = expf(m[r] - mn), theirs = expf(d[0] - mn);
        m[r] = mn;
        l[r] = l[r] * mine + d[THREADS] * theirs;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          f32x2 sum = pair(d[(2 + 2 * c) * THREADS] * theirs, d[(3 + 2 * c) * THREADS] * theirs);
          fma2(sum, o[r][c], pair(mine, mine));
          o[r][c] = sum;
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int qi = q0 + ti + 8 * r;
    float sum = l[r];
#pragma unroll
    for (int off = 1; off < 8; off *= 2) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    if (qi >= rows) continue;
    const bool valid = qi < len;                     // padded query rows of the padded form: zeros
    const float inv = valid ? 1.f / sum : 0.f;
    T* const orow = ob + (int64_t)qi * p.o_st;
    if (valid) {
      const float2 a = halves(o[r][0]), b2 = halves(o[r][1]), c = halves(o[r][2]), d = halves(o[r][3]);
      store4(orow + 4 * tj, a.x * inv, a.y * inv, b2.x * inv, b2.y * inv);
      store4(orow + 32 + 4 * tj, c.x * inv, c.y * inv, d.x * inv, d.y * inv);
    } else {
      store4(orow + 4 * tj, 0.f, 0.f, 0.f, 0.f);
      store4(orow + 32 + 4 * tj, 0.f, 0.f, 0.f, 0.f);
    }
    if (lse && tj == 0) lse[qi] = valid ? m[r] + logf(sum) : 0.f;
  }
}

template <typename T, int R, bool TABLES, int GROUPS>
int launch_variant(const AttnParams& p, cudaStream_t s) {
  constexpr int SMEM = smem_floats<R, TABLES, GROUPS> * 4;
  auto kern = attn_simt_kernel<T, R, TABLES, GROUPS>;
  if (SMEM > 47 * 1024) {
    int rc = opt_in_smem(reinterpret_cast<const void*>(kern), SMEM);
    if (rc) return rc;
  }
  dim3 grid((p.L + 8 * R - 1) / (8 * R), p.H, p.n_seqs);
  kern<<<grid, THREADS * GROUPS, SMEM, s>>>(p);
  return cuda_fail(cudaGetLastError(), "attn_simt launch");
}

template <typename T, bool TABLES>
int launch_rows(const AttnParams& p, cudaStream_t s) {
  // 32 query rows per block re-use each staged row twice as often as 16.  A block is bound by its own chain of key tiles, so two pairs of
  // warps share them (two blocks of 32 rows per SM instead of four: as many warps, and half the time to wait for the last block); four
  // pairs while blocks have SMs to themselves, of 16 rows where even those do.  us per call, 12 heads, rows x pairs:
  //   batch x length    blocks of 32 per SM    16 x 4    32 x 4    32 x 2    32 x 1    16 x 1
  //   1 x 128           0.3                      28.2      31.9      32.0      44.0      36.6
  //   1 x 256           0.6                      47.1      37.0      42.3      65.6      54.3
  //   2 x 256           1.3                      63.3      59.0      55.5      66.8      65.8
  //   3 x 192           1.5                      57.7      56.1      55.2      54.4      53.3
  //   4 x 256           2.6                     110.7      81.8      80.2      92.0     108.1
  //   4 x 300           3.2                     185.8     151.8     131.1     112.5     149.2
  //   6 x 256           3.9                     143.9     104.4      96.4      94.2     125.7
  //   16 x 128          5.2                     131.2     102.1      77.9      79.4      98.7
  //   8 x 512           10.4                    647.9     468.6     439.1     469.4     613.3
  //   14 x 384          13.6                    722.3     498.3     419.7     417.5     579.5
  // An SM runs four pairs at a time, so a call is rounds of four blocks of one pair, or of two blocks of two.  Where the last round of four is
  // nearly full, two pairs save nothing: they take twice as many rounds of half the length, adding their states up comes on top, and with an odd
  // number of tiles the second pair waits for a tile's time in each of them.  So rows that are all as long have one pair per block where more than
  // three of the last four slots are taken; with an odd number of tiles also beyond two (three tiles) or five blocks per SM; in long calls
  // also where the last round has more than one block and at most two, which is a whole round of two.  Three tiles and few blocks: 16 rows.
  // Among ragged rows those of one tile leave the second pair waiting, up to three tiles in all (one pair and two: 11 x 126 with 16 heads 49.5 and
  // 51.8, 31 x 128 84.8 and 94.6, 21 x 179 95.9 and 99.4; of four tiles, 15 x 32..256, 128.3 and 116.9, four draws of 14 x 256 0.97 to 1.14 times two pairs').  185 calls of
  // full rows and 178 of ragged ones take 7 and 8 % less time in the geometric mean than with one pair throughout (16 rows up to two
  // blocks per SM, then 32), and no full one takes longer; before the last round was looked at 20 of those took 2 to 17 % longer.
  // Gathered scores: the loads of the score rows are what a block waits for, and of 16 rows (168 registers for 250) six fit on an SM instead of four and
  // cover each other's; from two blocks of 32 per SM on, but for a single round that four fill.  16 x 1, 32 x 1 and 32 x 2:
  // 3 x 300 81.7, 109.2, 116.1; 8 x 256 130.5, 159.1, 144.3; 13 x 512 733, 918, 882; 4 x 300 123.7, 109.1, 126.4; 2 x 256 61.0, 82.2, 57.1.  Ragged
  // rows of more than three tiles gain from six blocks per SM on (four draws of 8 x 32..256 and up take 0.92 to 1.12 of the time of two pairs,
  // of 11 x 256 0.82 to 0.96, of 18 x 256 0.80 to 0.86).  Content alone stands between the two: 16 rows up to three blocks per SM (9 x 128 38.0, 42.3, 41.0), and then as with tables.
  // One tile leaves nothing to share: 16 rows where 32 would leave SMs without a block.
  int device = 0, rc;
  if ((rc = device_sms(&device))) return rc;
  const int64_t sms = device, rows = (int64_t)p.H * p.n_seqs, blocks16 = (p.L + 15) / 16 * rows, blocks32 = (p.L + 31) / 32 * rows;
  if (p.L <= KT) return blocks32 < 2 * sms ? launch_variant<T, 2, TABLES, 1>(p, s) : launch_variant<T, 4, TABLES, 1>(p, s);
  if (blocks16 <= sms) return launch_variant<T, 2, TABLES, 4>(p, s);
  if (blocks32 <= sms) return launch_variant<T, 4, TABLES, 4>(p, s);
  const int tiles = (p.L + KT - 1) / KT;
  const bool full = !p.varlen && !p.seqlens, gathers = p.c2p_scores || p.p2c_scores;
  if (tiles == 3 && blocks16 <= (TABLES ? 3 : 4) * sms) return launch_variant<T, 2, TABLES, 1>(p, s);
  if (!TABLES) {
    const bool by16 = full ? (blocks32 > 2 * sms && blocks32 <= 3 * sms) || (gathers && blocks32 > 4 * sms) : gathers && blocks32 > (tiles <= 3 ? 2 : 6) * sms;
    if (by16) return launch_variant<T, 2, TABLES, 1>(p, s);
  }
  const int64_t last = (blocks32 - 1) % (4 * sms) + 1;         // blocks of the last round of four per SM
  bool one;
  if (full) one = last > 3 * sms || (tiles % 2 ? blocks32 > (tiles == 3 ? 2 : 5) * sms : blocks32 > 8 * sms && last > sms && last <= 2 * sms);
  else one = tiles <= 3 && blocks32 > (tiles == 2 ? 4 : 5) * sms;
  return one ? launch_variant<T, 4, TABLES, 1>(p, s) : launch_variant<T, 4, TABLES, 2>(p, s);
}

template <typename T>
int launch_dtype(const AttnParams& p, cudaStream_t s) {
  return p.flags && !p.c2p_scores && !p.p2c_scores ? launch_rows<T, true>(p, s) : launch_rows<T, false>(p, s);
}

}  // namespace

int launch_attn_simt(const AttnParams& p, int dtype, cudaStream_t s) {
  if (p.n_seqs == 0 || p.L == 0) return TDB_OK;
  if (p.n_seqs > 65535 || p.H > 65535) { set_error("attn_simt: more than 65535 sequences or heads"); return TDB_ERR_SHAPE; }
  if (dtype == TDB_DTYPE_BF16 && (p.c2p_scores || p.p2c_scores)) return launch_attn_scores(p, s);
  return dtype == TDB_DTYPE_F32 ? launch_dtype<float>(p, s) : launch_dtype<__nv_bfloat16>(p, s);
}

}  // namespace tdb
