// The whole layer stack for a handful of tokens (a short request) in one kernel, bf16.
//
// Such a pass is bound by latency: the weights of a layer are 14 MB (hidden size 768), two microseconds of memory traffic, but as
// seven kernels a layer takes some forty, nearly all of it the way from one kernel's last store to the next one's first product.
// Here a persistent block per eight hidden columns walks all layers; the blocks meet at a counter in memory (1 us), five
// times per layer:
//
//   1  x = LN(z + a) of the layer before, every block for itself;  its 8 columns each of q, k and v    -> those that take a head
//   2  attention, one (sequence, head) per block (the other blocks only wait for the result)           -> all
//   3  its 8 columns of the output projection                                                          -> all
//   4  a = LN(y + x), every block for itself;  its 32 columns of the intermediate projection, GELU     -> all
//   5  its 8 columns of the second projection                                                          -> all
//
// A block's rows of the next weights are on their way to shared memory while the blocks meet (q, k, v and the intermediate
// projection take turns in one buffer, the other two in a second one, the norms' vectors in a third), so after a meeting only activations are waited for (L2).
// x and a live in shared memory (each block has all tokens), where they are the products' operand and the next residual.
// Products: warp-level tensor instruction; eight warps per 16 tokens share the columns in blocks of 32 and add their parts up
// through the weights' buffer.  The order of the columns inside a product is free as long as both operands share it, so a
// thread's fragments of two k16 steps are one 16-byte load.
//
// Base model, one pass of 32 tokens from ids to hidden states: 447 us as a replayed recording of 84 kernels, 306 here (with a new padding mask for
// each pass 508 and 354; the kernel itself 240: 20 us per layer, of which the five meetings 5.6, the LayerNorms 3.4, the products 5.0 - the second projection, whose 196 KB of
// activations come in at 55 bytes per clock, 2.6 - the sums of their parts with the way to memory 3.4, and the attention 2.4); 16 tokens 16 us
// per layer.  Tried and left out: clusters of four that share the LayerNorms over distributed shared memory (a row's four
// copies cost what forming it four times does) and split the second projection's columns (1.3 of its 5 thousand clocks).
// Passes per second of 1, 2, 4 and 6 threads with a stream each, here and as recordings whose small kernels run beside one another: base model, 32 tokens,
// 3226, 4116, 4162, 4154 and 2249, 3946, 5927, 5485; large model 1506, 1748, 1768, 1768 and 1066, 1818, 2677, 3203.  So one or two streams gain and many
// lose; a choice by what else is in flight would make a pass's rounding depend on timing, so there is none.
// The LayerNorm is out of line because in line, at two places, one of the copies ran in a warp that the compiler no longer
// took for converged: its ten shuffles cost 5 us.
//
// The blocks wait for one another, so the launch is a cooperative one (all of them run at the same time, or the launch
// fails: several streams' passes come one after the other), and every wait has a limit, after which all blocks leave, behind their own copies, and the host reports it.
#include "attn_warp_mma.cuh"
#include "gelu.cuh"
#include "ptx_sm100.cuh"
#include <math_constants.h>
#include <type_traits>

namespace tdb {
using namespace ptx;

namespace {

using bf16 = __nv_bfloat16;
constexpr int KS = 8;                                // warps that share a product's columns
constexpr int TT = SKINNY_TOKENS;                    // tokens at most, and rows of an attention tile
constexpr int TB = 52;                               // pitch of a band row in floats (48 distances)
constexpr uint32_t ATT_BYTES = 3 * TT * SP * 2 + 2 * TT * TB * 4, TAB_BYTES = 2 * 2 * TT * SP * 2;

// Rows in shared memory are 64 bytes longer than a multiple of 128, so that the 16-byte loads of two rows by four lanes each
// fall on different banks.
template <int MT, int NB> struct Plan {
  static constexpr int H = 256 * NB, THREADS = MT * KS * 32;
  static constexpr uint32_t PITCH = H * 2 + 64, PITCH4 = 4 * H * 2 + 64;
  static constexpr uint32_t PARTS = KS * MT * 16 * 40 * 4, A_LEAST = PARTS > ATT_BYTES ? PARTS : ATT_BYTES;
  static constexpr uint32_t A_BYTES = 32 * PITCH > A_LEAST ? 32 * PITCH : A_LEAST;
  static constexpr uint32_t OFF_X = 0, OFF_A = MT * 16 * PITCH, OFF_B = OFF_A + A_BYTES, OFF_N = OFF_B + 8 * PITCH4,
                            OFF_TAB = OFF_N + 2 * H * 2, OFF_BAR = OFF_TAB + TAB_BYTES;
  static constexpr uint32_t SMEM = OFF_BAR + 32;
  static_assert(SMEM <= 227 * 1024, "shared memory budget");
};

__device__ __forceinline__ uint4 ld16s(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ void st16s(uint32_t a, const uint4& v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
// What other blocks have written: from L2.
__device__ __forceinline__ uint4 ld16g(const bf16* p) { return __ldcg(reinterpret_cast<const uint4*>(p)); }
__device__ __forceinline__ void unpack8(const uint4& v, f32x2* f) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) f[i] = pair(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
}
__device__ __forceinline__ void warp_sums(float* x) {          // of two values
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    const float a = __shfl_xor_sync(0xffffffffu, x[0], off), b = __shfl_xor_sync(0xffffffffu, x[1], off);
    x[0] += a; x[1] += b;
  }
}
// Out of line, like the LayerNorm: the kernel's code runs once per layer, so what is not in it need not be fetched again.
__device__ __noinline__ bool wait_longer(uint32_t bar, uint32_t phase, volatile int* abort_flag, int32_t* status, uint64_t limit_ns) {
  return mbar_wait(bar, phase, abort_flag, status, 301, limit_ns);
}
// Until the counter has come to `expected`; gives up with the others, or after the limit.
__device__ __noinline__ void meet_others(int32_t* counter, int expected, int32_t* gave_up, int32_t* status, volatile int* abort_flag, uint64_t limit_ns) {
  const uint64_t t0 = globaltimer_ns();
#pragma unroll 1
  for (int i = 1;; ++i) {
    int now;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(now) : "l"(counter) : "memory");
    if (now >= expected) return;
    if (i % 64) continue;
    const bool late = globaltimer_ns() - t0 > limit_ns;
    if (!late && *reinterpret_cast<volatile int32_t*>(gave_up) == 0) continue;
    *abort_flag = 1;
    if (late) {
      *reinterpret_cast<volatile int32_t*>(gave_up) = 1;
      if (*reinterpret_cast<volatile int32_t*>(status) == 0) *reinterpret_cast<volatile int32_t*>(status) = 302;
    }
    return;
  }
}

// x <- LN(s + x) for the rows row0 and row0 + step (if it is below `rows`, as row0 is) of 256 NB columns, by one warp: s from L2, x
// and the norm's two vectors in shared memory.  Two rows at once, so that one's sums over the warp hide the other's.
template <int NB>
__device__ __noinline__ void norm_rows(const bf16* s, int row0, int step, int rows, uint32_t x, uint32_t pitch, uint32_t weight, uint32_t bias, float eps) {
  const int lane = threadIdx.x % 32;
  const bool two = row0 + step < rows;
  uint4 v[2][NB];
#pragma unroll
  for (int i = 0; i < NB; ++i) {
    v[0][i] = ld16g(s + (int64_t)row0 * 256 * NB + 8 * (lane + 32 * i));
    v[1][i] = two ? ld16g(s + (int64_t)(row0 + step) * 256 * NB + 8 * (lane + 32 * i)) : make_uint4(0, 0, 0, 0);
  }
  const uint32_t at[2] = {x + (uint32_t)row0 * pitch + 16u * (uint32_t)lane, x + (uint32_t)(two ? row0 + step : row0) * pitch + 16u * (uint32_t)lane};
  f32x2 f[2][NB][4], scale[2];
  float sum[2], sq[2];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    f32x2 total = 0ull;
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      f32x2 r[4];
      unpack8(v[j][i], f[j][i]);
      unpack8(ld16s(at[j] + 512u * (uint32_t)i), r);
#pragma unroll
      for (int e = 0; e < 4; ++e) { add2(f[j][i][e], r[e]); add2(total, f[j][i][e]); }
    }
    const float2 t = halves(total);
    sum[j] = t.x + t.y;
  }
  warp_sums(sum);
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const float mean = sum[j] * (1.f / (256 * NB));
    const f32x2 minus = pair(-mean, -mean);
    f32x2 total = 0ull;
#pragma unroll
    for (int i = 0; i < NB; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) { add2(f[j][i][e], minus); fma2(total, f[j][i][e], f[j][i][e]); }
    const float2 t = halves(total);
    sq[j] = t.x + t.y;
  }
  warp_sums(sq);
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const float inv = rsqrtf(fmaf(sq[j], 1.f / (256 * NB), eps));
    scale[j] = pair(inv, inv);
  }
#pragma unroll
  for (int i = 0; i < NB; ++i) {
    f32x2 g[4], b[4];
    unpack8(ld16s(weight + 16u * (uint32_t)(lane + 32 * i)), g);
    unpack8(ld16s(bias + 16u * (uint32_t)(lane + 32 * i)), b);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      uint32_t w[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        mul2(f[j][i][e], scale[j]);
        f32x2 y = b[e];
        fma2(y, f[j][i][e], g[e]);
        const float2 t = halves(y);
        w[e] = pack2(t.x, t.y);
      }
      if (j == 0 || two) st16s(at[j] + 512u * (uint32_t)i, make_uint4(w[0], w[1], w[2], w[3]));
    }
  }
}

// Rows of 64 bf16 to shared memory, by the whole block; those from `real` on become zeros.
__device__ __forceinline__ void copy_rows(bf16* dst, const bf16* src, int pitch, int rows, int real) {
  for (int e = threadIdx.x; e < rows * 8; e += blockDim.x) {
    const int row = e >> 3, c = e & 7;
    const bool r = row < real;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(saddr(dst + row * SP + c * 8)), "l"(src + (r ? row * pitch + c * 8 : 0)),
                 "r"(r ? 16 : 0) : "memory");
  }
}
// The distances -31 .. 32 of a head's tables.
__device__ __forceinline__ void copy_tables(bf16* dst, const ShortLayer& l, int h) {
  const int64_t at = ((int64_t)h * l.exp_rows + l.exp_delta_max - (TT - 1)) * 64;
  if (l.kr) copy_rows(dst, l.kr + at, 64, 2 * TT, 2 * TT);
  if (l.qr) copy_rows(dst + 2 * TT * SP, l.qr + at, 64, 2 * TT, 2 * TT);
}

// Attention of one head over one sequence of at most 16 MT tokens, by the whole block; `at`: ATT_BYTES of shared memory, `tab`: the
// head's tables.  The bands and their diagonal read are those of attn_small.cu, on 32-row tiles; a warp per 16 query rows forms the
// scores while the others form the bands, 16 rows x 16 distances each.
template <int MT>
__device__ __forceinline__ void short_attention(uint8_t* at, const bf16* tab, const bf16* qkv, int hidden, int h, int tok0, int len, const ShortLayer& l, bf16* ctx) {
  bf16 *const sQ = reinterpret_cast<bf16*>(at), *const sK = sQ + TT * SP, *const sV = sK + TT * SP;
  const bf16 *const sKr = tab, *const sQr = tab + 2 * TT * SP;
  float *const bC = reinterpret_cast<float*>(sV + TT * SP), *const bP = bC + TT * TB;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid / 32, 0), lane = tid % 32;
  const bf16* const base = qkv + (int64_t)tok0 * 3 * hidden + 64 * h;
  copy_rows(sQ, base, 3 * hidden, 16 * MT, len);
  copy_rows(sK, base + hidden, 3 * hidden, TT, len);
  copy_rows(sV, base + 2 * hidden, 3 * hidden, TT, len);
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const int r0 = lane / 4, kc = 2 * (lane % 4);
  float sc[4][4] = {};
  if (warp < MT) {
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      uint32_t a[4];
      ldsm4(a, sQ + (16 * warp + (lane & 15)) * SP + 16 * kk + 8 * (lane >> 4));
#pragma unroll
      for (int j = 0; j < 4; j += 2) {
        uint32_t k[4];
        ldsm4(k, sK + (8 * j + (lane & 7) + 8 * (lane >> 4)) * SP + 16 * kk + 8 * ((lane >> 3) & 1));
        mma(sc[j], a, k[0], k[1]);
        mma(sc[j + 1], a, k[2], k[3]);
      }
    }
  } else if (const int unit = warp - MT; unit < 6 * MT) {
    const int term = unit / (3 * MT), m = unit / 3 % MT, n = unit % 3;
    if (16 * m < len && (term ? l.qr : l.kr)) {
      const bf16 *const rows = (term ? sK : sQ) + 16 * m * SP, *const t = term ? sQr + (16 - 16 * m + 16 * n) * SP : sKr + (16 * m + 16 * n) * SP;
      float d[2][4] = {};
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        uint32_t a[4], k[4];
        ldsm4(a, rows + (lane & 15) * SP + 16 * kk + 8 * (lane >> 4));
        ldsm4(k, t + ((lane & 7) + 8 * (lane >> 4)) * SP + 16 * kk + 8 * ((lane >> 3) & 1));
        mma(d[0], a, k[0], k[1]);
        mma(d[1], a, k[2], k[3]);
      }
      float* const dst = (term ? bP : bC) + 16 * m * TB + 16 * n + kc;
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) *reinterpret_cast<float2*>(dst + (r0 + 8 * e) * TB + 8 * i) = make_float2(d[i][2 * e], d[i][2 * e + 1]);
    }
  }
  __syncthreads();
  if (warp < MT && 16 * warp < len) {
    float o[8][4] = {};
    const float sl2 = l.sm_scale * 1.4426950408889634f;
    float m[2] = {-CUDART_INF_F, -CUDART_INF_F}, sum[2] = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int il = r0 + 8 * (e >> 1), kl = 8 * j + kc + (e & 1);
        float x = sc[j][e];
        if (l.kr) x += bC[(16 * warp + il) * TB + il - kl + TT - 1];
        if (l.qr) x += bP[kl * TB + 16 * warp + il - (kl & 15) + 15];            // rows beyond the sequence are masked just below
        x = kl < len ? x * sl2 : -CUDART_INF_F;
        sc[j][e] = x;
        m[e >> 1] = fmaxf(m[e >> 1], x);
      }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      m[r] = fmaxf(m[r], __shfl_xor_sync(0xffffffffu, m[r], 1));
      m[r] = fmaxf(m[r], __shfl_xor_sync(0xffffffffu, m[r], 2));
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 2 * r; e < 2 * r + 2; ++e) { sc[j][e] = exp2f(sc[j][e] - m[r]); sum[r] += sc[j][e]; }
      sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 1);
      sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 2);
    }
#pragma unroll
    for (int kk = 0; kk < 2; ++kk) {                 // keys 16kk..+15
      const float *a = sc[2 * kk], *c = sc[2 * kk + 1];
      const uint32_t pf[4] = {pack2(a[0], a[1]), pack2(a[2], a[3]), pack2(c[0], c[1]), pack2(c[2], c[3])};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint32_t v[4];
        ldsm4t(v, sV + (16 * kk + (lane & 15)) * SP + 16 * i + 8 * (lane >> 4));
        mma(o[2 * i], pf, v[0], v[1]);
        mma(o[2 * i + 1], pf, v[2], v[3]);
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int row = 16 * warp + r0 + 8 * r;
      if (row >= len) continue;
      const float inv = 1.f / sum[r];
      uint32_t* const dst = reinterpret_cast<uint32_t*>(ctx + (int64_t)(tok0 + row) * hidden + 64 * h + kc);
#pragma unroll
      for (int i = 0; i < 8; ++i) dst[4 * i] = pack2(o[i][2 * r] * inv, o[i][2 * r + 1] * inv);
    }
  }
}

// MT: tiles of 16 tokens; NB: hidden size / 256.
template <int MT, int NB>
__global__ void __launch_bounds__(MT * KS * 32, 1) short_stack_kernel(const __grid_constant__ ShortStack p) {
  using P = Plan<MT, NB>;
  constexpr int H = P::H, ROWS = MT * 16;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ int s_abort;
  // the warp's number and everybody's verdict come out of warp-wide operations, so that the compiler sees branches on them as uniform
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid / 32, 0), lane = tid % 32, g = lane / 4, t = lane % 4;
  const int ks = warp % KS, mt = warp / KS, block = blockIdx.x, blocks = gridDim.x;
  const uint32_t base = smem_u32(smem), sX = base + P::OFF_X, sA = base + P::OFF_A, sB = base + P::OFF_B, sN = base + P::OFF_N;
  enum { A, B, N, BARS };                            // the barrier of each buffer that bulk copies go to
  const uint32_t bars = base + P::OFF_BAR;

  if (tid == 0) {
    s_abort = 0;
    for (int i = 0; i < BARS; ++i) mbar_init(bars + 8u * i, 1);
    fence_mbar_init();
  }
  __syncthreads();
  // This block's rows of a weight matrix to shared memory (by the first warp, a row per lane; whoever read or wrote the buffer is
  // behind a barrier).
  uint32_t phase[BARS] = {}, late = 0;               // late: a bit for each barrier whose wait was given up
  auto bring = [&](uint32_t dst, uint32_t pitch, int i, int rows, uint32_t bytes, const bf16* mine) {
    const uint32_t bar = bars + 8u * i;
    if (warp != 0 || (late >> i & 1u)) return;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (lane == 0) mbar_expect_tx(bar, (uint32_t)rows * bytes);
    __syncwarp();
    if (lane < rows) bulk_load(dst + (uint32_t)lane * pitch, mine, bytes, bar);
  };
  auto bring_qkv = [&](const ShortLayer& l) {
    bring(sA, P::PITCH, A, 24, 2 * H, l.qkv_w + ((int64_t)(lane >> 3) * H + 8 * block + (lane & 7)) * H);
  };
  auto bring_up = [&](const ShortLayer& l) { bring(sA, P::PITCH, A, 32, 2 * H, l.up_w + (int64_t)(32 * block + lane) * H); };
  auto bring_out = [&](const ShortLayer& l) { bring(sB, P::PITCH, B, 8, 2 * H, l.out_w + (int64_t)(8 * block + (lane & 7)) * H); };
  auto bring_down = [&](const ShortLayer& l) { bring(sB, P::PITCH4, B, 8, 8 * H, l.down_w + (int64_t)(8 * block + (lane & 7)) * 4 * H); };
  auto bring_norm = [&](const bf16* w, const bf16* b) { bring(sN, 2 * H, N, 2, 2 * H, lane ? b : w); };
  auto landed = [&](int i) {
    const uint32_t bar = bars + 8u * i;
    if (__any_sync(0xffffffffu, !mbar_try_wait(bar, phase[i])) &&
        __any_sync(0xffffffffu, !wait_longer(bar, phase[i], &s_abort, p.status, p.limit_ns))) {
      late |= 1u << i;
      phase[i] ^= 1;                                 // the copy's phase is still the one to wait for
    }
    __syncwarp();
    phase[i] ^= 1;
  };

  // The blocks' meeting: everything written before an arrival is there after a wait for it.
  int expected = 0;
  auto arrive = [&]() {
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      atomicAdd(p.counter, 1);
    }
  };
  auto meet = [&]() {                                // false: somebody gave up
    if (warp == 0) meet_others(p.counter, expected, p.gave_up, p.status, &s_abort, p.limit_ns);       // all its lanes, so that it stays in step
    __syncwarp();
    __syncthreads();
    return !__any_sync(0xffffffffu, *reinterpret_cast<volatile int*>(&s_abort));
  };

  // acc[f]: this warp's part (its blocks of 32 columns) of 16 tokens x 8 features; the activations from shared memory, or the
  // other blocks' from L2.
  auto product = [&](auto features, auto nb, uint32_t w, uint32_t pitch, auto&& row, float (*acc)[4]) {
    constexpr int F = decltype(features)::value, N = decltype(nb)::value, AHEAD = N > 8 ? N / 2 : N;       // blocks whose loads are in flight together
#pragma unroll
    for (int f = 0; f < F; ++f)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[f][e] = 0.f;
#pragma unroll 1
    for (int i0 = 0; i0 < N; i0 += AHEAD) {
      uint4 a[AHEAD][2];
      int b[AHEAD];                                  // the blocks of the grid begin at different columns, which lie in different parts of L2
#pragma unroll
      for (int i = 0; i < AHEAD; ++i) {
        b[i] = i0 + i + block % N;
        b[i] = ks + KS * (b[i] < N ? b[i] : b[i] - N);
#pragma unroll
        for (int r = 0; r < 2; ++r) a[i][r] = row(r, b[i]);
      }
#pragma unroll
      for (int i = 0; i < AHEAD; ++i) {
        const uint32_t lo[4] = {a[i][0].x, a[i][1].x, a[i][0].y, a[i][1].y}, hi[4] = {a[i][0].z, a[i][1].z, a[i][0].w, a[i][1].w};
#pragma unroll
        for (int f = 0; f < F; ++f) {
          const uint4 k = ld16s(w + (uint32_t)(8 * f + g) * pitch + 64u * (uint32_t)b[i] + 16u * (uint32_t)t);
          mma(acc[f], lo, k.x, k.y);
          mma(acc[f], hi, k.z, k.w);
        }
      }
    }
  };
  // The parts added up (in the buffer of the weights, which have been read), plus bias: store(token, column of the block, two values).
  auto finish = [&](auto features, uint32_t w, const float (*acc)[4], uint32_t bias, auto&& store) {
    constexpr int F = decltype(features)::value, STRIDE = F == 1 ? 8 : 40;
    static_assert(KS * ROWS * STRIDE * 4 <= (F == 1 ? 8 * P::PITCH : P::A_BYTES), "the parts fit");
    __syncthreads();
#pragma unroll
    for (int f = 0; f < F; ++f)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const uint32_t at = w + 4u * (uint32_t)((ks * ROWS + 16 * mt + g + 8 * r) * STRIDE + 8 * f + 2 * t);
        asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(at), "f"(acc[f][2 * r]), "f"(acc[f][2 * r + 1]) : "memory");
      }
    __syncthreads();
    constexpr int PAIRS = 4 * F;
    if (tid < ROWS * PAIRS) {
      const int row = tid / PAIRS, c = 2 * (tid % PAIRS);
      if (row < p.tokens) {
        float s0 = 0.f, s1 = 0.f;
#pragma unroll
        for (int k = 0; k < KS; ++k) {
          float a, b;
          asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(a), "=f"(b) : "r"(w + 4u * (uint32_t)((k * ROWS + row) * STRIDE + c)));
          s0 += a; s1 += b;
        }
        store(row, c, s0 + __uint_as_float(bias << 16), s1 + __uint_as_float(bias & 0xffff0000u));
      }
    }
  };
  // The bias of the two features that a thread will finish in a product with `pairs` pairs per block: asked for before a meeting.
  auto bias_of = [&](const bf16* b, int pairs, int stride) {
    const int c = 2 * (tid % pairs);
    uint32_t v;
    asm volatile("ld.global.nc.b32 %0, [%1];" : "=r"(v) : "l"(b + (c >> 3) * stride + (c & 7)));
    return v;
  };
  auto put = [](bf16* d, float a, float b) { *reinterpret_cast<uint32_t*>(d) = pack2(a, b); };
  // groups of 8 features
  constexpr std::integral_constant<int, 1> one;
  constexpr std::integral_constant<int, 3> three;
  constexpr std::integral_constant<int, 4> four;
  // blocks of 32 columns per warp
  constexpr std::integral_constant<int, NB> narrow;
  constexpr std::integral_constant<int, 4 * NB> wide;

  bring_qkv(p.layer[0]);
  bring_out(p.layer[0]);
  const int pairs = p.n_seqs * (H / 64), takers = pairs < blocks ? pairs : blocks;
  bf16* const tables = reinterpret_cast<bf16*>(smem + P::OFF_TAB);
  if (block < takers) copy_tables(tables, p.layer[0], block % (H / 64));       // of the first head that the block will take
  for (int e = tid; e < ROWS * (H / 8); e += P::THREADS) {
    const int row = e / (H / 8), c = e % (H / 8);
    st16s(sX + (uint32_t)row * P::PITCH + 16u * (uint32_t)c, row < p.tokens ? ld16g(p.x + (int64_t)row * H + 8 * c) : make_uint4(0, 0, 0, 0));
  }
  auto from_x = [&](int r, int b) { return ld16s(sX + (uint32_t)(16 * mt + g + 8 * r) * P::PITCH + 64u * (uint32_t)b + 16u * (uint32_t)t); };
  auto normalise = [&](const bf16* s, float eps) {
    landed(N);
    const int row = (warp + block) % (MT * KS);
    if (row < p.tokens) norm_rows<NB>(s, row, MT * KS, p.tokens, sX, P::PITCH, sN, sN + 2 * H, eps);
    __syncthreads();
  };
  // rows beyond the tokens repeat the last one; their results are dropped
  const bf16* rows_of[2];
  auto activations = [&](const bf16* s, int width) {
#pragma unroll
    for (int r = 0; r < 2; ++r) rows_of[r] = s + (int64_t)min(16 * mt + g + 8 * r, p.tokens - 1) * width + 8 * t;
  };
  auto from_l2 = [&](int r, int b) { return ld16g(rows_of[r] + 32 * b); };

  bool good = true;
  uint32_t due = 0;                                  // the barriers whose copies are on their way when the block gives up
  float acc[4][4];
  uint32_t bias = bias_of(p.layer[0].qkv_b + 8 * block, 12, H);
  __syncthreads();
  for (int i = 0; i < p.n_layers; ++i) {
    const ShortLayer& l = p.layer[i];
    const bool last = i + 1 == p.n_layers;
    // 1: q, k, v
    if (i > 0) normalise(p.z, p.layer[i - 1].eps2);
    landed(A);
    product(three, narrow, sA, P::PITCH, from_x, acc);
    finish(three, sA, acc, bias,
           [&](int row, int c, float a, float b) { put(p.qkv + (int64_t)row * 3 * H + (c >> 3) * H + 8 * block + (c & 7), a, b); });
    arrive();
    expected += blocks;
    bias = bias_of(l.out_b + 8 * block, 4, 0);
    // 2: attention
    if (block < takers) {
      if (!(good = meet())) { due = 1 << B; break; }
      for (int pair = block; pair < pairs; pair += blocks) {
        const int seq = pair / (H / 64), h = pair - seq * (H / 64);
        int tok0 = seq * p.length, len = p.length;
        if (p.cu_seqlens) {
          tok0 = max(0, min(__ldg(p.cu_seqlens + seq), p.tokens));
          len = min(__ldg(p.cu_seqlens + seq + 1) - tok0, p.tokens - tok0);
        }
        if (pair != block) {                         // behind the products that still read the head before
          __syncthreads();
          copy_tables(tables, l, h);
        }
        if (len > 0) short_attention<MT>(smem + P::OFF_A, tables, p.qkv, H, h, tok0, len, l, p.ctx);
      }
      arrive();
    }
    expected += takers;
    bring_up(l);
    if (!(good = meet())) { due = 1 << A | 1 << B; break; }
    // 3: output projection
    activations(p.ctx, H);
    landed(B);
    product(one, narrow, sB, P::PITCH, from_l2, acc);
    finish(one, sB, acc, bias,
           [&](int row, int c, float a, float b) { put(p.y + (int64_t)row * H + 8 * block + c, a, b); });
    arrive();
    expected += blocks;
    bring_down(l);
    bring_norm(l.ln1_w, l.ln1_b);
    bias = bias_of(l.up_b + 32 * block, 16, 8);
    if (!(good = meet())) { due = 1 << A | 1 << B | 1 << N; break; }
    // 4: intermediate projection
    normalise(p.y, l.eps1);
    landed(A);
    product(four, narrow, sA, P::PITCH, from_x, acc);
    finish(four, sA, acc, bias,
           [&](int row, int c, float a, float b) { put(p.u + (int64_t)row * 4 * H + 32 * block + c, gelu(a, bf16()), gelu(b, bf16())); });
    arrive();
    expected += blocks;
    if (!last) bring_qkv(p.layer[i + 1]);
    bias = bias_of(l.down_b + 8 * block, 4, 0);
    if (!(good = meet())) { due = (last ? 0 : 1 << A) | 1 << B; break; }
    // 5: second projection
    activations(p.u, 4 * H);
    landed(B);
    product(one, wide, sB, P::PITCH4, from_l2, acc);
    finish(one, sB, acc, bias, [&](int row, int c, float a, float b) { put(p.z + (int64_t)row * H + 8 * block + c, a, b); });
    arrive();
    expected += blocks;
    if (!last) bring_out(p.layer[i + 1]);
    bring_norm(l.ln2_w, l.ln2_b);
    if (!last) bias = bias_of(p.layer[i + 1].qkv_b + 8 * block, 12, H);
    if (!last && block < takers) copy_tables(tables, p.layer[i + 1], block % (H / 64));
    if (!(good = meet())) { due = (last ? 0 : 1 << A | 1 << B) | 1 << N; break; }
  }
  if (good) {                                        // the last layer's LayerNorm: a row per block
    landed(N);
    if (warp == 0 && block < p.tokens) {
      norm_rows<NB>(p.z, block, p.tokens, p.tokens, sX, P::PITCH, sN, sN + 2 * H, p.layer[p.n_layers - 1].eps2);
      __syncwarp();
      for (int c = lane; c < H / 8; c += 32)
        *reinterpret_cast<uint4*>(p.out + (int64_t)block * H + 8 * c) = ld16s(sX + (uint32_t)block * P::PITCH + 16u * (uint32_t)c);
    }
    // the last block to leave puts the counters back to zero: all have left their last meeting
    if (tid == 0 && atomicInc(reinterpret_cast<unsigned int*>(p.counter + 3), (unsigned int)(blocks - 1)) == (unsigned int)(blocks - 1))
      *reinterpret_cast<volatile int32_t*>(p.counter) = 0;
  }
  if (!good || late) {                               // copies that are still on their way come in before the block's memory is another's
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (tid == 0)
#pragma unroll
      for (int i = 0; i < BARS; ++i) {
        const uint64_t t0 = globaltimer_ns();
        while (((due | late) >> i & 1u) && !mbar_try_wait_parked(bars + 8u * i, phase[i], 20000u) && globaltimer_ns() - t0 < p.limit_ns) {}
      }
  }
}

template <int MT, int NB>
int launch_short(const ShortStack& p, cudaStream_t s) {
  auto kern = short_stack_kernel<MT, NB>;
  const int rc = opt_in_smem(reinterpret_cast<const void*>(kern), (int)Plan<MT, NB>::SMEM);
  if (rc) return rc;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeCooperative;
  attr.val.cooperative = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(32 * NB); cfg.blockDim = dim3(Plan<MT, NB>::THREADS); cfg.dynamicSmemBytes = Plan<MT, NB>::SMEM; cfg.stream = s;
  cfg.attrs = &attr; cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, p);
  const int failed = cuda_fail(e, "short stack launch");
  return e == cudaErrorCooperativeLaunchTooLarge ? TDB_ERR_UNSUPPORTED : failed;
}

// Whether all blocks can be resident at once on the current device; asked once per device.
template <int MT, int NB>
bool resident() {
  constexpr int MAX_DEV = 64;
  static int known[MAX_DEV] = {};                    // 1: they can, 2: they cannot; same value from every thread
  int dev = 0, sms = 0, cooperative = 0, per_sm = 0;
  if (cuda_fail(cudaGetDevice(&dev), "cudaGetDevice")) return false;
  if (dev < MAX_DEV && known[dev]) return known[dev] == 1;
  auto kern = short_stack_kernel<MT, NB>;
  if (device_sms(&sms) || opt_in_smem(reinterpret_cast<const void*>(kern), (int)Plan<MT, NB>::SMEM) ||
      cuda_fail(cudaDeviceGetAttribute(&cooperative, cudaDevAttrCooperativeLaunch, dev), "cudaDeviceGetAttribute") ||
      cuda_fail(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, Plan<MT, NB>::THREADS, Plan<MT, NB>::SMEM), "occupancy of the short stack"))
    return false;
  const bool fits = cooperative && per_sm * sms >= 32 * NB;
  if (dev < MAX_DEV) known[dev] = fits ? 1 : 2;
  return fits;
}

}  // namespace

}  // namespace tdb

using namespace tdb;

extern "C" {

// Hidden sizes whose columns the eight warps can share in whole blocks of 32, with a block per eight columns resident at once.  The tokens end at
// 32 because the attention has one tile of 32 keys, for which all score and band fragments are a warp's each; the shared memory would hold 48 at a hidden
// size of 768.  us per pass with a known mask on both sides of the line, 32 tokens here and 40 by the layer loop's recording: 165 and 200 (512, six layers), 306 and 416 (768,
// twelve), 639 and 874 (1024, 24).  Many short sequences cost a block several heads in turn: 32 sequences of one token 367 (768), as a recording 494.
int tdb_short_stack_applies(int64_t tokens, int64_t hidden, int64_t inner, int64_t layers) {
  if (tokens < 1 || tokens > SKINNY_TOKENS || layers < 1 || layers > SHORT_LAYERS || inner != 4 * hidden) return 0;
  const bool one = tokens <= 16;
  if (hidden == 512) return one ? resident<1, 2>() : resident<2, 2>();
  if (hidden == 768) return one ? resident<1, 3>() : resident<2, 3>();
  if (hidden == 1024) return one ? resident<1, 4>() : resident<2, 4>();
  return 0;
}

int tdb_short_stack(const ShortStack* p, int hidden, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  const bool one = p->tokens <= 16;
  if (hidden == 512) return one ? launch_short<1, 2>(*p, s) : launch_short<2, 2>(*p, s);
  if (hidden == 768) return one ? launch_short<1, 3>(*p, s) : launch_short<2, 3>(*p, s);
  if (hidden == 1024) return one ? launch_short<1, 4>(*p, s) : launch_short<2, 4>(*p, s);
  set_error("short stack: hidden size %d", hidden);
  return TDB_ERR_SHAPE;
}

}  // extern "C"
