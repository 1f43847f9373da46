// Far key tiles of long sequences on the sm_100a tensor cores (tcgen05 UMMA, accumulators in tensor memory).
//
// Where every distance of a 128x128 score tile lies at or beyond the saturation distance, on one side, all its scores use
// the same table row r of that side, and nothing has to be gathered:
//
//   s[i][j] = (Q[i].K[j] + Qr[r].K[j] + Q[i].Kr[r]) * scale
//
// The first two terms are two accumulating products (Qr[r] as an operand of 128 identical rows, which the expanded tables
// hold), the third is a constant of the query row that is added to its exponent.  What is left is plain attention, so this
// kernel is built like one: a persistent CTA takes pairs of query tiles (256 rows) of one head; two groups of eight warps own a
// tile each, two threads per row; while one group takes exponentials the tensor cores form the other's scores.
//
// The kernel for near key tiles (attn_umma.cu) has left each row's unnormalised output, reference exponent and sum in fp32;
// a group starts from that exponent, adds the near output at the end and writes the finished rows.  That state comes in as bulk
// copies while the item is at work (64 KB of outputs per pair of tiles, for which Q has one buffer and not two: the products run
// ahead of the exponentials by more than Q's way from memory), and the constants are formed one side per thread: read and formed by
// the groups at the item's ends, they took 6 of the 9.5 thousand clocks between two items.  Padded batches take the outer pairs
// first, which have most far tiles (far_work).  us per call before and after: 4 x 4096 tokens 512 and 502 (this kernel 252 and 237), 1 x 4096
// 212 and 170 (the order), 8 x 2048 350 and 337, 13 x 1200 286 and 270; 64 packed sequences of 2048 to 8192 the same, under the power cap.
//
// Bound: the special-function unit, 16384 exponentials per tile = 1024 clocks, beside 768 clocks of tensor work.  What matters
// is that neither waits for the other: three score buffers go round the two groups, so a group's next scores are complete
// before it has finished with the last ones, and only P.V follows its hand-off; and the two kinds of product are issued by two
// warps, because issuing blocks while the tensor pipe is busy and a lone issuing warp then adds its waits and commits (some
// 100 clocks each) to every batch.  A pair of tiles takes 2500 to 2800 clocks.  With one
// buffer per group and one issuing lane it took 4300, with three buffers and one issuing warp 3300; in the one kernel for all
// tiles, with one accumulator and all sixteen warps in step, 7400.  A quarter of the exponentials as polynomials on the FMA
// pipe, and tokens that let one group at a time take exponentials, were slower (254 us and 266 us against 242 of the version before).
//
// Error against float64: 2.392e-3 in the relative 2-norm at 1 x 4096, 2.379e-3 at 2 x 2048 with 64 buckets, against 2.389e-3 and
// 2.373e-3 of the one kernel for all tiles.  A pair of query tiles has its far tiles in common, so a tile more per side of each
// row is taken as a near one, whose bands are staged in bf16.
//
// Half-step t is group t & 1 at its tile t / 2.  Tensor-memory columns: three buffers of 128, S(t) in buffer t % 3 and P(t) (bf16)
// over the columns of S(t) that its own thread has read; O of the two groups at [384,448) [448,512).
// All hand-offs are mbarriers with bounded waits; a wait that gives up sets the CTA's abort flag, after which every role runs
// out its loops (the groups take their trip counts from one copy of the work item, so their named barriers still match), tensor
// memory is freed and the host reports it.
#include "attn_common.cuh"
#include <math_constants.h>
#include <algorithm>

namespace tdb {
using namespace ptx;

namespace {

constexpr int GW = 8, GT = GW * 32;                  // warps, threads of a group
constexpr int F_THREADS = 2 * GT + 3 * 32;           // + a warp of single lanes (Q and K; V; scheduler), two MMA warps
constexpr int F_RING = 3, STAGES = 2, BUFS = 3;
constexpr uint32_t TILE = BQ * HD * 2;               // bytes of a 128 x 64 bf16 tile
// of an item: query tiles A and B, left and right row of Qr; the near kernel's outputs of both tiles, its exponents and sums; both rows of Kr
constexpr uint32_t NEAR = BQ * HD * 4;
constexpr uint32_t F_OFF_Q = 0, F_OFF_K = 4 * TILE, F_OFF_V = F_OFF_K + STAGES * TILE, F_OFF_N = F_OFF_V + STAGES * TILE;
constexpr uint32_t F_OFF_ML = F_OFF_N + 2 * NEAR, F_OFF_KR = F_OFF_ML + 2 * BQ * 8, F_OFF_BAR = F_OFF_KR + 2 * HD * 2;
constexpr uint32_t F_OFF_WORK = F_OFF_BAR + 256, F_OFF_ITEM = F_OFF_WORK + F_RING * 64, F_OFF_X = F_OFF_ITEM + 8 * 64;
constexpr uint32_t F_OFF_FLAG = F_OFF_X + 2 * 2 * BQ * 4;    // exchange: [group][half][row]
constexpr uint32_t F_SMEM = F_OFF_FLAG + 64 + 1024;
static_assert(F_SMEM <= 227 * 1024, "shared memory budget");
constexpr uint32_t F_TM_S = 0, F_TM_O = 384, F_TM_COLS = 512;
constexpr uint64_t F_WAIT_NS = 1000ull * 1000ull * 1000ull;

enum FBar { FQ_FULL = 0, FQ_EMPTY, FN_FULL, FN_EMPTY, FK_FULL = 4, FK_EMPTY = 6, FV_FULL = 8, FV_EMPTY = 10, FS_FULL = 12 /* per buffer */,
            FP_READY = 15 /* per group */, FPV_DONE = 17, FWORK_FULL = 19, FWORK_EMPTY = 22, FDONE = 25 /* two */, FBUF_FREE = 27, F_NBARS = 30 };
constexpr int F_READERS = 4 + 1;                     // K lane, V lane, two MMA warps, the groups' leader

// A pair of query tiles of one head and its far key tiles: [0, n_left) and [right, right + n_far - n_left).
struct FarWork {
  int q0, len, rows, bcoord, h, n_left, right, n_far;          // n_far < 0: end of the stream
  int64_t tok0;
  int32_t seq, pad[5];
};
static_assert(sizeof(FarWork) == 64, "a ring slot");

// Index space: packed form, the listed tiles (of which every second one of a sequence has nothing to do); padded form, pairs of
// tiles, from the ends of the sequences inwards: the outer pairs have most far tiles, and the cheapest come last.  That order goes through
// one group of neighbouring sequences after another (p.far_group of them), because K and V of a whole group are in use at once.  32 MB of
// them is where more sequences stop helping the tail and begin to cost memory traffic.  us per call, 12 heads, groups of 1, 2, 4, 8 and all
// sequences (and pairs in their natural order): 16 x 4096 tokens (12.6 MB each) 1870, 1861, 1891, 1945, 1977 (1892); 8 x 8192 (25 MB) 3025,
// 3046, 3174, 3286 (3025); 64 x 2048 (6.3 MB) 2490, 2494, 2492, 2490, 2533 (2541); 48 x 1000..3000 (9.2 MB) 2292, 2301, 2309, 2321, 2376 (2331);
// 2 x 4096 265, 261 (312); 3 x 3000 249, 244, of three 240 (277).  Over 36 batches of at most 16384 tokens, 1152 and more each: 0.4 % faster than
// all sequences at once, from 6 % faster to 1.5 % slower (16 MB 0.3 %, 9 % to 3.3 %; 48 and 64 MB 0.1 %).
constexpr int64_t GROUP_BYTES = 32 << 20;
__device__ __forceinline__ int far_rows(const AttnParams& p) {
  return p.varlen ? reinterpret_cast<const int32_t*>(p.workspace)[0] : p.n_seqs * ((p.L + 2 * BQ - 1) / (2 * BQ));
}
// False: past the last index.  n_far == 0: nothing to do at this index.
__device__ __forceinline__ bool far_work(const AttnParams& p, int total, int w, FarWork& k) {
  const int tile = w / p.H;
  if (tile >= total) return false;
  k.h = w - tile * p.H;
  if (p.varlen) {
    const int2 e = reinterpret_cast<const int2*>(reinterpret_cast<const int32_t*>(p.workspace) + 4)[tile];
    const int c0 = p.cu_seqlens[e.x];
    k.len = p.cu_seqlens[e.x + 1] - c0; k.rows = k.len; k.tok0 = c0; k.bcoord = 0; k.q0 = e.y; k.seq = e.x;
  } else {
    const int pairs = (p.L + 2 * BQ - 1) / (2 * BQ), group = tile / (p.far_group * pairs), first = group * p.far_group;
    const int seqs = min(p.far_group, p.n_seqs - first), at = tile - first * pairs, rank = at / seqs, seq = first + at - rank * seqs;
    k.q0 = ((rank & 1) ? pairs - 1 - rank / 2 : rank / 2) * (2 * BQ);
    const int len = p.seqlens ? p.seqlens[seq] : p.L;
    k.len = len < 0 ? 0 : (len > p.L ? p.L : len);
    k.rows = p.L; k.tok0 = 0; k.bcoord = seq; k.seq = seq;
  }
  k.n_left = 0; k.right = 0; k.n_far = 0;
  if ((k.q0 & BQ) || k.q0 >= k.len) return true;     // the second tile of a pair, or padding
  const int all = (k.len + BK - 1) / BK;
  k.n_left = near_first(k.q0, p.split_sat);
  k.right = near_end(k.q0, p.split_sat);
  k.n_far = k.n_left + (all > k.right ? all - k.right : 0);
  return true;
}

__device__ __forceinline__ int far_tile(const FarWork& k, int it) { return it < k.n_left ? it : k.right + (it - k.n_left); }

__device__ __forceinline__ bool group_vote(int grp, bool flag) {
  uint32_t r;
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      "setp.ne.u32 q, %1, 0;\n"
      "bar.red.or.pred p, %2, %3, q;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}"
      : "=r"(r) : "r"((uint32_t)flag), "r"(1 + grp), "n"(GT) : "memory");
  return r != 0;
}
__device__ __forceinline__ void groups_sync() { asm volatile("bar.sync 11, %0;" ::"n"(2 * GT) : "memory"); }
__device__ __forceinline__ void group_sync(int grp) { asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "n"(GT) : "memory"); }

// A far score without the row's constant, from global memory (rare path only): key . (query row + saturated row of Qr).
template <bool P2C>
__device__ __noinline__ float far_score(const __nv_bfloat16* q, const __nv_bfloat16* k, const __nv_bfloat16* r) {
  float acc = 0.f;
#pragma unroll 1
  for (int d = 0; d < HD; ++d) {
    const float kv = __bfloat162float(k[d]);
    acc = fmaf(__bfloat162float(q[d]), kv, acc);
    if (P2C) acc = fmaf(__bfloat162float(r[d]), kv, acc);
  }
  return acc;
}

template <bool C2P, bool P2C>
__global__ void __launch_bounds__(F_THREADS, 1)
attn_far_kernel(const AttnParams p, int32_t* counter, const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_qr) {
  extern __shared__ uint8_t smem_raw[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gbase = smem_raw + (sbase - smem_u32(smem_raw));
  const uint32_t bars = sbase + F_OFF_BAR;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + F_OFF_FLAG);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gbase + F_OFF_FLAG + 8);
  FarWork* ring = reinterpret_cast<FarWork*>(gbase + F_OFF_WORK);
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  auto wait = [&](int i, uint32_t parity) { return mbar_wait(bar(i), parity, abort_flag, p.status, 201 + i, F_WAIT_NS); };
  if (tid == 0) {
    *abort_flag = 0;
    for (int i = 0; i < F_NBARS; ++i) {
      const bool by_warps = i >= FP_READY && i < FP_READY + 2, by_readers = i >= FWORK_EMPTY && i < FWORK_EMPTY + F_RING;
      // Q is free when its products are done and both groups have taken their rows' constants; what the near kernel left, when both have read it
      mbar_init(bar(i), by_readers ? (uint32_t)F_READERS : by_warps ? (uint32_t)GW : i == FQ_EMPTY ? 3u : i == FN_EMPTY ? 2u : 1u);
    }
    fence_mbar_init();
  }
  if (warp == 2 * GW && lane == 0) {
    prefetch_tmap(&tm_q); prefetch_tmap(&tm_k); prefetch_tmap(&tm_v);
    if (P2C) prefetch_tmap(&tm_qr);
  }
  if (warp == 2 * GW + 1) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), F_TM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  // For the near kernel, which lets this one start with the end of its last CTA.  Let in earlier, as SMs fall idle, the CTAs of this kernel
  // made 36 padded batches of 1152 tokens and more 1.0 % slower in the geometric mean (2.8 % slower to 0.3 % faster), packed ones 0 to 0.4 %.
  wait_for_stream();
  const int total = far_rows(p);
  int32_t gave_up_before = 0;
  if (warp == 2 * GW && lane == 2) gave_up_before = *reinterpret_cast<volatile int32_t*>(p.gave_up);

  auto fetch = [&](int n, FarWork& k) {
    wait(FWORK_FULL + (n % F_RING), (uint32_t)((n / F_RING) & 1));
    k = ring[n % F_RING];
    if (*abort_flag) k.n_far = -1;
    return k.n_far > 0;
  };
  auto release = [&](int n) { mbar_arrive(bar(FWORK_EMPTY + (n % F_RING))); };
  // where the near kernel has left the state of an item's tile
  auto state_of = [&](const FarWork& k, int tile) { return partial_tile(p, k.tok0, k.seq, k.bcoord, k.q0 + BQ * tile) * p.H + k.h; };

  if (warp == 2 * GW) {
    // ================================ TMA producers and scheduler ============================
    if (lane == 0) {                                 // per item what its products and its rows' constants need, then K
      FarWork k;
      int g = 0, n = 0;
      for (; fetch(n, k); release(n), ++n) {
        const uint32_t q = sbase + F_OFF_Q;
        const bool both = k.q0 + BQ < k.len;         // the near kernel has left something of the second tile too
        if (n >= 1) wait(FQ_EMPTY, (uint32_t)((n - 1) & 1));
        if (!*abort_flag) {
          mbar_expect_tx(bar(FQ_FULL), (P2C ? 4 : 2) * TILE + (C2P ? 2 * HD * 2 : 0) + (both ? 2 : 1) * BQ * 8);
          tma_load_4d(q, &tm_q, bar(FQ_FULL), 0, (int)k.tok0 + k.q0, k.h, k.bcoord);
          if (P2C) {
            tma_load_3d(q + 2 * TILE, &tm_qr, bar(FQ_FULL), 0, p.exp_rows - BQ, k.h);     // distances far above zero
            tma_load_3d(q + 3 * TILE, &tm_qr, bar(FQ_FULL), 0, 0, k.h);                    // far below
          }
          tma_load_4d(q + TILE, &tm_q, bar(FQ_FULL), 0, (int)k.tok0 + k.q0 + BQ, k.h, k.bcoord);
          if (C2P) {
            const __nv_bfloat16* kr = reinterpret_cast<const __nv_bfloat16*>(p.kr_exp) + (int64_t)k.h * p.exp_rows * HD;
            bulk_load(sbase + F_OFF_KR, kr + (int64_t)(p.exp_rows - 1) * HD, HD * 2, bar(FQ_FULL));
            bulk_load(sbase + F_OFF_KR + HD * 2, kr, HD * 2, bar(FQ_FULL));
          }
          for (int i = 0; i < (both ? 2 : 1); ++i)
            bulk_load(sbase + F_OFF_ML + (uint32_t)i * BQ * 8, p.part_ml + state_of(k, i) * (2 * BQ), BQ * 8, bar(FQ_FULL));
        }
        for (int it = 0; it < k.n_far; ++it, ++g) {
          const int st = g % STAGES;
          if (g >= STAGES) wait(FK_EMPTY + st, (uint32_t)((g / STAGES - 1) & 1));
          if (!*abort_flag) {
            mbar_expect_tx(bar(FK_FULL + st), TILE);
            tma_load_4d(sbase + F_OFF_K + st * TILE, &tm_k, bar(FK_FULL + st), 0, (int)k.tok0 + far_tile(k, it) * BK, k.h, k.bcoord);
          }
        }
      }
      release(n);
    } else if (lane == 1) {                          // V
      FarWork k;
      int g = 0, n = 0;
      for (; fetch(n, k); release(n), ++n)
        for (int it = 0; it < k.n_far; ++it, ++g) {
          const int st = g % STAGES;
          if (g >= STAGES) wait(FV_EMPTY + st, (uint32_t)((g / STAGES - 1) & 1));
          if (!*abort_flag) {
            mbar_expect_tx(bar(FV_FULL + st), TILE);
            tma_load_4d(sbase + F_OFF_V + st * TILE, &tm_v, bar(FV_FULL + st), 0, (int)k.tok0 + far_tile(k, it) * BK, k.h, k.bcoord);
          }
          if (it != (k.n_far > 1 ? 1 : 0)) continue;
          // the near kernel's outputs: needed at the item's end, the buffer is free since the end of the one before
          if (n >= 1) wait(FN_EMPTY, (uint32_t)((n - 1) & 1));
          if (*abort_flag) continue;
          const bool both = k.q0 + BQ < k.len;
          mbar_expect_tx(bar(FN_FULL), (both ? 2 : 1) * NEAR);
          for (int i = 0; i < (both ? 2 : 1); ++i)
            bulk_load(sbase + F_OFF_N + (uint32_t)i * NEAR, p.part_o + state_of(k, i) * (BQ * HD), NEAR, bar(FN_FULL));
        }
      release(n);
    } else if (lane == 2) {
      // Scheduler.  Every CTA with an index of its own draws until its first draw past the end: as many draws as indices, and
      // the counter wraps back to zero (see attn_umma.cu).
      const unsigned int last_item = (unsigned int)(total * p.H - 1);
      int n = 0;
      bool first = true;
      while (true) {
        const int w = (*abort_flag || gave_up_before != 0) ? 0x7fffffff
                      : first ? (int)blockIdx.x
                              : (int)gridDim.x + (int)atomicInc(reinterpret_cast<unsigned int*>(counter), last_item);
        first = false;
        FarWork k;
        if (!far_work(p, total, w, k)) k.n_far = -1;
        if (k.n_far == 0) continue;
        if (n >= F_RING) wait(FWORK_EMPTY + (n % F_RING), (uint32_t)(((n / F_RING) - 1) & 1));
        ring[n % F_RING] = k;
        mbar_arrive(bar(FWORK_FULL + (n % F_RING)));
        ++n;
        if (k.n_far < 0) break;
      }
    }
  } else if (warp >= 2 * GW + 1) {
    // ================================ MMA issuer ============================================
    // First warp: scores; second: P.V.  The whole warp walks its loop and one elected lane issues.
    constexpr uint32_t ID_S = make_idesc_bf16(128, BK, 0), ID_PV = make_idesc_bf16(128, HD, 1);
    const uint64_t dQ = smem_desc_sw128(sbase + F_OFF_Q), dK = smem_desc_sw128(sbase + F_OFF_K), dV = smem_desc_sw128(sbase + F_OFF_V);
    constexpr uint64_t STEP = TILE >> 4;
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
    struct Cur { int n, it, n_far, n_left; };          // item, its tile; n_far <= 0: end of the stream
    auto load_item = [&](Cur& c) {
      FarWork k;
      fetch(c.n, k);
      __syncwarp();
      c.n_far = __shfl_sync(0xffffffffu, k.n_far, 0);
      c.n_left = __shfl_sync(0xffffffffu, k.n_left, 0);
    };
    Cur c{0, 0, 0, 0};
    load_item(c);
    if (warp == 2 * GW + 1) {
#pragma unroll 1
      for (int t = 0; c.n_far > 0; ++t) {
        const int grp = t & 1, g = t >> 1, buf = t % BUFS;
        if (grp == 0) {
          if (c.it == 0) wait(FQ_FULL, (uint32_t)(c.n & 1));
          wait(FK_FULL + (g % STAGES), (uint32_t)((g / STAGES) & 1));
        }
        if (t >= BUFS) wait(FBUF_FREE + buf, (uint32_t)((t / BUFS - 1) & 1));
        tc_fence_after();
        const uint32_t tS = tm + F_TM_S + 128u * (uint32_t)buf;
        const uint64_t q = dQ, kd = dK + (uint64_t)(g % STAGES) * STEP;
#pragma unroll
        for (int i = 0; i < HD / 16; ++i) mma_ss_warp(tS, q + (uint64_t)grp * STEP + 2 * i, kd + 2 * i, ID_S, i > 0);
        if (P2C) {
          const uint64_t r = q + (c.it < c.n_left ? 2 : 3) * STEP;
#pragma unroll
          for (int i = 0; i < HD / 16; ++i) mma_ss_warp(tS, r + 2 * i, kd + 2 * i, ID_S, 1u);
        }
        tc_commit_warp(bar(FS_FULL + buf));
        if (grp == 1) {
          tc_commit_warp(bar(FK_EMPTY + (g % STAGES)));
          if (++c.it == c.n_far) {
            tc_commit_warp(bar(FQ_EMPTY));
            if (lane == 0) release(c.n);
            ++c.n; c.it = 0;
            load_item(c);
          }
        }
      }
    } else {
#pragma unroll 1
      for (int t = 0; c.n_far > 0; ++t) {
        const int grp = t & 1, g = t >> 1, buf = t % BUFS;
        if (grp == 0) wait(FV_FULL + (g % STAGES), (uint32_t)((g / STAGES) & 1));
        wait(FP_READY + grp, (uint32_t)(g & 1));
        tc_fence_after();
        const uint64_t vd = dV + (uint64_t)(g % STAGES) * STEP;
        const uint32_t tP = tm + F_TM_S + 128u * (uint32_t)buf, tO = tm + F_TM_O + 64u * (uint32_t)grp;
#pragma unroll
        for (int i = 0; i < BK / 16; ++i)                // keys 64.. of P lie over columns 64.. of the scores
          mma_ts_warp(tO, tP + 8u * (uint32_t)(i & 3) + 64u * (uint32_t)(i >> 2), vd + (uint64_t)(128 * i), ID_PV, (c.it > 0 || i > 0) ? 1u : 0u);
        tc_commit_warp(bar(FBUF_FREE + buf));
        tc_commit_warp(bar(FPV_DONE + grp));
        if (grp == 1) {
          tc_commit_warp(bar(FV_EMPTY + (g % STAGES)));
          if (++c.it == c.n_far) {
            if (lane == 0) release(c.n);
            ++c.n; c.it = 0;
            load_item(c);
          }
        }
      }
    }
    if (lane == 0) release(c.n);                       // the end-of-stream marker
    const int done = FDONE + (warp - 2 * GW - 1);
    tc_commit_warp(bar(done));
    int never = 0;                                     // this wait runs even after an abort, with its own limit
    mbar_wait(bar(done), 0, &never, p.status, 201 + FDONE, F_WAIT_NS);
  } else {
    // ================================ softmax groups ========================================
    const int grp = warp / GW, gw = warp % GW, gt = tid - grp * GT;
    const int qd = gw & 3, half = gw >> 2;
    const int row_t = qd * 32 + lane;
    const uint32_t lane_base = ((uint32_t)(qd * 32)) << 16;
    const uint32_t tO = tmem + lane_base + F_TM_O + 64u * (uint32_t)grp + 32u * (uint32_t)half;
    const uint32_t x_row = sbase + F_OFF_X + 4u * (uint32_t)(grp * 2 * BQ + row_t);             // + half * BQ * 4
    const float sl2 = p.sm_scale * 1.4426950408889634f;
    // Thread 0 takes the items from the ring one ahead of the stream (in an item's first tile it fetches the next); each
    // group's leader copies an item for its group before the barrier that ends the item before, so that all threads of a group
    // have the same trip count, also after an abort.
    FarWork* const items = reinterpret_cast<FarWork*>(gbase + F_OFF_ITEM);
    auto publish = [&](int n) {
      FarWork k;
      k.n_far = -1;
      if (n == 0 || items[(n - 1) & 3].n_far > 0) {    // nothing follows the end of the stream
        fetch(n, k);
        release(n);
      }
      items[n & 3] = k;
    };
    FarWork* const mine = items + 4 + 2 * grp;
    if (tid == 0) publish(0);
    groups_sync();
    if (gt == 0) mine[0] = items[0];
    group_sync(grp);
    int g = 0;
    for (int n = 0;; ++n) {
      const FarWork* const item = mine + (n & 1);
      const int n_far = item->n_far, n_left = item->n_left, right = item->right, len = item->len, h = item->h;
      const int row = item->q0 + BQ * grp + row_t;
      if (n_far <= 0) break;
      const int64_t tok = item->tok0 + row;                          // of the packed stream, or of its batch row
      const bool valid = row < len;
      wait(FQ_FULL, (uint32_t)(n & 1));
      float2 near = make_float2(0.f, 0.f);                           // the near tiles' exponent and sum
      if (valid) near = make_float2(lds_f32(sbase + F_OFF_ML + 8u * (uint32_t)(grp * BQ + row_t)), lds_f32(sbase + F_OFF_ML + 8u * (uint32_t)(grp * BQ + row_t) + 4u));
      float c_left = 0.f, c_right = 0.f;
      if (C2P) {                                                     // Q[i].Kr[r], a side by each of the row's two threads
        float c0 = 0.f, c1 = 0.f;
        if (half == 0 ? n_left > 0 : n_far > n_left) {
          const uint32_t qrow = sbase + F_OFF_Q + (uint32_t)grp * TILE + 128u * (uint32_t)row_t, kr = sbase + F_OFF_KR + (uint32_t)half * (HD * 2);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint4 a = lds_128(qrow + 16u * (uint32_t)(i ^ (row_t & 7))), b = lds_128(kr + 16u * (uint32_t)i);
            const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              c0 = fmaf(__uint_as_float(aw[e] << 16), __uint_as_float(bw[e] << 16), c0);
              c1 = fmaf(__uint_as_float(aw[e] & 0xffff0000u), __uint_as_float(bw[e] & 0xffff0000u), c1);
            }
          }
        }
        sts_f32(x_row + (uint32_t)half * (BQ * 4), (c0 + c1) * sl2);
        group_sync(grp);                                             // written again behind the first tile's vote at the earliest
        c_left = lds_f32(x_row);
        c_right = lds_f32(x_row + BQ * 4);
      }
      float m = near.x, l = 0.f;
      for (int it = 0; it < n_far; ++it, ++g) {
        const int kt = it < n_left ? it : right + (it - n_left);
        const int nv_tile = len - kt * BK, nvalid = nv_tile - 64 * half;   // keys e >= nvalid of this thread are masked
        const float c = it < n_left ? c_left : c_right;
        const int t = 2 * g + grp, buf = t % BUFS;
        const uint32_t tS = tmem + lane_base + F_TM_S + 128u * (uint32_t)buf + 64u * (uint32_t)half;
        wait(FS_FULL + buf, (uint32_t)((t / BUFS) & 1));
        tc_fence_after();
        if (it == 0 && tid == 0) publish(n + 1);
        // P of the thread's 64 keys: all scores first, so that nothing but the special-function unit paces the exponentials
        // (against the row's reference exponent); P goes over scores that have been read, sixteen keys at a time.
        float sum;
        {
          float x[64];
          const float bias = c - m;
          float s0 = 0.f, s1 = 0.f;
          tmem_ld32(tS, reinterpret_cast<uint32_t*>(x));
          tmem_ld32(tS + 32u, reinterpret_cast<uint32_t*>(x + 32));
          tmem_ld_wait32(reinterpret_cast<uint32_t*>(x));
          tmem_ld_wait32(reinterpret_cast<uint32_t*>(x + 32));
          if (nvalid < 64) {
#pragma unroll
            for (int e = 0; e < 64; ++e) x[e] = e < nvalid ? x[e] : -CUDART_INF_F;
          }
#pragma unroll
          for (int part = 0; part < 4; ++part) {
            uint32_t pk[8];
#pragma unroll
            for (int e = 0; e < 16; e += 2) {
              const float a = ex2(fmaf(x[16 * part + e], sl2, bias)), b = ex2(fmaf(x[16 * part + e + 1], sl2, bias));
              s0 += a; s1 += b;
              pk[e / 2] = pack_bf16x2(a, b);
            }
            tmem_st8(tS + 8u * (uint32_t)part, pk);
          }
          sum = s0 + s1;
        }
        if (g > 0) wait(FPV_DONE + grp, (uint32_t)((g - 1) & 1));    // done long ago; keeps the barrier's phases in step
        // A bf16 probability and an fp32 sum have room for 2^64 times the near tiles' exponent; a row beyond that (or the
        // overflow it led to) moves its exponent, and with it this tile's P and the output so far.  Its scores are gone, so
        // they are formed again, on the CUDA cores.
        if (group_vote(grp, valid && sum > 1.8e19f)) {
          const __nv_bfloat16* q = reinterpret_cast<const __nv_bfloat16*>(p.q) + (int64_t)item->bcoord * p.q_sb +
                                   (valid ? tok : item->tok0) * p.q_st + (int64_t)h * p.q_sh;
          const __nv_bfloat16* k = reinterpret_cast<const __nv_bfloat16*>(p.k) + (int64_t)item->bcoord * p.k_sb +
                                   (item->tok0 + kt * BK + 64 * half) * p.k_st + (int64_t)h * p.k_sh;
          const __nv_bfloat16* r = reinterpret_cast<const __nv_bfloat16*>(p.qr_exp) +
                                   ((int64_t)h * p.exp_rows + (it < n_left ? p.exp_rows - 1 : 0)) * HD;
          float mx = -CUDART_INF_F;
#pragma unroll 1
          for (int e = 0; e < 64 && e < nvalid; ++e) mx = fmaxf(mx, far_score<P2C>(q, k + e * p.k_st, r));
          sts_f32(x_row + (uint32_t)half * (BQ * 4), mx);
          group_sync(grp);
          const float top = fmaf(fmaxf(lds_f32(x_row), lds_f32(x_row + BQ * 4)), sl2, c);
          const bool redo = valid && top - m > 8.f;
          if (__any_sync(0xffffffffu, redo)) {
            const float m_new = redo ? top : m, alpha = redo ? ex2(m - top) : 1.f, bias = c - m_new;
            tmem_st_wait();
            sum = 0.f;
#pragma unroll 1
            for (int part = 0; part < 4; ++part) {
              uint32_t pk[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) {
                const int j = 16 * part + 2 * e;
                const float a = j < nvalid ? ex2(fmaf(far_score<P2C>(q, k + j * p.k_st, r), sl2, bias)) : 0.f;
                const float b = j + 1 < nvalid ? ex2(fmaf(far_score<P2C>(q, k + (j + 1) * p.k_st, r), sl2, bias)) : 0.f;
                sum += a + b;
                pk[e] = pack_bf16x2(a, b);
              }
              __syncwarp();
              tmem_st8(tS + 8u * (uint32_t)part, pk);
            }
            if (it > 0) {
              uint32_t o[32];
              tc_fence_after();
              tmem_ld32(tO, o);
              tmem_ld_wait32(o);
#pragma unroll
              for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
              tmem_st32(tO, o);
            }
            l *= alpha;
            m = m_new;
          }
        }
        l += sum;
        if (it == 0 && gt == 0) mbar_arrive(bar(FQ_EMPTY));                // behind the vote: the group has read its rows of Q
        // Keys beyond the sequence have exact zeros as probabilities, but their rows of V may hold anything (0 x NaN): group A
        // zeroes them in shared memory before it announces P, and the other group's product is issued after its own.
        if (grp == 0 && nv_tile < BK) {
          const int st = g % STAGES;
          wait(FV_FULL + st, (uint32_t)((g / STAGES) & 1));
          for (int i = gt; i < (BK - nv_tile) * 8; i += GT)
            sts_128(sbase + F_OFF_V + st * TILE + (uint32_t)(nv_tile + (i >> 3)) * 128u + 16u * (uint32_t)(i & 7), 0u, 0u, 0u, 0u);
          fence_proxy_async_smem();
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(FP_READY + grp));
      }
      // (far output + near output) / sum -> global
      group_sync(grp);                               // the last tile may have exchanged maxima in the same words
      sts_f32(x_row + (uint32_t)half * (BQ * 4), l);
      group_sync(grp);
      const float beta = ex2(near.x - m);
      const float l_tot = fmaf(near.y, beta, lds_f32(x_row) + lds_f32(x_row + BQ * 4));
      wait(FN_FULL, (uint32_t)(n & 1));
      float nr[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) nr[i] = valid ? lds_f32(sbase + F_OFF_N + (uint32_t)grp * NEAR + 4u * (uint32_t)((32 * half + i) * BQ + row_t)) : 0.f;
      wait(FPV_DONE + grp, (uint32_t)((g - 1) & 1));
      tc_fence_after();
      uint32_t r[32];
      tmem_ld32(tO, r);
      tmem_ld_wait32(r);
      tc_fence_before();
      if (row < item->rows) {
        float inv;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(l_tot));
        uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.o) + (int64_t)item->bcoord * p.o_sb + tok * p.o_st +
                                              (int64_t)h * p.o_sh + 32 * half);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float* v = nr + 8 * i;
          uint32_t w[4];
#pragma unroll
          for (int e = 0; e < 4; ++e)
            w[e] = valid ? pack_bf16x2(fmaf(v[2 * e], beta, __uint_as_float(r[8 * i + 2 * e])) * inv,
                                       fmaf(v[2 * e + 1], beta, __uint_as_float(r[8 * i + 2 * e + 1])) * inv) : 0u;
          dst[i] = make_uint4(w[0], w[1], w[2], w[3]);
        }
        if (p.lse && half == 0)
          p.lse[(int64_t)item->bcoord * p.lse_sb + (int64_t)h * p.lse_sh + tok] = valid ? m * 0.6931471805599453f + logf(l_tot) : 0.f;
      }
      if (gt == 0) mine[(n + 1) & 1] = items[(n + 1) & 3];
      group_sync(grp);                               // the exchange words are free again, and the near outputs have been read
      if (gt == 0) mbar_arrive(bar(FN_EMPTY));
    }
  }

  // ---- teardown ------------------------------------------------------------------------------
  if (*abort_flag) {                      // give copies that may still be in flight time to land
    if (tid == 0 && p.gave_up != p.status) *reinterpret_cast<volatile int32_t*>(p.gave_up) = 1;
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 2 * GW + 1) tmem_dealloc(tmem, F_TM_COLS);
}

template <bool C2P, bool P2C>
int launch_far_variant(const AttnParams& p, dim3 grid, const CUtensorMap* maps, cudaStream_t s) {
  auto kern = attn_far_kernel<C2P, P2C>;
  const int rc = opt_in_smem(reinterpret_cast<const void*>(kern), (int)F_SMEM);
  if (rc) return rc;
  return cuda_fail(launch_early(kern, grid, F_THREADS, F_SMEM, s, p, p.counter + 2, maps[0], maps[1], maps[2], maps[3]), "attn_far launch");
}

}  // namespace

// `tiles`: query tiles of the whole problem (an upper bound in the packed form, whose list says how many there are); at least as many as
// the kernel's indices.
int launch_attn_far(const AttnParams& given, int64_t tiles, int sms, cudaStream_t s) {
  AttnParams p = given;
  const int64_t kv_bytes = (int64_t)p.L * p.H * 2 * HD * 2;             // of a padded sequence
  const int most = (int)std::max<int64_t>(1, std::min<int64_t>(p.n_seqs, GROUP_BYTES / std::max<int64_t>(1, kv_bytes)));
  const int groups = (p.n_seqs + most - 1) / most;
  p.far_group = (p.n_seqs + groups - 1) / groups;                       // of about the same size
  CUtensorMap maps[4];
  const int64_t tokens = p.varlen ? p.total_tokens : p.L;
  const int B = p.varlen ? 1 : p.n_seqs;
  int rc;
  if ((rc = token_map(&maps[0], p.q, tokens, p.H, B, p.q_sb, p.q_st, p.q_sh, "q"))) return rc;
  if ((rc = token_map(&maps[1], p.k, tokens, p.H, B, p.k_sb, p.k_st, p.k_sh, "k"))) return rc;
  if ((rc = token_map(&maps[2], p.v, tokens, p.H, B, p.v_sb, p.v_st, p.v_sh, "v"))) return rc;
  const bool c2p = p.flags & TDB_FLAG_C2P, p2c = p.flags & TDB_FLAG_P2C;
  if (p2c) {
    if ((rc = table_map(&maps[3], p.qr_exp, p.exp_rows, p.H, BQ, "qr_exp (far tiles)"))) return rc;
  } else {
    maps[3] = maps[0];
  }
  const int64_t items = tiles * p.H;
  dim3 grid((unsigned)(items < sms ? items : sms), 1, 1);
  if (c2p && p2c) return launch_far_variant<true, true>(p, grid, maps, s);
  if (c2p) return launch_far_variant<true, false>(p, grid, maps, s);
  return launch_far_variant<false, true>(p, grid, maps, s);
}

}  // namespace tdb
