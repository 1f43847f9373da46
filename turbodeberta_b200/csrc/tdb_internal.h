// Internal declarations shared by the translation units of libtdb_b200.so.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include <stddef.h>
#include "../../include/tdb_b200.h"

namespace tdb {

// One attention problem in either form.  Padded form: sequence s is batch row s, tokens 0..L-1,
// valid length seqlens[s] (or L).  Packed form: sequence s is tokens cu_seqlens[s]..cu_seqlens[s+1]-1
// of batch row 0.
struct AttnParams {
  const void* q; const void* k; const void* v; void* o;
  int64_t q_sb, q_st, q_sh;
  int64_t k_sb, k_st, k_sh;
  int64_t v_sb, v_st, v_sh;
  int64_t o_sb, o_st, o_sh;
  const void* kr; const void* qr; int two_span;          // [H, two_span, D] of the I/O dtype
  const int16_t* idx; int idx_delta_max;                  // delta -> table row
  const void* kr_exp; const void* qr_exp;                 // [H, exp_rows, D] bf16, row x <-> delta = x - exp_delta_max
  // Materialised position scores (legacy op interface): c2p_scores[b, h, t, r] = Q[t].Kr[r], p2c_scores[b, h, t, r]
  // = K[t].Qr[r], rows of two_span contiguous elements of the I/O dtype.  When set they replace kr / qr.
  const void* c2p_scores; const void* p2c_scores;
  int64_t c2p_sb, c2p_st, c2p_sh, p2c_sb, p2c_st, p2c_sh;
  int exp_delta_max, exp_rows;
  const int32_t* seqlens;                                 // padded form, may be null
  const int32_t* cu_seqlens;                              // packed form
  int varlen;
  int n_seqs;                                             // B, or number of packed sequences
  int L;                                                  // padded length, or max_seqlen
  int64_t total_tokens;                                   // packed form: T
  int H, D;
  float sm_scale;
  int flags;
  float* lse; int64_t lse_sb, lse_sh;                     // lse[b*lse_sb + h*lse_sh + t] or null
  int32_t* status;                                        // device-visible words: 0 = gave-up code, 1 = malformed offsets (3: see tdb_embed)
  // Tensor-core kernel: the device-wide work counter (zero on entry, and zero again once the launch has finished) and the
  // flag that makes CTAs starting after a wait gave up hand out no work.  Null: status words 2 (reset by the launch) and 0.
  // counter[2] is a second counter, of the kernel for far tiles.
  int32_t* counter; int32_t* gave_up;
  void* workspace; size_t workspace_bytes;
  // Long sequences on the tensor cores: scratch for the softmax state that the kernel for near key tiles hands to the one for
  // far tiles, tdb_partial_floats() of fp32, part_ml behind part_o's tiles (null: one kernel does both).  split_sat and far_group are the launchers' own.
  float* part_o; float* part_ml; int split_sat; int far_group;
  int lengths_known;                                      // packed form: L is known to be the longest sequence's length
  int direct_tables;                                      // kr and qr are read by index; kr_exp and qr_exp do not exist (kernel for short sequences only)
  int tiles_listed;                                       // packed form: the workspace already holds this batch's tile list
};

// Launches a kernel that may start while the kernel in front of it on the stream is still running: its set-up (barriers,
// tensor memory, descriptors) then costs nothing.  The kernel calls wait_for_stream() before it touches anything that earlier
// work may have written or may still read.
template <typename... K, typename... A>
inline cudaError_t launch_stream(void (*kernel)(K...), dim3 grid, unsigned block, size_t smem, cudaStream_t s, bool early, A&&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid; cfg.blockDim = dim3(block); cfg.dynamicSmemBytes = smem; cfg.stream = s;
  cfg.attrs = &attr; cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<K>(args)...);
}
template <typename... K, typename... A>
inline cudaError_t launch_early(void (*kernel)(K...), dim3 grid, unsigned block, size_t smem, cudaStream_t s, A&&... args) {
  return launch_stream(kernel, grid, block, smem, s, true, static_cast<A&&>(args)...);
}
#ifdef __CUDACC__
__device__ __forceinline__ void wait_for_stream() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// From here on the next kernel may start (it waits by itself for what this one writes).  Called behind wait_for_stream(), or by a kernel that
// is launched behind the one in front and has nothing to wait for (the tile list), so that one kernel is ahead at a time: with the call in front of the wait five of a layer's kernels piled up on the SMs, and a
// pass of 32 tokens through the base model took 546 us instead of 496.
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

void set_error(const char* fmt, ...);
int cuda_fail(cudaError_t e, const char* what);

int device_sms(int* sms);                                            // of the current device; asked once per device
int opt_in_smem(const void* kernel, int bytes);                      // dynamic shared memory beyond 48 KB, set once per device

int launch_bucket_table(int buckets, int max_pos, int delta_max, int16_t* out, cudaStream_t s);
int launch_relpos_project(const void* rel, const void* W, const void* bias, int two_span, int hidden,
                          int H, int D, int dtype, void* out, cudaStream_t s);
bool relpos_umma_applicable(const void* rel, const void* W, const void* out, int hidden, int D, int dtype);
int launch_relpos_project_umma(const void* rel, const void* W, const void* bias, int two_span, int hidden, int H,
                               void* out, int32_t* status, cudaStream_t s);
int launch_relpos_expand(const void* table, const int16_t* idx, int idx_delta_max, int H, int two_span, int D,
                         int dtype, int exp_delta_max, int exp_rows, void* out, cudaStream_t s);
int launch_bounded_wait_selftest(int32_t* status, int code, uint64_t limit_ns, cudaStream_t s);
int launch_attn_simt(const AttnParams& p, int dtype, cudaStream_t s);
int launch_attn_scores(const AttnParams& p, cudaStream_t s);          // bf16, materialised position scores
bool small_applicable(const AttnParams& p);                            // short sequences: padded, or packed with a known longest
int launch_attn_small(const AttnParams& p, cudaStream_t s);
int launch_attn_umma(const AttnParams& p, cudaStream_t s);
bool has_far_tiles(const AttnParams& p);
size_t umma_workspace_bytes(int n_seqs, int64_t total_tokens);
int launch_relpos_expand_pair(const void* kr, const void* qr, const int16_t* idx, int idx_delta_max, int H, int two_span,
                              int exp_delta_max, int exp_rows, void* kr_out, void* qr_out, cudaStream_t s);
int static_tile_scratch(void** ptr);   // device address of the library's fixed tile-list array on the current device

}  // namespace tdb

constexpr int SKINNY_TOKENS = 32;
namespace tdb {
// The encoder's layers as encoder_short.cu takes them, all of them bf16: weights [features, columns], tables as in AttnParams (null: absent).
constexpr int SHORT_LAYERS = 48;
struct ShortLayer {
  const __nv_bfloat16 *qkv_w, *qkv_b, *out_w, *out_b, *ln1_w, *ln1_b, *up_w, *up_b, *down_w, *down_b, *ln2_w, *ln2_b, *kr, *qr;
  float eps1, eps2, sm_scale;
  int exp_delta_max, exp_rows;
};
struct ShortStack {
  ShortLayer layer[SHORT_LAYERS];
  int n_layers, tokens, n_seqs, length;               // length: of every sequence, where there are no offsets
  const __nv_bfloat16* x;                             // [tokens, hidden], like out, ctx, y and z; qkv: three times, u: four times as wide
  __nv_bfloat16 *out, *qkv, *ctx, *y, *u, *z;
  const int32_t* cu_seqlens;
  int32_t *status, *counter, *gave_up;                // as in AttnParams; counter[0] and counter[3] are zero on entry and again at the end
  uint64_t limit_ns;                                  // of a wait, after which the kernel gives up
};
}  // namespace tdb

// What the host extension calls (the checks and the launch behind the tdb_attn_fwd_* entry points on a filled AttnParams,
// and kernels that have no C entry point of their own).
#define TDB_HOST_API __attribute__((visibility("default")))
extern "C" {
TDB_HOST_API int tdb_run_attn(const tdb::AttnParams* p, int dtype, int kernel, void* stream);
// Floats of part_o and part_ml together that the call could use (0: none), for p as it will be passed to tdb_run_attn; part_ml
// starts at 64 / 66 of them.
TDB_HOST_API int64_t tdb_partial_floats(const tdb::AttnParams* p, int dtype, int kernel);
// Whether the call runs on the kernel that can do without expanded tables (AttnParams::direct_tables).
TDB_HOST_API int tdb_takes_direct_tables(const tdb::AttnParams* p, int dtype, int kernel);
TDB_HOST_API int tdb_expand_pair(const void* kr, const void* qr, const int16_t* idx, int idx_delta_max, int H, int two_span,
                                 int exp_delta_max, int exp_rows, void* kr_out, void* qr_out, void* stream);
// early: as for tdb_skinny, of w and b.
TDB_HOST_API int tdb_add_layernorm(const void* x, const void* res, const void* w, const void* b, float eps, int64_t rows, int hidden,
                                   int dtype, void* out, int early, void* stream);
// Embeddings of `rows` tokens (ids of 4 or 8 bytes, a mask of 1 or 8): see embed_kernel.  An id outside the vocabulary, which is the
// caller's mistake and not a failure of the device, has a status word of its own: 3.
TDB_HOST_API int tdb_embed(const void* ids, int id_bytes, const void* table, int64_t vocabulary, const void* w, const void* b, float eps, const void* mask,
                           int mask_bytes, int64_t rows, int hidden, int dtype, void* out, int32_t* status, void* stream);
TDB_HOST_API int tdb_gelu(void* x, int64_t elements, int dtype, void* stream);
// bf16 projection of a few tokens, y = x W^T + b, through GELU if asked.  early: may start beside the kernel in front, which
// then must not be what wrote W (W is read before the wait for it).
TDB_HOST_API int tdb_skinny_applies(int64_t T, int64_t K, int64_t N);
TDB_HOST_API int tdb_skinny(const void* x, const void* w, const void* b, int T, int K, int N, int gelu, int early, void* y, void* stream);
// All layers for at most SKINNY_TOKENS tokens in one kernel whose blocks wait for one another.  TDB_ERR_UNSUPPORTED: not all of them can be
// resident where the stream may run.
TDB_HOST_API int tdb_short_stack_applies(int64_t tokens, int64_t hidden, int64_t inner, int64_t layers);
TDB_HOST_API int tdb_short_stack(const tdb::ShortStack* p, int hidden, void* stream);
TDB_HOST_API int tdb_mask_rows(const void* mask, int elem_bytes, int B, int L, int32_t* seqlens, int32_t* cu, int32_t* ticket,
                               int32_t* out, void* stream);
TDB_HOST_API int tdb_mask_positions(const void* mask, int elem_bytes, const int32_t* cu, int B, int L, int32_t* pos, void* stream);
TDB_HOST_API int tdb_repack(int pack, const void* src, const int32_t* pos, int64_t rows, int row_bytes, void* dst, void* stream);
}
