// What the kernels with one block per (query tile, head, sequence) share: which sequence a block works on, and where it lies.
#pragma once
#include "tdb_internal.h"

namespace tdb {

// The sequence that block row z works on.  Blocks start in grid order, and those of a long sequence last longest: with the
// sequences taken by decreasing length (up to 64 of them, one per thread; a block has at least 64) the last blocks to start are the cheapest.
__device__ __forceinline__ int longest_first(const AttnParams& p, int z) {
  __shared__ int lens[64], mine;
  if (p.n_seqs == 1 || p.n_seqs > 64 || !(p.varlen || p.seqlens)) return z;
  const int t = threadIdx.x;
  int len = -1;
  if (t < p.n_seqs) len = p.varlen ? p.cu_seqlens[t + 1] - p.cu_seqlens[t] : p.seqlens[t];
  if (t < 64) lens[t] = len;
  __syncthreads();
  int rank = 0;
  for (int j = 0; j < p.n_seqs; ++j) rank += lens[j] > len || (lens[j] == len && j < t);
  if (t < p.n_seqs && rank == z) mine = t;
  __syncthreads();
  return mine;
}

// Length, rows that exist in the output, first token and batch row of sequence s.  False: malformed offsets, which are
// reported; nothing of the sequence is touched.
__device__ __forceinline__ bool sequence_of(const AttnParams& p, int s, int& len, int& rows, int64_t& tok0, int& b) {
  const bool reports = threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0;
  if (p.varlen) {
    const int c0 = p.cu_seqlens[s];
    len = p.cu_seqlens[s + 1] - c0; rows = len; tok0 = c0; b = 0;
    if (c0 < 0 || len < 0 || (int64_t)c0 + len > p.total_tokens) {
      if (reports) *reinterpret_cast<volatile int32_t*>(p.status + 1) = 1;
      return false;
    }
    // The grid covers max_seqlen rows per sequence: a longer sequence would leave rows unwritten, and offsets that
    // do not end at the token count leave tokens outside every sequence.  Both are reported, not guessed around.
    if (reports && (len > p.L || (s == p.n_seqs - 1 && (int64_t)c0 + len != p.total_tokens)))
      *reinterpret_cast<volatile int32_t*>(p.status + 1) = 1;
  } else {
    len = p.seqlens ? p.seqlens[s] : p.L; rows = p.L; tok0 = 0; b = s;
    len = len < 0 ? 0 : (len > p.L ? p.L : len);
  }
  return true;
}

}  // namespace tdb
