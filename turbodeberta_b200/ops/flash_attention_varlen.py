"""Packed (varlen) fused disentangled attention.

Same entry point as the reference's ``ops/flash_attention_varlen.py:348-374``::

    flash_attention_with_disentangled_varlen(q, k, v, q_pos, k_pos, cu_seqlens_q, cu_seqlens_k,
                                             max_seqlen_q, max_seqlen_k, causal=False, sm_scale=None,
                                             position_buckets=0, max_relative_distance=0)

q, k, v are ``(T, H, D)`` with the sequences back to back; ``cu_seqlens`` is int32 ``(n_seqs + 1)``.  As in the
fixed-length op, ``q_pos``/``k_pos`` are the projected tables ``(H, 2*span, D)`` rather than the per-token score
tensors ``(T, H, 2*span)`` of the reference.  Relative positions restart at every sequence.  The tile list is
built on the device from ``cu_seqlens``; nothing is read back except the status words at the end of the call.
Score tensors of shape ``(T, H, 2*span)`` are still accepted and only gathered, as in the padded form
(``p2c_mirrored=True`` reproduces the reference kernel's index, ``ops/flash_attention_varlen.py:144-152``).
"""
from __future__ import annotations

import math

import torch

from .. import _cabi as cabi
from .flash_attention import (_index_table_for_scores, _is_materialised, _tables_from_args, finish_status, needs_graph,
                              refuse_gradients)


def _call_varlen(q, k, v, tables, cu_seqlens, max_seqlen, sm_scale, kernel, return_lse, check, cu_seqlens_k=None):
    o, lse, st = cabi.host.attn_packed(q, k, v, None if tables is None else tables.native(), cu_seqlens, max_seqlen,
                                       sm_scale, kernel, return_lse, check)
    if st is not None:
        finish_status(st, check)
    _check_key_offsets(cu_seqlens, cu_seqlens_k, check)
    return o, lse


class _VarlenFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, *args):
        o, lse = _call_varlen(q, k, v, *args)
        if lse is not None:
            ctx.mark_non_differentiable(lse)
        return o, lse

    @staticmethod
    def backward(ctx, *grads):
        raise RuntimeError("turbodeberta_b200 attention is forward-only (as in the reference: no backward kernel)")


def _check_key_offsets(cu_q, cu_k, check) -> None:
    """Self-attention only: key offsets must equal the query offsets.  When the caller passes two different tensors
    the comparison runs on the device and counts as a malformed-offsets report of this call."""
    if cu_k is None or cu_k is cu_q or (cu_k.data_ptr() == cu_q.data_ptr() and cu_k.shape == cu_q.shape):
        return
    words = torch.zeros(4, dtype=torch.int32, device=cu_q.device)
    words[1:2].add_((cu_k.to(cu_q.device) != cu_q).any().to(torch.int32))
    finish_status(words, check)


def _scores_varlen(q, k, v, c2p_scores, p2c_scores, cu_seqlens, max_seqlen, sm_scale, position_buckets,
                   max_relative_distance, p2c_mirrored, return_lse, check_status, cu_seqlens_k=None):
    """Legacy form of the packed op: gather from materialised ``(T, H, 2*span)`` score tensors."""
    dev = cabi.require_cuda(q, k, v, cu_seqlens)
    refuse_gradients(q, k, v, c2p_scores, p2c_scores)
    some = c2p_scores if c2p_scores is not None else p2c_scores
    idx = _index_table_for_scores(some.shape[-1], position_buckets, max_relative_distance, dev)
    o, lse, st = cabi.host.attn_packed_scores(q, k, v, c2p_scores, p2c_scores, idx, p2c_mirrored, cu_seqlens, max_seqlen,
                                              sm_scale, return_lse, check_status)
    if st is not None:
        finish_status(st, check_status)
    _check_key_offsets(cu_seqlens, cu_seqlens_k, check_status)
    return o, lse


def flash_attention_with_disentangled_varlen(q, k, v, q_pos, k_pos, cu_seqlens_q, cu_seqlens_k, max_seqlen_q,
                                             max_seqlen_k, causal=False, sm_scale=None, position_buckets=0,
                                             max_relative_distance=0, *, tables=None, kernel=cabi.TDB_KERNEL_AUTO,
                                             return_lse=False, check_status=True, p2c_mirrored=False):
    """Fused disentangled attention on packed ``(T, H, D)`` inputs; returns ``o`` of the same shape."""
    if causal:
        raise NotImplementedError("causal masking is not part of the DeBERTa encoder path")
    if cu_seqlens_k is not None and cu_seqlens_k is not cu_seqlens_q:
        if cu_seqlens_k.shape != cu_seqlens_q.shape or cu_seqlens_k.dtype != cu_seqlens_q.dtype:
            raise ValueError("query and key offsets must be equal: only self-attention is supported")
    if sm_scale is None:
        sm_scale = 1.0 / math.sqrt(q.shape[-1])
    T = q.shape[0]
    max_seqlen = max(int(max_seqlen_q), int(max_seqlen_k if max_seqlen_k is not None else max_seqlen_q))
    max_seqlen = max(1, min(max_seqlen, T)) if T > 0 else 1
    if tables is None and (q_pos is not None or k_pos is not None):
        mat = [t is not None and _is_materialised(t, q, position_buckets, max_relative_distance) for t in (q_pos, k_pos)]
        if any(mat):
            if (q_pos is not None and not mat[0]) or (k_pos is not None and not mat[1]):
                raise ValueError("q_pos and k_pos must both be tables (H, 2*span, D) or both be score tensors (T, H, 2*span)")
            o, lse = _scores_varlen(q, k, v, q_pos, k_pos, cu_seqlens_q, max_seqlen, sm_scale, position_buckets,
                                    max_relative_distance, p2c_mirrored, return_lse, check_status, cu_seqlens_k)
            return (o, lse) if return_lse else o
    if p2c_mirrored:
        raise ValueError("p2c_mirrored applies to materialised score tensors only")
    tables = _tables_from_args(q_pos, k_pos, q, position_buckets, max_relative_distance, tables)
    call = _VarlenFn.apply if needs_graph(q, k, v) else _call_varlen
    o, lse = call(q, k, v, tables, cu_seqlens_q, max_seqlen, sm_scale, kernel, return_lse, check_status, cu_seqlens_k)
    if return_lse:
        return o, lse
    return o
