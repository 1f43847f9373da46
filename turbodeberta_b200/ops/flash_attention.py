"""Fixed-length (padded) fused disentangled attention.

Same entry point as the reference's ``ops/flash_attention.py:345-369``::

    flash_attention_with_disentangled(q, k, v, q_pos, k_pos, causal=False, sm_scale=None,
                                      position_buckets=0, max_relative_distance=0)

with q, k, v of logical shape ``(B, H, L, D)`` and arbitrary strides (a permuted view of the
``[B, L, H*D]`` projection output works without a copy).  One semantic change: the reference expects
``q_pos``/``k_pos`` to be the materialised score tensors ``Q.Kr^T`` / ``K.Qr^T`` of shape ``(B, H, L, 2*span)``
(``model.py:122-125``); here they are the projected tables ``Kr`` / ``Qr`` themselves, ``(H, 2*span, D)`` or
``(1, H, 2*span, D)`` (what ``model.py:95-100`` calls ``pos_key_layer`` / ``pos_query_layer``), or a prebuilt
``RelPosTables``; the products are formed on chip.  The keyword-only ``seqlens`` adds right-padding masking,
which the reference kernel does not have.  Forward only, like the reference (``ops/flash_attention.py:341-343``).

The reference's own calling convention still works: when ``q_pos`` / ``k_pos`` have the shape ``(B, H, L, 2*span)``
they are taken as the materialised scores and only gathered (``attn_scores.cu`` in bf16, the CUDA-core kernel in
fp32; both are bound by reading them).  The gather follows the eager module (same index for both terms) unless ``p2c_mirrored=True``, which
reproduces the reference kernel's mirrored position->content index (``ops/flash_attention.py:126-132``).
"""
from __future__ import annotations

import itertools
import math

import torch

from .. import _cabi as cabi
from .. import relpos as _relpos
from .. import status as _status


def _tables_from_args(q_pos, k_pos, q, position_buckets, max_relative_distance, tables):
    """Normalise the position arguments into something with a ``native()`` table object (None: no term is requested)."""
    if tables is not None:
        return tables
    if q_pos is None and k_pos is None:
        return None
    H, D = q.shape[-3] if q.dim() == 4 else q.shape[-2], q.shape[-1]

    def norm(t, name):
        if t is None:
            return None
        if t.dim() == 4 and t.shape[0] == 1:
            t = t[0]
        if t.dim() != 3 or t.shape[0] != H or t.shape[-1] != D:
            raise ValueError(
                f"{name} must be the projected relative table of shape (H, 2*span, D) = ({H}, 2*span, {D}) or the "
                f"materialised score tensor of q's leading shape with 2*span columns; got {tuple(t.shape)}.")
        return t

    kr, qr = norm(q_pos, "q_pos"), norm(k_pos, "k_pos")
    two_span = (kr if kr is not None else qr).shape[1]
    if position_buckets > 0:
        if two_span != 2 * position_buckets:
            raise ValueError(f"table has {two_span} rows but position_buckets={position_buckets}")
        if max_relative_distance <= 0:
            raise ValueError("max_relative_distance must be given with position_buckets")
    else:
        if max_relative_distance <= 0:
            max_relative_distance = two_span // 2
        if two_span != 2 * max_relative_distance:
            raise ValueError(f"table has {two_span} rows but max_relative_distance={max_relative_distance}")
    if D != 64:
        raise ValueError(f"head_dim {D}: only 64 is supported")
    idx, exp_dm = _geometry(position_buckets, max_relative_distance, q.device)
    return _CallTables(cabi.host.call_tables(kr, qr, q, idx, exp_dm))


class _CallTables:
    """Tables made for one call."""
    __slots__ = ("_native",)

    def __init__(self, native):
        self._native = native

    def native(self):
        return self._native


_GEOMETRY: dict = {}


def _geometry(position_buckets, max_relative_distance, device):
    """(index table, delta_max of the expanded tables), kept per geometry and device."""
    key = (position_buckets, max_relative_distance, device)
    g = _GEOMETRY.get(key)
    if g is None:
        sat = _relpos.saturation_distance(position_buckets, max_relative_distance)
        idx = _relpos.bucket_index_table(position_buckets, max_relative_distance, sat + 1, device)
        g = _GEOMETRY[key] = (idx, sat + cabi.TDB_EXPAND_MARGIN)
    return g


def _is_materialised(t, q, position_buckets=0, max_relative_distance=0) -> bool:
    """True when ``t`` is a per-token score tensor (``q.shape[:-1] + (2*span,)``) rather than a projected table
    (``(H, 2*span, D)``, optionally with a leading 1).  Where both readings fit the shape, the geometry arguments
    decide (a table has 2*span rows, a score tensor 2*span columns); if they do not, it is taken as a table."""
    if t is None or t.dim() != q.dim():
        return False
    shape, qs = t.shape, q.shape
    if shape[:-1] != qs[:-1]:
        return False
    H, D = qs[-3] if len(qs) == 4 else qs[-2], qs[-1]
    table = shape[0] == 1 and shape[1] == H and shape[3] == D if len(shape) == 4 else (shape[0] == H and shape[2] == D)
    if not table:
        return True
    want = 2 * position_buckets if position_buckets > 0 else 2 * max_relative_distance
    return want > 0 and t.shape[-1] == want and t.shape[-2] != want


def _index_table_for_scores(two_span, position_buckets, max_relative_distance, dev):
    if position_buckets > 0:
        if two_span != 2 * position_buckets:
            raise ValueError(f"score tensors have {two_span} columns but position_buckets={position_buckets}")
        if max_relative_distance <= 0:
            raise ValueError("max_relative_distance must be given with position_buckets")
    else:
        if max_relative_distance <= 0:
            max_relative_distance = two_span // 2
        if two_span != 2 * max_relative_distance:
            raise ValueError(f"score tensors have {two_span} columns but max_relative_distance={max_relative_distance}")
    return _geometry(position_buckets, max_relative_distance, dev)[0]


def refuse_gradients(*tensors) -> None:
    """The score-tensor form runs outside any autograd function, so nothing would stop a training loop from getting
    an output without a gradient path; refuse it up front (the fused form raises in ``backward`` instead, like the
    reference, ``ops/flash_attention.py:341-343``)."""
    if torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in tensors):
        raise RuntimeError("turbodeberta_b200 attention is forward-only (as in the reference: no backward kernel); "
                           "call it under torch.no_grad() or with detached inputs")


def _scores_fixed(q, k, v, c2p_scores, p2c_scores, seqlens, sm_scale, position_buckets, max_relative_distance,
                  p2c_mirrored, return_lse, check_status):
    """Legacy form of the fixed-length op: gather from materialised ``(B, H, L, 2*span)`` score tensors."""
    refuse_gradients(q, k, v, c2p_scores, p2c_scores)
    if not q.is_cuda:
        cabi.require_cuda(q, k, v, seqlens)
    some = c2p_scores if c2p_scores is not None else p2c_scores
    idx = _index_table_for_scores(some.shape[-1], position_buckets, max_relative_distance, q.device)
    o, lse, st = cabi.host.attn_fixed_scores(q, k, v, c2p_scores, p2c_scores, idx, p2c_mirrored, seqlens, sm_scale,
                                             return_lse, check_status)
    if st is not None:
        finish_status(st, check_status)
    return o, lse


# Status words of calls made with check_status=False; read by check_pending_status().
_PENDING_STATUS = _status.PENDING


def check_pending_status() -> None:
    """Read (one synchronisation) the device status words of every call since the last check that was made
    with ``check_status=False`` and raise if any bounded device wait gave up or any ``cu_seqlens`` was malformed."""
    _check_pending(None)


def _check_pending(report) -> None:
    """``check_pending_status()`` that also reads a report of the caller's own (a native ``Report``, or a tensor of words)."""
    own = report.tolist() if isinstance(report, torch.Tensor) else ()
    pooled, blocks = cabi.host.drain_pending() if report is None or own else cabi.host.drain_pending(report), {}
    for st in _PENDING_STATUS.drain():
        blocks.setdefault(st.device, []).append(st)
    if pooled is None and not blocks and not own:
        return
    words = [torch.stack(sts).amax(dim=0).tolist() for sts in blocks.values()]
    _raise_for([max(w) for w in itertools.zip_longest(pooled or (0,), own, *words, fillvalue=0)])


def _check_status(status: torch.Tensor):
    """Read the device status words (synchronises); raise if a wait gave up or cu_seqlens was invalid."""
    _raise_for(status.tolist())


def _raise_for(st):
    """The error that status words stand for, if any.  Words of several calls may have come together: the message names
    every kind, and a wait that gave up, after which no output can be relied on, decides the type before a mistake of a caller's."""
    found = []
    if st[0]:
        found.append((f"a device-side wait gave up (barrier code {st[0]})", lambda text: cabi.TdbError(cabi.ERR_TIMEOUT, text)))
    if len(st) > 1 and st[1]:
        found.append(("cu_seqlens is not a non-decreasing sequence ending at the token count (or the key offsets "
                      "differ from the query offsets, or max_seqlen is smaller than the longest sequence)", ValueError))
    if len(st) > 3 and st[3]:
        found.append(("a token id lies outside the vocabulary", IndexError))
    if found:
        raise found[0][1]("; and ".join(text for text, _ in found))


def finish_status(st, check: bool) -> None:
    """What a native call left to the caller: an error code of the library, the words of a report, or (during a stream
    capture, or with every pooled word in use) a tensor of words that nobody has read yet."""
    if isinstance(st, torch.Tensor):
        if check:
            _check_status(st)
        else:
            _PENDING_STATUS.append(st)
    elif isinstance(st, int):
        cabi.check(st)
    else:
        _raise_for(st)


def needs_graph(*tensors) -> bool:
    """Whether autograd would record the call (its backward then raises)."""
    return torch.is_grad_enabled() and any(t.requires_grad for t in tensors)


def _call_fixed(q, k, v, tables, seqlens, sm_scale, kernel, return_lse, check):
    o, lse, st = cabi.host.attn_fixed(q, k, v, None if tables is None else tables.native(), seqlens, sm_scale, kernel,
                                      return_lse, check)
    if st is not None:
        finish_status(st, check)
    return o, lse


class _FixedFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, *args):
        o, lse = _call_fixed(q, k, v, *args)
        if lse is not None:
            ctx.mark_non_differentiable(lse)
        return o, lse

    @staticmethod
    def backward(ctx, *grads):
        raise RuntimeError("turbodeberta_b200 attention is forward-only (as in the reference: no backward kernel)")


def flash_attention_with_disentangled(q, k, v, q_pos, k_pos, causal=False, sm_scale=None, position_buckets=0,
                                      max_relative_distance=0, *, seqlens=None, tables=None,
                                      kernel=cabi.TDB_KERNEL_AUTO, return_lse=False, check_status=True,
                                      p2c_mirrored=False):
    """Fused disentangled attention on padded ``(B, H, L, D)`` inputs; returns ``o`` with the shape of ``q``
    (memory layout ``[B, L, H, D]``, so ``o.transpose(1, 2).reshape(B, L, H*D)`` is a free view).

    ``q_pos`` feeds the content->position term (table ``Kr``), ``k_pos`` the position->content term (``Qr``);
    either may be None.  ``seqlens`` (int ``[B]``) masks keys beyond each row's length and zeroes its padded
    query rows.  ``check_status=False`` skips the end-of-call read of the device status words (no host sync);
    the caller then owns checking ``status``.
    """
    if causal:
        raise NotImplementedError("causal masking is not part of the DeBERTa encoder path")
    if sm_scale is None:
        sm_scale = 1.0 / math.sqrt(q.shape[-1])
    if tables is None and (q_pos is not None or k_pos is not None):
        mat = [t is not None and _is_materialised(t, q, position_buckets, max_relative_distance) for t in (q_pos, k_pos)]
        if any(mat):
            if (q_pos is not None and not mat[0]) or (k_pos is not None and not mat[1]):
                raise ValueError("q_pos and k_pos must both be tables (H, 2*span, D) or both be score tensors (B, H, L, 2*span)")
            o, lse = _scores_fixed(q, k, v, q_pos, k_pos, seqlens, sm_scale, position_buckets, max_relative_distance,
                                   p2c_mirrored, return_lse, check_status)
            return (o, lse) if return_lse else o
    if p2c_mirrored:
        raise ValueError("p2c_mirrored applies to materialised score tensors only")
    tables = _tables_from_args(q_pos, k_pos, q, position_buckets, max_relative_distance, tables)
    call = _FixedFn.apply if needs_graph(q, k, v) else _call_fixed
    o, lse = call(q, k, v, tables, seqlens, sm_scale, kernel, return_lse, check_status)
    if return_lse:
        return o, lse
    return o
