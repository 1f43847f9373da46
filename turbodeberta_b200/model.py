"""HF DeBERTa-v2/v3 model patch: same class names as the reference's ``model.py``.

``FlashDisentangledSelfAttention`` keeps the eager module's parameters and signature
(``model.py:34-39`` of the reference, HF ``modeling_deberta_v2.py:191-199``) and replaces its arithmetic by
one fused kernel call.  Differences from the reference module, all on the host side:

* the ``Q.Kr^T`` / ``K.Qr^T`` tensors of ``model.py:122-125,143-148`` are never built; the projected
  relative tables are computed by the library once and cached until a weight changes;
* Q, K, V stay in the ``[B, L, H*D]`` layout the Linear layers produce (no ``transform`` copies,
  ``model.py:70-73,118-120``) and the output is produced directly in ``[B, L, H*D]``;
* the attention mask HF's encoder passes (``[B,1,L,L] = m (x) m^T``) is reduced to per-row key validity
  once per forward (cached on the mask tensor), instead of the per-layer ``sum == numel`` test of
  ``model.py:55-63``; right-padded batches use the padded kernel with lengths, any other token-validity
  pattern goes through pack -> packed kernel -> re-pad (``model.py:138-183``);
* the stray ``print`` of ``model.py:145`` is gone.
"""
from __future__ import annotations

import math
import threading
import warnings
import weakref

import torch
from torch import nn
from transformers.models.deberta_v2.modeling_deberta_v2 import (
    DebertaV2Attention, DebertaV2Embeddings, DebertaV2Encoder, DebertaV2ForMaskedLM, DebertaV2ForMultipleChoice,
    DebertaV2ForQuestionAnswering, DebertaV2ForSequenceClassification, DebertaV2ForTokenClassification,
    DebertaV2Intermediate, DebertaV2Layer, DebertaV2Model, DebertaV2Output, DebertaV2SelfOutput,
    DisentangledSelfAttention)

from . import relpos as _relpos
from ._cabi import host
from .ops.flash_attention import _PENDING_STATUS, _check_pending, flash_attention_with_disentangled
from .ops.flash_attention_varlen import flash_attention_with_disentangled_varlen
from .padding import _get_unpad_data, _upad_input, index_first_axis, pad_input


class PackedSequences:
    """Stands in for the attention mask when the encoder runs on the packed token stream: hidden states are
    ``[1, T, hidden]`` with the sequences back to back, ``cu_seqlens`` (int32 ``[n_seqs + 1]``) marks them."""
    __slots__ = ("cu_seqlens", "max_seqlen")

    def __init__(self, cu_seqlens: torch.Tensor, max_seqlen: int):
        self.cu_seqlens, self.max_seqlen = cu_seqlens, int(max_seqlen)


class MaskInfo:
    """Key validity derived from an attention mask: lengths, and the packing indices when needed.  ``packed`` (only from
    the native analysis of a 2-D mask): token count, longest sequence and the sequences' offsets."""
    __slots__ = ("all_ones", "right_padded", "seqlens", "key_mask", "packed")

    def __init__(self, all_ones, right_padded, seqlens, key_mask, packed=None):
        self.all_ones, self.right_padded, self.seqlens, self.key_mask = all_ones, right_padded, seqlens, key_mask
        self.packed = packed


_MASK_CACHE: dict = {}
_MASK_LOCK = threading.Lock()


def _mask_cache_put(tensor: torch.Tensor, info) -> None:
    """Remember the analysis of a live mask tensor.  Entries of tensors that have been freed are dropped first; only
    if more than 64 live masks are tracked does the oldest entry go (so a mask that is passed again and again, e.g.
    the static input of a captured graph, is never re-analysed because other masks came and went)."""
    with _MASK_LOCK:
        dead = [k for k, (ref, _, _) in _MASK_CACHE.items() if ref() is None]
        for k in dead:
            del _MASK_CACHE[k]
        while len(_MASK_CACHE) >= 64:
            del _MASK_CACHE[next(iter(_MASK_CACHE))]
        _MASK_CACHE[id(tensor)] = (weakref.ref(tensor), tensor._version, info)


def analyse_mask(attention_mask: torch.Tensor | None, batch: int, length: int, refresh: bool = False) -> MaskInfo:
    """Reduce a ``[B,L]``, ``[B,L,L]`` or ``[B,1,L,L]`` mask to per-row key validity.

    The first analysis of a mask costs one device synchronisation (two booleans are read back: all ones? right
    padded?); the result is cached on the mask tensor object (weak reference) and its version, so the 24 layers of
    one forward share it.  A mask that is not the outer product of a token-validity vector (i.e. whose valid queries
    disagree about the keys) is rejected.

    ``refresh=True`` (what the encoder passes once per forward) keeps the cached pair of booleans but recomputes the
    length and validity tensors from the mask with synchronisation-free operations.  Inside a CUDA-graph capture that
    puts the recomputation into the graph: replays then follow the lengths currently in the (static) mask buffer,
    while the choice between the all-ones, right-padded and packed routes stays the one made at capture."""
    if attention_mask is None:
        return MaskInfo(True, True, None, None)
    key = id(attention_mask)
    hit = _MASK_CACHE.get(key)
    flags = None
    if hit is not None:
        ref, version, cached = hit
        if ref() is attention_mask and version == attention_mask._version:     # same live tensor object, unmodified
            if not refresh and cached.key_mask is not None:            # the native analysis leaves it out
                return cached
            flags = (cached.all_ones, cached.right_padded)
    m = attention_mask
    if m.dim() == 4:
        if m.shape[1] != 1:
            raise ValueError("per-head attention masks are not supported")
        m = m[:, 0]
    if m.dim() == 3:
        full = m != 0
        key_mask = full.any(dim=1)                                  # a key is valid if any query may see it
        if flags is None:
            query_mask = full.any(dim=2)
            outer = key_mask[:, None, :] & query_mask[:, :, None]
            consistent = torch.equal(outer, full) and torch.equal(key_mask, query_mask)
            if not consistent:
                raise ValueError("attention_mask is not of the form m (x) m^T for a token-validity vector m; "
                                 "the fused kernels support token padding masks only")
    elif m.dim() == 2:
        key_mask = m != 0
    else:
        raise ValueError(f"unsupported attention_mask rank {attention_mask.dim()}")
    if key_mask.shape != (batch, length):
        raise ValueError("attention_mask does not match the hidden states")
    seqlens = key_mask.sum(-1, dtype=torch.int32)
    if flags is None:
        prefix = torch.arange(length, device=key_mask.device)[None, :] < seqlens[:, None]
        flags = torch.stack([key_mask.all(), (prefix == key_mask).all()]).tolist()      # the one sync
    info = MaskInfo(bool(flags[0]), bool(flags[1]), seqlens, key_mask)
    _mask_cache_put(attention_mask, info)
    return info


def _analyse_2d(attention_mask: torch.Tensor, batch: int, length: int) -> MaskInfo | None:
    """``analyse_mask`` of a CUDA ``[B, L]`` mask in one kernel and one synchronisation, offsets of the packed stream
    included.  A mask that is already known to be all ones costs neither."""
    if attention_mask.shape != (batch, length) or batch == 0 or length == 0:
        return None
    hit = _MASK_CACHE.get(id(attention_mask))
    if hit is not None and hit[0]() is attention_mask and hit[1] == attention_mask._version and hit[2].all_ones:
        return hit[2]
    rows = host.mask_rows(attention_mask)
    if rows is None:
        return None
    all_ones, right, tokens, longest, seqlens, cu = rows
    info = MaskInfo(all_ones, right, seqlens, None, (tokens, longest, cu))      # who needs the validity itself asks analyse_mask
    if all_ones and not attention_mask.is_inference():
        _mask_cache_put(attention_mask, info)
    return info


_WARNED: set = set()


def _warn_once(key: str, message: str) -> None:
    if key not in _WARNED:
        _WARNED.add(key)
        warnings.warn(message, stacklevel=3)


class FlashDisentangledSelfAttention(DisentangledSelfAttention):
    """Drop-in for HF's ``DisentangledSelfAttention`` running the fused sm_100a kernels."""

    def __init__(self, *args, **kwargs):
        super().__init__(*args, **kwargs)
        self._tables = None
        self._tables_key = None
        self._qkv = None
        self._qkv_key = None

    # -- fused Q/K/V projection ------------------------------------------------------------------
    def _project_qkv(self, hidden_states: torch.Tensor, query_states: torch.Tensor):
        """Q, K, V as ``[..., H, D]`` views.  For inference self-attention the three Linear layers run as one GEMM
        over a cached concatenation of their weights (rebuilt when a weight changes); the result is consumed through
        strided views, so no copy follows.  With gradients enabled, or a separate query input, the layers run as is."""
        H, D = self.num_attention_heads, self.attention_head_size
        lead = hidden_states.shape[:-1]
        if query_states is hidden_states and not torch.is_grad_enabled():
            qkv = torch.nn.functional.linear(hidden_states, *self._qkv_weights()).view(*lead, 3, H, D)
            return qkv.select(-3, 0), qkv.select(-3, 1), qkv.select(-3, 2)
        q = self.query_proj(query_states).view(*query_states.shape[:-1], H, D)
        k = self.key_proj(hidden_states).view(*lead, H, D)
        v = self.value_proj(hidden_states).view(*lead, H, D)
        return q, k, v

    def _qkv_weights(self):
        """Weight and bias of the three projections as one GEMM's (cached until one of them changes)."""
        params = (self.query_proj.weight, self.query_proj.bias, self.key_proj.weight, self.key_proj.bias,
                  self.value_proj.weight, self.value_proj.bias)
        key = tuple((t.data_ptr(), t._version, t.dtype, t.device) for t in params)
        if self._qkv is None or self._qkv_key != key:
            w = torch.cat([params[0], params[2], params[4]], 0).detach()
            b = torch.cat([params[1], params[3], params[5]], 0).detach()
            self._qkv, self._qkv_key = (w, b), key
        return self._qkv

    # -- relative tables ---------------------------------------------------------------------------
    def _relative_tables(self, rel_embeddings: torch.Tensor, dtype: torch.dtype):
        c2p, p2c = "c2p" in self.pos_att_type, "p2c" in self.pos_att_type
        if not self.relative_attention or not (c2p or p2c) or rel_embeddings is None:
            return None
        if self.share_att_key:
            kp, qp = self.key_proj, self.query_proj
        else:
            kp = self.pos_key_proj if c2p else None
            qp = self.pos_query_proj if p2c else None
        stamp = getattr(rel_embeddings, "_tdb_stamp", None)
        params = [t for lin in (kp, qp) if lin is not None for t in (lin.weight, lin.bias) if t is not None]
        key = (stamp, dtype, rel_embeddings.device, tuple((t.data_ptr(), t._version) for t in params), c2p, p2c,
               self.share_att_key, self.num_attention_heads, self.position_buckets, self.max_relative_positions)
        if stamp is not None and self._tables is not None and self._tables_key == key:
            return self._tables
        rel = rel_embeddings.detach().to(dtype)
        tables = _relpos.build_tables(
            rel, num_heads=self.num_attention_heads, position_buckets=self.position_buckets,
            max_relative_positions=self.max_relative_positions,
            key_weight=None if kp is None else kp.weight.detach(), key_bias=None if kp is None else kp.bias,
            query_weight=None if qp is None else qp.weight.detach(), query_bias=None if qp is None else qp.bias,
            c2p=c2p, p2c=p2c)
        if stamp is not None:
            self._tables, self._tables_key = tables, key
        return tables

    # -- forward ------------------------------------------------------------------------------------
    def forward(self, hidden_states, attention_mask, output_attentions=False, query_states=None,
                relative_pos=None, rel_embeddings=None):
        """Same contract as the reference (``model.py:34-186``): returns ``(context [B, L, H*D], None)``.
        ``relative_pos`` is accepted and ignored (positions are implied by the token order), and attention
        probabilities are never materialised, so the second element is always None."""
        if query_states is None:
            query_states = hidden_states
        B, L, _ = hidden_states.shape
        if query_states.shape[1] != L:
            raise NotImplementedError("query and key lengths must match (encoder self-attention)")
        H, D = self.num_attention_heads, self.attention_head_size
        if self.training and float(getattr(self.dropout, "p", 0.0)) > 0.0:
            _warn_once("dropout", "the fused attention has no dropout on the attention probabilities (neither has the "
                       "reference's kernel) and no backward pass: attention_probs_dropout_prob is ignored")
        q, k, v = self._project_qkv(hidden_states, query_states)
        if q.dtype == torch.float32 and B * L >= 4096:
            _warn_once("fp32", "float32 inputs run on the exact CUDA-core attention kernel, some ten times slower than the bf16 "
                       "tensor-core kernel; "
                       "convert the model with .bfloat16() for throughput")
        scale_factor = 1 + int("c2p" in self.pos_att_type) + int("p2c" in self.pos_att_type)
        sm_scale = 1.0 / math.sqrt(D * scale_factor)
        tables = None
        if self.relative_attention:
            rel_embeddings = self.pos_dropout(rel_embeddings)
            tables = self._relative_tables(rel_embeddings, q.dtype)
        buckets = self.position_buckets if self.relative_attention else 0
        max_rel = self.max_relative_positions if self.relative_attention else 0
        if isinstance(attention_mask, PackedSequences):                  # packed stream from the encoder: [1, T, hidden]
            cu = attention_mask.cu_seqlens
            out = flash_attention_with_disentangled_varlen(
                q[0], k[0], v[0], None, None, cu, cu, attention_mask.max_seqlen, attention_mask.max_seqlen, False,
                sm_scale, buckets, max_rel, tables=tables, check_status=False)
            return (out.reshape(1, L, H * D), None)
        info = analyse_mask(attention_mask, B, L)
        if info.all_ones or info.right_padded:
            out = flash_attention_with_disentangled(
                q.permute(0, 2, 1, 3), k.permute(0, 2, 1, 3), v.permute(0, 2, 1, 3), None, None, False, sm_scale,
                buckets, max_rel, seqlens=None if info.all_ones else info.seqlens, tables=tables,
                check_status=False)
            out = out.transpose(1, 2).reshape(B, L, H * D)
        else:
            (qu, ku, vu, _, _, indices, (cu_q, cu_k), (max_q, max_k)) = _upad_input(
                q, k, v, None, None, info.key_mask, L, H)
            out_unpad = flash_attention_with_disentangled_varlen(
                qu, ku, vu, None, None, cu_q, cu_k, max_q, max_k, False, sm_scale, buckets, max_rel, tables=tables,
                check_status=False)
            out = pad_input(out_unpad, indices, B, L).reshape(B, L, H * D)
        return (out, None)


class FlashDebertaV2Attention(DebertaV2Attention):
    def __init__(self, config):
        super().__init__(config)
        self.self = FlashDisentangledSelfAttention(config)


class FlashDebertaV2Layer(DebertaV2Layer):
    def __init__(self, config):
        super().__init__(config)
        self.attention = FlashDebertaV2Attention(config)


# Native plans of live encoders and models; kept outside the modules, which stay plain data to copy and pickle.  A plan
# holds modules below its key, never the key itself, so it goes when the key goes.
_PLANS: "weakref.WeakKeyDictionary" = weakref.WeakKeyDictionary()
# Held while a plan is made or brought up to date: one thread does it, the others find it done.
_PLAN_LOCK = threading.RLock()

#: what the native loop takes over from the modules besides their weights
_ATTENTION_SETTINGS = ("num_attention_heads", "attention_head_size", "pos_att_type", "share_att_key", "relative_attention",
                       "position_buckets", "max_relative_positions")
_NORM_SETTINGS = ("eps", "normalized_shape")
_GELU_SETTINGS = ("act", "approximate")


class _EncoderPlan:
    """The native form of an encoder's layer list, valid for that list object as long as ``watch`` holds."""
    __slots__ = ("layers", "watch", "native", "attns", "stamp")

    def __init__(self, layers, watch, native, attns):
        self.layers, self.watch, self.native, self.attns = layers, watch, native, attns
        self.stamp = None                    # of the relative embeddings behind the tables that ``native`` has


class FlashDebertaV2Encoder(DebertaV2Encoder):
    """HF encoder whose layers use the fused attention.  Two host-side savings: the ``[L, L]`` relative
    position matrix is not built (the kernels do not read it), and in eval mode the LayerNorm'd relative
    embeddings are computed once and stamped so that every layer can keep its derived tables."""

    def __init__(self, config):
        super().__init__(config)
        self.layer = nn.ModuleList([FlashDebertaV2Layer(config) for _ in range(config.num_hidden_layers)])
        self._rel_cache = None
        self._rel_cache_key = None
        self._rel_stamp = 0

    def get_rel_pos(self, hidden_states, query_states=None, relative_pos=None):
        return relative_pos

    #: run padded batches on the packed token stream (unpad once after the embeddings, re-pad once at the end)
    pack_padded_batches = True
    #: with packing, re-pad only the last layer's output; earlier entries of ``hidden_states`` stay ``[1, T, hidden]``
    skip_intermediate_padding = False

    def forward(self, hidden_states, attention_mask, output_hidden_states=True, output_attentions=False,
                query_states=None, relative_pos=None, return_dict=True):
        self._mask_info = None
        if (query_states is None and self.conv is None and not output_attentions
                and hidden_states.is_cuda and hidden_states.dim() == 3):
            if not torch.is_grad_enabled():
                out = self._forward_native(hidden_states, attention_mask, output_hidden_states, return_dict)
                if out is not None:
                    self._check_status_unless_capturing()
                    return out
            # One analysis of the user's mask per forward (cached per mask tensor, so a repeated call with the same
            # tensor - e.g. while the forward is being captured into a CUDA graph - costs no synchronisation); the
            # expanded mask that the HF encoder builds from it inherits the result in get_attention_mask().
            info = analyse_mask(attention_mask, hidden_states.shape[0], hidden_states.shape[1], refresh=True)
            if self.pack_padded_batches and not info.all_ones:
                out = self._forward_packed(hidden_states, info, output_hidden_states, return_dict)
                self._check_status_unless_capturing()
                return out
            self._mask_info = info
        out = super().forward(hidden_states, attention_mask, output_hidden_states=output_hidden_states,
                              output_attentions=output_attentions, query_states=query_states,
                              relative_pos=relative_pos, return_dict=return_dict)
        self._check_status_unless_capturing()   # one synchronisation per encoder forward instead of one per layer
        return out

    def get_attention_mask(self, attention_mask):
        out = super().get_attention_mask(attention_mask)
        info = getattr(self, "_mask_info", None)
        if info is not None and isinstance(out, torch.Tensor) and out is not attention_mask:
            _mask_cache_put(out, info)
        return out

    @staticmethod
    def _check_status_unless_capturing():
        """Reading the device status words synchronises, which a stream capture does not allow: while the forward is
        being captured into a CUDA graph the words stay pending (the graph's replays rewrite them) and the next
        ``check_pending_status()`` outside a capture reads them."""
        if not torch.cuda.is_current_stream_capturing():
            report, _PASS.report = _PASS.report, None
            _check_pending(report)

    # -- the whole layer loop in one native call -------------------------------------------------------
    def _native_layers(self):
        """The plan of a stack made of the stock modules only, else None."""
        layers = list(self.layer)
        native, attns, settings = None, [], []
        for layer in layers:
            att, up, down = layer.attention, layer.intermediate, layer.output
            sa, so, act = att.self, att.output, layer.intermediate.intermediate_act_fn
            stock = (type(layer) in (DebertaV2Layer, FlashDebertaV2Layer)
                     and type(att) in (DebertaV2Attention, FlashDebertaV2Attention)
                     and type(sa) is FlashDisentangledSelfAttention and type(so) is DebertaV2SelfOutput
                     and type(up) is DebertaV2Intermediate and type(down) is DebertaV2Output
                     and (getattr(act, "act", None) is nn.functional.gelu
                          or (type(act) is nn.GELU and act.approximate == "none")))
            if not stock or sa.attention_head_size != 64:
                return None
            lins = [sa.query_proj, sa.key_proj, sa.value_proj, so.dense, up.dense, down.dense]
            if not sa.share_att_key and sa.relative_attention:
                lins += [lin for lin in (getattr(sa, "pos_key_proj", None), getattr(sa, "pos_query_proj", None)) if lin is not None]
            norms = [so.LayerNorm, down.LayerNorm]
            if any(type(m) is not nn.Linear or m.bias is None for m in lins):
                return None
            if any(type(m) is not nn.LayerNorm or m.weight is None or m.bias is None for m in norms):
                return None
            drops = [so._modules.get("dropout"), down._modules.get("dropout")]
            drops += [sa._modules.get("pos_dropout")] if sa.relative_attention else []
            if any(type(m) not in (nn.Dropout, nn.Identity) for m in drops):         # in eval mode both do nothing
                return None
            hidden = so.dense.out_features
            widest = 1024 if so.dense.weight.dtype == torch.float32 else 2048
            if hidden % 8 or hidden > widest or up.dense.out_features % 8 or hidden != 64 * sa.num_attention_heads:
                return None
            if native is None:
                native = host.Encoder(sa.num_attention_heads)
            terms = 1 + int("c2p" in sa.pos_att_type) + int("p2c" in sa.pos_att_type)
            native.add_layer([so.dense.weight, so.dense.bias, norms[0].weight, norms[0].bias, up.dense.weight, up.dense.bias,
                              down.dense.weight, down.dense.bias, norms[1].weight, norms[1].bias], norms[0].eps,
                             norms[1].eps, 1.0 / math.sqrt(64 * terms), [t for m in lins[:3] + lins[6:] for t in (m.weight, m.bias)])
            attns.append(sa)
            settings += [(sa, _ATTENTION_SETTINGS), (norms[0], _NORM_SETTINGS), (norms[1], _NORM_SETTINGS), (act, _GELU_SETTINGS)]
        if native is None:
            return None
        return _EncoderPlan(self.layer, host.Watch(list(self.layer.modules()), settings), native, attns)

    def _native_plan(self, hidden_states, rel_embeddings):
        """The plan with every layer's derived tensors up to date, or None where the native loop does not apply.  Whether a
        kept plan still matches the modules in its list is for the caller to ask (``watch.holds()``), once the GPU is busy."""
        plan = _PLANS.get(self)
        if plan is None or plan.layers is not self._modules["layer"]:
            plan = self._native_layers()
            if plan is None or not plan.watch.holds():
                return None
            _PLANS[self] = plan
        native, attns = plan.native, plan.attns
        if not native.fits(hidden_states):
            return None
        dtype = hidden_states.dtype
        stamp_now = (getattr(rel_embeddings, "_tdb_stamp", None), dtype)
        if plan.stamp != stamp_now:
            todo = range(len(attns))
            if rel_embeddings is not None and stamp_now[0] is None:
                return None
        else:
            todo = native.stale()
        made = False
        for i in todo:
            made = True
            w, b = attns[i]._qkv_weights()
            tables = attns[i]._relative_tables(rel_embeddings, dtype) if attns[i].relative_attention else None
            if not native.set_derived(i, hidden_states, w, b, None if tables is None else tables.native()):
                return None
        if made and hidden_states.is_cuda and not torch.cuda.is_current_stream_capturing():
            native.set_ready(hidden_states)      # passes on other streams wait for this
        plan.stamp = stamp_now
        return plan

    def _forward_native(self, hidden_states, attention_mask, output_hidden_states, return_dict):
        """The encoder as one native call on the token-major stream: packed (valid tokens only) for padded batches,
        ``[B * L, hidden]`` otherwise.  None where the generic route has to take over."""
        if (self.training or hidden_states.dtype not in (torch.float32, torch.bfloat16) or torch.is_autocast_enabled()
                or torch.nn.modules.module._has_any_global_hook() or hidden_states.numel() == 0):
            return None
        B, L, hid = hidden_states.shape
        if (torch.cuda.is_current_stream_capturing() or attention_mask is None or attention_mask.dim() != 2
                or attention_mask.device != hidden_states.device):
            info = analyse_mask(attention_mask, B, L, refresh=True)
            if not info.all_ones:
                return None
        else:
            info = _analyse_2d(attention_mask, B, L)
            if info is None or (not info.all_ones and (not self.pack_padded_batches or info.packed[0] == 0)):
                return None
        with _PLAN_LOCK:
            plan = self._native_plan(hidden_states, self.get_rel_embedding())
        if plan is None:
            return None
        native = plan.native
        every = output_hidden_states and _WANTED.hidden_states
        if info.all_ones:
            outs, words = native.run(hidden_states.reshape(B * L, hid), None, L, every)
            padded = [o.view(B, L, hid) for o in outs]
        else:
            tokens, longest, cu = info.packed
            x, pos = host.pack_rows(hidden_states, attention_mask, cu, tokens)
            outs, words = native.run(x, cu, longest, every)
            keep = [o[None] for o in outs[:-1]] if self.skip_intermediate_padding else [host.unpack_rows(o, pos, B, L) for o in outs[:-1]]
            padded = keep + [host.unpack_rows(outs[-1], pos, B, L)]
        for w in words:
            _PENDING_STATUS.append(w)
        # The look at some two hundred modules takes the host 90 us, so it runs behind the launches, beside the GPU; the
        # result has no side effects and is simply dropped when somebody has changed the modules since the last forward.
        if not plan.watch.holds():
            _PLANS.pop(self, None)               # another thread may have been first
            return self._forward_native(hidden_states, attention_mask, output_hidden_states, return_dict)
        all_hidden = None
        if output_hidden_states:
            all_hidden = (hidden_states, *padded) if every else (padded[-1],)
        from transformers.modeling_outputs import BaseModelOutput
        if not return_dict:
            return tuple(v for v in [padded[-1], all_hidden, None] if v is not None)
        return BaseModelOutput(last_hidden_state=padded[-1], hidden_states=all_hidden, attentions=None)

    def _forward_packed(self, hidden_states, info: MaskInfo, output_hidden_states: bool, return_dict: bool):
        """The layer loop of the HF encoder (``modeling_deberta_v2.py:630-682``) on valid tokens only.  The reference
        packs and re-pads inside every attention call (``model.py:157-183``); here the whole stack (attention, both
        projections, FFN, LayerNorms) sees ``[1, T, hidden]`` and padding costs nothing.  Padded positions of the
        returned tensors are zero."""
        from transformers.modeling_outputs import BaseModelOutput
        B, L, hid = hidden_states.shape
        indices, cu_seqlens, max_seqlen = _get_unpad_data(info.key_mask)
        x = index_first_axis(hidden_states.reshape(B * L, hid), indices)[None]
        seqs = PackedSequences(cu_seqlens, max_seqlen)
        rel_embeddings = self.get_rel_embedding()
        all_hidden = (hidden_states,) if output_hidden_states else None
        n = len(self.layer)
        for i, layer in enumerate(self.layer):
            x, _ = layer(x, seqs, query_states=None, relative_pos=None, rel_embeddings=rel_embeddings,
                         output_attentions=False)
            if output_hidden_states:
                last = i == n - 1
                all_hidden = all_hidden + ((pad_input(x[0], indices, B, L) if (last or not self.skip_intermediate_padding)
                                            else x),)
        output_states = all_hidden[-1] if output_hidden_states else pad_input(x[0], indices, B, L)
        if not return_dict:
            return tuple(v for v in [output_states, all_hidden, None] if v is not None)
        return BaseModelOutput(last_hidden_state=output_states, hidden_states=all_hidden, attentions=None)

    def get_rel_embedding(self):
        if not self.relative_attention:
            return None
        params, eps = [self.rel_embeddings.weight], None
        if "layer_norm" in self.norm_rel_ebd:
            params += [self.LayerNorm.weight, self.LayerNorm.bias]
            eps = getattr(self.LayerNorm, "eps", None)
        if self.training or torch.is_grad_enabled():
            return super().get_rel_embedding()
        key = (eps, *((t.data_ptr(), t._version, t.dtype, t.device) for t in params))
        if self._rel_cache is None or key != self._rel_cache_key:
            rel = super().get_rel_embedding().detach()
            self._rel_stamp += 1
            rel._tdb_stamp = (id(self), self._rel_stamp)
            self._rel_cache, self._rel_cache_key = rel, key
        return self._rel_cache


class _Wanted(threading.local):
    """What the model around the encoder will use of the layers' outputs (the HF model asks its encoder for all of them and
    then drops them unless its caller asked, which for a padded batch costs one re-padding per layer)."""
    hidden_states = True


_WANTED = _Wanted()


class _Pass(threading.local):
    """The report of the embeddings of this thread's pass, until its check: a bad id is an error of this caller's, whoever else checks."""
    report = None


_PASS = _Pass()
_PLAIN_TENSORS = frozenset((torch.Tensor, nn.Parameter))      # other classes may keep their values elsewhere (quantised, sharded)
_MASK_TYPES = (torch.int64, torch.bool, torch.uint8)
_PLAIN_ARGUMENTS = frozenset(("input_ids", "attention_mask", "output_hidden_states", "output_attentions", "return_dict"))


class FlashDebertaV2Model(DebertaV2Model):
    def __init__(self, config):
        super().__init__(config)
        self.encoder = FlashDebertaV2Encoder(config)
        self.post_init()

    def forward(self, *args, **kwargs):
        wanted = kwargs.get("output_hidden_states")
        if wanted is None:
            wanted = len(args) > 1 or bool(getattr(self.config, "output_hidden_states", False))
        before = _WANTED.hidden_states
        _WANTED.hidden_states = bool(wanted) or getattr(self, "z_steps", 0) != 0
        try:
            if not args and not wanted and _PLAIN_ARGUMENTS.issuperset(kwargs):
                out = self._forward_plain(kwargs.get("input_ids"), kwargs.get("attention_mask"), kwargs)
                if out is not None:
                    return out
            return super().forward(*args, **kwargs)
        finally:
            _WANTED.hidden_states = before

    def _forward_plain(self, input_ids, attention_mask, kwargs):
        """Ids and a 2-D mask in, last hidden states out, for inference with the stock embeddings (words and LayerNorm
        only): the same operations as the HF model's forward without its argument handling, which takes the host as long as
        a short text takes the GPU.  None where that forward has to run."""
        if (self.training or torch.is_grad_enabled() or getattr(self, "z_steps", 0) != 0 or not isinstance(input_ids, torch.Tensor)
                or not input_ids.is_cuda or input_ids.dim() != 2 or kwargs.get("output_attentions")
                or kwargs.get("return_dict", True) is False or not getattr(self.config, "use_return_dict", True)
                or getattr(self.config, "output_attentions", False) or torch.is_autocast_enabled()
                or torch.nn.modules.module._has_any_global_hook()):
            return None
        if attention_mask is not None and (attention_mask.dim() != 2 or attention_mask.shape != input_ids.shape
                                           or attention_mask.device != input_ids.device):
            return None
        emb = self.embeddings
        watch, of, plain = _PLANS.get(self, (None, None, None))
        if watch is None or of is not emb:
            if (type(emb) is not DebertaV2Embeddings or type(emb.word_embeddings) is not nn.Embedding
                    or type(emb.LayerNorm) is not nn.LayerNorm or emb.word_embeddings.max_norm is not None
                    or any(getattr(emb, n, None) is not None for n in ("position_embeddings", "token_type_embeddings", "embed_proj"))):
                return None
            watch = host.Watch(list(emb.modules()), [(emb.word_embeddings, ("max_norm",))])
            plain = all(type(p) is nn.Parameter for p in emb.parameters())      # the watch knows them by identity
            _PLANS[self] = (watch, emb, plain)
        if not watch.holds():
            _PLANS.pop(self, None)
            return None
        if attention_mask is None:
            attention_mask = torch.ones(input_ids.shape, dtype=torch.long, device=input_ids.device)
        table, norm = emb.word_embeddings.weight, emb.LayerNorm
        embedded = None
        if (plain and type(input_ids) in _PLAIN_TENSORS and type(attention_mask) in _PLAIN_TENSORS and norm.weight is not None
                and norm.bias is not None and tuple(norm.normalized_shape) == table.shape[1:]):
            # Rows of a wider tensor, or a mask of another type, must not change what an id outside the vocabulary does: torch's own
            # embedding ends in an assertion on the device.
            known = attention_mask.dtype in _MASK_TYPES
            embedded = host.embed(input_ids, table, norm.weight, norm.bias, norm.eps,
                                  attention_mask if known else torch.ones(input_ids.shape, dtype=torch.bool, device=input_ids.device), True)
            if embedded is not None and not known:
                embedded[0].mul_(attention_mask.to(table.dtype)[..., None])
        report = None
        if embedded is not None:
            x, report = embedded
            if isinstance(report, torch.Tensor) and torch.cuda.is_current_stream_capturing():       # each replay writes it: left to the next check
                _PENDING_STATUS.append(report)
                report = None
        else:
            x = nn.functional.embedding(input_ids, table)
            x = nn.functional.layer_norm(x, norm.normalized_shape, norm.weight, norm.bias, norm.eps)
            x.mul_(attention_mask.to(x.dtype)[..., None])
        before, _PASS.report = _PASS.report, report
        try:
            out = self.encoder(x, attention_mask, output_hidden_states=False, output_attentions=False, return_dict=True)
            if _PASS.report is not None:             # an encoder that does not check
                FlashDebertaV2Encoder._check_status_unless_capturing()
            return out
        finally:
            _PASS.report = before


def patch_model(model: nn.Module) -> nn.Module:
    """Swap, in place, every eager ``DisentangledSelfAttention`` of an already built HF DeBERTa-v2 model for
    the fused module (parameters are shared, not copied) and give its encoder the cached relative embeddings."""
    for name, mod in list(model.named_modules()):
        if isinstance(mod, DebertaV2Attention) and not isinstance(mod.self, FlashDisentangledSelfAttention):
            old = mod.self
            new = FlashDisentangledSelfAttention.__new__(FlashDisentangledSelfAttention)
            new.__dict__.update(old.__dict__)
            new._tables, new._tables_key, new._qkv, new._qkv_key = None, None, None, None
            mod.self = new
        if type(mod) is DebertaV2Encoder:
            mod.__class__ = FlashDebertaV2Encoder
            mod._rel_cache, mod._rel_cache_key, mod._rel_stamp = None, None, 0
        if type(mod) is DebertaV2Model:
            mod.__class__ = FlashDebertaV2Model
    return model


class FlashDebertaV2ForMaskedLM(DebertaV2ForMaskedLM):
    def __init__(self, config):
        super().__init__(config)
        self.deberta = FlashDebertaV2Model(config)
        self.post_init()


class FlashDebertaV2ForSequenceClassification(DebertaV2ForSequenceClassification):
    def __init__(self, config):
        super().__init__(config)
        self.deberta = FlashDebertaV2Model(config)
        self.post_init()


class FlashDebertaV2ForTokenClassification(DebertaV2ForTokenClassification):
    def __init__(self, config):
        super().__init__(config)
        self.deberta = FlashDebertaV2Model(config)
        self.post_init()


class FlashDebertaV2ForQuestionAnswering(DebertaV2ForQuestionAnswering):
    def __init__(self, config):
        super().__init__(config)
        self.deberta = FlashDebertaV2Model(config)
        self.post_init()


class FlashDebertaV2ForMultipleChoice(DebertaV2ForMultipleChoice):
    def __init__(self, config):
        super().__init__(config)
        self.deberta = FlashDebertaV2Model(config)
        self.post_init()
