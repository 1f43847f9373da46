"""Performance cases: what a user of this package runs, over the sizes they run it at.

Four entry points, all forward only (the package has no backward pass):

* ``fixed``   ``flash_attention_with_disentangled`` on padded batches, bf16 and fp32
* ``packed``  ``flash_attention_with_disentangled_varlen`` on back-to-back sequences, bf16
* ``scores``  the fixed-length operator in the calling convention of the original package: the caller has already
              multiplied Q and K with the projected position tables and passes the two score tensors
* ``model``   ``FlashDebertaV2Model`` from token ids to the last hidden states, bf16

``listed()`` gives the reference points, ``draw(rng)`` more cases of the same ranges.  Lengths are part of a case (their
seed is one of its fields), values come from the seed that ``prepare`` is given.
"""
import math

import numpy as np
import torch

from turbodeberta_b200 import relpos
from turbodeberta_b200.model import FlashDebertaV2Model
from turbodeberta_b200.ops.flash_attention import flash_attention_with_disentangled
from turbodeberta_b200.ops.flash_attention_varlen import flash_attention_with_disentangled_varlen

HEAD_DIM = 64
DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}


def _fixed(name, batch, length, heads=12, **more):
    """Padded batch.  lo: shortest valid length (0: every row is full, no lengths are passed).  pos: the position
    terms.  tables: "kept" (projected and expanded once per layer, as the model does) or "per_call" (the projected
    tables are the q_pos / k_pos arguments of each call).  span 0: no log buckets, max_dist distances each way."""
    c = dict(entry="fixed", dtype="bf16", batch=batch, length=length, heads=heads, lo=0, len_seed=0, pos="c2p+p2c",
             tables="kept", span=256, max_dist=512)
    c.update(more)
    return dict(c, name=name) if name else c


def _packed(name, n_seqs, lo, hi, heads, spread, len_seed):
    """Packed stream of n_seqs sequences, lengths in [lo, hi], spread evenly or evenly over their logarithm."""
    c = dict(entry="packed", dtype="bf16", n_seqs=n_seqs, lo=lo, hi=hi, heads=heads, spread=spread, len_seed=len_seed,
             pos="c2p+p2c", span=256, max_dist=512)
    return dict(c, name=name) if name else c


def _scores(name, batch, length, heads, lo=0, len_seed=0):
    c = dict(entry="scores", dtype="bf16", batch=batch, length=length, heads=heads, lo=lo, len_seed=len_seed,
             pos="c2p+p2c", span=256, max_dist=512)
    return dict(c, name=name) if name else c


def _model(name, size, batch, length, lo=0, len_seed=0):
    """size: "base" (12 layers, hidden 768, 12 heads) or "large" (24 layers, hidden 1024, 16 heads)."""
    c = dict(entry="model", dtype="bf16", size=size, batch=batch, length=length, lo=lo, len_seed=len_seed)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one short sentence through one layer's attention: an interactive request
        _fixed("fixed_one_sentence", 1, 40),
        # a small batch of medium texts, projected tables handed over with each call
        _fixed("fixed_tables_per_call", 8, 128, tables="per_call"),
        # the benchmark's batch: base model's heads, 32 right-padded rows of 64 to 512 tokens
        _fixed("fixed_base_ragged", 32, 512, lo=64, len_seed=1002),
        # full rows on the large model's heads: one GPU's share of a 256-row encoder batch on eight GPUs
        _fixed("fixed_large_full", 32, 512, heads=16),
        # long documents, every row full
        _fixed("fixed_long", 4, 4096),
        # fp32: two full rows (the parity configuration), and an ordinary ragged batch of an odd padded length
        _fixed("fixed_fp32_base", 2, 128, dtype="fp32"),
        _fixed("fixed_fp32_ragged", 8, 387, dtype="fp32", lo=48, len_seed=7),
        # the packed stream of a corpus with mixed lengths, large model's heads
        _packed("packed_mixed", 256, 16, 1024, 16, "log", 1003),
        # packed long documents: the largest call
        _packed("packed_long", 64, 2048, 8192, 12, "even", 1005),
        # a caller that still multiplies out the position scores itself
        _scores("scores_batch", 8, 256, 12),
        # whole models: one short request, and a padded batch of mixed lengths
        _model("model_base_one", "base", 1, 32),
        _model("model_large_ragged", "large", 32, 512, lo=64, len_seed=1004),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fixed", "fixed", "fixed", "fp32", "packed", "packed", "scores", "model"])
    seed = rng.randrange(1 << 20)
    pos = rng.choice(["c2p+p2c"] * 6 + ["c2p", "p2c"])
    span, max_dist = rng.choice([(256, 512)] * 6 + [(64, 128), (0, 512)])
    if kind in ("fixed", "fp32"):
        fp32 = kind == "fp32"
        length = _log_int(rng, 16, 512 if fp32 else 4096)
        batch = min(_log_int(rng, 1, 32), max(1, (4096 if fp32 else 16384) // length))
        return _fixed(None, batch, length, rng.choice([12, 16]), dtype="fp32" if fp32 else "bf16",
                      lo=rng.choice([0, max(1, length // 8), max(1, length // 2)]), len_seed=seed, pos=pos,
                      tables=rng.choice(["kept", "kept", "kept", "per_call"]), span=span, max_dist=max_dist)
    if kind == "packed":
        hi = _log_int(rng, 64, 8192)
        n_seqs = max(1, min(_log_int(rng, 2, 256), 131072 // hi))
        c = _packed(None, n_seqs, max(1, hi // rng.choice([2, 4, 16, 64])), hi, rng.choice([12, 16]),
                    rng.choice(["even", "log"]), seed)
        return dict(c, pos=pos, span=span, max_dist=max_dist)
    if kind == "scores":
        length = _log_int(rng, 16, 512)
        batch = min(_log_int(rng, 1, 32), max(1, 4096 // length))
        return _scores(None, batch, length, rng.choice([12, 16]), rng.choice([0, max(1, length // 4)]), seed)
    length = _log_int(rng, 16, 512)
    batch = min(_log_int(rng, 1, 32), max(1, 8192 // length))
    return _model(None, rng.choice(["base", "base", "large"]), batch, length, rng.choice([0, max(1, length // 8)]), seed)


# ------------------------------------------------------------------------------------------------------------- sizes
def _lengths(case):
    rng = np.random.default_rng(case["len_seed"])
    if case["entry"] == "packed":
        if case["spread"] == "log":
            x = np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), case["n_seqs"]))
            return np.floor(x).astype(np.int64).clip(1)
        return rng.integers(case["lo"], case["hi"] + 1, case["n_seqs"])
    if not case["lo"]:
        return np.full(case["batch"], case["length"], dtype=np.int64)
    return rng.integers(case["lo"], case["length"] + 1, case["batch"])


def _two_span(case):
    return 2 * (case["span"] or case["max_dist"])


def _sm_scale(case):
    return 1.0 / math.sqrt(HEAD_DIM * (2 + case["pos"].count("+")))


def _model_size(case):
    return dict(base=(768, 12, 12), large=(1024, 24, 16))[case["size"]]              # hidden, layers, heads


def _attention_flops(lengths, heads, two_span, terms):
    """Q.K and P.V, and one product per position term with the table rows that the sequence's distances can reach."""
    n = lengths.astype(np.float64)
    reach = np.minimum(two_span, np.maximum(2 * n - 1, 0))
    return float((4 * n * n * HEAD_DIM + terms * 2 * n * reach * HEAD_DIM).sum() * heads)


def work(case):
    n = _lengths(case)
    tokens = float(n.sum())
    if case["entry"] == "model":
        hidden, layers, heads = _model_size(case)
        flops = layers * (2 * tokens * 12 * hidden * hidden + _attention_flops(n, heads, 512, 2))
        return {"flops": flops, "bytes": 2.0 * layers * 12 * hidden * hidden + 2 * 2 * tokens * hidden + 16 * tokens}
    e = 4 if case["dtype"] == "fp32" else 2
    heads, two_span, terms = case["heads"], _two_span(case), 1 + case["pos"].count("+")
    bytes_ = 4.0 * e * tokens * heads * HEAD_DIM + 4 * len(n)
    if case["entry"] == "scores":
        reach = np.minimum(two_span, np.maximum(2 * n - 1, 0))
        bytes_ += terms * e * float((n * reach).sum()) * heads
        return {"flops": _attention_flops(n, heads, two_span, 0), "bytes": bytes_}
    bytes_ += terms * e * two_span * heads * HEAD_DIM
    return {"flops": _attention_flops(n, heads, two_span, terms), "bytes": bytes_}


def tolerance(case):
    if case["entry"] == "model":            # every layer rounds its activations to bf16 several times
        return {"rel": 2e-2 if case["size"] == "base" else 3e-2}
    return {"rel": 1e-5 if case["dtype"] == "fp32" else 1e-2}


# ------------------------------------------------------------------------------------------------------------ inputs
def _tables(case, gen):
    """Projected tables of one layer, [heads, 2*span, 64] each (None for an absent term), in the call's dtype."""
    shape = (case["heads"], _two_span(case), HEAD_DIM)
    t = {}
    for term in ("c2p", "p2c"):
        x = torch.randn(shape, generator=gen, device="cuda").mul_(0.5).to(DTYPES[case["dtype"]])
        t[term] = x if term in case["pos"].split("+") else None
    return t["c2p"], t["p2c"]


def _kept_tables(case, gen):
    """The tables as a layer keeps them: projected from the relative embeddings and expanded, once."""
    dt, hidden = DTYPES[case["dtype"]], case["heads"] * HEAD_DIM
    rel = torch.randn(_two_span(case), hidden, generator=gen, device="cuda").to(dt)
    w = [(torch.randn(hidden, hidden, generator=gen, device="cuda") * (0.5 / math.sqrt(hidden))).to(dt) for _ in range(2)]
    return relpos.build_tables(rel, num_heads=case["heads"], position_buckets=case["span"],
                               max_relative_positions=case["max_dist"], key_weight=w[0], query_weight=w[1],
                               c2p="c2p" in case["pos"], p2c="p2c" in case["pos"])


def _prepare_model(case, gen):
    from transformers import DebertaV2Config
    hidden, layers, heads = _model_size(case)
    cfg = DebertaV2Config(vocab_size=128100, hidden_size=hidden, num_hidden_layers=layers, num_attention_heads=heads,
                          intermediate_size=4 * hidden, hidden_act="gelu", relative_attention=True, position_buckets=256,
                          max_relative_positions=-1, max_position_embeddings=512, norm_rel_ebd="layer_norm",
                          share_att_key=True, pos_att_type=["p2c", "c2p"], position_biased_input=False, type_vocab_size=0)
    before = torch.get_default_dtype()
    torch.set_default_dtype(torch.bfloat16)
    try:
        with torch.device("cuda"):
            model = FlashDebertaV2Model(cfg).eval()
    finally:
        torch.set_default_dtype(before)
    with torch.no_grad():
        for name, p in sorted(model.named_parameters()):
            if "LayerNorm" in name and name.endswith("weight"):
                p.fill_(1.0)
            else:
                p.normal_(0.0, 0.02, generator=gen)
    lens = torch.as_tensor(_lengths(case), device="cuda")
    ids = torch.randint(1, cfg.vocab_size, (case["batch"], case["length"]), generator=gen, device="cuda")
    ids[torch.arange(case["length"], device="cuda")[None] >= lens[:, None]] = 0      # padding token
    return {"model": model, "ids": ids}


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    if case["entry"] == "model":
        return {"case": case, **_prepare_model(case, gen)}
    dt, heads, n = DTYPES[case["dtype"]], case["heads"], _lengths(case)
    s = {"case": case, "sm_scale": _sm_scale(case), "tables": None, "q_pos": None, "k_pos": None, "seqlens": None}
    lead = (int(n.sum()),) if case["entry"] == "packed" else (case["batch"], case["length"])
    # q, k and v as a layer has them: views of one projection output [.., 3, heads, 64]
    qkv = torch.randn(*lead, 3, heads, HEAD_DIM, generator=gen, device="cuda", dtype=dt)
    q, k, v = (qkv.select(-3, i) for i in range(3))
    if case["entry"] == "packed":
        s["cu"] = torch.as_tensor(np.concatenate([[0], np.cumsum(n)]).astype(np.int32), device="cuda")
        s["max_seqlen"] = int(n.max())
        s["tables"] = _kept_tables(case, gen)
    else:
        q, k, v = (t.permute(0, 2, 1, 3) for t in (q, k, v))
        if case["lo"]:
            s["seqlens"] = torch.as_tensor(n.astype(np.int32), device="cuda")
        if case["entry"] == "scores":           # (batch, heads, length, 64), contiguous, as that convention has them
            q, k, v = (t.contiguous() for t in (q, k, v))
            kr, qr = _tables(case, gen)
            s["q_pos"] = torch.matmul(q, kr.transpose(-1, -2))
            s["k_pos"] = torch.matmul(k, qr.transpose(-1, -2))
        elif case["tables"] == "per_call":
            s["q_pos"], s["k_pos"] = _tables(case, gen)
        else:
            s["tables"] = _kept_tables(case, gen)
    s["q"], s["k"], s["v"] = q, k, v
    return s


# --------------------------------------------------------------------------------------------------------------- run
def run(s):
    case = s["case"]
    if case["entry"] == "model":
        ids = s["ids"]
        with torch.no_grad():
            return s["model"](input_ids=ids, attention_mask=ids.ne(0).long()).last_hidden_state
    if case["entry"] == "packed":
        return flash_attention_with_disentangled_varlen(
            s["q"], s["k"], s["v"], None, None, s["cu"], s["cu"], s["max_seqlen"], s["max_seqlen"], False, s["sm_scale"],
            case["span"], case["max_dist"], tables=s["tables"])
    return flash_attention_with_disentangled(
        s["q"], s["k"], s["v"], s["q_pos"], s["k_pos"], False, s["sm_scale"], case["span"], case["max_dist"],
        seqlens=s["seqlens"], tables=s["tables"])
