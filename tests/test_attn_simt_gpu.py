"""GPU parity of the CUDA-core attention kernel (the full-precision path) against the oracle."""
import os

import numpy as np
import pytest
import torch

from tests import util
from tests.golden import make_golden as G
from turbodeberta_b200 import workloads

pytestmark = pytest.mark.gpu
SIMT = 1


def _run_fixed(w, dtype, c2p=True, p2c=True, share=True, kernel=SIMT, with_lens=True):
    from turbodeberta_b200.ops.flash_attention import flash_attention_with_disentangled
    q, k, v, rel, P = util.device_inputs(w, dtype)
    tables = util.make_tables(w, rel, P, c2p, p2c, share) if (c2p or p2c) else None
    d = w.head_dim
    scale = 1.0 / (d * (1 + int(c2p) + int(p2c))) ** 0.5
    lens = torch.as_tensor(np.asarray(w.lengths), dtype=torch.int32, device="cuda") if with_lens else None
    o = flash_attention_with_disentangled(q.permute(0, 2, 1, 3), k.permute(0, 2, 1, 3), v.permute(0, 2, 1, 3),
                                          None, None, False, scale, w.position_buckets, w.max_relative_positions,
                                          seqlens=lens, tables=tables, kernel=kernel)
    ref = util.oracle_fixed(q, k, v, tables, w.lengths if with_lens else None, w, c2p, p2c, scale)
    return o.permute(0, 2, 1, 3), ref


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("name", sorted(G.SMALL_CASES))
def test_simt_small_cases(name, dtype):
    spec = G.SMALL_CASES[name]
    w = G.small_workload(name)
    c2p, p2c = "c2p" in spec[7], "p2c" in spec[7]
    o, ref = _run_fixed(w, dtype, c2p, p2c, share=spec[6])
    util.assert_close(o, ref, dtype, name)


def test_simt_config1_fp32_matches_eager_fixture():
    """Configuration 1 end to end at the op level: fp32, batch 2 x 128, against the committed eager output."""
    w = workloads.config1()
    o, ref = _run_fixed(w, torch.float32)
    util.assert_close(o, ref, torch.float32, "config1 vs oracle")
    gold = np.load(os.path.join(os.path.dirname(__file__), "golden", "attention_eager.npz"))["config1_every8th"]
    got = o.reshape(2, 128, 768)[:, ::8].float().cpu().numpy()
    assert np.abs(got - gold).max() / np.abs(gold).max() < util.FP32_REL_TOL


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_simt_varlen(dtype):
    from turbodeberta_b200.ops.flash_attention_varlen import flash_attention_with_disentangled_varlen
    w = workloads.make_attention_workload("v", seed=21, hidden_size=128, num_heads=2,
                                          lengths=[5, 1, 33, 17, 128, 129, 600], padded_len=None, dtype=dtype)
    q, k, v, rel, P = util.device_inputs(w, dtype)
    tables = util.make_tables(w, rel, P)
    cu = torch.as_tensor(w.cu_seqlens, device="cuda")
    scale = 1.0 / (3 * 64) ** 0.5
    o, lse = flash_attention_with_disentangled_varlen(q, k, v, None, None, cu, cu, 600, 600, False, scale, 256, 512,
                                                      tables=tables, kernel=SIMT, return_lse=True)
    ref = util.oracle_varlen(q, k, v, tables, w.cu_seqlens, w, sm_scale=scale)
    util.assert_close(o, ref, dtype, "varlen")
    assert torch.isfinite(lse).all()


def test_argument_errors():
    from turbodeberta_b200.ops.flash_attention import flash_attention_with_disentangled
    q = torch.zeros(1, 2, 16, 32, device="cuda")
    with pytest.raises(ValueError):
        flash_attention_with_disentangled(q, q, q, None, None)                  # head_dim 32
    q = torch.zeros(1, 2, 16, 64, device="cuda", dtype=torch.float16)
    with pytest.raises(ValueError):
        flash_attention_with_disentangled(q, q, q, None, None)                  # fp16
    q = torch.zeros(1, 2, 16, 64, device="cuda")
    with pytest.raises(ValueError):
        flash_attention_with_disentangled(q, q, q, torch.zeros(1, 2, 16, 300, device="cuda"), None,
                                          position_buckets=256, max_relative_distance=512)   # 300 columns are neither
    o = flash_attention_with_disentangled(q, q, q, torch.zeros(1, 2, 16, 512, device="cuda"), None,
                                          position_buckets=256, max_relative_distance=512)   # materialised scores
    assert o.shape == q.shape and torch.isfinite(o).all()
    with pytest.raises(RuntimeError):
        flash_attention_with_disentangled(q.cpu(), q.cpu(), q.cpu(), None, None)            # no CPU path
    with pytest.raises(NotImplementedError):
        flash_attention_with_disentangled(q, q, q, None, None, causal=True)


def test_understated_max_seqlen_and_short_offsets_are_reported():
    """The CUDA-core kernel sizes its grid from max_seqlen: a value below the longest sequence, or offsets that stop
    short of the token count, must come back as an error instead of rows that were never written."""
    from turbodeberta_b200.ops.flash_attention_varlen import flash_attention_with_disentangled_varlen
    w = workloads.make_attention_workload("v", seed=22, hidden_size=128, num_heads=2, lengths=[40, 200],
                                          padded_len=None, dtype=torch.float32)
    q, k, v, rel, P = util.device_inputs(w, torch.float32)
    tables = util.make_tables(w, rel, P)
    cu = torch.as_tensor(w.cu_seqlens, device="cuda")
    args = (False, 1.0 / (3 * 64) ** 0.5, 256, 512)
    with pytest.raises(ValueError, match="max_seqlen"):
        flash_attention_with_disentangled_varlen(q, k, v, None, None, cu, cu, 64, 64, *args, tables=tables, kernel=SIMT)
    short = cu.clone()
    short[-1] -= 8
    with pytest.raises(ValueError, match="cu_seqlens"):
        flash_attention_with_disentangled_varlen(q, k, v, None, None, short, short, 200, 200, *args, tables=tables,
                                                 kernel=SIMT)
    other = cu.clone()
    other[1] += 1                                          # key offsets that differ from the query offsets
    with pytest.raises(ValueError, match="key offsets"):
        flash_attention_with_disentangled_varlen(q, k, v, None, None, cu, other, 200, 200, *args, tables=tables)
    o = flash_attention_with_disentangled_varlen(q, k, v, None, None, cu, cu.clone(), 200, 200, *args, tables=tables)
    assert torch.isfinite(o).all()


def test_backward_raises_like_the_reference():
    """Forward-only (the reference raises in backward, ``ops/flash_attention.py:341-343``): a loss built on the output
    must fail loudly instead of training with no gradient through the attention."""
    from turbodeberta_b200.ops.flash_attention import flash_attention_with_disentangled
    from turbodeberta_b200.ops.flash_attention_varlen import flash_attention_with_disentangled_varlen
    q = torch.randn(1, 2, 16, 64, device="cuda", requires_grad=True)
    o = flash_attention_with_disentangled(q, q.detach(), q.detach(), None, None)
    assert o.requires_grad
    with pytest.raises(RuntimeError, match="forward-only"):
        o.sum().backward()
    qp = torch.randn(16, 2, 64, device="cuda", requires_grad=True)
    cu = torch.tensor([0, 16], dtype=torch.int32, device="cuda")
    o = flash_attention_with_disentangled_varlen(qp, qp.detach(), qp.detach(), None, None, cu, cu, 16, 16)
    with pytest.raises(RuntimeError, match="forward-only"):
        o.sum().backward()
    scores = torch.zeros(1, 2, 16, 512, device="cuda")
    with pytest.raises(RuntimeError, match="forward-only"):           # score-tensor form: refused before the launch
        flash_attention_with_disentangled(q, q, q, scores, None, position_buckets=256, max_relative_distance=512)
    with torch.no_grad():
        o = flash_attention_with_disentangled(q, q, q, scores, None, position_buckets=256, max_relative_distance=512)
    assert not o.requires_grad


@pytest.mark.parametrize("lengths,c2p,p2c", [([16], True, True), ([387, 300, 130, 65], True, True), ([512, 64], True, False), ([2048], True, True)])
def test_fp32_error_does_not_grow_with_the_sequence(lengths, c2p, p2c):
    """Relative 2-norm against float64 within four units of fp32 rounding (2^-24): the scores of unit variance bring about two, the
    output's own rounding half of one, and sums over 16 keys, the tile and the tiles are short enough to stay below those."""
    from turbodeberta_b200 import relpos
    from turbodeberta_b200.ops.flash_attention import flash_attention_with_disentangled
    from oracle import disentangled_oracle as orc
    g = torch.Generator(device="cuda").manual_seed(31)
    H, L = 4, max(lengths)
    q, k, v = (torch.randn(len(lengths), L, H, 64, generator=g, device="cuda") for _ in range(3))
    rel = torch.randn(512, H * 64, generator=g, device="cuda")
    w = [torch.randn(H * 64, H * 64, generator=g, device="cuda") * (0.5 / (H * 64) ** 0.5) for _ in range(2)]
    t = relpos.build_tables(rel, num_heads=H, position_buckets=256, max_relative_positions=512, key_weight=w[0], query_weight=w[1],
                            c2p=c2p, p2c=p2c)
    scale = 1 / (64 * (1 + c2p + p2c)) ** 0.5
    got = flash_attention_with_disentangled(*(x.permute(0, 2, 1, 3) for x in (q, k, v)), None, None, False, scale, 256, 512, tables=t,
                                            seqlens=torch.tensor(lengths, device="cuda", dtype=torch.int32))
    f64 = lambda x: None if x is None else x.double().cpu().numpy()      # noqa: E731
    want = orc.attention_fixed(f64(q), f64(k), f64(v), f64(t.kr), f64(t.qr), lengths, position_buckets=256, max_relative_positions=512,
                               c2p=c2p, p2c=p2c, sm_scale=scale)
    err = np.linalg.norm(got.permute(0, 2, 1, 3).double().cpu().numpy() - want) / np.linalg.norm(want)
    assert err <= 4 * 2.0 ** -24, err


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lengths,padded,heads", [([65], 65, 2), ([128, 64, 1], 128, 2), ([129, 0, 63], 129, 2), ([300, 192, 193], 300, 2),
                                                  ([257, 320, 64, 0], 320, 3), ([200, 65, 128, 1], 200, 12), ([128, 64, 1, 0] * 20, 128, 3),
                                                  ([128, 64, 1, 0] * 20, 128, 4)])
@pytest.mark.parametrize("c2p,p2c", [(True, True), (True, False), (False, True), (False, False)])
def test_pairs_of_warps_share_the_key_tiles(lengths, padded, heads, c2p, p2c, dtype):
    """One, two and four pairs, 16 and 32 rows, at the tiles' edges; sequences with no tile for some of the pairs, and none at all."""
    w = workloads.make_attention_workload("g", seed=24, hidden_size=64 * heads, num_heads=heads, lengths=lengths, padded_len=padded,
                                          position_buckets=32, max_relative_positions=64, dtype=dtype)
    o, ref = _run_fixed(w, dtype, c2p, p2c)
    util.assert_close(o, ref, dtype, f"{lengths} c2p={c2p} p2c={p2c}")
    for b, n in enumerate(lengths):
        assert torch.count_nonzero(o[b, n:]).item() == 0


def test_a_calls_own_tables_are_not_expanded_for_the_exact_kernel():
    """It reads them by index in either type: the call allocates its output, not the tensor-core kernels' copies of the tables (0.8 MB here)."""
    from turbodeberta_b200.ops.flash_attention import flash_attention_with_disentangled
    w = workloads.make_attention_workload("own", seed=23, hidden_size=128, num_heads=2, lengths=[40], padded_len=40, dtype=torch.bfloat16)
    q, k, v, rel, P = util.device_inputs(w, torch.bfloat16)
    t = util.make_tables(w, rel, P)
    q, k, v = (x.permute(0, 2, 1, 3) for x in (q, k, v))
    run = lambda **kw: flash_attention_with_disentangled(q, k, v, kw.pop("q_pos", None), kw.pop("k_pos", None), False, 0.07, w.position_buckets,
                                                         w.max_relative_positions, kernel=SIMT, **kw)
    run(q_pos=t.kr, k_pos=t.qr)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    got = run(q_pos=t.kr, k_pos=t.qr)
    assert torch.cuda.max_memory_allocated() - before < 100_000
    assert torch.equal(got, run(tables=t))


@pytest.mark.parametrize("form", ["tables", "content", "scores"])
@pytest.mark.parametrize("ragged", [False, True])
@pytest.mark.parametrize("batch,length", [(3, 192), (4, 192), (4, 129), (9, 65), (12, 128), (4, 300), (3, 449), (14, 128), (27, 128), (14, 256), (40, 65)])
def test_both_sides_of_the_rule_for_rows_and_pairs(batch, length, ragged, form):
    """Around the lines between 16 and 32 rows and between one and two pairs of warps (148 SMs, 12 heads): every block's rows, against torch in float64."""
    from turbodeberta_b200.ops.flash_attention import flash_attention_with_disentangled
    g = torch.Generator(device="cuda").manual_seed(37)
    q, k, v = (torch.randn(batch, 12, length, 64, generator=g, device="cuda") for _ in range(3))
    lens = torch.randint(1, length + 1, (batch,), generator=g, device="cuda", dtype=torch.int32) if ragged else None
    kr, qr = (torch.randn(12, 64, 64, generator=g, device="cuda") for _ in range(2))
    at = torch.arange(length, device="cuda")
    row = (at[:, None] - at[None, :] + 32).clamp(0, 63)                      # of query i and key j, without buckets
    pos, both = None, None
    if form != "content":
        c = torch.einsum("bhid,hrd->bhir", q.double(), kr.double()).float()
        p = torch.einsum("bhjd,hrd->bhjr", k.double(), qr.double()).float()
        pos = c.double().gather(-1, row.expand(batch, 12, -1, -1)) + p.double().gather(-1, row.t().expand(batch, 12, -1, -1)).transpose(-1, -2)
        both = (kr, qr) if form == "tables" else (c, p)
    got = flash_attention_with_disentangled(q, k, v, *(both or (None, None)), False, 0.07, 0, 32, seqlens=lens)
    s = torch.einsum("bhid,bhjd->bhij", q.double(), k.double())
    s = (s if pos is None else s + pos) * 0.07
    if ragged:
        s.masked_fill_(at >= lens[:, None, None, None], float("-inf"))
    want = torch.einsum("bhij,bhjd->bhid", s.softmax(-1), v.double())
    if ragged:
        want.masked_fill_((at >= lens[:, None])[:, None, :, None], 0.0)
    assert ((got.double() - want).norm() / want.norm()).item() < 1e-6            # fp32 sums: some 2e-7
