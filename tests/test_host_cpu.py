"""Host-side logic that needs no GPU: pack/unpack glue, mask analysis, model patch wiring, sharding (gloo, 2 ranks)."""
import os
import socket

import numpy as np
import pytest
import torch
import torch.distributed as dist
import torch.multiprocessing as mp


def test_pad_unpad_round_trip():
    from turbodeberta_b200 import padding
    g = torch.Generator().manual_seed(0)
    x = torch.randn(3, 7, 2, 4, generator=g)
    mask = torch.tensor([[1, 1, 1, 0, 0, 0, 0], [1, 1, 1, 1, 1, 1, 1], [0, 1, 0, 1, 1, 0, 0]])
    toks, idx, cu, mx = padding.unpad_input(x, mask)
    assert toks.shape == (13, 2, 4) and cu.tolist() == [0, 3, 10, 13] and mx == 7 and cu.dtype == torch.int32
    assert torch.equal(toks, x.reshape(21, 2, 4)[mask.flatten().bool()])
    back = padding.pad_input(toks, idx, 3, 7)
    assert torch.equal(back, x * mask[:, :, None, None])
    q, k, v, pk, pq, iq, (cq, ck), (mq, mk) = padding._upad_input(x, x + 1, x + 2, "kr", "qr", mask, 7, 2)
    assert torch.equal(k, toks + 1) and torch.equal(v, toks + 2) and pk == "kr" and pq == "qr"
    assert torch.equal(cq, cu) and mq == mk == 7 and torch.equal(iq, idx)
    with pytest.raises(NotImplementedError):
        padding._upad_input(x[:, :1], x, x, None, None, mask, 1, 2)


def test_mask_analysis():
    from turbodeberta_b200.model import analyse_mask

    def ext(m):
        e = m[:, None, None, :]
        return e * e.squeeze(-2).unsqueeze(-1)

    i = analyse_mask(ext(torch.ones(2, 5)), 2, 5)
    assert i.all_ones and i.right_padded
    i = analyse_mask(ext(torch.tensor([[1, 1, 0, 0, 0], [1, 1, 1, 1, 1]])), 2, 5)
    assert not i.all_ones and i.right_padded and i.seqlens.tolist() == [2, 5]
    i = analyse_mask(torch.tensor([[0, 0, 1, 1, 1], [1, 1, 1, 1, 1]]), 2, 5)
    assert not i.right_padded and i.seqlens.tolist() == [3, 5]
    with pytest.raises(ValueError):
        analyse_mask(torch.tril(torch.ones(1, 1, 5, 5)), 1, 5)
    assert analyse_mask(None, 1, 5).all_ones


def test_patch_classes_keep_hf_parameter_names():
    from transformers import DebertaV2Config
    from transformers.models.deberta_v2.modeling_deberta_v2 import DebertaV2Model
    from turbodeberta_b200 import model as M
    cfg = DebertaV2Config(vocab_size=300, hidden_size=128, num_hidden_layers=2, num_attention_heads=2,
                          intermediate_size=256, relative_attention=True, position_buckets=256,
                          max_relative_positions=-1, norm_rel_ebd="layer_norm", share_att_key=True,
                          pos_att_type=["p2c", "c2p"], position_biased_input=False, type_vocab_size=0)
    hf = DebertaV2Model(cfg)
    fl = M.FlashDebertaV2Model(cfg)
    assert list(fl.state_dict()) == list(hf.state_dict())
    fl.load_state_dict(hf.state_dict())
    assert all(isinstance(l.attention.self, M.FlashDisentangledSelfAttention) for l in fl.encoder.layer)
    for cls in (M.FlashDebertaV2ForMaskedLM, M.FlashDebertaV2ForSequenceClassification,
                M.FlashDebertaV2ForTokenClassification, M.FlashDebertaV2ForQuestionAnswering,
                M.FlashDebertaV2ForMultipleChoice):
        assert isinstance(cls(cfg).deberta.encoder, M.FlashDebertaV2Encoder)
    patched = M.patch_model(DebertaV2Model(cfg))
    assert isinstance(patched.encoder, M.FlashDebertaV2Encoder)
    assert all(isinstance(l.attention.self, M.FlashDisentangledSelfAttention) for l in patched.encoder.layer)
    # eval-mode relative embeddings are computed once and stamped
    patched.eval()
    with torch.no_grad():
        a, b = patched.encoder.get_rel_embedding(), patched.encoder.get_rel_embedding()
    assert a is b and hasattr(a, "_tdb_stamp")


def test_shard_planner():
    from turbodeberta_b200 import sharding
    sl = [sharding.shard_batch(10, 4, r) for r in range(4)]
    assert [s.stop - s.start for s in sl] == [3, 3, 2, 2] and sl[0].start == 0 and sl[-1].stop == 10
    lengths = [1000, 10, 20, 900, 30, 500, 480, 40]
    plan = sharding.shard_packed(lengths, 2)
    assert sorted(sum(plan, [])) == list(range(8))
    cost = [sum(lengths[i] ** 2 for i in p) for p in plan]
    assert max(cost) / min(cost) < 1.35


def _free_port():
    s = socket.socket(); s.bind(("127.0.0.1", 0)); p = s.getsockname()[1]; s.close(); return p


def _gather_worker(rank, world, port, ret):
    from turbodeberta_b200 import sharding
    os.environ.update(MASTER_ADDR="127.0.0.1", MASTER_PORT=str(port))
    dist.init_process_group("gloo", rank=rank, world_size=world)
    try:
        full = torch.arange(5 * 3 * 2, dtype=torch.float32).view(5, 3, 2)
        sl = sharding.shard_batch(5, world, rank)
        got = sharding.gather_padded(full[sl] * 1.0, 5)
        ok1 = torch.equal(got, full)
        lengths = [4, 1, 7, 2, 5]
        plan = sharding.shard_packed(lengths, world)
        cu = np.concatenate([[0], np.cumsum(lengths)])
        stream = torch.arange(int(cu[-1]) * 2, dtype=torch.float32).view(-1, 2)
        local = torch.cat([stream[cu[s]:cu[s + 1]] for s in plan[rank]], 0) if plan[rank] else stream[:0]
        got2 = sharding.gather_packed(local, lengths, plan)
        ok2 = torch.equal(got2, stream)
        ret[rank] = bool(ok1 and ok2)
    finally:
        dist.destroy_process_group()


def test_gather_two_ranks_gloo():
    world = 2
    mgr = mp.Manager()
    ret = mgr.dict()
    port = _free_port()
    mp.spawn(_gather_worker, args=(world, port, ret), nprocs=world, join=True)
    assert dict(ret) == {0: True, 1: True}


def test_reference_import_paths_resolve_to_this_package():
    """Code written against the reference imports ``turbodeberta.*`` (``src/turbodeberta/`` there): the alias package
    serves the same module paths and names from this implementation."""
    import turbodeberta.model as m
    import turbodeberta.ops.flash_attention as fa
    import turbodeberta.ops.flash_attention_varlen as fav
    import turbodeberta.padding as pad
    import turbodeberta_b200.model as ours
    from turbodeberta_b200.ops.flash_attention import flash_attention_with_disentangled
    from turbodeberta_b200.ops.flash_attention_varlen import flash_attention_with_disentangled_varlen
    assert m.FlashDebertaV2Model is ours.FlashDebertaV2Model
    assert m.FlashDisentangledSelfAttention is ours.FlashDisentangledSelfAttention
    for name in ("FlashDebertaV2Attention", "FlashDebertaV2Layer", "FlashDebertaV2Encoder", "FlashDebertaV2ForMaskedLM",
                 "FlashDebertaV2ForSequenceClassification", "FlashDebertaV2ForTokenClassification",
                 "FlashDebertaV2ForQuestionAnswering", "FlashDebertaV2ForMultipleChoice"):
        assert getattr(m, name) is getattr(ours, name)
    assert fa.flash_attention_with_disentangled is flash_attention_with_disentangled
    assert fav.flash_attention_with_disentangled_varlen is flash_attention_with_disentangled_varlen
    for name in ("pad_input", "unpad_input", "_upad_input", "index_first_axis", "index_put_first_axis", "_get_unpad_data"):
        assert callable(getattr(pad, name))


def test_pending_status_blocks_are_folded_never_dropped():
    """Unchecked status blocks pile up only to a bound, and a report in the very first one survives the folding."""
    from turbodeberta_b200.status import PendingStatus
    q = PendingStatus()
    first = torch.tensor([7, 0, 0, 0], dtype=torch.int32)
    q.append(first)
    for _ in range(3 * PendingStatus.FOLD_AT):
        q.append(torch.zeros(4, dtype=torch.int32))
    assert len(q) < PendingStatus.FOLD_AT
    blocks = q.drain()
    assert len(q) == 0
    assert int(torch.stack(blocks).amax(dim=0)[0]) == 7


def test_reports_of_several_kinds_are_all_named(monkeypatch):
    """Words of several calls come together in one check: none of them hides another, from the pool or from a block of a call's own."""
    from turbodeberta_b200 import _cabi as cabi
    from turbodeberta_b200.ops import flash_attention as fa
    pool = []
    monkeypatch.setattr(cabi.host, "drain_pending", lambda: pool.pop() if pool else None)
    wait, offsets, token = (302, 0, 0, 0), (0, 1, 0, 0), (0, 0, 0, 1)
    for pooled, own, error, texts in ((token, None, IndexError, ["vocabulary"]), (offsets, None, ValueError, ["cu_seqlens"]),
                                      (token, wait, cabi.TdbError, ["302", "vocabulary"]), (wait, token, cabi.TdbError, ["302", "vocabulary"]),
                                      ((401, 1, 0, 1), offsets, cabi.TdbError, ["401", "cu_seqlens", "vocabulary"]),
                                      (token, offsets, ValueError, ["cu_seqlens", "vocabulary"])):
        pool.append(pooled)
        if own:
            fa._PENDING_STATUS.append(torch.tensor(own, dtype=torch.int32))
        with pytest.raises(error) as e:
            fa.check_pending_status()
        assert all(t in str(e.value) for t in texts)
        fa.check_pending_status()                    # nothing is reported twice


def test_mask_analysis_refresh_recomputes_lengths_without_changing_the_route():
    from turbodeberta_b200.model import analyse_mask
    m = torch.zeros(2, 6, dtype=torch.long)
    m[0, :6] = 1
    m[1, :3] = 1
    a = analyse_mask(m, 2, 6)
    assert (a.all_ones, a.right_padded) == (False, True) and a.seqlens.tolist() == [6, 3]
    b = analyse_mask(m, 2, 6, refresh=True)
    assert b is not a and (b.all_ones, b.right_padded) == (False, True) and b.seqlens.tolist() == [6, 3]
    assert analyse_mask(m, 2, 6) is b                      # the refreshed analysis is what later calls see


def test_mask_analysis_after_the_native_one_has_the_validity_too():
    """The native analysis of a mask of ones keeps what the encoder needs of it; whoever asks for the rest afterwards gets it."""
    from turbodeberta_b200 import model as M
    m = torch.ones(2, 6, dtype=torch.long)
    M._mask_cache_put(m, M.MaskInfo(True, True, torch.tensor([6, 6], dtype=torch.int32), None, (12, 6, None)))
    info = M.analyse_mask(m, 2, 6)
    assert info.all_ones and info.right_padded and info.seqlens.tolist() == [6, 6] and torch.equal(info.key_mask, m != 0)
    assert M.analyse_mask(m, 2, 6) is info


@pytest.mark.parametrize("tokens,columns,features,own", [(32, 1024, 4096, 1), (33, 1024, 4096, 0), (32, 4096, 1024, 1), (8, 1024, 4104, 1), (1, 1280, 3840, 0), (1, 1280, 1280, 1),
                                                         (32, 768, 3072, 1), (16, 768, 4, 0), (16, 760, 8, 0)])
def test_which_projections_are_kernels_of_our_own(tokens, columns, features, own):
    import ctypes as C
    from turbodeberta_b200 import _cabi as cabi
    assert cabi.lib.tdb_skinny_applies(C.c_int64(tokens), C.c_int64(columns), C.c_int64(features)) == own


def _small_config(**kw):
    from transformers import DebertaV2Config
    return DebertaV2Config(**{**dict(vocab_size=50, hidden_size=128, num_hidden_layers=4, num_attention_heads=2,
                                     intermediate_size=256, relative_attention=True, position_buckets=32,
                                     max_relative_positions=64, norm_rel_ebd="layer_norm", share_att_key=True,
                                     pos_att_type=["p2c", "c2p"], position_biased_input=False, type_vocab_size=0), **kw})


@pytest.mark.parametrize("name,value", [("pos_att_type", ["c2p"]), ("pos_att_type", ["p2c"]), ("position_buckets", 16),
                                        ("max_relative_positions", 128), ("num_attention_heads", 1)])
def test_kept_tables_follow_the_modules_settings(name, value, monkeypatch):
    """The tables that a layer keeps are those of its present settings, not of the ones it had when they were made."""
    from turbodeberta_b200 import model as M
    monkeypatch.setattr(M._relpos, "build_tables", lambda rel, **kw: {k: v for k, v in kw.items() if "weight" not in k and "bias" not in k})
    sa = M.FlashDisentangledSelfAttention(_small_config()).eval()
    rel = torch.randn(64, 128)
    rel._tdb_stamp = (0, 1)
    before = sa._relative_tables(rel, rel.dtype)
    assert sa._relative_tables(rel, rel.dtype) is before and before["c2p"] and before["p2c"]
    setattr(sa, name, value)
    after = sa._relative_tables(rel, rel.dtype)
    assert after == dict(before, **(dict(c2p="c2p" in value, p2c="p2c" in value) if name == "pos_att_type" else
                                    {name.replace("num_attention_heads", "num_heads"): value}))
    assert sa._relative_tables(rel, rel.dtype) is after


def test_kept_relative_embeddings_follow_the_encoders_norm():
    """eps alone changes no weight; without the norm in norm_rel_ebd the embeddings go as they are."""
    from turbodeberta_b200 import model as M
    enc = M.FlashDebertaV2Encoder(_small_config()).eval()
    with torch.no_grad():
        enc.get_rel_embedding()
        enc.LayerNorm.eps = 0.5
        assert torch.equal(enc.get_rel_embedding(), enc.LayerNorm(enc.rel_embeddings.weight))
        enc.norm_rel_ebd = ["none"]
        assert torch.equal(enc.get_rel_embedding(), enc.rel_embeddings.weight)


def _set_eps(enc):
    enc.layer[1].output.LayerNorm.eps = 0.25


def _append_in_place(enc):
    enc.layer[0].attention.self.pos_att_type.append("p2c")


def _plain_gelu(enc):
    act = enc.layer[3].intermediate.intermediate_act_fn
    act.act = act._gelu_python


@pytest.mark.parametrize("change,native_after", [
    (lambda e: setattr(e, "layer", torch.nn.ModuleList(e.layer[:2])), True),          # pruned layers
    (lambda e: setattr(e, "layer", torch.nn.ModuleList(list(e.layer)[::-1])), True),
    (lambda e: e.layer.__delitem__(3), True),
    (_set_eps, True), (_append_in_place, True), (_plain_gelu, False),
    (lambda e: setattr(e.layer[0].attention.self, "share_att_key", False), True),
    (lambda e: setattr(e.layer[2].attention.output, "dropout", torch.nn.ReLU().eval()), False)])
def test_a_plan_is_of_the_encoders_present_layers(change, native_after):
    """What the native loop was made from, and what it is made from after a change (on the CPU a stack without position
    terms gets as far as that)."""
    from turbodeberta_b200 import model as M
    enc = M.FlashDebertaV2Encoder(_small_config(relative_attention=False, pos_att_type=[])).eval()
    x = torch.zeros(1, 128)
    with torch.no_grad():
        first = enc._native_plan(x, None)
        assert first.watch.holds() and enc._native_plan(x, None) is first and len(first.attns) == 4
        change(enc)
        kept = enc._native_plan(x, None)
        assert kept is not first or not kept.watch.holds()       # the encoder's forward asks both
        M._PLANS.pop(enc, None)
        made = enc._native_plan(x, None)
        assert (made is not None) == native_after
        if native_after:
            assert made.watch.holds() and made.attns == [layer.attention.self for layer in enc.layer]


class _FakePlan:
    """A plan that runs nothing; its watch fails the first time, after another thread has dropped the plan."""

    def __init__(self):
        self.native, self.watch, self.asked = self, self, 0

    def run(self, x, *_):
        return [x + 1], []

    def holds(self):
        self.asked += 1
        return self.asked > 1


def test_a_plan_that_another_thread_has_dropped(monkeypatch):
    from turbodeberta_b200 import model as M
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    enc = M.FlashDebertaV2Encoder(_small_config()).eval()
    plan = _FakePlan()
    enc._native_plan = lambda *_: plan
    with torch.no_grad():
        out = enc._forward_native(torch.zeros(1, 3, 128), None, False, True)
    assert plan.asked == 2 and torch.equal(out.last_hidden_state, torch.ones(1, 3, 128))


def test_one_thread_at_a_time_brings_a_plan_up_to_date(monkeypatch):
    import threading
    import time
    from turbodeberta_b200 import model as M
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    enc = M.FlashDebertaV2Encoder(_small_config()).eval()
    inside, most, plan = [], [0], _FakePlan()
    plan.asked = 1

    def slow(*_):
        inside.append(1)
        most[0] = max(most[0], len(inside))
        time.sleep(0.02)
        inside.pop()
        return plan
    enc._native_plan = slow

    def work():
        with torch.no_grad():
            enc._forward_native(torch.zeros(1, 3, 128), None, False, True)
    threads = [threading.Thread(target=work) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert most[0] == 1


def test_masks_of_several_threads():
    """Masks that come and go in many threads: the cache of their analyses drops entries that others drop too."""
    import sys
    import threading
    from turbodeberta_b200 import model as M
    before, failed = sys.getswitchinterval(), []

    def work():
        try:
            for i in range(400):
                m = torch.ones(1, 2)
                M._mask_cache_put(m, i)
                keep = [torch.ones(1, 2) for _ in range(3)]
                for t in keep:
                    M._mask_cache_put(t, i)
        except Exception as e:      # noqa: BLE001
            failed.append(e)
    sys.setswitchinterval(1e-6)
    try:
        threads = [threading.Thread(target=work) for _ in range(8)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        sys.setswitchinterval(before)
    assert not failed


def _shift(p):
    buf = torch.empty(p.numel() + 1)
    p.data = buf[1:].view_as(p).copy_(p.data)


@pytest.mark.parametrize("change,width,fits", [
    (lambda layer: None, 128, True), (lambda layer: None, 64, False), (lambda layer: None, 192, False),
    (lambda layer: _shift(layer.output.LayerNorm.weight), 128, False),
    (lambda layer: _shift(layer.output.dense.weight), 128, True),           # products look at that themselves
    (lambda layer: setattr(layer.output.dense.weight, "data", layer.output.dense.weight.data[:, :64].contiguous()), 128, False),
    (lambda layer: setattr(layer.intermediate.dense.bias, "data", layer.intermediate.dense.bias.data[:64]), 128, False),
    (lambda layer: setattr(layer.attention.self.key_proj.weight, "data", torch.zeros(64, 128)), 128, False)])
def test_the_native_loop_takes_only_what_it_can_read(change, width, fits):
    from turbodeberta_b200 import model as M
    enc = M.FlashDebertaV2Encoder(_small_config(relative_attention=False, pos_att_type=[])).eval()
    with torch.no_grad():
        assert enc._native_plan(torch.zeros(1, 128), None) is not None
        change(enc.layer[1])
        assert (enc._native_plan(torch.zeros(1, width), None) is not None) == fits


def test_a_mask_on_another_device_is_not_for_the_mask_kernel(monkeypatch):
    from turbodeberta_b200 import model as M
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(M, "analyse_mask", lambda *_, **__: M.MaskInfo(False, True, None, None))
    monkeypatch.setattr(M, "_analyse_2d", lambda *_: pytest.fail("another device's mask"))
    enc = M.FlashDebertaV2Encoder(_small_config()).eval()
    with torch.no_grad():
        assert enc._forward_native(torch.zeros(1, 3, 128), torch.ones(1, 3, device="meta"), False, True) is None
