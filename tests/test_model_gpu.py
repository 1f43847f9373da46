"""GPU parity of the patched HF modules against the eager modules they replace."""
import numpy as np
import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu


def _cfg(**kw):
    from transformers import DebertaV2Config
    base = dict(vocab_size=500, hidden_size=128, num_hidden_layers=2, num_attention_heads=2, intermediate_size=256,
                relative_attention=True, position_buckets=256, max_relative_positions=-1, norm_rel_ebd="layer_norm",
                share_att_key=True, pos_att_type=["p2c", "c2p"], position_biased_input=False, type_vocab_size=0,
                hidden_dropout_prob=0.0, attention_probs_dropout_prob=0.0)
    base.update(kw)
    return DebertaV2Config(**base)


def _ext(mask2d):
    e = mask2d[:, None, None, :]
    return e * e.squeeze(-2).unsqueeze(-1)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("mask_kind", ["ones", "right", "left"])
@pytest.mark.parametrize("share,pos", [(True, ["c2p", "p2c"]), (False, ["c2p", "p2c"]), (True, ["c2p"]), (True, [])])
def test_attention_module_matches_eager(dtype, mask_kind, share, pos):
    from transformers.models.deberta_v2.modeling_deberta_v2 import DisentangledSelfAttention
    from turbodeberta_b200.model import FlashDisentangledSelfAttention
    torch.manual_seed(3)
    cfg = _cfg(share_att_key=share, pos_att_type=pos, relative_attention=len(pos) > 0)
    ref = DisentangledSelfAttention(cfg).eval()
    with torch.no_grad():
        for p in ref.parameters():
            p.normal_(0, 0.05)
    B, L = 3, 200
    x = torch.randn(B, L, 128)
    rel = torch.randn(512, 128) * 0.1
    lens = {"ones": [L, L, L], "right": [200, 37, 129], "left": [200, 37, 129]}[mask_kind]
    m = torch.zeros(B, L, dtype=torch.long)
    for b, n in enumerate(lens):
        if mask_kind == "left":
            m[b, L - n:] = 1
        else:
            m[b, :n] = 1
    # reference: fp32 eager on the same (dtype-rounded) parameters and inputs
    ref_r = DisentangledSelfAttention(cfg).eval()
    ref_r.load_state_dict({k: v.to(dtype).float() for k, v in ref.state_dict().items()})
    xr, relr = x.to(dtype).float(), rel.to(dtype).float()
    with torch.no_grad():
        want, _ = ref_r(xr, _ext(m).bool(), relative_pos=None, rel_embeddings=relr)
    fl = FlashDisentangledSelfAttention(cfg).eval()
    fl.load_state_dict(ref.state_dict())
    fl = fl.to("cuda", dtype)
    with torch.no_grad():
        got, probs = fl(x.to("cuda", dtype), _ext(m).to("cuda"), rel_embeddings=rel.to("cuda", dtype))
    assert probs is None and got.shape == (B, L, 128)
    valid = m.bool()
    g, w = got.float().cpu()[valid].numpy(), want[valid].numpy()
    if dtype == torch.float32:
        assert np.abs(g - w).max() / np.abs(w).max() < util.FP32_REL_TOL
    else:
        # Q/K/V are rounded to bf16 after the projection in the fused path only; allow for it on top of the kernel tolerance
        assert np.abs(g - w).max() < 2 * util.BF16_ABS_TOL
    assert torch.count_nonzero(got.float().cpu()[~valid]).item() == 0


def test_whole_model_matches_eager_fp32():
    from transformers.models.deberta_v2.modeling_deberta_v2 import DebertaV2Model
    from turbodeberta_b200.model import FlashDebertaV2Model, patch_model
    torch.manual_seed(5)
    cfg = _cfg()
    hf = DebertaV2Model(cfg).eval()
    fl = FlashDebertaV2Model(cfg).eval()
    fl.load_state_dict(hf.state_dict())
    ids = torch.randint(0, 500, (3, 160))
    mask = torch.ones(3, 160, dtype=torch.long)
    mask[1, 100:] = 0
    mask[2, 33:] = 0
    with torch.no_grad():
        want = hf(input_ids=ids, attention_mask=mask).last_hidden_state
        got = fl.cuda()(input_ids=ids.cuda(), attention_mask=mask.cuda()).last_hidden_state.cpu()
        got2 = fl(input_ids=ids.cuda(), attention_mask=mask.cuda()).last_hidden_state.cpu()      # cached tables
    v = mask.bool()
    assert (got[v] - want[v]).abs().max().item() / want[v].abs().max().item() < 2e-4
    assert torch.equal(got, got2)
    patched = patch_model(DebertaV2Model(cfg).eval())
    patched.load_state_dict(hf.state_dict())
    with torch.no_grad():
        got3 = patched.cuda()(input_ids=ids.cuda(), attention_mask=mask.cuda()).last_hidden_state.cpu()
    assert (got3[v] - want[v]).abs().max().item() / want[v].abs().max().item() < 2e-4


def test_tables_follow_weight_updates():
    """The cached relative tables must be rebuilt when a projection weight changes in place."""
    from turbodeberta_b200.model import FlashDebertaV2Model
    torch.manual_seed(6)
    fl = FlashDebertaV2Model(_cfg()).eval().cuda()
    ids = torch.randint(0, 500, (1, 64)).cuda()
    with torch.no_grad():
        a = fl(input_ids=ids).last_hidden_state.clone()
        fl.encoder.layer[0].attention.self.key_proj.weight.mul_(1.5)
        b = fl(input_ids=ids).last_hidden_state
    assert not torch.equal(a, b)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_packed_encoder_route_matches_padded_route(dtype):
    """Padded batches run on the packed token stream by default; both routes and the eager model must agree on
    every valid token, for the last layer and for the intermediate hidden states."""
    from transformers.models.deberta_v2.modeling_deberta_v2 import DebertaV2Model
    from turbodeberta_b200.model import FlashDebertaV2Model
    torch.manual_seed(8)
    cfg = _cfg(num_hidden_layers=3)
    hf = DebertaV2Model(cfg).eval()
    fl = FlashDebertaV2Model(cfg).eval()
    fl.load_state_dict(hf.state_dict())
    fl = fl.to("cuda", dtype)
    ids = torch.randint(0, 500, (4, 300))
    mask = torch.zeros(4, 300, dtype=torch.long)
    for b, n in enumerate([300, 17, 129, 256]):
        mask[b, :n] = 1
    v = mask.bool()
    with torch.no_grad():
        want = hf(input_ids=ids, attention_mask=mask, output_hidden_states=True)
        assert fl.encoder.pack_padded_batches
        packed = fl(input_ids=ids.cuda(), attention_mask=mask.cuda(), output_hidden_states=True)
        fl.encoder.pack_padded_batches = False
        padded = fl(input_ids=ids.cuda(), attention_mask=mask.cuda(), output_hidden_states=True)
        fl.encoder.pack_padded_batches = True
    assert len(packed.hidden_states) == len(want.hidden_states) == 4
    tol = 2e-4 if dtype == torch.float32 else 6e-2
    for a, b_, c in zip(packed.hidden_states, padded.hidden_states, want.hidden_states):
        a, b_ = a.float().cpu(), b_.float().cpu()
        scale = c[v].abs().max().item()
        assert (a[v] - c[v]).abs().max().item() / scale < tol
        assert (a[v] - b_[v]).abs().max().item() / scale < tol
    assert torch.count_nonzero(packed.last_hidden_state.float().cpu()[~v]).item() == 0
    assert torch.equal(packed.last_hidden_state, packed.hidden_states[-1])


def test_encoder_forward_captures_into_a_cuda_graph():
    """After a warm-up with the same mask tensor (tables, fused weights and the mask analysis are cached) the whole
    model forward records into a CUDA graph: no allocation in the library, no synchronisation on the path; the
    replay reproduces the eager forward bit for bit and leaves the status words for the next check."""
    from turbodeberta_b200.model import FlashDebertaV2Model
    from turbodeberta_b200.ops.flash_attention import check_pending_status
    torch.manual_seed(9)
    model = FlashDebertaV2Model(_cfg(num_hidden_layers=3)).eval().cuda().to(torch.bfloat16)
    ids = torch.randint(0, 500, (4, 256), device="cuda")
    mask = torch.ones_like(ids)

    @torch.no_grad()
    def fwd():
        return model(input_ids=ids, attention_mask=mask).last_hidden_state

    eager = fwd().clone()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        fwd()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = fwd()
    ids.copy_(torch.randint(0, 500, (4, 256), device="cuda"))        # new contents in the captured input buffer
    graph.replay()
    torch.cuda.synchronize()
    check_pending_status()                                           # the replay's status words are readable now
    fresh = fwd()
    assert torch.equal(out, fresh)
    assert not torch.equal(out, eager)


def _config4():
    """Configuration 4's model: DeBERTa-v3-large geometry, random init."""
    from transformers import DebertaV2Config
    return DebertaV2Config(vocab_size=128100, hidden_size=1024, num_hidden_layers=24, num_attention_heads=16,
                           intermediate_size=4096, hidden_act="gelu", relative_attention=True, position_buckets=256,
                           max_relative_positions=-1, max_position_embeddings=512, norm_rel_ebd="layer_norm",
                           share_att_key=True, pos_att_type=["p2c", "c2p"], position_biased_input=False, type_vocab_size=0)


def test_config4_model_at_full_size_matches_eager():
    """The 24-layer, hidden-1024, 16-head model of configuration 4 on 512-token sequences against the eager model in
    fp32 on the host: bf16 on 2 x 512 tokens (tensor-core kernel), fp32 on 1 x 512 tokens (exact kernel)."""
    from transformers.models.deberta_v2.modeling_deberta_v2 import DebertaV2Model
    from turbodeberta_b200.model import FlashDebertaV2Model
    torch.manual_seed(1004)
    cfg = _config4()
    hf = DebertaV2Model(cfg).eval()
    sd_bf = {k: v.to(torch.bfloat16) for k, v in hf.state_dict().items()}
    hf.load_state_dict({k: v.float() for k, v in sd_bf.items()})          # fp32 model holding the bf16-rounded weights
    gen = torch.Generator().manual_seed(1004)
    ids = torch.randint(0, 128100, (2, 512), generator=gen)
    mask = torch.ones_like(ids)
    with torch.no_grad():
        want = hf(input_ids=ids, attention_mask=mask).last_hidden_state
    fl = FlashDebertaV2Model(cfg).eval()
    fl.load_state_dict(hf.state_dict())
    # fp32, one sequence
    fl32 = fl.to("cuda")
    with torch.no_grad():
        got32 = fl32(input_ids=ids[:1].cuda(), attention_mask=mask[:1].cuda()).last_hidden_state.cpu()
    rel = (got32 - want[:1]).abs().max().item() / want[:1].abs().max().item()
    assert rel < util.MODEL_FP32_REL_TOL, rel
    # bf16, both sequences; yardstick: the eager model in bf16 on the same GPU
    flbf = fl32.to(torch.bfloat16)
    with torch.no_grad():
        got = flbf(input_ids=ids.cuda(), attention_mask=mask.cuda()).last_hidden_state.float().cpu()
    del flbf, fl32, fl
    eager_bf = DebertaV2Model(cfg).eval()
    eager_bf.load_state_dict(hf.state_dict())
    eager_bf = eager_bf.to("cuda", torch.bfloat16)
    with torch.no_grad():
        eag = eager_bf(input_ids=ids.cuda(), attention_mask=mask.cuda()).last_hidden_state.float().cpu()
    del eager_bf
    torch.cuda.empty_cache()
    assert torch.isfinite(got).all()
    err_ours, err_eager = (got - want).abs(), (eag - want).abs()
    f = util.MODEL_BF16_VS_EAGER_FACTOR
    assert err_ours.max().item() <= f * err_eager.max().item(), (err_ours.max().item(), err_eager.max().item())
    assert err_ours.pow(2).mean().sqrt().item() <= f * err_eager.pow(2).mean().sqrt().item()


def test_task_head_classes_run_on_the_gpu():
    """The five head classes (broken constructors upstream, ``model.py:244-314``) through the fused kernels against
    their eager counterparts with the same weights, fp32, padded batch."""
    import transformers.models.deberta_v2.modeling_deberta_v2 as hfm
    import turbodeberta_b200.model as ours
    torch.manual_seed(11)
    cfg = _cfg(num_labels=2)                 # the question-answering head splits its output in two
    ids = torch.randint(0, 500, (3, 96))
    mask = torch.ones_like(ids)
    mask[1, 50:] = 0
    for name in ("ForMaskedLM", "ForSequenceClassification", "ForTokenClassification", "ForQuestionAnswering",
                 "ForMultipleChoice"):
        hf = getattr(hfm, "DebertaV2" + name)(cfg).eval()
        fl = getattr(ours, "FlashDebertaV2" + name)(cfg).eval()
        fl.load_state_dict(hf.state_dict())
        x, m = (ids[None], mask[None]) if name == "ForMultipleChoice" else (ids, mask)       # [1, choices, L]
        with torch.no_grad():
            want = hf(input_ids=x, attention_mask=m)
            got = fl.cuda()(input_ids=x.cuda(), attention_mask=m.cuda())
        outs = [("start_logits", "end_logits")] if name == "ForQuestionAnswering" else [("logits",)]
        for fields in outs:
            for f in fields:
                a, b = getattr(got, f).float().cpu(), getattr(want, f)
                if name in ("ForMaskedLM", "ForTokenClassification", "ForQuestionAnswering"):       # per-token outputs
                    v = mask.bool()
                    a, b = a[v], b[v]
                assert (a - b).abs().max().item() / max(b.abs().max().item(), 1e-6) < 5e-4, (name, f)
        del hf, fl


def _generic_route(model, **kw):
    """The layer-by-layer route: a hook anywhere in the stack takes the native layer loop out of the way."""
    handle = model.encoder.layer[0].register_forward_hook(lambda *a: None)
    try:
        return model(**kw)
    finally:
        handle.remove()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lengths,L", [([1], 1), ([128, 128], 128), ([129, 1, 64], 129), ([33, 0, 7, 200], 200), ([64, 1, 0, 17], 64)])
def test_native_layer_loop_matches_the_module_route(dtype, lengths, L):
    """The encoder's native loop against the modules it stands in for: one token, full rows, ragged rows, an empty row,
    holes in the mask; hooks and replaced parameters must be seen."""
    import copy
    from turbodeberta_b200.model import FlashDebertaV2Model
    torch.manual_seed(12)
    model = FlashDebertaV2Model(_cfg(num_hidden_layers=3)).eval().to("cuda", dtype)
    ids = torch.randint(0, 500, (len(lengths), L), device="cuda")
    mask = (torch.arange(L, device="cuda")[None] < torch.tensor(lengths, device="cuda")[:, None]).long()
    if L == 129:
        mask[0, 5:40] = 0                                            # not right padded
    v = mask.bool()
    tol = 1e-4 if dtype == torch.float32 else 4e-2
    with torch.no_grad():
        for _ in range(2):
            got = model(input_ids=ids, attention_mask=mask, output_hidden_states=True)
            want = _generic_route(model, input_ids=ids, attention_mask=mask, output_hidden_states=True)
            assert len(got.hidden_states) == len(want.hidden_states) == 4
            for a, b in zip(got.hidden_states, want.hidden_states):
                assert a.shape == b.shape
                assert (a.float() - b.float())[v].abs().max().item() <= tol * b.float()[v].abs().max().item()
            assert torch.equal(got.last_hidden_state, got.hidden_states[-1])
            assert torch.count_nonzero(got.last_hidden_state[~v]).item() == 0
            # a replaced parameter and an in-place update, both behind a plan that was made before
            model.encoder.layer[1].output.dense.weight = torch.nn.Parameter(model.encoder.layer[1].output.dense.weight * 1.25)
            model.encoder.layer[0].attention.self.key_proj.weight.mul_(1.1)
        plain = model(input_ids=ids, attention_mask=mask)
        assert plain.hidden_states is None
        twin = copy.deepcopy(model)
        assert torch.equal(twin(input_ids=ids, attention_mask=mask).last_hidden_state, plain.last_hidden_state)
        called = []
        model.encoder.layer[2].output.dense.register_forward_hook(lambda *a: called.append(1))
        model(input_ids=ids, attention_mask=mask)
        assert called


@pytest.mark.parametrize("rows,hidden", [(1, 8), (3, 768), (2400, 1024), (2401, 264), (5, 2048)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_residual_layernorm_kernel(rows, hidden, dtype):
    from turbodeberta_b200 import _cabi as cabi
    if dtype == torch.float32 and hidden > 1024:
        pytest.skip("fp32 rows go up to 1024 columns")
    torch.manual_seed(13)
    x, r = (torch.randn(rows, hidden, device="cuda").to(dtype) * 3 for _ in range(2))
    w, b = (torch.randn(hidden, device="cuda").to(dtype) for _ in range(2))
    out = torch.empty_like(x)
    cabi.check(cabi.host.add_layernorm(x, r, w, b, 1e-7, out))
    want = torch.nn.functional.layer_norm(x.double() + r.double(), (hidden,), w.double(), b.double(), 1e-7)
    tol = 1e-5 if dtype == torch.float32 else 1e-2
    assert (out.double() - want).abs().max().item() <= tol * want.abs().max().item()


@pytest.mark.parametrize("n", [8, 4096, 8 * 257])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gelu_kernel(n, dtype):
    from turbodeberta_b200 import _cabi as cabi
    x = torch.linspace(-9, 9, n, device="cuda").to(dtype)
    want = torch.nn.functional.gelu(x.double())
    cabi.check(cabi.host.gelu_(x))
    bound = (1e-6 if dtype == torch.float32 else 5e-3) * want.abs() + (2e-7 if dtype == torch.float32 else 1e-6)
    assert ((x.double() - want).abs() <= bound).all()


@pytest.mark.parametrize("lengths,L", [([40], 40), ([1, 90, 33], 90), ([128, 128], 128)])
def test_repeated_shapes_replay_a_recorded_graph(lengths, L):
    """From its second pass on a small shape runs as a recorded graph: new inputs, more shapes than are kept, other
    streams and replaced weights must all give what the first (unrecorded) pass gives."""
    from turbodeberta_b200.model import FlashDebertaV2Model
    from turbodeberta_b200.ops.flash_attention import check_pending_status
    torch.manual_seed(14)
    model = FlashDebertaV2Model(_cfg(num_hidden_layers=2)).eval().to("cuda", torch.bfloat16)

    def inputs(extra=0):
        ids = torch.randint(1, 500, (len(lengths), L + extra), device="cuda")
        mask = (torch.arange(L + extra, device="cuda")[None] < torch.tensor(lengths, device="cuda")[:, None] + extra).long()
        return dict(input_ids=ids, attention_mask=mask)

    @torch.no_grad()
    def fresh(kw):
        with torch.cuda.stream(torch.cuda.Stream()):                 # a stream's first pass is not recorded
            out = model(**kw).last_hidden_state
        torch.cuda.synchronize()
        return out

    with torch.no_grad():
        for step in range(4):
            kw = inputs()
            assert torch.equal(model(**kw).last_hidden_state, fresh(kw)), step
        for extra in list(range(1, 12)) * 2:
            kw = inputs(extra)
            a = model(**kw).last_hidden_state
            assert torch.equal(a, model(**kw).last_hidden_state)
        model.encoder.layer[1].intermediate.dense.weight = torch.nn.Parameter(model.encoder.layer[1].intermediate.dense.weight * 1.5)
        model.encoder.layer[0].attention.self.value_proj.weight.mul_(0.5)
        kw = inputs()
        a = model(**kw).last_hidden_state
        assert torch.equal(a, fresh(kw))
    check_pending_status()


def test_plans_do_not_keep_models_alive():
    """A model that is dropped takes its native plan, recorded graphs and weights along."""
    import gc
    from turbodeberta_b200 import model as M
    model = M.FlashDebertaV2Model(_cfg(num_hidden_layers=2)).eval().to("cuda", torch.bfloat16)
    ids = torch.randint(1, 500, (2, 40), device="cuda")
    gc.collect()
    before = len(M._PLANS)
    with torch.no_grad():
        for _ in range(3):
            model(input_ids=ids, attention_mask=torch.ones_like(ids))
    assert len(M._PLANS) == before + 2                   # the model's and its encoder's
    del model
    gc.collect()
    assert len(M._PLANS) == before


def test_replaced_embeddings_and_hooks_on_them_are_seen():
    from turbodeberta_b200.model import FlashDebertaV2Model
    torch.manual_seed(15)
    model = FlashDebertaV2Model(_cfg(num_hidden_layers=2)).eval().to("cuda", torch.bfloat16)
    ids = torch.randint(1, 500, (2, 40), device="cuda")
    mask = torch.ones_like(ids)
    mask[1, 20:] = 0
    with torch.no_grad():
        a = model(input_ids=ids, attention_mask=mask).last_hidden_state
        assert torch.equal(a, model(ids, mask).last_hidden_state)          # positional arguments: the HF model's own forward
        assert torch.equal(a, model(input_ids=ids, attention_mask=mask, return_dict=False)[0])
        called = []
        handle = model.embeddings.LayerNorm.register_forward_hook(lambda *x: called.append(1))
        assert torch.equal(a, model(input_ids=ids, attention_mask=mask).last_hidden_state) and called
        handle.remove()
        model.embeddings.word_embeddings = torch.nn.Embedding(500, 128).to("cuda", torch.bfloat16)
        b = model(input_ids=ids, attention_mask=mask).last_hidden_state
        assert not torch.equal(a, b)
        assert torch.equal(b, model(ids, mask).last_hidden_state)


@pytest.mark.parametrize("tokens", [1, 16, 17, 32])
@pytest.mark.parametrize("columns,features", [(32, 8), (768, 2304), (1024, 1000), (2080, 768), (3072, 776), (4096, 64)])
@pytest.mark.parametrize("gelu", [False, True])
def test_skinny_projection(tokens, columns, features, gelu):
    """The projection kernel for few tokens at the edges of its token tiles, column blocks per warp and feature groups."""
    from turbodeberta_b200 import _cabi as cabi
    torch.manual_seed(16)
    x = torch.randn(tokens, columns, device="cuda").bfloat16()
    w = (torch.randn(features, columns, device="cuda") / columns ** 0.5).bfloat16()
    b = torch.randn(features, device="cuda").bfloat16()
    y = torch.full((tokens, features), float("nan"), device="cuda", dtype=torch.bfloat16)
    cabi.check(cabi.host.skinny(x, w, b, gelu, y))
    want = torch.nn.functional.linear(x.double(), w.double(), b.double())
    want = torch.nn.functional.gelu(want) if gelu else want
    assert ((y.double() - want).abs() <= 5e-3 * want.abs() + 1e-5).all()
    big = torch.zeros(33, columns, device="cuda", dtype=torch.bfloat16)
    assert cabi.host.skinny(big, w, b, gelu, y) == cabi.ERR_SHAPE


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_changed_stacks_and_settings_are_seen(dtype):
    """After a first pass: fewer layers in a new list, another eps, another set of position terms; each result is the
    module route's for the model as it then is."""
    import copy
    from turbodeberta_b200.model import FlashDebertaV2Model
    torch.manual_seed(17)
    model = FlashDebertaV2Model(_cfg(num_hidden_layers=4)).eval().to("cuda", dtype)
    ids = torch.randint(1, 500, (2, 40), device="cuda")
    mask = torch.ones_like(ids)
    mask[1, 20:] = 0
    v = mask.bool()
    enc = model.encoder
    with torch.no_grad():                            # scores of some size, so that the position terms matter
        for layer in enc.layer:
            layer.attention.self.query_proj.weight.mul_(10)
            layer.attention.self.key_proj.weight.mul_(10)
            layer.attention.self.value_proj.weight.mul_(10)

    def prune():
        enc.layer = torch.nn.ModuleList(enc.layer[:2])

    def eps():
        enc.layer[-1].output.LayerNorm.eps = 0.5

    def terms():
        for layer in enc.layer:
            layer.attention.self.pos_att_type = ["c2p"]

    tol = 1e-4 if dtype == torch.float32 else 4e-2
    with torch.no_grad():
        before = None
        for change in (lambda: None, prune, eps, terms):
            change()
            for _ in range(3):                       # the last ones replay a recording in bf16
                got = model(input_ids=ids, attention_mask=mask).last_hidden_state
            # by the modules of a copy: a hook on this model's would make it drop its plan
            want = _generic_route(copy.deepcopy(model), input_ids=ids, attention_mask=mask).last_hidden_state
            err = (got.float() - want.float())[v].abs().max().item()
            assert err <= tol * want.float()[v].abs().max().item()
            if before is not None:                   # and the change is no matter of rounding
                assert (got.float() - before)[v].abs().max().item() > 4 * err
            before = got.float()


def test_first_passes_of_several_threads():
    """Threads on streams of their own, all of them on a model without a plan and then on its recordings."""
    import threading
    from turbodeberta_b200.model import FlashDebertaV2Model
    torch.manual_seed(18)
    for _ in range(3):
        model = FlashDebertaV2Model(_cfg(num_hidden_layers=3)).eval().to("cuda", torch.bfloat16)
        ids = torch.randint(1, 500, (2, 60), device="cuda")
        mask = torch.ones_like(ids)
        torch.cuda.synchronize()
        outs, failed = [], []

        def work():
            try:
                with torch.no_grad(), torch.cuda.stream(torch.cuda.Stream()):
                    for _ in range(4):
                        out = model(input_ids=ids, attention_mask=mask).last_hidden_state
                        torch.cuda.current_stream().synchronize()
                        outs.append(out)
            except Exception as e:      # noqa: BLE001
                failed.append(e)
        threads = [threading.Thread(target=work) for _ in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not failed
        with torch.no_grad():
            want = model(input_ids=ids, attention_mask=mask).last_hidden_state
        assert len(outs) == 16 and all(torch.equal(o, want) for o in outs)


class _room:
    """At most this many more bytes from the device while it lasts."""

    def __init__(self, room):
        self.room = room

    def __enter__(self):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        total = torch.cuda.get_device_properties(0).total_memory
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + self.room) / total)

    def __exit__(self, *_):
        torch.cuda.set_per_process_memory_fraction(1.0)


def test_status_slots_survive_calls_that_run_out_of_memory():
    """More failing calls than there are slots: 32 MB of mask whose 256 MB of lengths and offsets do not fit."""
    from turbodeberta_b200._cabi import host
    mask = torch.ones(1 << 25, 1, dtype=torch.uint8, device="cuda")
    small = torch.ones(2, 3, dtype=torch.uint8, device="cuda")
    with _room(64 << 20):
        for _ in range(300):
            with pytest.raises(torch.OutOfMemoryError):
                host.mask_rows(mask)
    assert host.mask_rows(small)[:4] == (True, True, 6, 3)


def test_streams_that_their_owner_destroys():
    """Deferred checks and recordings of a stream of the caller's that is gone when they are looked at, or whose handle has
    passed to a new stream."""
    import ctypes
    from turbodeberta_b200.model import FlashDebertaV2Model
    from turbodeberta_b200.ops.flash_attention import check_pending_status, flash_attention_with_disentangled
    torch.manual_seed(19)
    model = FlashDebertaV2Model(_cfg(num_hidden_layers=2)).eval().to("cuda", torch.bfloat16)
    rt = torch.cuda.cudart()
    q = torch.randn(1, 2, 40, 64, device="cuda").bfloat16()
    want = flash_attention_with_disentangled(q, q, q, None, None)
    for _ in range(4):
        ids = torch.randint(1, 500, (2, 40), device="cuda")
        with torch.no_grad():
            ref = model(input_ids=ids, attention_mask=torch.ones_like(ids)).last_hidden_state
        torch.cuda.synchronize()
        handle = ctypes.c_void_p(0)
        assert int(rt.cudaStreamCreate(ctypes.addressof(handle))) == 0
        with torch.no_grad(), torch.cuda.stream(torch.cuda.ExternalStream(handle.value)):
            outs = [model(input_ids=ids, attention_mask=torch.ones_like(ids)).last_hidden_state for _ in range(3)]
            o = flash_attention_with_disentangled(q, q, q, None, None, check_status=False)
            torch.cuda.current_stream().synchronize()
            outs = [t.cpu() for t in outs]
            same = torch.equal(o, want)
        assert int(rt.cudaStreamDestroy(handle.value)) == 0
        check_pending_status()
        assert same and all(torch.equal(t, ref.cpu()) for t in outs)


def _flatten_parameters(model, shift):
    """All parameters as views of one buffer, each `shift` bytes behind a 256-byte boundary."""
    params = list(model.parameters())
    size = params[0].element_size()
    step = 256 // size
    flat = torch.empty(sum((p.numel() // step + 2) * step for p in params), dtype=params[0].dtype, device="cuda")
    at = 0
    for p in params:
        view = flat[at + shift // size:][:p.numel()].view_as(p)
        view.copy_(p.data)
        p.data = view
        at += (p.numel() // step + 2) * step
    assert all(p.data_ptr() % 256 == shift for p in params)


def test_parameters_in_one_flat_buffer():
    """Weights, biases and norms that start on 16-byte boundaries only: the native loop takes them, with library products chosen
    for that alignment (72 tokens) and with the projection kernels (24)."""
    from turbodeberta_b200 import model as M
    torch.manual_seed(20)
    model = M.FlashDebertaV2Model(_cfg(num_hidden_layers=2)).eval().to("cuda", torch.bfloat16)
    aligned = [torch.randint(1, 500, (2, n), device="cuda") for n in (36, 12)]
    with torch.no_grad():
        before = [model(input_ids=i, attention_mask=torch.ones_like(i)).last_hidden_state for i in aligned]
        _flatten_parameters(model, 16)
        for ids, want in zip(aligned, before):
            for _ in range(3):
                got = model(input_ids=ids, attention_mask=torch.ones_like(ids)).last_hidden_state
                assert (got.float() - want.float()).abs().max().item() <= 4e-2 * want.float().abs().max().item()
        assert M._PLANS.get(model.encoder) is not None


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("padded", [False, True])
def test_encoder_inputs_of_any_layout(dtype, padded):
    """Hidden states that are a slice of wider rows or start between two 16-byte pieces; rows of the wrong width are refused as
    by the modules."""
    from turbodeberta_b200.model import FlashDebertaV2Encoder
    torch.manual_seed(21)
    enc = FlashDebertaV2Encoder(_cfg(num_hidden_layers=2)).eval().to("cuda", dtype)
    B, L = 2, 40
    mask = torch.ones(B, L, dtype=torch.long, device="cuda")
    if padded:
        mask[1, 20:] = 0
    x = torch.randn(B, L, 128, device="cuda").to(dtype)
    wide = torch.randn(B, L, 256, device="cuda").to(dtype)
    wide[..., :128] = x
    flat = torch.empty(B * L * 128 + 1, device="cuda", dtype=dtype)
    flat[1:] = x.flatten()
    with torch.no_grad():
        for every in (True, False, False, False):
            want = enc(x, mask, output_hidden_states=every).last_hidden_state
            for y in (wide[..., :128], flat[1:].view(B, L, 128), x.transpose(0, 1).contiguous().transpose(0, 1)):
                assert torch.equal(enc(y, mask, output_hidden_states=every).last_hidden_state, want)
        for width in (64, 192):
            with pytest.raises(RuntimeError):
                enc(torch.randn(B, L, width, device="cuda").to(dtype), mask)
        norm = enc.layer[0].output.LayerNorm
        shifted = torch.empty(129, device="cuda", dtype=dtype)[1:]
        norm.weight.data = shifted.copy_(norm.weight.data)
        got = enc(x, mask).last_hidden_state
    tol = 1e-4 if dtype == torch.float32 else 4e-2
    assert (got.float() - want.float()).abs().max().item() <= tol * want.float().abs().max().item()


def test_recordings_are_kept_for_shapes_that_come_back():
    """Eight recordings.  More shapes than that in turn push none of them out; a shape that keeps coming while another stays
    away takes its place; weights that change with every pass are not recorded for.  Every pass gives the first one's result."""
    from turbodeberta_b200 import model as M
    torch.manual_seed(22)
    model = M.FlashDebertaV2Model(_cfg(num_hidden_layers=2)).eval().to("cuda", torch.bfloat16)
    ids = [torch.randint(1, 500, (1, n), device="cuda") for n in range(20, 32)]

    @torch.no_grad()
    def run(x):
        out = model(input_ids=x, attention_mask=torch.ones_like(x)).last_hidden_state
        return out, M._PLANS[model.encoder].native.recordings

    want = [run(x)[0] for x in ids]
    assert run(ids[0])[1] == 1                       # the second appearance
    for _ in range(20):
        for x, w in zip(ids, want):
            out, made = run(x)
            assert torch.equal(out, w)
    assert made == 8
    for i in range(12):
        out, made = run(ids[11])                     # one of the four without a recording
        assert torch.equal(out, want[11])
    assert made == 9
    made = run(ids[0])[1]
    with torch.no_grad():
        for _ in range(6):
            model.encoder.layer[0].attention.self.key_proj.bias.add_(0.01)
            assert run(ids[1])[1] == made


def test_long_sequences_without_room_for_scratch_say_so():
    """24 MB of output fit, 49 MB of scratch do not: a warning, and the same attention."""
    import warnings
    from turbodeberta_b200 import relpos
    from turbodeberta_b200.ops.flash_attention import flash_attention_with_disentangled
    torch.manual_seed(23)
    q, k, v = (torch.randn(4, 4096, 12, 64, device="cuda").bfloat16().permute(0, 2, 1, 3) for _ in range(3))
    w = [(torch.randn(768, 768, device="cuda") / 56).bfloat16() for _ in range(2)]
    tables = relpos.build_tables(torch.randn(512, 768, device="cuda").bfloat16(), num_heads=12, position_buckets=256,
                                 max_relative_positions=512, key_weight=w[0], query_weight=w[1])

    def call():
        return flash_attention_with_disentangled(q, k, v, None, None, False, 1 / 192 ** 0.5, 256, 512, tables=tables)
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        want = call()
        with _room(40 << 20):
            with pytest.raises(RuntimeWarning, match="49 MB of scratch"):
                call()
    with _room(40 << 20), pytest.warns(RuntimeWarning, match="49 MB of scratch"):
        got = call()
    # both round P to bf16 against reference exponents of their own: two roundings of half a unit, outputs below 1
    assert (got.float() - want.float()).abs().max().item() < 8e-3


def test_a_pass_that_fits_once_fits_again():
    """The buffers of a recording may not fit where the pass itself does."""
    from turbodeberta_b200.model import FlashDebertaV2Encoder
    torch.manual_seed(24)
    enc = FlashDebertaV2Encoder(_cfg(num_hidden_layers=2)).eval().to("cuda", torch.bfloat16)
    x = torch.randn(32, 256, 128, device="cuda").bfloat16()          # 2 MB
    mask = torch.ones(32, 256, dtype=torch.long, device="cuda")
    fitted = 0
    with torch.no_grad():
        want = enc(x, mask, output_hidden_states=False).last_hidden_state
        for room in range(32, 96, 4):
            with torch.cuda.stream(torch.cuda.Stream()):
                with _room(room << 20):
                    try:
                        first = enc(x, mask, output_hidden_states=False).last_hidden_state
                    except torch.OutOfMemoryError:
                        continue
                    del first
                    fitted += 1
                    second = enc(x, mask, output_hidden_states=False).last_hidden_state
                assert torch.equal(second, want)
    assert fitted


@pytest.mark.parametrize("tokens,features", [(16, 3552), (16, 3560), (1, 4104), (17, 1184), (17, 1192), (32, 4096)])
@pytest.mark.parametrize("columns", [32, 768, 1024])
def test_skinny_projection_on_both_sides_of_its_rule(tokens, features, columns):
    """8 features per block up to three (one token tile) or one (two) of them per SM, 16 beyond; also a last block that is half full."""
    from turbodeberta_b200 import _cabi as cabi
    torch.manual_seed(25)
    x = torch.randn(tokens, columns, device="cuda").bfloat16()
    w = (torch.randn(features, columns, device="cuda") / columns ** 0.5).bfloat16()
    b = torch.randn(features, device="cuda").bfloat16()
    y = torch.full((tokens + 1, features), float("nan"), device="cuda", dtype=torch.bfloat16)
    cabi.check(cabi.host.skinny(x, w, b, False, y))
    want = torch.nn.functional.linear(x.double(), w.double(), b.double())
    assert ((y[:tokens].double() - want).abs() <= 5e-3 * want.abs() + 1e-5).all()
    assert y[tokens].isnan().all()
