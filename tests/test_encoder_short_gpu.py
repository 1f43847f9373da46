"""The encoder's layers as one kernel (at most 32 tokens, bf16) against the modules in fp32 and the kernel-by-kernel loop."""
import copy

import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(hidden, layers, pos=("c2p", "p2c"), **kw):
    from transformers import DebertaV2Config
    from turbodeberta_b200.model import FlashDebertaV2Model
    cfg = DebertaV2Config(vocab_size=300, hidden_size=hidden, num_hidden_layers=layers, num_attention_heads=hidden // 64,
                          intermediate_size=4 * hidden, relative_attention=True, position_buckets=256, max_relative_positions=-1,
                          norm_rel_ebd="layer_norm", share_att_key=True, pos_att_type=list(pos), position_biased_input=False,
                          type_vocab_size=0, hidden_dropout_prob=0.0, attention_probs_dropout_prob=0.0, **kw)
    torch.manual_seed(31)
    model = FlashDebertaV2Model(cfg).eval().cuda()
    with torch.no_grad():
        for name, p in model.named_parameters():
            if name.endswith("bias"):
                p.normal_(0.0, 0.1)
            elif "LayerNorm" in name:
                p.normal_(1.0, 0.1)
    return model.to(torch.bfloat16)


def _inputs(lengths):
    L = max(lengths)
    ids = torch.randint(1, 300, (len(lengths), L), device="cuda")
    mask = (torch.arange(L, device="cuda")[None] < torch.tensor(lengths, device="cuda")[:, None]).long()
    return dict(input_ids=ids, attention_mask=mask)


def _recordings(model):
    from turbodeberta_b200 import model as M
    return M._PLANS[model.encoder].native.recordings


@pytest.mark.parametrize("hidden", [512, 768, 1024])
@pytest.mark.parametrize("lengths", [[1], [16], [17], [32], [20, 12], [9, 1, 16, 5], [1] * 32, [2] * 16], ids=str)
def test_one_kernel_is_as_exact_as_the_loop(hidden, lengths):
    """Both round the same tensors to bf16, so their distances to the fp32 modules are those of two draws of the same roundings:
    half as much again is far outside of what a 2-norm over at least 512 values varies by."""
    model = _model(hidden, 2)
    kw = _inputs(lengths)
    v = kw["attention_mask"].bool()
    with torch.no_grad():
        got = model(**kw).last_hidden_state
        assert torch.equal(got, model(**kw).last_hidden_state) and torch.equal(got, model(**kw).last_hidden_state)
        assert _recordings(model) == 0               # no other route repeats a shape without one
        loop = model(**kw, output_hidden_states=True).last_hidden_state
        want = copy.deepcopy(model).float()(**kw).last_hidden_state[v]
    assert torch.count_nonzero(got[~v]).item() == 0
    off = [(x[v].float() - want).norm().item() / want.norm().item() for x in (got, loop)]
    assert off[0] <= 1.5 * off[1] < 3e-2, off


@pytest.mark.parametrize("pos", [["c2p"], ["p2c"], []], ids=str)
def test_position_terms_of_the_one_kernel(pos):
    model = _model(512, 2, pos)
    kw = _inputs([19, 13])
    v = kw["attention_mask"].bool()
    with torch.no_grad():
        got = model(**kw).last_hidden_state
        want = copy.deepcopy(model).float()(**kw).last_hidden_state
    assert ((got.float() - want)[v].norm() / want[v].norm()).item() < 1.5e-2


def test_the_one_kernel_on_several_streams_and_in_a_graph():
    """Passes on two streams at once, and a captured one: it takes the counters it meets at from zero to zero each time."""
    from turbodeberta_b200.ops.flash_attention import check_pending_status
    model = _model(768, 3)
    kw = _inputs([32])
    kw["attention_mask"] = torch.ones_like(kw["input_ids"])
    streams = [torch.cuda.Stream() for _ in range(2)]
    with torch.no_grad():
        want = model(**kw).last_hidden_state
        torch.cuda.synchronize()
        outs = []
        for i in range(12):
            with torch.cuda.stream(streams[i % 2]):
                outs.append(model(**kw).last_hidden_state)
        torch.cuda.synchronize()
        assert all(torch.equal(o, want) for o in outs)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = model(**kw).last_hidden_state
        for _ in range(3):
            out.zero_()
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(out, want)
        check_pending_status()
        model.encoder.layer[1].output.dense.weight.mul_(1.5)
        assert not torch.equal(model(**kw).last_hidden_state, want)
