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


def _stack_of(tokens, hidden, layers, words, limit_ns):
    """The arguments of tdb_short_stack for one sequence without position terms, as the library lays them out, with random weights."""
    import ctypes as C

    class Layer(C.Structure):
        _fields_ = [("tensors", C.c_void_p * 14), ("eps1", C.c_float), ("eps2", C.c_float), ("sm_scale", C.c_float),
                    ("exp_delta_max", C.c_int), ("exp_rows", C.c_int)]

    class Stack(C.Structure):
        _fields_ = [("layer", Layer * 48), ("n_layers", C.c_int), ("tokens", C.c_int), ("n_seqs", C.c_int), ("length", C.c_int),
                    ("x", C.c_void_p), ("out", C.c_void_p), ("scratch", C.c_void_p * 5), ("cu_seqlens", C.c_void_p),
                    ("status", C.c_void_p), ("counter", C.c_void_p), ("gave_up", C.c_void_p), ("limit_ns", C.c_uint64)]

    def random(*shape):
        return torch.randn(shape, device="cuda", dtype=torch.bfloat16) * 0.05
    shapes = [(3 * hidden, hidden), (3 * hidden,), (hidden, hidden), (hidden,), (hidden,), (hidden,), (4 * hidden, hidden), (4 * hidden,),
              (hidden, 4 * hidden), (hidden,), (hidden,), (hidden,)]                  # q/k/v, output, norm, up, down, norm
    p, keep = Stack(), []
    torch.manual_seed(5)
    for i in range(layers):
        w = [random(*s) for s in shapes]
        keep += w
        p.layer[i] = Layer((C.c_void_p * 14)(*[t.data_ptr() for t in w]), 1e-7, 1e-7, 0.07, 0, 0)
    x, out = random(tokens, hidden), torch.zeros(tokens, hidden, device="cuda", dtype=torch.bfloat16)
    scratch = [torch.zeros(tokens, n * hidden, device="cuda", dtype=torch.bfloat16) for n in (3, 1, 1, 4, 1)]
    p.n_layers, p.tokens, p.n_seqs, p.length, p.limit_ns = layers, tokens, 1, tokens, limit_ns
    p.x, p.out, p.scratch = x.data_ptr(), out.data_ptr(), (C.c_void_p * 5)(*[t.data_ptr() for t in scratch])
    p.status, p.counter, p.gave_up = words.data_ptr(), words.data_ptr() + 16, words.data_ptr() + 20       # as a call's own words lie
    return p, out, keep + [x] + scratch


@pytest.mark.parametrize("tokens", [16, 32])
@pytest.mark.parametrize("hidden", [512, 768, 1024])
def test_a_meeting_that_nobody_completes_is_given_up(hidden, tokens):
    """The counter begins one short, so the first meeting's limit of 5 ms runs out: every block leaves, the code is reported, and with the
    words cleared the next pass on them is right."""
    import ctypes as C
    import time
    from turbodeberta_b200 import _cabi as cabi
    words = torch.zeros(8, dtype=torch.int32, device="cuda")
    p, out, keep = _stack_of(tokens, hidden, 2, words, 5_000_000)

    def run():
        cabi.check(cabi.lib.tdb_short_stack(C.byref(p), hidden, C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        torch.cuda.synchronize()
    run()
    want = out.clone()
    assert words.tolist() == [0] * 8 and torch.isfinite(want.float()).all() and torch.count_nonzero(want).item() > 0
    out.zero_()
    words[4] = -1
    torch.cuda.synchronize()
    t0 = time.time()
    run()
    assert time.time() - t0 < 0.5
    assert words[0].item() == 302 and words[5].item() == 1 and torch.count_nonzero(out).item() == 0
    words.zero_()
    run()
    assert words.tolist() == [0] * 8 and torch.equal(out, want)


def test_a_launch_that_fails_is_reported_once():
    """What a refused launch leaves behind is not the next kernel's error.  (The launch takes its grid from the feature count: 0 is refused on
    the host.)  A capture that has become invalid refuses the whole-stack kernel, which is not the answer of a device that is too small."""
    import ctypes as C
    from turbodeberta_b200 import _cabi as cabi
    rt = C.CDLL("libcudart.so.12")                    # the one that torch has loaded
    words = torch.zeros(8, dtype=torch.int32, device="cuda")
    p, out, keep = _stack_of(16, 512, 1, words, 5_000_000)
    idx = torch.full((513,), -1, device="cuda", dtype=torch.int16)
    torch.cuda.synchronize()
    current = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    where = C.c_void_p(out.data_ptr())
    assert cabi.lib.tdb_skinny(where, where, where, 16, 512, 0, 0, 0, where, current) == cabi.ERR_CUDA
    assert cabi.lib.tdb_bucket_table(0, 256, 256, cabi.ptr(idx), current) == 0
    stream, graph = C.c_void_p(), C.c_void_p()
    assert rt.cudaStreamCreateWithFlags(C.byref(stream), 1) == 0
    assert rt.cudaStreamBeginCapture(stream, 2) == 0              # relaxed
    assert rt.cudaStreamSynchronize(stream) != 0                  # not allowed in a capture, which ends it
    assert cabi.lib.tdb_short_stack(C.byref(p), 512, stream) == cabi.ERR_CUDA
    assert rt.cudaStreamEndCapture(stream, C.byref(graph)) != 0 and not graph.value
    rt.cudaGetLastError()
    assert rt.cudaStreamDestroy(stream) == 0
    torch.cuda.synchronize()
    assert (idx >= 0).all() and torch.count_nonzero(out).item() == 0
