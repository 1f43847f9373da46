"""The model's input in one kernel: gather, LayerNorm, padding mask."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape,hidden", [((1, 1), 8), ((3, 7), 264), ((2, 33), 768), ((40, 61), 1024)])
@pytest.mark.parametrize("ids_type,mask_type", [(torch.long, torch.long), (torch.int32, torch.bool), (torch.long, torch.uint8)])
def test_embeddings(shape, hidden, dtype, ids_type, mask_type):
    """Against the four operations that it stands for, in float64.  Errors are relative to the two terms that are added, which may
    cancel: bf16 rounds the sum once (2^-9 of it), fp32 carries some ten roundings (2^-24 each) of mean, variance and products."""
    from turbodeberta_b200._cabi import host
    torch.manual_seed(41)
    table = torch.randn(97, hidden, device="cuda").to(dtype)
    w, b = (torch.randn(hidden, device="cuda").to(dtype) for _ in range(2))
    ids = torch.randint(0, 97, shape, device="cuda")
    ids.view(-1)[:1] = 96
    mask = torch.rand(shape, device="cuda") < 0.7
    out, words = host.embed(ids.to(ids_type), table, w, b, 1e-7, mask.to(mask_type))
    product = torch.nn.functional.layer_norm(table.double()[ids], (hidden,), w.double(), None, 1e-7)
    want = (product + b.double()) * mask[..., None]
    bound = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-6
    assert ((out.double() - want).abs() <= bound * (product.abs() + b.double().abs()) + 1e-7).all()
    assert words is None and host.drain_pending() is None


def test_embeddings_leave_other_tensors_to_torch():
    from turbodeberta_b200._cabi import host
    table, v = torch.randn(9, 16, device="cuda"), torch.ones(16, device="cuda")
    ids, mask = torch.zeros(2, 4, dtype=torch.long, device="cuda"), torch.ones(2, 4, dtype=torch.long, device="cuda")
    assert host.embed(ids, table, v, v, 1e-7, mask) is not None
    wide = torch.randn(9, 32, device="cuda")
    for bad in ((ids.t(), table, v, v, mask.t()), (ids, wide[:, :16], v, v, mask), (ids, wide.view(-1)[1:145].view(9, 16), v, v, mask), (ids, table, v, v.bfloat16(), mask),
                (ids, table, v, v, mask.float()), (ids, table.half(), v.half(), v.half(), mask), (ids[:0], table, v, v, mask[:0])):
        assert host.embed(*bad[:4], 1e-7, bad[4]) is None
    host.drain_pending()


def test_ids_outside_the_vocabulary_are_reported():
    from tests.test_model_gpu import _cfg
    from turbodeberta_b200.model import FlashDebertaV2Model
    model = FlashDebertaV2Model(_cfg()).eval().to("cuda", torch.bfloat16)
    ids = torch.randint(0, 500, (2, 20), device="cuda")
    with torch.no_grad():
        want = model(input_ids=ids).last_hidden_state
        for bad in (500, -1, 1 << 40):
            wrong = ids.clone()
            wrong[1, 3] = bad
            with pytest.raises(IndexError):
                model(input_ids=wrong)
        assert torch.equal(model(input_ids=ids).last_hidden_state, want)


def test_the_report_of_a_bad_id_leaves_the_others_words_alone():
    from turbodeberta_b200 import _cabi as cabi
    from turbodeberta_b200.ops import flash_attention as fa
    table, v = torch.randn(9, 16, device="cuda"), torch.ones(16, device="cuda")
    ids, mask = torch.full((2, 4), 9, dtype=torch.long, device="cuda"), torch.ones(2, 4, dtype=torch.long, device="cuda")
    cabi.host.embed(ids, table, v, v, 1e-7, mask)
    assert cabi.host.drain_pending() == (0, 0, 0, 1)
    cabi.host.embed(ids, table, v, v, 1e-7, mask)
    timed_out = torch.zeros(4, dtype=torch.int32, device="cuda")
    cabi.check(cabi.lib.tdb_selftest_bounded_wait(cabi.ptr(timed_out), 77, 2000, cabi.stream_ptr(ids.device)))
    fa._PENDING_STATUS.append(timed_out)
    with pytest.raises(cabi.TdbError, match="77.*vocabulary"):
        fa.check_pending_status()
    fa.check_pending_status()


def _model():
    from tests.test_model_gpu import _cfg
    from turbodeberta_b200.model import FlashDebertaV2Model
    return FlashDebertaV2Model(_cfg()).eval().to("cuda", torch.bfloat16)


def test_a_bad_id_is_reported_to_its_own_caller():
    """Another thread's pass checks between this pass's embeddings and its own check: it gets its result, and this one the error."""
    import threading
    mine, others = _model(), _model()
    good = torch.randint(0, 500, (2, 20), device="cuda")
    bad = good.clone()
    bad[1, 3] = 500
    run = mine.encoder.forward
    seen = []

    def other_pass():
        try:
            with torch.no_grad():
                seen.append(others(input_ids=good).last_hidden_state)
        except Exception as e:                                   # noqa: BLE001
            seen.append(e)

    def forward(*a, **kw):
        t = threading.Thread(target=other_pass)
        t.start()
        t.join()
        return run(*a, **kw)

    with torch.no_grad():
        want = others(input_ids=good).last_hidden_state
        mine(input_ids=good)
        mine.encoder.forward = forward
        with pytest.raises(IndexError):
            mine(input_ids=bad)
        assert torch.equal(seen.pop(), want)
        mine(input_ids=good)
        assert torch.equal(seen.pop(), want)


def test_a_pass_that_ends_early_gives_its_report_back():
    """More passes than there are pooled words, each with a bad id and an encoder that fails: the words come back clean."""
    from turbodeberta_b200._cabi import host
    model = _model()
    bad = torch.full((2, 20), 1000, device="cuda")

    def fail(*a, **kw):
        raise RuntimeError("not today")

    run = model.encoder.forward
    model.encoder.forward = fail
    with torch.no_grad():
        for _ in range(300):
            with pytest.raises(RuntimeError, match="not today"):
                model(input_ids=bad)
        model.encoder.forward = run
        model(input_ids=bad.clamp(max=499))
        table, v = torch.randn(9, 16, device="cuda"), torch.ones(16, device="cuda")
        ids = torch.zeros(2, 4, dtype=torch.long, device="cuda")
        report = host.embed(ids, table, v, v, 1e-7, ids, True)[1]
        assert isinstance(report, host.Report) and host.drain_pending(report) is None and host.drain_pending(report) is None


def test_an_encoder_that_does_not_check_leaves_the_report_to_the_model():
    model = _model()
    bad = torch.full((2, 20), 1000, device="cuda")
    with torch.no_grad():
        model.encoder.forward = lambda x, *a, **kw: x
        with pytest.raises(IndexError):
            model(input_ids=bad)
        assert model(input_ids=bad.clamp(max=499)).shape[:2] == (2, 20)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("ids_of", [lambda x: x, lambda x: x.t().contiguous().t(), lambda x: torch.cat([x, x], 1)[:, :20], lambda x: x.repeat_interleave(2, 1)[:, ::2],
                                    lambda x: x.int().t().contiguous().t()], ids=["rows", "columns", "wider", "strided", "int32"])
@pytest.mark.parametrize("mask_of", [lambda m: m, lambda m: m.t().contiguous().t(), lambda m: m.int(), lambda m: m.float(), lambda m: m.bfloat16() * 0.5, lambda m: m.bool().t().contiguous().t()],
                         ids=["int64", "columns", "int32", "float", "halves", "bool columns"])
def test_ids_and_masks_of_any_layout_and_type(ids_of, mask_of, dtype, monkeypatch):
    """The same input as torch's operations form, and the same error for an id outside the vocabulary."""
    model = _model().to(dtype)
    ids = torch.randint(0, 500, (3, 20), device="cuda")
    mask = (torch.arange(20, device="cuda")[None] < torch.tensor([[20], [7], [1]], device="cuda")).long()
    seen = []
    model.encoder.forward = lambda x, *a, **kw: seen.append(x) or x
    with torch.no_grad():
        emb = model.embeddings
        want = emb.LayerNorm(emb.word_embeddings(ids)) * mask_of(mask).to(dtype)[..., None]

        def refuse(*a, **kw):                        # a bad id must not get there: its assertion would end the context
            raise AssertionError("torch's embedding")

        monkeypatch.setattr(torch.nn.functional, "embedding", refuse)
        model(input_ids=ids_of(ids), attention_mask=mask_of(mask))
        # bf16: both round the LayerNorm's result and the product once (half a unit each way: 2^-7); fp32: ten roundings of sums
        assert ((seen[0] - want).abs() <= (2.0 ** -7 if dtype == torch.bfloat16 else 1e-5) * want.abs() + 1e-6).all()
        ids[2, 0] = 500
        with pytest.raises(IndexError):
            model(input_ids=ids_of(ids), attention_mask=mask_of(mask))


class _Halves(torch.Tensor):
    """A tensor that holds half of its values: it has no memory of its own for a kernel to read."""
    @staticmethod
    def __new__(cls, inner):
        return torch.Tensor._make_wrapper_subclass(cls, inner.shape, dtype=inner.dtype, device=inner.device)

    def __init__(self, inner):
        self.inner = inner

    @classmethod
    def __torch_dispatch__(cls, func, types, args=(), kwargs=None):
        if func is torch.ops.aten.detach.default:
            return cls(args[0].inner)
        return func(*[a.inner * 2 if isinstance(a, cls) else a for a in args], **(kwargs or {}))


def test_a_table_of_another_tensor_class_is_left_to_torch(monkeypatch):
    from turbodeberta_b200 import model as M
    model = _model()
    ids = torch.randint(0, 500, (2, 20), device="cuda")
    with torch.no_grad():
        want = model(input_ids=ids).last_hidden_state.float()
        words = model.embeddings.word_embeddings
        words.weight = torch.nn.Parameter(_Halves(words.weight.detach() / 2), requires_grad=False)
        monkeypatch.setattr(M.host, "embed", lambda *a: pytest.fail("not a tensor that the kernel can read"))
        got = model(input_ids=ids).last_hidden_state.float()
    assert ((got - want).norm() / want.norm()).item() < 1e-2         # the two routes round the same tensors to bf16
