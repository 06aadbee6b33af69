"""Host-side rules that pick a kernel, and what they remember about a rulebook.  No GPU: the kernels are not run."""
import pytest
import torch

from pointelligence_b200 import _cabi


@pytest.fixture
def rulebook():
    """27 taps of 40 triplets, rows ascending inside each tap."""
    g = torch.Generator().manual_seed(0)
    i = torch.sort(torch.randint(0, 200, (27, 40), generator=g), dim=1).values.int().flatten()
    j = torch.randint(0, 200, (1080,), generator=g).int()
    return i, j, torch.arange(28) * 40


def test_row_order_is_remembered_with_the_cut_into_taps(rulebook):
    i, j, seg = rulebook
    _cabi.mark_built(i, j, seg, 27, symmetric=True)
    assert _cabi._rows_ascend(i, j, seg, 27) and _cabi.is_symmetric(i, j) and _cabi.is_symmetric(i, j, 27)
    merged = seg[::3].contiguous()      # nine taps of the same triplets: rows fall at the seams
    assert not _cabi._rows_ascend(i, j, merged, 9) and not _cabi.is_symmetric(i, j, 9)
    assert not _cabi._rows_ascend(i, j, seg.clone(), 27)
    seg += 0                            # written to since
    assert not _cabi._rows_ascend(i, j, seg, 27) and _cabi.is_symmetric(i, j, 27)
    i += 0
    assert not _cabi.is_symmetric(i, j, 27)


@pytest.mark.parametrize("words,want", [((-1, -1), -1), ((5, -1), -1), ((-1, 0), -1), ((5, 0), 5), ((0, 0), 0), ((5, 1), -2)])
def test_words_of_a_plan_that_is_not_waited_for(words, want):
    assert _cabi.host().peek(torch.tensor(words, dtype=torch.int32)) == want


def test_a_rulebook_takes_the_same_engine_however_often_it_is_used(rulebook, monkeypatch):
    """5.4 triplets per row and a small accumulator: the scatter engine, whose operands stay exact, at every pass; no
    plan is built under way, where the stream may be capturing."""
    i, j, seg = rulebook

    def no_plan(*args):
        raise AssertionError("a plan was built by a feature pass")

    monkeypatch.setattr(_cabi, "cached_mvmr_plan", no_plan)
    assert all(_cabi._plan_hook(i, j, seg, 27, 200, 64, 64, False) is None for _ in range(40))


@pytest.mark.parametrize("C,M,G,transpose,takes", [
    (64, 64, 1, False, True), (1024, 256, 1, False, True), (256, 256, 1, True, True), (16, 512, 1, True, True),
    (64, 272, 1, False, False), (512, 64, 1, True, False), (64, 64, 2, False, False), (6, 32, 1, False, False),
    (32, 20, 1, False, False), (1040, 64, 1, False, False)])
def test_layers_that_may_sum_in_16_bits(rulebook, C, M, G, transpose, takes):
    i, j, seg = rulebook
    w, x = torch.empty(27, G, C, M, dtype=torch.bfloat16), torch.empty(1, 1, dtype=torch.bfloat16)
    assert _cabi.planned_supported(w, x, j, i, seg, 200, transpose) is takes


class _Words:
    """Stands in for the host module: what the words of a plan say, call by call (the last value from then on)."""

    def __init__(self, *values, then=lambda: None):
        self.values, self.then, self.seen = list(values), then, []

    def peek(self, word):
        self.seen.append(word)
        value = self.values.pop(0) if len(self.values) > 1 else self.values[0]
        self.then()
        return value


def _plan(word="word", stream="built here"):
    return _cabi.MvmrPlan(torch.empty(0), 10, 3, 4, 2, 5, word, stream)


def test_another_thread_may_drop_the_word_of_a_plan(monkeypatch):
    plan = _plan()

    def other_thread():
        plan._multi, plan._word = 2, None

    words = _Words(-1, 2, then=other_thread)
    monkeypatch.setattr(_cabi, "host", lambda: words)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: "elsewhere")
    assert plan.multi_buckets == 2 and None not in words.seen


def test_a_plan_is_waited_for_without_calls_that_a_capture_refuses(monkeypatch):
    def refused(device=None):
        raise RuntimeError("operation not permitted when stream is capturing")

    words = _Words(-1, -1, -1, 3)
    monkeypatch.setattr(_cabi, "host", lambda: words)
    monkeypatch.setattr(torch.cuda, "synchronize", refused)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: "elsewhere")
    assert _plan().multi_buckets == 3
    words.values = [-1]
    assert _plan(stream="elsewhere").multi_buckets == 5      # the build's own stream: the bound, no wait
    monkeypatch.setattr(_cabi, "_PLAN_WAIT_SECONDS", 0.01)
    with pytest.raises(RuntimeError, match="not ready"):
        _plan().multi_buckets
    words.values = [-2]
    with pytest.raises(RuntimeError, match="ascend"):
        _plan().multi_buckets


def test_rulebooks_of_inference_mode(monkeypatch):
    """Inference tensors have no version: a rulebook of them is used, and nothing is remembered about it."""
    with torch.inference_mode():
        i, j, seg = (torch.arange(n, dtype=t) for n, t in ((3000, torch.int32), (3000, torch.int32), (28, torch.int64)))
    _cabi.mark_built(i, j, seg, 27, symmetric=True)
    assert not _cabi._rows_ascend(i, j, seg, 27) and not _cabi.is_symmetric(i, j, 27)
    built = []
    monkeypatch.setattr(_cabi, "mvmr_plan", lambda *args: built.append(args) or _plan(word=None))
    assert _cabi._planned_pays(3000, 100, 64, 27)
    assert _cabi._plan_hook(i, j, seg, 27, 100, 64, 64, False) is None and not built
    for _ in range(2):                       # asked for by name: a plan for every pass
        assert _cabi._plan_hook(i, j, seg, 27, 100, 64, 64, True)[1:] == (2, 5)
    assert len(built) == 2 and not any(refs[0]() is i for refs, _, _ in _cabi._PLAN_CACHE.values())


def test_biases_the_kernels_add():
    from pointelligence_b200.sparse_engines.tig import _fuses

    w, x = torch.empty(27, 2, 8, 16), torch.empty(10, 16)
    assert _fuses(torch.empty(32), w, x) and _fuses(torch.empty(64)[::2], w, x) and _fuses(torch.empty(16), w[:, 0], x)
    for bias in (torch.empty(31), torch.empty(1), torch.empty(()), torch.empty(1, 32), torch.empty(32).half()):
        assert not _fuses(bias, w, x)


def test_what_watches_operators_sees_the_operator(monkeypatch):
    """The compiled path is for plain eager calls; tracers, modes and transforms get the registered operator."""
    from torch.fx.experimental.proxy_tensor import make_fx
    from torch.utils._python_dispatch import TorchDispatchMode

    from pointelligence_b200.sparse_engines import tig

    class Watch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    seen = []

    def call(x):
        seen.append(tig._takes_host_path())      # (what the tensors are is looked at after these)
        return x * 2

    x = torch.ones(3)
    call(x)
    with Watch():
        call(x)
    make_fx(call)(x)
    torch.jit.trace(call, (x,), check_trace=False)
    torch.func.vmap(call)(x)
    torch.func.grad(lambda v: call(v).sum())(x)
    torch.func.jvp(call, (x,), (x,))
    with torch.autograd.forward_ad.dual_level():
        call(x)
    call(x)
    assert seen == [True] + [False] * 7 + [True]


def test_transforms_of_the_fused_layer_norm_are_refused():
    """The node has one derivative rule, backward; a transform must not get past it to the kernels."""
    from pointelligence_b200.layers.norm import fused_layer_norm

    x, lengths = torch.randn(4, 8), torch.tensor([4])
    with pytest.raises(RuntimeError, match="functorch"):
        torch.func.vmap(lambda v: fused_layer_norm(v, lengths))(x[None])
    with torch.no_grad(), pytest.raises(RuntimeError, match="functorch"):
        torch.func.jvp(lambda v: fused_layer_norm(v, lengths), (x,), (x,))


def test_layer_norm_takes_rows_only():
    from pointelligence_b200.layers.norm import fused_layer_norm

    for shape in ((4, 8, 3), (8,)):
        with pytest.raises(ValueError):
            fused_layer_norm(torch.randn(shape), torch.tensor([4]))


def _dense(monkeypatch):
    monkeypatch.setattr(_cabi, "mvmr_plan", lambda *args: _plan(word=None))
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: "here")
    return lambda: tuple(torch.arange(n, dtype=t) for n, t in ((3000, torch.int32), (3000, torch.int32), (28, torch.int64)))


@pytest.mark.parametrize("forced", [False, True])
def test_a_plan_that_a_capture_reads_lives_as_long_as_its_rulebook(monkeypatch, forced):
    """Sixty-four other plans, or a write to the index tensors, push it out of the cache; a graph goes on reading it."""
    import gc
    import weakref

    dense = _dense(monkeypatch)
    i, j, seg = dense()
    call = lambda capturing: _cabi._plan_hook(i, j, seg, 27, 100, 64, 64, forced, False, capturing)
    remembered = lambda: _cabi._remembered_plan(_cabi._plan_key(i, j, seg, 27, 100, _cabi.plan_group_blocks(64)), i, j, seg)
    assert call(False) is not None
    plan = weakref.ref(remembered())
    assert call(True)[0] is plan().buffer and call(True)[0] is plan().buffer
    others = [dense() for _ in range(_cabi._PLAN_CACHE_MAX + 1)]
    for other in others:
        _cabi._plan_hook(*other, 27, 100, 64, 64, forced)
    i += 1
    assert call(False) is not None
    gc.collect()
    assert plan() is not None and remembered() is not plan()
    del i, call, remembered
    gc.collect()
    assert plan() is None


def test_wide_and_grouped_layers_are_captured_on_the_scatter_kernels(monkeypatch):
    """... with a remembered plan too: what a graph reads are the caller's tensors."""
    i, j, seg = _dense(monkeypatch)()
    monkeypatch.setattr(_cabi, "_split_pays", lambda *args: True)
    assert _cabi._plan_hook(i, j, seg, 27, 100, 512, 64, False, True, False) is not None
    assert _cabi._plan_hook(i, j, seg, 27, 100, 512, 64, False, True, True) is None


@pytest.mark.parametrize("T,n,outw,inw,pays", [
    (605_000, 120_000, 288, 1024, False), (1_300_000, 260_000, 288, 1024, False),    # thin, and a long contraction
    (294_000, 60_000, 512, 512, False), (605_000, 120_000, 512, 1024, True),         # thin: from a gigabyte
    (409_000, 60_000, 512, 512, True), (450_000, 60_000, 288, 1024, False), (847_000, 120_000, 288, 1024, True),
    (18_900_000, 141_000, 384, 128, True), (18_900_000, 141_000, 384, 1024, False)])  # 15 GB of sums
def test_rulebooks_on_which_two_part_sums_pay(T, n, outw, inw, pays):
    assert _cabi._planned_pays(T, n, outw, 27) and _cabi._split_pays(T, n, outw, inw, 27) is pays


def test_joined_casts_are_those_of_the_weights_as_they_are(monkeypatch):
    """(The library's kernels do not run: the check for CUDA tensors is taken out.)"""
    from torch.nn.utils import prune

    from pointelligence_b200 import backbone

    monkeypatch.setattr(backbone, "_takes_host_path", lambda *tensors: True)
    make = lambda: torch.nn.Sequential(*(backbone.Bf16PointConv3d(16, width, 3) for width in (16, 24, 8)))
    changes = [lambda c: c.weight.add_(1), lambda c: setattr(c.weight, "data", torch.zeros_like(c.weight)),
               lambda c: setattr(c, "weight", torch.nn.Parameter(c.weight.clone()))]
    for change in changes:
        net = make()
        with torch.no_grad(), backbone.weights_cast_together(net):
            assert all(torch.equal(backbone._joint_cast(c), c.weight.bfloat16()) for c in net)
            with torch.enable_grad():
                assert backbone._joint_cast(net[0]) is None
            change(net[1])
            assert backbone._joint_cast(net[1]) is None and backbone._joint_cast(net[0]) is not None
    nets = [make() for _ in range(3)]
    prune.random_unstructured(nets[0][2], "weight", 0.3)
    nets[1].register_forward_pre_hook(lambda *_: None)
    nets[2][1].register_forward_hook(lambda *_: None)
    for net in nets:
        with torch.no_grad(), backbone.weights_cast_together(net):
            assert all(backbone._joint_cast(c) is None for c in net)
