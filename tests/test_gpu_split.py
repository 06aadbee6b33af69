"""GPU tests of what wide and grouped bf16 layers get by way of a plan: bucket sums in two parts and, where an operand is not
finite, the scatter kernels over the same output (``pcx_mvmr_split``)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _rulebook(seed, n_in, n_out, K, T, distinct=False):
    """Tap-sorted triplets; ``distinct``: no (row, tap) pair twice, so that no sums are taken."""
    rng = np.random.default_rng(seed)
    if distinct:
        pair = rng.permutation(n_out * K)[:T]
        i, k = pair // K, pair % K
    else:
        i, k = rng.integers(0, n_out, T), rng.integers(0, K, T)
        k[rng.random(T) < 0.5] = K // 2
    j = rng.integers(0, n_in, T)
    order = np.lexsort((i, k))
    i, j, k = i[order].astype(np.int32), j[order].astype(np.int32), k[order]
    seg = np.searchsorted(k, np.arange(K + 1)).astype(np.int64)
    return tuple(torch.from_numpy(a).to(DEV) for a in (i, j, seg))


@pytest.fixture
def always(monkeypatch):
    """Every wide or grouped bf16 layer takes the plan, whatever its size."""
    from pointelligence_b200 import _cabi

    monkeypatch.setattr(_cabi, "_planned_pays", lambda *a: True)
    monkeypatch.setattr(_cabi, "_split_pays", lambda *a: True)
    return _cabi


def _kernels(cabi, fn):
    cabi.profile_enable(True)
    try:
        out = fn()
        torch.cuda.synchronize()
        return out, [name for name, _ in cabi.profile_records()]
    finally:
        cabi.profile_enable(False)


@pytest.mark.parametrize("K,G,C,M,transpose", [(27, 1, 64, 288, False), (27, 1, 288, 64, True), (27, 2, 32, 48, False), (8, 4, 16, 16, True)])
@pytest.mark.parametrize("what", ["feature inf", "feature -inf and inf", "feature nan", "weight inf", "weight nan", "sum beyond bf16",
                                  "weight inf, no sums"])
def test_operands_that_are_not_finite(always, what, K, G, C, M, transpose):
    """Infinities and NaN are exactly where the scatter kernels put them; all else is as close as ever."""
    n_in, n_out = 300, 700
    distinct = what.endswith("no sums")
    i, j, seg = _rulebook(C + M, n_in, n_out, K, 4000 if distinct else 14000, distinct)
    inw = M if transpose else C
    g = torch.Generator(device=DEV).manual_seed(1)
    w = torch.rand(K, G, C, M, device=DEV, generator=g).bfloat16() / 8    # of one sign: an infinity stays one
    x = torch.rand(n_in, G * inw, device=DEV, generator=g).bfloat16()
    if what == "feature inf":
        x[17, 3] = float("inf")
    elif what == "feature -inf and inf":
        x[17, 3], x[18, 3], x[19, 5] = float("inf"), -float("inf"), -float("inf")
    elif what == "feature nan":
        x[17, 3] = float("nan")
    elif what == "sum beyond bf16":
        x.fill_(3e38)
        w *= 1e-4
    else:
        w[1, 0, 3, 7] = float("nan") if what == "weight nan" else float("inf")
    out, names = _kernels(always, lambda: always.mvmr(w, x, j, i, seg, None, n_out, transpose))
    assert [n for n in names if n != "bucket_sum_kernel"] == [f"mvmr_os_kernel({'dgrad' if transpose else 'fwd'})"]
    want = always.mvmr(w, x, j, i, seg, None, n_out, transpose, always.ENGINE_TENSOR)
    finite = torch.isfinite(want)
    assert torch.equal(torch.isnan(out), torch.isnan(want))
    assert torch.equal(out[torch.isinf(want)], want[torch.isinf(want)]) and torch.equal(finite, torch.isfinite(out))
    if what == "sum beyond bf16":
        assert bool(finite.all())
    else:
        assert not bool(finite.all()) and bool(finite.all(1).any())    # rows that do not meet it stay whole
    # as the scatter kernels' sums, in another order: the one rounding may fall to the other side (2^-7 of a value of one sign)
    assert bool(((out - want).abs() <= 2.0 ** -7 * want.abs())[finite].all())
    assert always.device_status() == 0


def test_finite_operands_are_not_done_again(always):
    """What follows the output-stationary kernel leaves its rows alone: they are those of the kernel by itself."""
    i, j, seg = _rulebook(3, 500, 900, 27, 20000)
    w = (torch.randn(27, 2, 48, 64, device=DEV) / 7).bfloat16()
    x = torch.randn(500, 96, device=DEV).bfloat16()
    plan = always.mvmr_plan(i, j, seg, 27, 900, always.plan_group_blocks(128))
    assert torch.equal(always.mvmr(w, x, j, i, seg, None, 900, False), always.mvmr_planned(w, x, plan, False, True))


@pytest.mark.parametrize("room,T", [(64, 8000000), (150, 400000)])   # MB: the plan does not fit; the plan does, the sums do not
def test_a_device_without_room_for_plan_or_sums(always, room, T):
    """The scatter kernels take the call, as they did before there was a choice."""
    n = 20000
    i, j, seg = _rulebook(4, n, n, 27, T)
    w = (torch.randn(27, 1, 1024, 288, device=DEV) / 32).bfloat16()
    x = torch.randn(n, 1024, device=DEV).bfloat16()
    plan = lambda: always._remembered_plan(always._plan_key(i, j, seg, 27, n, always.plan_group_blocks(288)), i, j, seg)
    want = always.mvmr(w, x, j, i, seg, None, n, False, always.ENGINE_TENSOR)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (room << 20)) / total)
    try:
        out, names = _kernels(always, lambda: always.mvmr(w, x, j, i, seg, None, n, False))
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert names == ["mvmr_tc_kernel(fwd)"] and (plan() is not None) is (room == 150)
    assert float((out.float() - want.float()).norm() / want.float().norm()) < 1e-3     # ties of the one rounding


@pytest.mark.parametrize("G,C,M", [(2, 32, 48), (1, 64, 288), (1, 288, 64)])
def test_layer_on_a_self_search_rulebook(always, G, C, M):
    """A bias, and the input gradient over the forward plan with the taps of the weight reversed.  Bounds as for two-part sums
    in general: 2^-8 of an element for its one rounding, 2^-16 + 2^-19 of the magnitudes that made it up."""
    from pointelligence_b200.layers import PointConv3d

    g = torch.Generator(device=DEV).manual_seed(C)
    pts = torch.rand(900, 3, device=DEV, generator=g)
    i, j, k, seg, _ = always.radius_search(pts, pts, 0.25, None, None, 0, 3, 0.1, want_k=True)
    always.mark_built(i, j, seg, 27, True)
    conv = PointConv3d(G * C, G * M, 3, groups=G, bias=True, device=DEV, dtype=torch.bfloat16)
    with torch.no_grad():
        conv.bias.normal_()
    x = torch.randn(900, G * C, device=DEV, generator=g).bfloat16().requires_grad_()
    go = torch.randn(900, G * M, device=DEV, generator=g).bfloat16()

    def step():
        y = conv(x, i, j, k, 900, seg_offs=seg)
        return y.detach(), torch.autograd.grad(y, x, go)[0]

    (y, gx), names = _kernels(always, step)
    assert [n for n in names if "mvmr" in n] == ["mvmr_os_kernel(fwd)", "mvmr_os_kernel(dgrad)"]
    w = conv.weight.detach().double().view(27, G, C, M)
    bias = conv.bias.detach().double()

    def sums(x, w, scatter, gather, width):
        out = torch.zeros(900, G, width, dtype=torch.float64, device=DEV)
        for t in range(27):
            s = slice(int(seg[t]), int(seg[t + 1]))
            out.index_add_(0, scatter[s].long(), torch.einsum("tgc,gcm->tgm", x.view(900, G, -1)[gather[s].long()], w[t]))
        return out.flatten(1)

    xd, god = x.detach().double(), go.double()
    for got, want, size, part in ((y, sums(xd, w, i, j, M) + bias, sums(xd.abs(), w.abs(), i, j, M) + bias.abs(), M),
                                  (gx, sums(god, w.transpose(2, 3), j, i, C), sums(god.abs(), w.abs().transpose(2, 3), j, i, C), C)):
        if G == 1 and part <= 256:
            continue    # sums rounded to 16 bits, as the layers of that width have them
        lost = size * (2.0 ** -16 + 2.0 ** -19)
        assert bool(((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + lost * (1 + 2.0 ** -8)).all())
    assert always.device_status() == 0


def _captured(fn):
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        fn()                                  # the usual warm-up: a plan is built and remembered
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = fn()
    return graph, out


@pytest.mark.parametrize("G,C,M", [(1, 64, 288), (2, 32, 48)])
def test_a_replay_of_a_wide_or_grouped_layer_follows_its_index_tensors(always, G, C, M):
    i, j, seg = _rulebook(8, 500, 900, 27, 20000)
    w, x = (torch.randn(27, G, C, M, device=DEV) / 8).bfloat16(), torch.randn(500, G * C, device=DEV).bfloat16()
    graph, out = _captured(lambda: always.mvmr(w, x, j, i, seg, None, 900, False))
    for t, other in zip((i, j, seg), _rulebook(9, 500, 900, 27, 20000)):
        t.copy_(other)
    graph.replay()
    want = always.mvmr(w, x, j, i, seg, None, 900, False, always.ENGINE_TENSOR)
    assert float((out.float() - want.float()).norm() / want.float().norm()) < 1e-3


def test_a_replay_reads_a_plan_that_the_cache_has_dropped(always):
    i, j, seg = _rulebook(10, 500, 900, 27, 20000)
    w, x = (torch.randn(27, 1, 64, 64, device=DEV) / 8).bfloat16(), torch.randn(500, 64, device=DEV).bfloat16()
    graph, out = _captured(lambda: always.mvmr(w, x, j, i, seg, None, 900, False))
    want = always.mvmr(w, x, j, i, seg, None, 900, False)
    plan = always._remembered_plan(always._plan_key(i, j, seg, 27, 900, always.plan_group_blocks(64)), i, j, seg)
    size, address = plan.buffer.numel(), plan.buffer.data_ptr()
    del plan
    always._PLAN_CACHE.clear()
    taken = [torch.empty(size, dtype=torch.uint8, device=DEV) for _ in range(8)]    # what a freed buffer's place would go to
    assert address not in [t.data_ptr() for t in taken]
    graph.replay()
    assert torch.equal(out, want)
