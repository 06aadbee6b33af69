"""Which kernel a call takes, at the limits of what each kernel may be given."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TOL = {torch.bfloat16: 2.9e-3, torch.float16: 3.7e-4}   # one rounding of the result: 2^-9 and 2^-12 at most


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm().clamp_min(1e-30))


@pytest.mark.parametrize("C,M,G", [(272 * 2, 64, 1), (64, 512, 1), (512, 512, 1), (288, 32, 2), (256, 256, 1)])
def test_one_triplet_per_row_with_contractions_of_several_parts(C, M, G):
    """Rows of more than 256 input channels are summed by several passes: they must not be stored by each of them."""
    from pointelligence_b200 import _cabi

    n, K, dtype = 300, 8, torch.bfloat16
    g = torch.Generator(device=DEV).manual_seed(1)
    k = torch.sort(torch.randint(0, K, (n,), device=DEV, generator=g)).values
    seg = torch.searchsorted(k, torch.arange(K + 1, device=DEV))
    once, any_row = torch.randperm(n, device=DEV, generator=g).int(), torch.randint(0, 70, (n,), device=DEV, generator=g).int()
    w = (torch.randn(K, G, C, M, device=DEV, generator=g) / C ** 0.5).to(dtype)
    for transpose in (False, True):
        x = torch.randn(70, G * (M if transpose else C), device=DEV, generator=g).to(dtype)
        out = _cabi.mvmr(w, x, any_row, once, seg, None, n, transpose, _cabi.ENGINE_FLAG_FAN_IN_ONE)
        wd = w.double().transpose(2, 3) if transpose else w.double()
        ref = torch.zeros(n, out.shape[1], dtype=torch.float64, device=DEV)
        ref[once.long()] = torch.einsum("tgc,tgcm->tgm", x.double().view(70, G, -1)[any_row.long()], wd[k]).reshape(n, -1)
        assert _rel(out, ref) < TOL[dtype], transpose


def test_geometry_built_triplets_with_merged_taps():
    """Rows ascend inside the 27 taps of the search, not inside nine merged ones: that plan has to sort."""
    from pointelligence_b200 import _cabi
    from pointelligence_b200.layers.triplets import build_triplets_segmented

    n = 3000
    g = torch.Generator(device=DEV).manual_seed(2)
    pts = torch.rand(n, 3, device=DEV, generator=g) * n ** (1 / 3)
    i, j, _, seg, _ = build_triplets_segmented(pts, torch.zeros(n, dtype=torch.int32, device=DEV),
                                               torch.tensor([n], device=DEV), 1.5, 3, radius_scaler=2.5)
    merged = seg[::3].contiguous()
    w = torch.randn(9, 1, 64, 64, device=DEV, generator=g).bfloat16() / 8
    x = torch.randn(n, 64, device=DEV, generator=g).bfloat16()
    out = _cabi.mvmr(w, x, j, i, merged, None, n, False, _cabi.ENGINE_PLANNED)
    ref = torch.zeros(n, 64, dtype=torch.float64, device=DEV)
    for tap in range(9):
        a, b = int(merged[tap]), int(merged[tap + 1])
        ref.index_add_(0, i[a:b].long(), x[j[a:b].long()].double() @ w[tap, 0].double())
    assert _rel(out, ref) < TOL[torch.bfloat16]


def test_a_chain_of_layers_on_one_sparse_rulebook_is_captured():
    """Six layers on one rulebook of a few triplets per row: twelve passes by the end of the capture, the same bits as
    the eager chain's engine gives."""
    from pointelligence_b200 import _cabi
    from pointelligence_b200.internals.two_phase import GeometryScheduler
    from pointelligence_b200.layers.conv import PointConv3d
    from pointelligence_b200.layers.metadata import MetaData
    from pointelligence_b200.layers.two_phase_conv import ConvOp

    g = torch.Generator(device=DEV).manual_seed(0)
    pts, batch = torch.rand(4096, 3, generator=g, device=DEV) * 5.0, torch.arange(4096, device=DEV) // 2048
    torch.manual_seed(1)
    ops = [ConvOp(PointConv3d(32, 32, kernel_size=3, device=DEV, dtype=torch.bfloat16), stride=1.0) for _ in range(6)]
    with torch.no_grad():
        metas = [MetaData(points=pts.clone(), sample_inds=batch.clone(), sample_sizes=torch.bincount(batch), grid_size=0.2)
                 for _ in range(2)]
        eager = GeometryScheduler().prepare(ops, metas[0])
        graphed = GeometryScheduler().prepare(ops, metas[1], compile_segments=True)
        for seed in range(2):
            x = torch.randn(4096, 32, device=DEV, generator=g.manual_seed(seed)).bfloat16()
            want, got = eager(x), graphed(x)
            assert torch.allclose(got.float(), want.float(), atol=2e-2, rtol=2e-2)
    assert _cabi.device_status() == 0


@pytest.mark.parametrize("C,M,G", [(20, 20, 1), (6, 32, 1), (32, 64, 2), (512, 512, 1), (272, 320, 1)])
def test_dense_rulebooks_of_padded_grouped_and_wide_layers_keep_exact_operands(C, M, G):
    """Buckets of several rows of 30 000 leave the range of fp16; the products of these rows do not."""
    from pointelligence_b200.sparse_engines.tig import TigIndex, tig_mvmr

    n, K, T = 500, 9, 10000
    g = torch.Generator(device=DEV).manual_seed(3)
    k = torch.sort(torch.randint(0, K, (T,), device=DEV, generator=g)).values
    i, j = (torch.randint(0, n, (T,), device=DEV, generator=g).int() for _ in range(2))
    seg = torch.searchsorted(k, torch.arange(K + 1, device=DEV))
    w = (torch.randn(K, G, C, M, device=DEV, generator=g) * 1e-4).half().requires_grad_()
    x = (30000 + 1000 * torch.randn(n, G * C, device=DEV, generator=g)).half().requires_grad_()
    y = tig_mvmr(w, x, TigIndex.from_flat(i, j, seg, n, n, K))
    rows = torch.einsum("tgc,tgcm->tgm", x.detach().double().view(n, G, C)[j.long()], w.detach().double()[k])
    ref = torch.zeros(n, G, M, dtype=torch.float64, device=DEV).index_add_(0, i.long(), rows).view(n, -1)
    assert torch.isfinite(y).all() and _rel(y.detach(), ref) < TOL[torch.float16]
    go = torch.full_like(y, 30000.0)
    gx, = torch.autograd.grad(y, x, go)
    back = torch.einsum("tgm,tgcm->tgc", go.double().view(n, G, M)[i.long()], w.detach().double()[k])
    ref = torch.zeros(n, G, C, dtype=torch.float64, device=DEV).index_add_(0, j.long(), back).view(n, -1)
    assert torch.isfinite(gx).all() and _rel(gx, ref) < TOL[torch.float16]


@pytest.mark.parametrize("density", [4.0, 40.0])
def test_layers_under_inference_mode(density):
    """Strided and stride-1 layers on sparse and dense clouds whose index tensors are inference tensors."""
    from pointelligence_b200.layers import MetaData, PointConv3d, conv_with_stride

    n = 3000
    g = torch.Generator(device=DEV).manual_seed(5)
    pts = torch.rand(n, 3, device=DEV, generator=g) * (n / density) ** (1 / 3)
    inds, x = torch.zeros(n, dtype=torch.int64, device=DEV), torch.randn(n, 64, device=DEV, generator=g).bfloat16()
    torch.manual_seed(6)
    convs = [PointConv3d(64, 64, 3, device=DEV, dtype=torch.bfloat16) for _ in range(3)]
    results = []
    for mode in (torch.no_grad, torch.inference_mode):
        with mode():
            m = MetaData(points=pts, sample_inds=inds, sample_sizes=torch.bincount(inds), grid_size=0.5)
            y, m = conv_with_stride(convs[0], x, m, 1.0)
            m.dirty_triplets()
            y, m = conv_with_stride(convs[1], y, m, 2.0)
            m.dirty_triplets()
            y, m = conv_with_stride(convs[2], y, m, 1.0)
        results.append((y, m.i, m.j))
    assert all(torch.equal(a, b) for a, b in zip(results[0][1:], results[1][1:]))
    assert _rel(results[1][0], results[0][0].double()) < 6 * TOL[torch.bfloat16]   # three layers, two engines


@pytest.mark.parametrize("M,dtype", [(32, torch.bfloat16), (20, torch.float16), (32, torch.float32)])
def test_strided_broadcast_and_misfitting_biases(M, dtype):
    from pointelligence_b200.sparse_engines.tig import TigIndex, tig_mvmr

    n, K, T = 200, 8, 900
    g = torch.Generator(device=DEV).manual_seed(7)
    k = torch.sort(torch.randint(0, K, (T,), device=DEV, generator=g)).values
    i, j = (torch.randint(0, n, (T,), device=DEV, generator=g).int() for _ in range(2))
    index = TigIndex.from_flat(i, j, torch.searchsorted(k, torch.arange(K + 1, device=DEV)), n, n, K)
    w = torch.randn(K, 1, 32, M, device=DEV, generator=g).to(dtype) / 6
    x = torch.randn(n, 32, device=DEV, generator=g).to(dtype)
    wide = torch.randn(2 * M, device=DEV, generator=g).to(dtype)
    plain = tig_mvmr(w, x, index)
    for bias in (wide[::2], wide[:1], wide[0], wide[:M].view(1, M)):
        bias = bias.detach().requires_grad_()
        y = tig_mvmr(w, x, index, bias=bias)
        # at most: the sum rounded, and rounded again with the bias
        assert _rel(y.detach(), plain.double() + bias.detach().double()) < 2 * TOL.get(dtype, 3e-6)
        grad, = torch.autograd.grad(y.sum(), bias)
        assert grad.shape == bias.shape and _rel(grad, torch.full_like(bias, y.numel() / bias.numel()).double()) < 1e-6
    for bias in (wide[:M - 1], wide):
        with pytest.raises(RuntimeError):
            tig_mvmr(w, x, index, bias=bias)


def test_vmap_and_tracing_of_a_convolution():
    from torch.fx.experimental.proxy_tensor import make_fx

    from pointelligence_b200.sparse_engines.tig import TigIndex, tig_mvmr

    n, K, T = 100, 8, 500
    g = torch.Generator(device=DEV).manual_seed(8)
    k = torch.sort(torch.randint(0, K, (T,), device=DEV, generator=g)).values
    i, j = (torch.randint(0, n, (T,), device=DEV, generator=g).int() for _ in range(2))
    index = TigIndex.from_flat(i, j, torch.searchsorted(k, torch.arange(K + 1, device=DEV)), n, n, K)
    w, b = torch.randn(K, 1, 32, 32, device=DEV, generator=g), torch.randn(32, device=DEV, generator=g)
    xs = torch.randn(3, n, 32, device=DEV, generator=g)
    want = torch.stack([tig_mvmr(w, x, index, bias=b) for x in xs])
    assert _rel(torch.func.vmap(lambda x: tig_mvmr(w, x, index, bias=b))(xs), want.double()) < 4e-6
    traced = make_fx(lambda x: tig_mvmr(w, x, index, bias=b))(xs[0])
    assert "pointelligence_b200.tig_mvmr" in traced.code
    assert _rel(traced(xs[1]), want[1].double()) < 4e-6    # and not the values it was traced with


@pytest.mark.parametrize("grad", [False, True])
def test_forward_mode_of_the_fused_layer_norm_is_refused(grad):
    import torch.autograd.forward_ad as fa

    from pointelligence_b200.layers.norm import fused_layer_norm

    x, lengths = torch.randn(5, 8, device=DEV), torch.tensor([5], device=DEV)
    with fa.dual_level(), torch.set_grad_enabled(grad), pytest.raises((RuntimeError, NotImplementedError), match="jvp"):
        fused_layer_norm(fa.make_dual(x, torch.ones_like(x)), lengths)


def test_operands_of_other_shapes_are_refused():
    from pointelligence_b200 import _cabi
    from pointelligence_b200.layers.norm import fused_layer_norm
    from pointelligence_b200.sparse_engines.tig import TigIndex, tig_mvmr

    i = j = torch.arange(10, device=DEV, dtype=torch.int32)
    seg, w, x = torch.tensor([0, 4, 10], device=DEV), torch.randn(2, 1, 8, 8, device=DEV), torch.randn(10, 8, device=DEV)
    index = TigIndex.from_flat(i, j, seg, 10, 10, 2)
    assert tig_mvmr(w, x, index).shape == tig_mvmr(w[:, 0], x, index).shape == (10, 8)
    for weight in (w[:, 0], w[..., None]):
        with pytest.raises(ValueError):
            _cabi.mvmr(weight, x, j, i, seg, None, 10, False)
    with pytest.raises(AssertionError):
        _cabi.mvmr(w, x.half(), j, i, seg, None, 10, False)
    with pytest.raises(AssertionError):
        _cabi.vvor(x[:, None], j, x[:, None].half(), i, seg, None, 2)
    for feat in (x[:, :7], x[:9], torch.randn(10, 9, device=DEV)):
        with pytest.raises(AssertionError):
            tig_mvmr(w, feat, index)
    with pytest.raises(ValueError):
        fused_layer_norm(torch.randn(10, 8, 2, device=DEV), torch.tensor([10], device=DEV))


@pytest.mark.parametrize("ids", [(0, 3), (7, 2 ** 31 - 2), (5, 2 ** 40 + 1), (-4, 9)])
def test_grid_sampling_of_points_with_any_sample_ids(ids):
    """Ids come back as they went in, and no array is made for every id up to the largest."""
    from pointelligence_b200.internals.grid_sample import grid_sample_filter

    g = torch.Generator(device=DEV).manual_seed(9)
    pts = torch.rand(2000, 3, device=DEV, generator=g)
    inds = torch.tensor(ids, device=DEV).repeat_interleave(1000)
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    _, sample, indices, _ = grid_sample_filter(pts, 0.2, inds)
    assert torch.cuda.max_memory_allocated() - before < 2 ** 20 * 8
    assert torch.equal(sample, inds[indices]) and sample.dtype == inds.dtype
    if max(ids) < 2 ** 31:
        sizes = getattr(sample, "pcx_sample_sizes", None)
        assert (sizes is not None) == (ids == (0, 3))
        assert sizes is None or torch.equal(sizes, torch.bincount(sample))


def test_clouds_of_alternating_extents_are_sorted_once():
    """Rooms whose cell keys need some bits more and less (here 20 and 28): from the third call on every call launches
    the same kernels, and all of them find the cells of a cloud sorted for its own bits."""
    from pointelligence_b200 import _cabi

    g = torch.Generator(device=DEV).manual_seed(10)
    clouds = [torch.rand(5000, 3, device=DEV, generator=g) * side for side in (4.1, 26.0)]
    cell = 0.0413       # of this test alone: what a size needed is remembered
    first = [_cabi.grid_sample_center_nearest(c, cell, None, True) for c in clouds]
    launches = []
    for n in range(8):
        _cabi.launch_count(reset=True)
        out = _cabi.grid_sample_center_nearest(clouds[n % 2], cell, None, True)
        launches.append(_cabi.launch_count())
        assert torch.equal(out[0], first[n % 2][0]) and torch.equal(out[3], first[n % 2][3])
    assert len(set(launches)) == 1, launches
    key = torch.div(clouds[1], cell, rounding_mode="floor").long()
    assert first[1][0].numel() == torch.unique(key, dim=0).shape[0]


def test_geometry_handed_to_two_streams_is_known_to_both(monkeypatch):
    """The allocator has to hear of every stream that a result of the geometry stream is used on."""
    from pointelligence_b200 import _cabi

    real, heard = _cabi.host(), []

    class Host:
        def __getattr__(self, name):
            return getattr(real, name)

        def record_streams(self, tensors):
            heard.extend((id(t), torch.cuda.current_stream().cuda_stream) for t in tensors)
            real.record_streams(tensors)

    monkeypatch.setattr(_cabi, "host", Host)
    result = torch.ones(8, device=DEV)
    build = _cabi.on_geometry_stream(lambda x: result)     # as a builder that finds its rulebook in the cache
    side = torch.cuda.Stream()
    with _cabi.geometry_overlap(torch.device(DEV)):
        for stream in (torch.cuda.current_stream(), torch.cuda.current_stream(), side):
            with torch.cuda.stream(stream):
                build(result)
    assert heard == [(id(result), s.cuda_stream) for s in (torch.cuda.current_stream(), side)]


@pytest.mark.parametrize("C", [64, 384])
def test_features_at_odd_addresses_on_a_dense_rulebook(C):
    from pointelligence_b200 import _cabi

    n, K, T = 300, 9, 6000
    g = torch.Generator(device=DEV).manual_seed(11)
    k = torch.sort(torch.randint(0, K, (T,), device=DEV, generator=g)).values
    i, j = (torch.randint(0, n, (T,), device=DEV, generator=g).int() for _ in range(2))
    seg = torch.searchsorted(k, torch.arange(K + 1, device=DEV))
    w = torch.randn(K, 1, C, 64, device=DEV, generator=g).bfloat16() / C ** 0.5
    x = torch.randn(n * C + 1, device=DEV, generator=g).bfloat16()[1:].view(n, C)
    out = _cabi.mvmr(w, x, j, i, seg, None, n, False)
    rows = torch.einsum("tc,tcm->tm", x.double()[j.long()], w[:, 0].double()[k])
    assert _rel(out, torch.zeros(n, 64, dtype=torch.float64, device=DEV).index_add_(0, i.long(), rows)) < TOL[torch.bfloat16]


@pytest.mark.parametrize("C,M", [(32, 32), (70, 96), (256, 64)])
def test_short_chunks_of_the_cuda_core_engine(C, M):
    """Taps of no, one and around 16, 32, 64 and 128 triplets: what is multiplied of a chunk goes by its rows.  fp32
    sums of at most 256 products of size one over 129 rows each, 2^-24 relative each: below 4e-6."""
    from pointelligence_b200 import _cabi

    sizes = [0, 1, 15, 16, 17, 31, 32, 33, 0, 63, 64, 65, 127, 128, 129, 200]
    seg = torch.tensor([0] + sizes, device=DEV).cumsum(0)
    T, n = int(seg[-1]), 301
    g = torch.Generator(device=DEV).manual_seed(12)
    k = torch.repeat_interleave(torch.arange(len(sizes), device=DEV), torch.tensor(sizes, device=DEV))
    i, j = (torch.randint(0, n, (T,), device=DEV, generator=g).int() for _ in range(2))
    w = torch.randn(len(sizes), 1, C, M, device=DEV, generator=g)
    x, go = torch.randn(n, C, device=DEV, generator=g), torch.randn(n, M, device=DEV, generator=g)
    y, gx = _cabi.mvmr(w, x, j, i, seg, None, n, False), _cabi.mvmr(w, go, i, j, seg, None, n, True)
    wd = w[:, 0].double()[k]
    y_ref = torch.zeros(n, M, dtype=torch.float64, device=DEV).index_add_(0, i.long(), torch.einsum("tc,tcm->tm", x.double()[j.long()], wd))
    gx_ref = torch.zeros(n, C, dtype=torch.float64, device=DEV).index_add_(0, j.long(), torch.einsum("tm,tcm->tc", go.double()[i.long()], wd))
    assert _rel(y, y_ref) < 4e-6 and _rel(gx, gx_ref) < 4e-6


def test_weight_gradient_of_one_tap_over_many_chunks():
    """One tap and more chunks than CTAs add to it, in fp32: sums of up to 30 011 products of size one, whose partial
    sums grow like the root of their number, stay below 4e-6 relative."""
    from pointelligence_b200 import _cabi

    n = 30011
    g = torch.Generator(device=DEV).manual_seed(13)
    ai, bi = (torch.randint(0, n, (n,), device=DEV, generator=g).int() for _ in range(2))
    a, b = torch.randn(n, 1, 32, device=DEV, generator=g), torch.randn(n, 1, 29, device=DEV, generator=g)
    out = _cabi.vvor(a, ai, b, bi, torch.tensor([0, n], device=DEV), None, 1)
    assert _rel(out[0, 0], a[ai.long(), 0].double().T @ b[bi.long(), 0].double()) < 4e-6


def test_time_of_the_layer_norm_is_recorded():
    """The event timer that the benchmark's split of a training step reads: one record per pass, all kernels inside."""
    from pointelligence_b200 import _cabi
    from pointelligence_b200.layers.norm import RaggedLayerNorm

    norm, x = RaggedLayerNorm(64).to(DEV), torch.randn(200000, 64, device=DEV, requires_grad=True)
    lengths = torch.tensor([120000, 80000], device=DEV)
    norm(x, lengths).sum().backward()
    _cabi.profile_enable(True)
    norm(x, lengths).sum().backward()
    records = _cabi.profile_records()
    _cabi.profile_enable(False)
    # 51 MB in, 51 MB out at 8 TB/s: more than 5 us each way even from the caches
    assert [name for name, ms in records if ms > 5e-3] == ["layer_norm(fwd)", "layer_norm(bwd)"]


@pytest.mark.parametrize("C", [112, 176, 208, 224, 240])
def test_bucket_sums_of_widths_between_the_powers_of_two(C):
    """Rows of 14, 22, 26, 28 and 30 pieces of 16 bytes: the last lanes of a row have nothing to do."""
    from pointelligence_b200 import _cabi

    n, K, T = 300, 9, 6000
    g = torch.Generator(device=DEV).manual_seed(14)
    k = torch.sort(torch.randint(0, K, (T,), device=DEV, generator=g)).values
    i, j = (torch.randint(0, n, (T,), device=DEV, generator=g).int() for _ in range(2))
    seg = torch.searchsorted(k, torch.arange(K + 1, device=DEV))
    w = torch.randn(K, 1, C, 64, device=DEV, generator=g).bfloat16() / C ** 0.5
    x = torch.randn(n, C, device=DEV, generator=g).bfloat16()
    out = _cabi.mvmr(w, x, j, i, seg, None, n, False, _cabi.ENGINE_PLANNED)
    rows = torch.einsum("tc,tcm->tm", x.double()[j.long()], w[:, 0].double()[k])
    assert _rel(out, torch.zeros(n, 64, dtype=torch.float64, device=DEV).index_add_(0, i.long(), rows)) < TOL[torch.bfloat16]
