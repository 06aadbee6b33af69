"""Layers of few input channels (``pcx_mvmr_thin``) against fp64, over the sizes where its tiles end."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# one rounding of the result: at most the type's unit roundoff in every element, and so in the norm; sums in fp32 are below
BOUND = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}


def _rulebook(n_out, n_in, K, ratio, seed, empty=()):
    """Tap-sorted, rows ascending inside a tap, with (row, tap) buckets of several triplets."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    T = max(int(n_out * ratio), 1)
    i = torch.randint(0, n_out, (T,), device="cuda", generator=g)
    j = torch.randint(0, n_in, (T,), device="cuda", generator=g)
    k = torch.randint(0, K, (T,), device="cuda", generator=g)
    for e in empty:
        k = torch.where(k == e, (e + 1) % K, k)
    order = torch.argsort(k * n_out + i, stable=True)
    i, j, k = i[order], j[order], k[order]
    seg = torch.searchsorted(k.contiguous(), torch.arange(K + 1, device="cuda"))
    return i.int().contiguous(), j.int().contiguous(), k, seg


def _exact(w, x, i, j, k, n_out):
    out = torch.zeros(n_out, w.shape[-1], dtype=torch.float64, device="cuda")
    for tap in range(w.shape[0]):
        t = k == tap
        if bool(t.any()):
            out.index_add_(0, i[t].long(), x[j[t].long()].double() @ w[tap].double())
    return out


def _thin(weight, feat, i, j, seg, bias, n_out, flags=0, keep=False):
    from pointelligence_b200 import _cabi

    K, C, M = weight.shape
    width = C if flags & 1 else M
    out = torch.full((n_out, width), float("nan"), device="cuda", dtype=feat.dtype)
    L, ptr = _cabi.lib(), _cabi.ptr
    ws = _cabi.workspace(L.pcx_mvmr_thin_workspace_bytes(feat.shape[0], n_out, K, C, M, flags & 1), feat.device)
    _cabi.check(L.pcx_mvmr_thin(ptr(weight), ptr(feat), ptr(j), ptr(i), ptr(seg), ptr(bias), ptr(out), i.numel(), feat.shape[0],
                                n_out, K, C, M, flags, _cabi.dtype_code(feat.dtype), ptr(ws), ws.numel(), _cabi.stream_ptr()))
    return (out, ws) if keep else out


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm().clamp_min(1e-300))


@pytest.mark.parametrize("n_out,K,C,M,ratio,empty", [
    (1, 2, 1, 16, 1.0, ()), (127, 8, 8, 16, 3.0, ()), (128, 9, 3, 32, 4.0, (0,)), (129, 27, 3, 20, 6.0, (0, 13, 26)),
    (1000, 27, 6, 64, 40.0, ()), (5000, 125, 6, 32, 25.0, (7, 8, 9)), (5000, 125, 8, 48, 25.0, ()), (20000, 27, 7, 96, 6.0, ()),
    (30000, 27, 2, 256, 5.0, ()), (3000, 27, 4, 3, 200.0, ()), (40001, 125, 5, 72, 3.0, ()), (300, 343, 6, 1000, 30.0, (342,)),
    (150, 27, 8, 24, 900.0, ())])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_against_fp64(n_out, K, C, M, ratio, empty, dtype):
    g = torch.Generator(device="cuda").manual_seed(n_out)
    n_in = n_out + 37
    i, j, k, seg = _rulebook(n_out, n_in, K, ratio, n_out + K, empty)
    w = (torch.randn(K, C, M, device="cuda", generator=g) / C ** 0.5).to(dtype)
    x = torch.randn(n_in, C, device="cuda", generator=g).to(dtype)
    b = torch.randn(M, device="cuda", generator=g).to(dtype)
    assert _rel(_thin(w, x, i, j, seg, None, n_out), _exact(w, x, i, j, k, n_out)) <= BOUND[dtype]
    assert _rel(_thin(w, x, i, j, seg, b, n_out), _exact(w, x, i, j, k, n_out) + b.double()) <= BOUND[dtype]
    wt, flipped = w.transpose(1, 2).contiguous(), w.flip(0).contiguous()
    assert _rel(_thin(wt, x, i, j, seg, None, n_out, 1), _exact(w, x, i, j, k, n_out)) <= BOUND[dtype]
    assert _rel(_thin(flipped, x, i, j, seg, None, n_out, 2), _exact(w, x, i, j, k, n_out)) <= BOUND[dtype]


@pytest.mark.parametrize("K,C,M", [(27, 6, 32), (125, 8, 80)])
def test_odd_addresses_and_operands_that_are_not_finite(K, C, M):
    from pointelligence_b200 import _cabi

    g = torch.Generator(device="cuda").manual_seed(K)
    n = 3001
    i, j, k, seg = _rulebook(n, n, K, 8.0, K)
    w = (torch.randn(K, C, M, device="cuda", generator=g) / C ** 0.5).bfloat16()
    x = torch.randn(n, C, device="cuda", generator=g).bfloat16()
    exact = _exact(w, x, i, j, k, n)
    # operands that begin at an odd element
    odd = lambda t: torch.cat([t.new_zeros(1), t.flatten()])[1:].view(t.shape)
    assert _rel(_thin(odd(w), odd(x), i, j, seg, None, n), exact) <= BOUND[torch.bfloat16]
    # infinities and NaN reach the rows whose triplets meet them, and no others
    for spoil_w, spoil_x in ((True, False), (False, True), (True, True)):
        w2, x2 = w.clone(), x.clone()
        if spoil_w:
            w2[5, 1, 3], w2[K - 1, 0, 0] = float("inf"), float("nan")
        if spoil_x:
            x2[17, 0], x2[1234, C - 1] = float("nan"), float("-inf")
        got = _thin(w2, x2, i, j, seg, None, n)
        ref = _cabi.mvmr(w2.unsqueeze(1), x2, j, i, seg, None, n, False, _cabi.ENGINE_CUDA_CORE)
        assert torch.equal(got.isnan(), ref.isnan()) and torch.equal(got.isinf(), ref.isinf())
        ok = ref.isfinite()
        assert _rel(got[ok], ref[ok].double()) <= 2 * BOUND[torch.bfloat16]


def test_the_layers_that_take_it():
    """Rulebooks of the search, forward and, where the rulebook is its own mirror image, the input gradient."""
    from pointelligence_b200 import _cabi
    from pointelligence_b200.layers import MetaData, PointConv3d

    pts = torch.rand(20000, 3, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    m = MetaData(points=pts, sample_inds=torch.zeros(len(pts), dtype=torch.int64, device="cuda"),
                 sample_sizes=torch.tensor([len(pts)], device="cuda"), grid_size=0.025, kernel_size=(5, 5, 5), receptive_field_scaler=2.5)
    def kernels(call):
        _cabi.profile_enable(True)
        out = call()
        torch.cuda.synchronize()
        names = [n for n, _ in _cabi.profile_records()]
        _cabi.profile_enable(False)
        return out, names

    i, j, k = m.i, m.j, m.k
    conv = PointConv3d(6, 64, 5, device="cuda", dtype=torch.bfloat16)
    x = torch.randn(len(pts), 6, device="cuda", dtype=torch.bfloat16)
    with torch.no_grad():
        y, names = kernels(lambda: conv(x, i, j, k, len(pts), contract=m.contract, seg_offs=m.seg_offs))
    assert names == ["mvmr_thin_kernel"]
    assert _rel(y, _exact(conv.weight[:, 0], x, i, j, k, len(pts)) + conv.bias.double()) <= BOUND[torch.bfloat16]
    narrow = PointConv3d(64, 6, 5, device="cuda", dtype=torch.float16)
    x64 = torch.randn(len(pts), 64, device="cuda", dtype=torch.float16, requires_grad=True)
    z = narrow(x64, i, j, k, len(pts), contract=m.contract, seg_offs=m.seg_offs)
    go = torch.randn_like(z)
    (gx,), names = kernels(lambda: torch.autograd.grad(z, (x64,), go))
    assert names == ["mvmr_thin_kernel"]
    assert _rel(gx, _exact(narrow.weight[:, 0].transpose(1, 2), go, j, i, k, len(pts))) <= BOUND[torch.float16]
    with torch.no_grad():
        few = PointConv3d(6, 4, 5, device="cuda", dtype=torch.bfloat16)      # too few sums to save
        _, names = kernels(lambda: few(x, i, j, k, len(pts), contract=m.contract, seg_offs=m.seg_offs))
        assert "mvmr_thin_kernel" not in names
        i.add_(0)      # written to since the search: nothing is known about the order
        _, names = kernels(lambda: conv(x, i, j, k, len(pts), contract=m.contract, seg_offs=m.seg_offs))
        assert "mvmr_thin_kernel" not in names


def _clumped(n, members, K, C, ratio, seed, spread=1):
    """``_rulebook`` with, for the first ``members`` of ``n`` points in random order, triplets of each with each of them
    in ``spread`` taps from the middle on: rows of which every one has as many triplets in a tap."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    i, j, k, _ = _rulebook(n, n, K, ratio, seed)
    clump = torch.randperm(n, device="cuda", generator=g)[:members]
    a, b = (t.flatten() for t in torch.meshgrid(clump, clump, indexing="ij"))
    i = torch.cat([i.long()] + [a] * spread)
    j = torch.cat([j.long()] + [b] * spread)
    k = torch.cat([k] + [torch.full_like(a, K // 2 + s) for s in range(spread)])
    order = torch.argsort(k * n + i, stable=True)
    i, j, k = i[order], j[order], k[order]
    seg = torch.searchsorted(k.contiguous(), torch.arange(K + 1, device="cuda"))
    return i.int().contiguous(), j.int().contiguous(), k, seg


def _steps(ws, n_out, K):
    """Steps of every (block, slot of eight taps), from the workspace of a call."""
    up = lambda n: (n + 255) // 256 * 256
    blocks = (n_out + 127) // 128
    at = up(4 * 8 * torch.cuda.get_device_properties(0).multi_processor_count) + up(4 * blocks * K * 128)
    return ws[at:at + 8 * blocks * ((K + 7) // 8)].view(torch.int32)[::2]


@pytest.mark.parametrize("members,K,C,spread", [(8, 27, 3, 1), (9, 27, 6, 1), (10, 27, 6, 14), (33, 27, 8, 2), (64, 125, 6, 1), (65, 125, 3, 3),
                                                (400, 27, 6, 1), (1000, 27, 8, 2)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("sign", [False, True])
def test_rows_of_many_triplets_in_a_tap(members, K, C, spread, dtype, sign):
    """Points within a centimetre of each other: a block takes eight steps at most for eight taps, as long as the sums of such
    a (row, tap) stay within the type's range, and loses nothing (fp32 sums before the product, handed on in three parts)."""
    n, M = 5000, 48
    g = torch.Generator(device="cuda").manual_seed(members)
    i, j, k, seg = _clumped(n, members, K, C, 6.0, members + K, spread)
    w = (torch.randn(K, C, M, device="cuda", generator=g) / C ** 0.5).to(dtype)
    x = torch.randn(n, C, device="cuda", generator=g).to(dtype)
    if sign:
        w, x = w.abs(), x.abs()
    got, ws = _thin(w, x, i, j, seg, None, n, keep=True)
    assert _rel(got, _exact(w, x, i, j, k, n)) <= BOUND[dtype]
    assert 3 <= int(_steps(ws, n, K).max()) <= 8


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_sums_that_leave_the_range_or_are_no_numbers(dtype):
    """Those of a (row, tap) are then taken triplet by triplet: infinities and NaN as the scatter kernel has them, and finite
    rows where the sum of the features alone would be infinite."""
    from pointelligence_b200 import _cabi

    n, K, C, M, members = 1000, 27, 6, 32, 40
    g = torch.Generator(device="cuda").manual_seed(5)
    i, j, k, seg = _clumped(n, members, K, C, 4.0, 9)
    top = torch.finfo(dtype).max
    x = torch.randn(n, C, device="cuda", generator=g).to(dtype)
    x[:, 1] = top / 4
    w = (torch.randn(K, C, M, device="cuda", generator=g) / 64).to(dtype)
    got = _thin(w, x, i, j, seg, None, n)
    exact = _exact(w, x, i, j, k, n)
    fits = exact.abs() < top / 2
    assert bool(fits.any()) and bool(got[fits].isfinite().all()) and _rel(got[fits], exact[fits]) <= 4 * BOUND[dtype]
    heavy = torch.bincount(i[k == K // 2].long(), minlength=n).argmax()
    x = torch.randn(n, C, device="cuda", generator=g).to(dtype)
    members_of = j[(k == K // 2) & (i == heavy)].long()
    x[members_of[7], 2], x[members_of[30], 3] = float("inf"), float("nan")
    got = _thin(w, x, i, j, seg, None, n)
    ref = _cabi.mvmr(w.unsqueeze(1), x, j, i, seg, None, n, False, _cabi.ENGINE_CUDA_CORE)
    assert torch.equal(got.isnan(), ref.isnan()) and torch.equal(got.isinf(), ref.isinf()) and bool(got.isnan().any())
    ok = ref.isfinite()
    assert _rel(got[ok], ref[ok].double()) <= 2 * BOUND[dtype]


@pytest.mark.parametrize("room", [0, 1, 30, 100000])   # sums that the workspace holds
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_sums_that_find_no_room(room, dtype):
    """Triplets of those are taken one by one, in the same eight taps as sums that found room."""
    from pointelligence_b200 import _cabi

    n, K, C, M, members = 1500, 27, 5, 40, 50
    g = torch.Generator(device="cuda").manual_seed(room)
    i, j, k, seg = _clumped(n, members, K, C, 5.0, 3, 4)
    w = (torch.randn(K, C, M, device="cuda", generator=g) / C ** 0.5).to(dtype)
    x = torch.randn(n, C, device="cuda", generator=g).to(dtype)
    L, ptr = _cabi.lib(), _cabi.ptr
    bare = L.pcx_mvmr_thin_workspace_bytes(n, n, K, C, M, 0) - 48 * n      # (with room for a sum a row)
    ws = torch.empty(bare + 48 * room + 256, dtype=torch.uint8, device="cuda")
    out = torch.full((n, M), float("nan"), device="cuda", dtype=dtype)
    code = _cabi.dtype_code(dtype)
    call = lambda size: L.pcx_mvmr_thin(ptr(w), ptr(x), ptr(j), ptr(i), ptr(seg), None, ptr(out), i.numel(), n, n, K, C, M, 0, code, ptr(ws), size,
                                        _cabi.stream_ptr())
    _cabi.check(call(bare + 48 * room + 256))
    assert _rel(out, _exact(w, x, i, j, k, n)) <= BOUND[dtype]
    most = int(_steps(ws, n, K).max())
    assert most <= 8 if room == 100000 else most >= members
    assert call(bare - 512) == -4      # PCX_E_CAPACITY


def test_too_little_memory_for_the_table():
    """A call that the scatter kernels have room for is no error where the table of this one does not fit."""
    from pointelligence_b200 import _cabi
    from pointelligence_b200.layers.triplets import build_triplets_segmented

    n, K = 200_000, 125
    pts = torch.rand(n, 3, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    pts = pts * torch.tensor([1.0, 1.0, 0.02], device="cuda")
    ids, sizes = torch.zeros(n, dtype=torch.int64, device="cuda"), torch.tensor([n], device="cuda")
    i, j, k, seg, _ = build_triplets_segmented(pts, ids, sizes, 0.0115, 5, radius_scaler=2.1)
    w = (torch.randn(K, 1, 4, 32, device="cuda") / 2).bfloat16()
    x = torch.randn(n, 4, device="cuda").bfloat16()

    def call():
        _cabi.profile_enable(True)
        y = _cabi.mvmr(w, x, j, i, seg, None, n, False)
        names = [name for name, _ in _cabi.profile_records()]
        _cabi.profile_enable(False)
        return y, names

    want, names = call()
    assert names == ["mvmr_thin_kernel"], (names, i.numel() / n)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    limit = torch.cuda.memory_reserved() + (84 << 20)      # the table takes 100 MB, the scatter kernel's sums 26
    torch.cuda.set_per_process_memory_fraction(limit / total)
    try:
        got, names = call()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert "mvmr_thin_kernel" not in names
    assert _rel(got, want.double()) < 1e-2
