"""Layers whose widths the tensor engines take in parts or padded: channel counts that are not multiples of 16,
rows wider than 256 channels, grouped weights -- on the scatter kernel, the output-stationary kernel (split by
taps where the cloud is small, whole groups where it is not) and the weight-gradient kernel, against fp64.

Tolerance: the operands are exact in the reference.  A result is rounded once (2^-9 relative at most, bf16;
2^-12, fp16), a bucket sum of the output-stationary kernel once more; relative Frobenius errors stay below
2^-8.5 = 2.8e-3 (bf16) and 2^-11.5 = 3.5e-4 (fp16), the fp32 sums add less than 1e-5."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TOL = {torch.bfloat16: 2.9e-3, torch.float16: 3.7e-4}


def _rulebook(n_out, n_in, K, T, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    k = torch.sort(torch.randint(0, K, (T,), device=DEV, generator=g)).values
    i = torch.randint(0, n_out, (T,), device=DEV, generator=g)
    order = torch.argsort(k * n_out + i, stable=True)
    i, j = i[order].int(), torch.randint(0, n_in, (T,), device=DEV, generator=g).int()
    seg = torch.searchsorted(k, torch.arange(K + 1, device=DEV)).to(torch.int64)
    return i, j, k, seg


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm().clamp_min(1e-30))


CASES = [  # n_out, n_in, K, T, G, C, M, dtype
    (1, 1, 1, 1, 1, 3, 16, torch.bfloat16),
    (300, 257, 27, 4000, 1, 6, 32, torch.bfloat16),
    (129, 200, 27, 5000, 1, 20, 20, torch.float16),
    (500, 400, 125, 9000, 1, 3, 272, torch.bfloat16),
    (400, 380, 27, 12000, 1, 512, 512, torch.float16),
    (260, 300, 8, 2500, 1, 384, 320, torch.bfloat16),
    (513, 513, 27, 9000, 2, 48, 256, torch.bfloat16),
    (300, 300, 27, 3000, 2, 3, 10, torch.float16),
    (200, 220, 27, 4000, 4, 16, 320, torch.bfloat16),
    (80000, 80000, 27, 500000, 1, 32, 48, torch.bfloat16),
    (40000, 40000, 27, 600000, 1, 256, 256, torch.bfloat16),   # fewer slots than copy teams, many steps a block
    (20001, 20000, 125, 600000, 1, 5, 32, torch.bfloat16),     # steps of four taps, of two on the way back
    (3000, 3000, 70, 60000, 2, 32, 16, torch.float16),         # steps that end in a part of their taps
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(str(v) for v in c[:7]))
def test_padded_wide_and_grouped_layers(case):
    from pointelligence_b200 import _cabi
    from pointelligence_b200.sparse_engines.tig import TigIndex, tig_mvmr

    n_out, n_in, K, T, G, C, M, dtype = case
    i, j, k, seg = _rulebook(n_out, n_in, K, T, 3)
    g = torch.Generator(device=DEV).manual_seed(4)
    w = (torch.randn(K, G, C, M, device=DEV, generator=g) / C ** 0.5).to(dtype)
    x = torch.randn(n_in, G * C, device=DEV, generator=g).to(dtype)
    go = torch.randn(n_out, G * M, device=DEV, generator=g).to(dtype)
    b = torch.randn(G * M, device=DEV, generator=g).to(dtype)
    y_ref = torch.zeros(n_out, G, M, dtype=torch.float64, device=DEV)
    gx_ref = torch.zeros(n_in, G, C, dtype=torch.float64, device=DEV)
    gw_ref = torch.zeros(K, G, C, M, dtype=torch.float64, device=DEV)
    xd, gd, wd = x.double().view(n_in, G, C), go.double().view(n_out, G, M), w.double()
    for tap in range(K):
        a, e = int(seg[tap]), int(seg[tap + 1])
        ii, jj = i[a:e].long(), j[a:e].long()
        y_ref.index_add_(0, ii, torch.einsum("tgc,gcm->tgm", xd[jj], wd[tap]))
        gx_ref.index_add_(0, jj, torch.einsum("tgm,gcm->tgc", gd[ii], wd[tap]))
        gw_ref[tap] = torch.einsum("tgc,tgm->gcm", xd[jj], gd[ii])
    tol = TOL[dtype]
    # the layer: bias, forward and the three gradients
    index = TigIndex.from_flat(i, j, seg, n_out, n_in, K)
    ws, xs, bs = (t.clone().requires_grad_() for t in (w, x, b))
    y = tig_mvmr(ws, xs, index, bias=bs)
    y.backward(go)
    assert _rel(y, y_ref.view(n_out, -1) + b.double()) < tol
    assert _rel(xs.grad, gx_ref.view(n_in, -1)) < tol and _rel(ws.grad, gw_ref) < tol
    assert _rel(bs.grad, go.double().sum(0)) < tol
    # every engine that takes these widths
    if C % 16 == 0 and M % 16 == 0 and C != 320:
        for engine in (_cabi.ENGINE_TENSOR, _cabi.ENGINE_PLANNED):
            out = _cabi.mvmr(w, x, j, i, seg, None, n_out, False, engine)
            assert _rel(out, y_ref.view(n_out, -1)) < tol, engine
            gx = _cabi.mvmr(w, go, i, j, seg, None, n_in, True, engine)
            assert _rel(gx, gx_ref.view(n_in, -1)) < tol, engine
        again = _cabi.mvmr(w, x, j, i, seg, None, n_out, False, _cabi.ENGINE_PLANNED)
        assert torch.equal(out, again)            # fixed order of every sum, split or not
    assert _cabi.device_status() == 0


def test_output_row_count_one_above_a_whole_wave_of_groups():
    """75 777 rows: 297 groups, the first count that is not split, and a last block of one row."""
    from pointelligence_b200 import _cabi

    n, K, T = 296 * 256 + 1, 27, 300000
    i, j, k, seg = _rulebook(n, n, K, T, 9)
    i[-1] = n - 1
    w = torch.randn(K, 1, 32, 32, device=DEV).bfloat16() / 6
    x = torch.randn(n, 32, device=DEV).bfloat16()
    out = _cabi.mvmr(w, x, j, i, seg, None, n, False, _cabi.ENGINE_PLANNED)
    ref = torch.zeros(n, 32, dtype=torch.float64, device=DEV)
    for tap in range(K):
        a, e = int(seg[tap]), int(seg[tap + 1])
        ref.index_add_(0, i[a:e].long(), x[j[a:e].long()].double() @ w[tap, 0].double())
    assert _rel(out, ref) < TOL[torch.bfloat16]


def test_plan_of_rows_out_of_order_inside_a_tap():
    """The counting path and the sorting path of the plan builder regroup the same triplets."""
    from pointelligence_b200 import _cabi

    n, K, T = 700, 27, 9000
    i, j, k, seg = _rulebook(n, n, K, T, 13)
    shuffle = torch.argsort(k * T + torch.randperm(T, device=DEV))
    counted = _cabi.mvmr_plan(i, j, seg, K, n, 2)
    sorted_ = _cabi.mvmr_plan(i[shuffle], j[shuffle], seg, K, n, 2)
    a, b = counted.views(), sorted_.views()
    assert torch.equal(a["perm"], b["perm"]) and torch.equal(a["tile_offs"], b["tile_offs"])
    assert counted.multi_buckets == sorted_.multi_buckets > 0
    assert torch.equal(a["entries"][:, 0], b["entries"][:, 0])
    assert torch.equal(a["tile_rows"] < -1, b["tile_rows"] < -1) and torch.equal(a["tile_rows"].clamp_min(-1), b["tile_rows"].clamp_min(-1))
    w, x = torch.randn(K, 1, 64, 64, device=DEV).bfloat16() / 8, torch.randn(n, 64, device=DEV).bfloat16()
    assert _rel(_cabi.mvmr_planned(w, x, counted, False), _cabi.mvmr_planned(w, x, sorted_, False).double()) < TOL[torch.bfloat16]


@pytest.mark.parametrize("Ma,Cb", [(16, 16), (64, 64), (96, 160), (256, 256)])
@pytest.mark.parametrize("scale", [1, 16])
def test_weight_gradient_at_the_edges_of_chunks(Ma, Cb, scale):
    """Taps of no, one, and around a multiple of 16 / 64 / 256 triplets, between taps of many chunks (which are
    longer where the rulebook is); fp32 sums of exact products, rounded once."""
    from pointelligence_b200 import _cabi

    sizes = [0, 1, 15, 16, 17, 0, 63, 64, 65, 255, 256, 257, 12000 * scale, 3, 0, 127 * scale, 128, 129, 0]
    seg = torch.tensor([0] + sizes, device=DEV).cumsum(0)
    T, n = int(seg[-1]), 3001
    g = torch.Generator(device=DEV).manual_seed(9)
    ai, bi = (torch.randint(0, n, (T,), device=DEV, generator=g).int() for _ in range(2))
    a, b = (torch.randn(n, 1, c, device=DEV, generator=g).to(torch.bfloat16) for c in (Ma, Cb))
    out = _cabi.vvor(a, ai, b, bi, seg, None, len(sizes))
    ref = torch.zeros(len(sizes), 1, Ma, Cb, dtype=torch.float64, device=DEV)
    for k in range(len(sizes)):
        s, e = int(seg[k]), int(seg[k + 1])
        ref[k, 0] = a[ai[s:e].long(), 0].double().T @ b[bi[s:e].long(), 0].double()
        assert _rel(out[k], ref[k]) < TOL[torch.bfloat16], k


@pytest.mark.parametrize("n", [300, 5000])
def test_plan_of_a_geometry_built_rulebook_is_not_waited_for(n):
    """The plan whose bucket count arrives later, used at once, later and on another stream, gives the bits of the
    plan that was waited for."""
    from pointelligence_b200 import _cabi
    from pointelligence_b200.layers.triplets import build_triplets_segmented

    g = torch.Generator(device=DEV).manual_seed(n)
    pts = torch.rand(n, 3, device=DEV, generator=g) * n ** (1 / 3)
    inds, sizes = torch.zeros(n, dtype=torch.int32, device=DEV), torch.tensor([n], device=DEV)
    i, j, k, seg, _ = build_triplets_segmented(pts, inds, sizes, 1.5, 3, radius_scaler=2.5)
    want = _cabi.mvmr_plan(i.clone(), j.clone(), seg, 27, n, 2)
    assert want._word is None and want.multi_buckets > 0
    w, x = torch.randn(27, 1, 64, 64, device=DEV).bfloat16() / 8, torch.randn(n, 64, device=DEV).bfloat16()
    ref = _cabi.mvmr_planned(w, x, want, False)
    torch.cuda.synchronize()
    plan = _cabi.cached_mvmr_plan(i, j, seg, 27, n, 2)
    assert want.multi_buckets <= plan.multi_buckets <= i.numel() // 2
    assert torch.equal(_cabi.mvmr_planned(w, x, plan, False), ref)
    fresh = _cabi.cached_mvmr_plan(i, j, seg.clone(), 27, n, 2)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        assert fresh.multi_buckets == want.multi_buckets
        assert torch.equal(_cabi.mvmr_planned(w, x, fresh, False), ref)
    side.synchronize()
    torch.cuda.synchronize()
    assert plan.multi_buckets == want.multi_buckets and plan._word is None


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T", [1, 300, 9000])
@pytest.mark.parametrize("C,M,G", [(512, 64, 1), (320, 288, 1), (768, 288, 1), (2048, 16, 1), (384, 512, 2)])
def test_parts_of_a_contraction_in_one_block(C, M, G, T, dtype):
    """Few tiles: each part a block of its own; many: one block takes them one after another.  Operands of -1, 0 and 1
    keep every sum a whole number below 2^8, exact in fp32 and after the rounding, in any order."""
    from pointelligence_b200 import _cabi

    n = max(2, T // 4)
    i, j, k, seg = _rulebook(n, n, 27, T, 7)
    g = torch.Generator(device=DEV).manual_seed(8)

    def few(*shape):   # one in eight is -1 or 1
        sign = 2 * torch.randint(0, 2, shape, device=DEV, generator=g) - 1
        return (torch.randint(0, 8, shape, device=DEV, generator=g) // 7 * sign).to(dtype)

    w, x, go = few(27, G, C, M), few(n, G * C), few(n, G * M)
    y_ref = torch.zeros(n, G, M, dtype=torch.float64, device=DEV)
    gx_ref = torch.zeros(n, G, C, dtype=torch.float64, device=DEV)
    for t in range(27):
        s = slice(int(seg[t]), int(seg[t + 1]))
        y_ref.index_add_(0, i[s].long(), torch.einsum("tgc,gcm->tgm", x[j[s].long()].view(-1, G, C).double(), w[t].double()))
        gx_ref.index_add_(0, j[s].long(), torch.einsum("tgm,gcm->tgc", go[i[s].long()].view(-1, G, M).double(), w[t].double()))
    assert max(y_ref.abs().max(), gx_ref.abs().max()) < 256
    y = _cabi.mvmr(w, x, j, i, seg, None, n, False, _cabi.ENGINE_TENSOR)
    gx = _cabi.mvmr(w, go, i, j, seg, None, n, True, _cabi.ENGINE_TENSOR)
    assert torch.equal(y.double(), y_ref.flatten(1)) and torch.equal(gx.double(), gx_ref.flatten(1))


def _whole_numbers(dtype, seed, T, n, C, M, n_in=None):
    """Operands of -1, 0 and 1, one in eight not 0: every sum a whole number, exact in fp32 and, below 2^8, after the rounding."""
    n_in = n_in or n
    i, j, k, seg = _rulebook(n, n_in, 27, T, seed)
    g = torch.Generator(device=DEV).manual_seed(seed)

    def few(*shape):
        sign = 2 * torch.randint(0, 2, shape, device=DEV, generator=g) - 1
        return (torch.randint(0, 8, shape, device=DEV, generator=g) // 7 * sign).to(dtype)

    w, x, go = few(27, 1, C, M), few(n_in, C), few(n, M)
    y, gx = (torch.zeros(rows, width, dtype=torch.float64, device=DEV) for rows, width in ((n, M), (n_in, C)))
    for t in range(27):
        s = slice(int(seg[t]), int(seg[t + 1]))
        y.index_add_(0, i[s].long(), x[j[s].long()].double() @ w[t, 0].double())
        gx.index_add_(0, j[s].long(), go[i[s].long()].double() @ w[t, 0].double().T)
    assert max(y.abs().max(), gx.abs().max()) < 256
    return i, j, seg, w, x, go, y, gx


# parts of the contraction, what tensor memory holds of them, links: 3 / 4 / 1, 4 / 4 / 1, 5 / 4 / 5, 6 / 4 / 2, 7 / 4 / 7, 8 / 4 / 2;
# 3 / 2 / 3, 4 / 2 / 2; three narrow parts
@pytest.mark.parametrize("C,M", [(768, 128), (1024, 128), (1280, 80), (1536, 128), (1792, 96), (2048, 128), (768, 512), (1024, 256), (528, 80)])
@pytest.mark.parametrize("T", [20000, 60000])   # too few tiles for links of several parts, and enough
def test_links_of_a_contraction(C, M, T):
    from pointelligence_b200 import _cabi

    i, j, seg, w, x, go, y, gx = _whole_numbers(torch.float16, C + M, T, T // 4, C, M)
    assert torch.equal(_cabi.mvmr(w, x, j, i, seg, None, T // 4, False, _cabi.ENGINE_TENSOR).double(), y)
    assert torch.equal(_cabi.mvmr(w, go, i, j, seg, None, T // 4, True, _cabi.ENGINE_TENSOR).double(), gx)
    wt = w.transpose(2, 3).contiguous()     # the same links in the other direction
    assert torch.equal(_cabi.mvmr(wt, x, j, i, seg, None, T // 4, True, _cabi.ENGINE_TENSOR).double(), y)
    assert _cabi.device_status() == 0


@pytest.mark.parametrize("n", [163840, 163841])   # accumulators of 160 MB and a row more: eight warps a block, and four
def test_accumulators_about_the_size_that_keeps_four_warps(n):
    from pointelligence_b200 import _cabi

    i, j, seg, w, x, go, y, gx = _whole_numbers(torch.float16, 3, 30000, n, 256, 256, n_in=9000)
    assert torch.equal(_cabi.mvmr(w, x, j, i, seg, None, n, False, _cabi.ENGINE_TENSOR).double(), y)
    assert torch.equal(_cabi.mvmr(w, go, i, j, seg, None, 9000, True, _cabi.ENGINE_TENSOR).double(), gx)


@pytest.mark.parametrize("rows", [1, 2, 3, 5, 170, 171, 1365, 1366, 30001])
@pytest.mark.parametrize("offset", [0, 1, 8])   # of the first element of the output, in elements: 8 is a 16-byte boundary again
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_sums_are_rounded_to_rows_of_any_size_and_address(rows, offset, dtype):
    """No triplets and a bias: every row is the bias, exactly, and nothing beyond the rows is written."""
    from pointelligence_b200 import _cabi

    lib, M = _cabi.lib(), 3
    bias = torch.tensor([1.5, -2.0, 0.25], dtype=dtype, device=DEV)
    w = torch.zeros(1, 1, 3, M, dtype=dtype, device=DEV)
    seg = torch.zeros(2, dtype=torch.int64, device=DEV)
    out = torch.full((rows * M + 24,), 7.0, dtype=dtype, device=DEV)
    code = 1 if dtype == torch.float16 else 2
    need = lib.pcx_mvmr_workspace_bytes(rows, 1, 1, 3, M, 0, code)
    ws = torch.empty(need, dtype=torch.uint8, device=DEV)
    _cabi.check(lib.pcx_mvmr_bias(w.data_ptr(), None, None, None, seg.data_ptr(), None, bias.data_ptr(), out.data_ptr() + 2 * offset,
                                  0, 1, rows, 1, 1, 3, M, 0, code, 0, ws.data_ptr(), need, torch.cuda.current_stream().cuda_stream))
    assert torch.equal(out[offset:offset + rows * M].view(rows, M), bias.expand(rows, M))
    assert (out[:offset] == 7).all() and (out[offset + rows * M:] == 7).all()
