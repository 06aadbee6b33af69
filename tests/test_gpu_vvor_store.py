"""The weight gradient of few triplets a tap, whose blocks store what they have summed, against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n,K,G,C,M,ratio,empty", [
    (1, 27, 1, 256, 256, 1.0, ()), (63, 27, 1, 256, 256, 9.0, (0, 26)), (300, 8, 1, 512, 384, 6.0, (3,)), (942, 27, 1, 512, 512, 30.0, ()),
    (500, 27, 2, 208, 112, 12.0, (5,)), (700, 125, 1, 96, 1024, 40.0, (124,)), (400, 27, 1, 144, 288, 20.0, ()), (200, 300, 1, 112, 80, 20.0, (0, 1, 2))])
def test_blocks_of_whole_taps(n, K, G, C, M, ratio, empty, dtype):
    from pointelligence_b200 import _cabi

    g = torch.Generator(device="cuda").manual_seed(n + K)
    T = max(int(n * ratio), 1)
    k = torch.sort(torch.randint(0, K, (T,), device="cuda", generator=g))[0]
    for e in empty:
        k = torch.where(k == e, K // 2 + 1, k)
    k = torch.sort(k)[0]
    seg = torch.searchsorted(k, torch.arange(K + 1, device="cuda"))
    i, j = (torch.randint(0, n, (T,), device="cuda", generator=g).int() for _ in range(2))
    a = torch.randn(n, G, C, device="cuda", generator=g).to(dtype)
    b = torch.randn(n, G, M, device="cuda", generator=g).to(dtype)
    _cabi.launch_count(reset=True)
    got = _cabi.vvor(a, i, b, j, seg, None, K)
    assert _cabi.launch_count() == 1      # no sums cleared or rounded
    at = [int(s) for s in seg]
    ref = torch.stack([torch.einsum("tgc,tgm->gcm", a[i[at[t]:at[t + 1]].long()].double(), b[j[at[t]:at[t + 1]].long()].double())
                       for t in range(K)])
    # one rounding of fp32 sums: the type's unit roundoff in every element
    assert float((got.double() - ref).norm() / ref.norm()) <= (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11)
    for e in empty:
        assert not bool(got[e].any())


def _strided(n_in, n_out, K, T, seed, share):
    """Tap-sorted triplets of ``n_out`` rows on ``n_in`` points; ``share`` of them in the middle tap."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    k = torch.randint(0, K, (T,), device="cuda", generator=g)
    k = torch.where(torch.rand(T, device="cuda", generator=g) < share, K // 2, k)
    k = torch.sort(k)[0]
    seg = torch.searchsorted(k, torch.arange(K + 1, device="cuda"))
    i = torch.randint(0, n_out, (T,), device="cuda", generator=g).int()
    return i, torch.randint(0, n_in, (T,), device="cuda", generator=g).int(), seg


# 512 x 512 channels: 3131 triplets of the fullest tap take as long as the fp32 sums
@pytest.mark.parametrize("n_in,n_out,T,share,known,stores", [
    (942, 942, 20000, 0.0, None, True),        # a self-search by its sizes: twice the average, 1481, and the points
    (942, 942, 20000, 0.9, 18000, False),      # ... known to crowd in a tap
    (942, 942, 20000, 0.0, 800, True),
    (3000, 900, 20000, 0.0, None, True),       # strided: twice the average
    (3000, 900, 60000, 0.0, None, False),
    (3000, 900, 60000, 0.0, 2300, True),       # known to hold fewer
    (3000, 900, 80000, 0.9, 72000, False),
    (3000, 900, 3000, 1.0, None, True)])       # all triplets in a tap are few enough
def test_the_fullest_tap_decides(n_in, n_out, T, share, known, stores):
    from pointelligence_b200 import _cabi

    K, C, M = 27, 512, 512
    i, j, seg = _strided(n_in, n_out, K, T, n_in + T, share)
    if known is not None:
        _cabi.mark_built(i, j, seg, K, symmetric=False, fullest=known)
    x = torch.randn(n_in, 1, C, device="cuda").bfloat16()
    go = torch.randn(n_out, 1, M, device="cuda").bfloat16()
    _cabi.vvor(x, j, go, i, seg, None, K)
    for _ in range(2):      # the rulebook of a layer, and of the up-sampling layer that mirrors it
        _cabi.launch_count(reset=True)
        got = _cabi.vvor(x, j, go, i, seg, None, K)
        assert _cabi.launch_count() == (1 if stores else 3)
        at = [int(s) for s in seg]
        for t in (0, K // 2):
            ref = x[j[at[t]:at[t + 1]].long(), 0].double().t() @ go[i[at[t]:at[t + 1]].long(), 0].double()
            assert float((got[t, 0].double() - ref).norm()) <= 2.0 ** -8 * float(ref.norm())
        x, go, i, j = go, x, j, i


def test_searches_tell_their_fullest_tap():
    from pointelligence_b200 import _cabi
    from pointelligence_b200.layers import MetaData
    from pointelligence_b200.layers.triplets import build_triplets_segmented, handle_stride_and_build_triplets

    g = torch.Generator(device="cuda").manual_seed(0)
    for clump in (0, 200):
        pts = torch.rand(3000, 3, device="cuda", generator=g)
        pts[:clump] = pts[:clump] * 1e-3 + 0.5
        ids, sizes = torch.zeros(3000, dtype=torch.int64, device="cuda"), torch.tensor([3000], device="cuda")
        for _ in range(2):      # counted first, then with a capacity
            i, j, k, seg, _ = build_triplets_segmented(pts, ids, sizes, 0.1, 3, radius_scaler=2.5)
            full = int((seg[1:] - seg[:-1]).max())
            assert _cabi.fullest_tap(i, j, seg, 27) == full == _cabi.fullest_tap(j, i, seg, 27)
            assert _cabi.fullest_tap(i, j, seg.clone(), 27) is None and _cabi.fullest_tap(i.clone(), j, seg, 27) is None
        m = MetaData(points=pts, sample_inds=ids, sample_sizes=sizes, grid_size=0.05)
        m = handle_stride_and_build_triplets(m, 2.0, (3, 3, 3), 2.5)
        assert _cabi.fullest_tap(m.i, m.j, m.seg_offs, 27) == int((m.seg_offs[1:] - m.seg_offs[:-1]).max())
        i.add_(0)
        assert _cabi.fullest_tap(i, j, seg, 27) is None
