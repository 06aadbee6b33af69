"""The one-hand-over tap-segmented search (``pcx_radius_taps_*``) against the two-call search
(``pcx_radius_count`` + ``pcx_radius_fill``), which the golden vectors and the oracle pin elsewhere.

The two paths bin the points differently (hashed buckets against injective cell keys), walk the
candidates differently (one lane per cell against one warp per query) and place the pairs
differently (direct tap-major placement against a radix sort by tap), so bit-equal ``i, j, k``,
segment offsets and neighbour counts on the same inputs is a strong check of each.  Cases: both
distances, kernel sizes 3 and 5, batched samples with separate queries, negative coordinates,
a run far longer than the 64-candidate mask (identical points), the boundary shell of pairs within
3 ulp of the radius under all three predicate roundings, and the capacity protocol of the C ABI.
"""
import os

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _both(pts, qry, ps, qs, radius, k, grid, dt=0):
    from pointelligence_b200 import _cabi

    old = os.environ.get("PCX_RADIUS_TAPS")
    try:
        os.environ["PCX_RADIUS_TAPS"] = "0"
        ref = _cabi.radius_search(pts, qry, radius, ps, qs, dt, k, grid, want_k=True)
        os.environ["PCX_RADIUS_TAPS"] = "1"
        got = _cabi.radius_search(pts, qry, radius, ps, qs, dt, k, grid, want_k=True)
    finally:
        if old is None:
            os.environ.pop("PCX_RADIUS_TAPS", None)
        else:
            os.environ["PCX_RADIUS_TAPS"] = old
    return ref, got


def _assert_same(ref, got):
    for name, a, b in zip(("i", "j", "k", "seg_offs", "num_neighbors"), ref, got):
        assert a.dtype == b.dtype and a.shape == b.shape, name
        assert torch.equal(a, b), name


@pytest.mark.parametrize("n,radius,k,dt", [(60000, 0.05, 3, 0), (60000, 0.05, 3, 1), (20000, 0.08, 5, 0),
                                           (20000, 0.08, 5, 1), (37, 0.3, 3, 0), (1, 0.1, 3, 0)])
def test_scene_equals_two_call_search(n, radius, k, dt):
    from pointelligence_b200 import _cabi
    from pointelligence_b200.synthetic import indoor_scene

    dev = torch.device("cuda:0")
    torch.manual_seed(n)
    pts = torch.from_numpy(indoor_scene(n, 1)).to(dev) if n > 100 else torch.rand(n, 3, device=dev)
    grid = radius / 2.5 if k == 3 else radius / 4.5
    _cabi._TAPS_RATIO.clear()
    ref, got = _both(pts, pts, None, None, radius, k, grid, dt)       # counted first call
    _assert_same(ref, got)
    assert got[0].numel() == int(got[4].sum())
    ref, got = _both(pts, pts, None, None, radius, k, grid, dt)       # estimated capacity
    _assert_same(ref, got)


def test_batched_samples_separate_queries_and_capacity_retry():
    from pointelligence_b200 import _cabi
    from pointelligence_b200.synthetic import indoor_scene

    dev = torch.device("cuda:0")
    torch.manual_seed(0)
    pts = torch.cat([torch.from_numpy(indoor_scene(30000, s)) for s in range(3)]).to(dev)
    smp = torch.arange(3, device=dev).repeat_interleave(30000)
    qi = torch.randperm(pts.shape[0], device=dev)[:40000].sort().values
    qry, qs = pts[qi] + 0.003 * torch.randn(40000, 3, device=dev), smp[qi]
    _cabi._TAPS_RATIO.clear()
    _assert_same(*_both(pts, qry, smp, qs, 0.05, 3, 0.02))
    # every sample holds the same coordinates: a query's bucket mixes the three samples
    same = torch.from_numpy(indoor_scene(20000, 7)).to(dev).repeat(3, 1)
    smp3 = torch.arange(3, device=dev).repeat_interleave(20000)
    ref, got = _both(same, same, smp3, smp3, 0.05, 3, 0.02)
    _assert_same(ref, got)
    assert bool((smp3[got[0].long()] == smp3[got[1].long()]).all())
    # an estimate that is far too small: the wrapper retries the fill pass with the exact size
    _cabi._TAPS_RATIO[(3, 0, 0.05)] = 0.01
    _assert_same(*_both(pts, qry, smp, qs, 0.05, 3, 0.02))
    assert _cabi._TAPS_RATIO[(3, 0, 0.05)] > 1.0


def test_long_runs_and_negative_coordinates():
    from pointelligence_b200 import _cabi
    from pointelligence_b200.synthetic import indoor_scene

    dev = torch.device("cuda:0")
    _cabi._TAPS_RATIO.clear()
    same = torch.zeros(1500, 3, device=dev) + 0.5              # one bucket, 1500 candidates per lane
    ref, got = _both(same, same, None, None, 0.05, 3, 0.02)
    _assert_same(ref, got)
    assert got[0].numel() == 1500 * 1500
    _cabi._TAPS_RATIO.clear()
    neg = torch.from_numpy(indoor_scene(50000, 3)).to(dev) - 5.0
    _assert_same(*_both(neg, neg, None, None, 0.05, 3, 0.02))


def test_boundary_shell_all_predicate_roundings():
    from pointelligence_b200 import _cabi

    dev = torch.device("cuda:0")
    rng = np.random.default_rng(0)
    nq, per, radius = 2048, 64, 0.05
    q = (rng.random((nq, 3)) * 50).astype(np.float32)
    d = rng.standard_normal((nq, per, 3))
    d /= np.linalg.norm(d, axis=-1, keepdims=True)
    scale = radius * (1 + rng.integers(-3, 4, (nq, per, 1)) * 2.0 ** -24)
    p = (q[:, None, :].astype(np.float64) + d * scale).astype(np.float32).reshape(-1, 3)
    qt, pt = torch.from_numpy(q).to(dev), torch.from_numpy(p).to(dev)
    totals = []
    try:
        for variant in (0, 1, 2):
            _cabi.check(_cabi.lib().pcx_set_radius_predicate(variant))
            _cabi._TAPS_RATIO.clear()
            ref, got = _both(pt, qt, None, None, radius, 3, 0.02)
            _assert_same(ref, got)
            totals.append(got[0].numel())
    finally:
        _cabi.check(_cabi.lib().pcx_set_radius_predicate(1))
    assert 0 < totals[1] < nq * per and totals[0] != totals[1]   # the shell separates the roundings


def test_c_abi_capacity_protocol_and_argument_errors():
    from pointelligence_b200 import _cabi
    from pointelligence_b200._cabi import c_int64, ptr, stream_ptr, workspace
    from pointelligence_b200.synthetic import indoor_scene

    dev = torch.device("cuda:0")
    L = _cabi.lib()
    pts = torch.from_numpy(indoor_scene(5000, 2)).to(dev)
    n = pts.shape[0]
    assert L.pcx_radius_taps_supported(3) == 1 and L.pcx_radius_taps_supported(5) == 1
    assert L.pcx_radius_taps_supported(7) == 0 and L.pcx_radius_taps_supported(4) == 0
    assert L.pcx_radius_taps_workspace_bytes(n, n, 7) == 0
    ws = workspace(L.pcx_radius_taps_workspace_bytes(n, n, 3), dev)
    nn = torch.empty(n, dtype=torch.int64, device=dev)
    seg = torch.empty(28, dtype=torch.int64, device=dev)
    args = (ptr(pts), ptr(pts), None, None, n, n, 0.05, 0, 3, 0.02, ptr(nn), ptr(seg))
    assert L.pcx_radius_taps_count(*args, ptr(ws), 128, stream_ptr()) == _cabi.PCX_E_CAPACITY   # workspace too small
    assert L.pcx_radius_taps_count(ptr(pts), ptr(pts), None, None, n, n, -1.0, 0, 3, 0.02, ptr(nn), ptr(seg),
                                   ptr(ws), ws.numel(), stream_ptr()) == -1                    # PCX_E_ARG
    assert L.pcx_radius_taps_count(ptr(pts), ptr(pts), None, None, n, n, 0.05, 0, 7, 0.02, ptr(nn), ptr(seg),
                                   ptr(ws), ws.numel(), stream_ptr()) == -6                    # PCX_E_UNSUPPORTED
    _cabi.check(L.pcx_radius_taps_count(*args, ptr(ws), ws.numel(), stream_ptr()))
    total = (c_int64 * 3)()
    _cabi.check(L.pcx_radius_taps_total(n, n, 3, total, ptr(ws), ws.numel(), stream_ptr()))
    t = int(total[0])
    assert t == int(nn.sum()) and int(seg[-1]) == t and int(total[1]) == 0
    small = torch.full((t - 1,), -7, dtype=torch.int32, device=dev)
    got = (c_int64 * 3)()
    rc = L.pcx_radius_taps_fill(ptr(pts), None, None, n, n, 0.05, 0, 3, 0.02, t - 1, ptr(small), ptr(small), None,
                                got, ptr(ws), ws.numel(), stream_ptr())
    assert rc == _cabi.PCX_E_CAPACITY and int(got[0]) == t
    assert bool((small == -7).all())                         # nothing was written
    oi = torch.empty(t, dtype=torch.int32, device=dev)
    oj = torch.empty_like(oi)
    _cabi.check(L.pcx_radius_taps_fill(ptr(pts), None, None, n, n, 0.05, 0, 3, 0.02, t, ptr(oi), ptr(oj), None,
                                       got, ptr(ws), ws.numel(), stream_ptr()))
    os.environ["PCX_RADIUS_TAPS"] = "0"
    try:
        ref = _cabi.radius_search(pts, pts, 0.05, None, None, 0, 3, 0.02, want_k=False)
    finally:
        os.environ.pop("PCX_RADIUS_TAPS", None)
    assert torch.equal(oi, ref[0]) and torch.equal(oj, ref[1])
    # queries with no neighbour are counted for the caller
    far = torch.cat([pts[:100], pts[:7] + 100.0])
    ws = workspace(L.pcx_radius_taps_workspace_bytes(n, 107, 3), dev)
    nn = torch.empty(107, dtype=torch.int64, device=dev)
    _cabi.check(L.pcx_radius_taps_count(ptr(pts), ptr(far), None, None, n, 107, 0.05, 0, 3, 0.02, ptr(nn), ptr(seg),
                                        ptr(ws), ws.numel(), stream_ptr()))
    _cabi.check(L.pcx_radius_taps_total(n, 107, 3, total, ptr(ws), ws.numel(), stream_ptr()))
    assert int(total[1]) == 7 and int((nn == 0).sum()) == 7


def test_builder_raises_for_a_query_without_neighbour():
    from pointelligence_b200.layers.triplets import build_triplets_segmented
    from pointelligence_b200.synthetic import indoor_scene

    dev = torch.device("cuda:0")
    pts = torch.from_numpy(indoor_scene(3000, 4)).to(dev)
    smp = torch.zeros(3000, dtype=torch.int64, device=dev)
    qry = torch.cat([pts[:50], pts[:1] + 100.0])
    qsm = torch.zeros(51, dtype=torch.int64, device=dev)
    with pytest.raises(AssertionError):
        build_triplets_segmented(pts, smp, torch.tensor([3000], device=dev), 0.05, 3, query_points=qry,
                                 query_sample_inds=qsm, query_sample_sizes=torch.tensor([51], device=dev),
                                 radius_scaler=2.5)


def test_tap_ties_on_a_half_grid_lattice():
    """Points on a lattice of half the tap grid: every offset divided by the tap grid is an integer
    or a half-integer, the round-half-even cases the division-free tap computation must hand to
    the exact division."""
    from pointelligence_b200 import _cabi

    dev = torch.device("cuda:0")
    g = 0.02
    axis = torch.arange(24, device=dev, dtype=torch.float32) * (g / 2)
    pts = torch.cartesian_prod(axis, axis, axis).contiguous()
    pts = pts + torch.tensor([0.3, -0.2, 1.7], device=dev)          # lattice offsets that are not representable exactly
    for k, radius in ((3, 0.05), (5, 0.045)):
        _cabi._TAPS_RATIO.clear()
        ref, got = _both(pts, pts, None, None, radius, k, g)
        _assert_same(ref, got)
        assert got[0].numel() > 20 * pts.shape[0]


# neighbours about the number that is kept of a query (64, 128), the pairs a block places at a time (1024 or 1536 for 32
# queries) and the fours of candidates a warp lists at a time (64 for four queries); clusters a cell apart keep the runs apart
@pytest.mark.parametrize("per", [1, 7, 31, 32, 33, 63, 64, 65, 127, 128, 129, 260])
@pytest.mark.parametrize("k", [3, 5])
def test_lists_of_any_length(per, k):
    from pointelligence_b200 import _cabi

    dev = torch.device("cuda:0")
    gen = torch.Generator().manual_seed(per * k)
    centre = torch.arange(41).float()[:, None] * torch.tensor([[0.11, 0.07, 0.0]])
    size = torch.randint(max(1, per - 1), per + 2, (41,), generator=gen)
    pts = torch.repeat_interleave(centre, size, 0)
    pts = (pts + 0.01 * torch.randn(pts.shape, generator=gen))[torch.randperm(pts.shape[0], generator=gen)].to(dev)
    _cabi._TAPS_RATIO.clear()
    _assert_same(*_both(pts, pts, None, None, 0.05, k, 0.02))


@pytest.mark.parametrize("shift", [0.0, -3.0, 1000.0, -20000.0])
def test_cells_out_of_reach(shift):
    """Points and queries on the faces, edges and corners of the search cells and a few ulp off them, where a cell is left out
    of the search if it is farther than the radius."""
    from pointelligence_b200 import _cabi

    dev, radius = torch.device("cuda:0"), 0.05
    rng = np.random.default_rng(5)
    p = (np.round(rng.uniform(-8, 8, (6000, 3))) * radius + shift).astype(np.float32)   # cells are two radii wide
    for _ in range(3):
        p = np.where(rng.random(p.shape) < 0.3, np.nextafter(p, np.float32(np.inf) * rng.choice([-1, 1], p.shape).astype(np.float32)), p)
    q = p[rng.permutation(len(p))][:3000]
    q = np.where(rng.random(q.shape) < 0.3, q + rng.uniform(-radius, radius, q.shape).astype(np.float32), q).astype(np.float32)
    _cabi._TAPS_RATIO.clear()
    _assert_same(*_both(torch.from_numpy(p).to(dev), torch.from_numpy(q).to(dev), None, None, radius, 3, 0.02))


@pytest.mark.parametrize("at", [5e6, -5e6, 1e30, 2.0 ** 30 * 2e-3, -(2.0 ** 30) * 2e-3, 2.0 ** 31 * 2e-3])
@pytest.mark.parametrize("axis", [0, 2])
def test_cells_beyond_the_integers(at, axis):
    """Coordinates whose cell number does not fit 32 bits, or lies about where the search stops trusting it: all of them share
    a cell at the end, and a point still finds itself and its copies."""
    dev, radius = torch.device("cuda:0"), 1e-3
    g = torch.Generator().manual_seed(7)
    p = torch.rand(50, 3, generator=g) * 0.01
    p[:, axis] = (at + abs(at) * 2e-5 * torch.rand(50, generator=g)).float()
    p = torch.cat([p, p[:20]]).to(dev)
    ref, got = _both(p, p, None, None, radius, 3, 1e-3)
    _assert_same(ref, got)
    assert got[0].numel() >= p.shape[0]


@pytest.mark.parametrize("k", [3, 5])
@pytest.mark.parametrize("long", [300, 1600])
def test_long_lists_among_short_ones(long, k):
    """Queries with more pairs than a block places at a time among queries with few or none: a warp walks its runs again in
    the rounds that hold pairs of its queries, and in those alone."""
    from pointelligence_b200 import _cabi

    dev = torch.device("cuda:0")
    gen = torch.Generator().manual_seed(long + k)
    centre = torch.arange(4).float()[:, None] * torch.tensor([[0.31, 0.0, 0.0]])
    pts = torch.repeat_interleave(centre, torch.tensor([long, 3, long // 2, 70]), 0)
    pts = (pts + 0.008 * torch.randn(pts.shape, generator=gen)).to(dev)
    which = torch.randint(0, 6, (200,), generator=gen)        # clusters 4 and 5: nothing there
    qry = (which.float()[:, None] * torch.tensor([[0.31, 0.0, 0.0]]) + 0.004 * torch.randn(200, 3, generator=gen)).to(dev)
    _cabi._TAPS_RATIO.clear()
    ref, got = _both(pts, qry, None, None, 0.05, k, 0.02)
    _assert_same(ref, got)
    assert int(got[4].max()) > long // 2 and int(got[4].min()) == 0


@pytest.mark.parametrize("crowd", [(1023,), (1024,), (1025, 1024, 3), (5000, 1, 2049, 700)])
def test_crowded_cells_keep_their_points_in_order(crowd):
    """Up to 1024 points of a bucket are ordered by counting, more by going through all points; the order of the points
    inside a cell decides the order of the pairs."""
    from pointelligence_b200 import _cabi

    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(sum(crowd))
    pts = torch.cat([torch.rand(n, 3, device=dev, generator=g) * 0.19 + 0.005 + 0.6 * c for c, n in enumerate(crowd)])
    pts = torch.cat([pts, torch.rand(3000, 3, device=dev, generator=g) * 4.0 - 1.0])
    pts = pts[torch.randperm(pts.shape[0], device=dev, generator=g)].contiguous()
    qry = pts[::17].contiguous()
    _cabi._TAPS_RATIO.clear()
    for _ in range(2):      # counted, then with a capacity from the first
        _assert_same(*_both(pts, qry, None, None, 0.1, 3, 0.08))
    smp = torch.arange(pts.shape[0], device=dev) // ((pts.shape[0] + 2) // 3)
    _assert_same(*_both(pts, qry, smp, smp[::17].contiguous(), 0.1, 3, 0.08))


@pytest.mark.parametrize("crowd", [(1025,), (1024 + 256, 5000), (2048, 2049), (70000, 40000, 1100), (33000, 16385, 2500)])
@pytest.mark.parametrize("filler", [0, 90000, 1200000])
@pytest.mark.parametrize("in_order", [False, True])
def test_crowded_cells_of_any_size_keep_their_points_in_order(crowd, filler, in_order):
    """More than 1024 points of a bucket are merged from tiles of 256, or, where that is more work, found by going through
    all points."""
    from pointelligence_b200 import _cabi

    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(sum(crowd) + filler)
    pts = torch.cat([torch.rand(n, 3, device=dev, generator=g) * 0.19 + 0.005 + 0.6 * c for c, n in enumerate(crowd)])
    pts = torch.cat([pts, torch.rand(filler, 3, device=dev, generator=g) * 40.0 - 41.0])
    if not in_order:
        pts = pts[torch.randperm(pts.shape[0], device=dev, generator=g)].contiguous()
    qry = pts[:: pts.shape[0] // 40].contiguous()
    for smp in (None, torch.arange(pts.shape[0], device=dev) // ((pts.shape[0] + 2) // 3)):
        _cabi._TAPS_RATIO.clear()
        ref, got = _both(pts, qry, smp, None if smp is None else smp[:: pts.shape[0] // 40].contiguous(), 0.1, 3, 0.08)
        _assert_same(ref, got)


def test_many_crowded_cells_and_few_queries():
    """Four million points, 1100 in every cell: putting them in order takes no longer than a few sorts of as many keys."""
    from pointelligence_b200 import _cabi

    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(0)
    n = 4_000_000
    side = (n / 1100) ** (1 / 3) * 0.2
    pts = torch.rand(n, 3, device=dev, generator=g) * side
    qry = pts[:32] + 1000.0      # near none of them: what is left is the order
    keys = torch.randint(0, 1 << 40, (n,), device=dev, generator=g)

    def best(call):
        times = []
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            call()
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    search = best(lambda: _cabi.radius_search(pts, qry, 0.1, None, None, 0, kernel_size=3, kernel_grid_size=0.08))
    assert search < 5 * best(lambda: torch.sort(keys)), search


@pytest.mark.parametrize("lowest", [-1, -2, -7, -2**31])
@pytest.mark.parametrize("samples", [1, 3])
def test_samples_numbered_below_zero(lowest, samples):
    """A query in the last cell of sample -1 along every axis looks at a cell whose key is that of an empty slot."""
    from pointelligence_b200 import _cabi

    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(samples)
    pts = torch.cat([torch.rand(400, 3, device=dev, generator=g), torch.full((20, 3), 1.15, device=dev)] * samples)
    ids = torch.arange(samples, device=dev).repeat_interleave(420)
    ref, got = _both(pts, pts, ids + lowest, ids + lowest, 0.1, 3, 0.08)
    _assert_same(ref, got)
    _assert_same(_both(pts, pts, ids, ids, 0.1, 3, 0.08)[0], ref)
    below = _cabi.radius_search(pts, pts, 0.1, ids + lowest, ids + lowest, 0, return_distances=True)
    above = _cabi.radius_search(pts, pts, 0.1, ids, ids, 0, return_distances=True)
    for a, b in zip(below, above):
        assert torch.equal(a, b)
