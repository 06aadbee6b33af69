"""Down-sampling: how points are put in the order of their cells, whatever clouds of the same cell size came before."""
import numpy as np
import pytest
import torch

from oracle import geometry as og

pytestmark = pytest.mark.gpu


def _room(n, cell, seed):
    rng = np.random.default_rng(seed)
    pts = rng.random((n, 3)) * cell * 40
    pts[:, 2] *= 0.1
    return pts.astype(np.float32), np.sort(rng.integers(0, 3, n)).astype(np.int32)


def _crowd(n, cell, seed, corner):
    """Most points in a few cells of a wide extent."""
    pts, ids = _room(n, cell, seed)
    pts[: n - 2] *= 0.02
    pts[n - 1] = [corner * cell, -corner * cell, corner * cell]
    return pts, ids


def _check(pts, ids, cell, want):
    from pointelligence_b200 import _cabi

    idx, p, smp, mapping = _cabi.grid_sample_center_nearest(torch.from_numpy(pts).cuda(), cell, torch.from_numpy(ids).cuda(), True)
    ref_p, ref_i, ref_idx, ref_map = want
    assert torch.equal(idx.cpu(), torch.from_numpy(np.asarray(ref_idx)).long()) and torch.equal(p.cpu(), torch.from_numpy(np.asarray(ref_p)))
    assert torch.equal(mapping.cpu(), torch.from_numpy(np.asarray(ref_map)).long())
    assert torch.equal(smp.cpu(), torch.from_numpy(np.asarray(ref_i)).int())


@pytest.mark.parametrize("corner", [2e4, 1.3e6])   # a key space of 2^46 cells, and one of more than 2^62
def test_crowded_clouds_among_ordinary_ones(corner):
    """Two ranges a point, sixteen, sorted at once for sixteen clouds, and counting again: every call finds the same cells."""
    cell = 0.0371 + corner * 1e-9
    clouds = [_room(5000, cell, 1), _crowd(6000, cell, 2, corner), _crowd(4097, cell, 3, corner)]
    want = [og.grid_sample_center_nearest(p, cell, i, True) for p, i in clouds]
    for which in [0, 1, 1, 1, 0, 2] + [1] * 20 + [0] * 20 + [1, 0, 1, 2, 0]:
        _check(*clouds[which], cell, want[which])


def _ranges_used(pts, ids, cell):
    """Ranges that a call counts its points in, told from what it leaves of a filled workspace."""
    import ctypes

    from pointelligence_b200 import _cabi

    lib, n = _cabi.lib(), pts.shape[0]
    pts, ids = torch.from_numpy(pts).cuda(), torch.from_numpy(ids).cuda()
    num = 4096
    while num < 2 * n and num < 1 << 21:
        num *= 2
    more = min(8 * num, 1 << 23)
    ws = torch.full((int(lib.pcx_grid_sample_workspace_bytes(n)),), 0x5a, dtype=torch.uint8, device="cuda")
    info = (ctypes.c_int64 * 3)()
    _cabi.check(lib.pcx_grid_sample_count_samples(pts.data_ptr(), ids.data_ptr(), n, cell, info, ws.data_ptr(), ws.numel(),
                                                  torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    words = ws[256:256 + 4 * more].view(torch.int32)
    used = int((words != 0x5a5a5a5a).sum())
    assert used in (num, more)
    return used // num


def test_more_ranges_are_given_up_where_clouds_do_not_need_them():
    """A cloud of a spinning sensor crowds in two ranges a point and not in sixteen; rooms of the same cell size after it go back
    to two."""
    cell, n = 0.0467, 100_000
    room = _room(n, cell, 4)
    rng = np.random.default_rng(5)
    radius = cell * (5 + 15 * rng.random(n) + 8000 * (rng.random(n) < 0.01))     # dense in the middle
    angle = rng.random(n) * 2 * np.pi
    sweep = np.stack([radius * np.cos(angle), radius * np.sin(angle), rng.random(n) * cell * 30], 1).astype(np.float32)
    sweep = sweep, room[1]
    _ranges_used(*room, cell)
    assert _ranges_used(*room, cell) == 1
    _ranges_used(*sweep, cell)                                          # crowded: sorted, and remembered
    assert _ranges_used(*sweep, cell) == 8 and _ranges_used(*sweep, cell) == 8
    used = [_ranges_used(*room, cell) for _ in range(12)]
    assert used[0] == 8 and used[-1] == 1 and used == sorted(used, reverse=True)
    _ranges_used(*sweep, cell)
    # both in turn: the sweeps keep what they need
    used = [_ranges_used(*(sweep, room)[t % 2], cell) for t in range(12)]
    assert used == [8] * 12
