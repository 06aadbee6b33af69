"""Layers of different widths that several threads run for the first time, at once: the shared memory that one of them asks
for is not taken back by another that needs less."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import threading, torch
from pointelligence_b200 import _cabi
from pointelligence_b200.layers.triplets import build_triplets_segmented

g = torch.Generator(device="cuda").manual_seed(0)
n, K = 4000, 27
pts = torch.rand(n, 3, device="cuda", generator=g)
ids, sizes = torch.zeros(n, dtype=torch.int64, device="cuda"), torch.tensor([n], device="cuda")
i, j, k, seg, _ = build_triplets_segmented(pts, ids, sizes, 0.12, 3, radius_scaler=2.5)
plan = _cabi.cached_mvmr_plan(i, j, seg, K, n, _cabi.plan_group_blocks(64))
plan.multi_buckets
torch.cuda.synchronize()
errors, start = [], threading.Barrier(9)

def layer(width):
    try:
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            w6 = torch.randn(K, 1, 6, width, device="cuda").bfloat16()
            w = torch.randn(K, 1, 64, width, device="cuda").bfloat16()
            x6, x = torch.randn(n, 6, device="cuda").bfloat16(), torch.randn(n, 64, device="cuda").bfloat16()
            a, b = torch.randn(n, 1, 4 * width, device="cuda").bfloat16(), torch.randn(n, 1, 2 * width, device="cuda").bfloat16()
            stream.synchronize()
            start.wait()
            for _ in range(20):
                _cabi.mvmr(w6, x6, j, i, seg, None, n, False)
                _cabi.mvmr(w, x, j, i, seg, None, n, False)
                _cabi.mvmr(w, x, j, i, seg, None, n, False, _cabi.ENGINE_TENSOR)
                _cabi.vvor(a, i, b, j, seg, None, K)
            stream.synchronize()
    except Exception as e:
        errors.append(f"{width}: {e}")

threads = [threading.Thread(target=layer, args=(16 * (t % 8 + 1),)) for t in range(9)]
[t.start() for t in threads]
[t.join() for t in threads]
assert not errors, errors
assert _cabi.device_status() == 0
"""


@pytest.mark.parametrize("run", range(3))
def test_first_calls_of_several_threads(run):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    done = subprocess.run([sys.executable, "-c", PROGRAM], cwd=root, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
