"""Layer norms of small batches, which take one kernel forward and one backward, at the line and against the larger ones."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(x, lengths, w, b, res, relu, eps):
    at, out = 0, []
    for n in lengths:
        part = x[at:at + n]
        at += n
        if n == 0:
            continue
        mu = part.mean()
        out.append((part - mu) / torch.sqrt(((part - mu) ** 2).mean() + eps))
    y = torch.cat(out) if out else x
    y = y * w + b if w is not None else y
    y = y if res is None else y + res
    return y.relu() if relu else y


@pytest.mark.parametrize("lengths,C", [([1], 8), ([3, 0, 5], 24), ([0, 700, 0, 0, 33, 1], 64), ([65536], 64), ([65537], 64), ([200] * 32, 96),
                                       ([100] * 33, 96), ([5000, 1, 8000], 20), ([300, 500], 2048), ([40, 60], 4096), ([17, 4], 2056)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tail", [False, True])
def test_against_fp64(lengths, C, dtype, tail):
    from pointelligence_b200.layers.norm import fused_layer_norm

    g = torch.Generator(device="cuda").manual_seed(sum(lengths) + C)
    N = sum(lengths)
    make = lambda *shape: torch.randn(*shape, device="cuda", generator=g)
    x, res, go = (make(N, C) * 2 + 3).to(dtype).requires_grad_(), make(N, C).to(dtype).requires_grad_(), make(N, C).to(dtype)
    w, b = (make(C) * 0.2 + 1).requires_grad_(), make(C).requires_grad_()
    y = fused_layer_norm(x, torch.tensor(lengths, device="cuda"), w, b, 1e-5, residual=res if tail else None, relu=tail)
    leaves = [t.detach().double().requires_grad_() for t in (x, w, b, res)]
    ref = _reference(leaves[0], lengths, leaves[1], leaves[2], leaves[3] if tail else None, tail, 1e-5)
    # one rounding of the result; in the gradient the mask of the ReLU is that of the rounded result, and rows of few elements cancel
    unit = {torch.float32: 2e-6, torch.bfloat16: 2.0 ** -8}[dtype]
    assert float((y.double() - ref).norm() / ref.norm()) <= unit
    mask = (y.double() > 0) if tail else torch.ones_like(ref)
    wants = (x, w, b) + ((res,) if tail else ())
    got = torch.autograd.grad(y, wants, go)
    inner = _reference(leaves[0], lengths, leaves[1], leaves[2], leaves[3] if tail else None, False, 1e-5)
    want = torch.autograd.grad(inner, [leaves[0], leaves[1], leaves[2]] + ([leaves[3]] if tail else []), go.double() * mask)
    for a, r in zip(got, want):
        assert float((a.double() - r).norm()) <= 4 * unit * float(r.norm()) + 1e-4 * float(go.double().norm()) * (1 if N * C < 64 else 1e-2)


PART_OF_THE_CHIP = """
import torch
from pointelligence_b200.layers.norm import fused_layer_norm

part = torch.cuda.GreenContext.create(num_sms=16, device_id=0)
stream = part.Stream()
g = torch.Generator(device="cuda").manual_seed(0)
x = (torch.randn(20000, 64, device="cuda", generator=g) * 2 + 3).bfloat16().requires_grad_()
go = torch.randn(20000, 64, device="cuda", generator=g).bfloat16()
w, b = torch.ones(64, device="cuda").requires_grad_(), torch.zeros(64, device="cuda").requires_grad_()
lengths = torch.tensor([15000, 5000], device="cuda")
whole = torch.autograd.grad(fused_layer_norm(x, lengths, w, b, 1e-5), (x, w, b), go)
torch.cuda.synchronize()
with torch.cuda.stream(stream):
    got = torch.autograd.grad(fused_layer_norm(x, lengths, w, b, 1e-5), (x, w, b), go)
stream.synchronize()
assert all(float((a.double() - r.double()).norm() / r.double().norm()) < 1e-3 for a, r in zip(got, whole))
"""


def test_on_a_part_of_the_chip():
    """A stream that has fewer multiprocessors than the blocks of one launch would take together."""
    import os
    import subprocess
    import sys

    if not hasattr(torch.cuda, "GreenContext"):
        pytest.skip("no green contexts")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    done = subprocess.run([sys.executable, "-c", PART_OF_THE_CHIP], cwd=root, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
