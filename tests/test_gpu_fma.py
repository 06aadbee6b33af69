"""CUDA-core engines of tap-sorted triplets against fp64: widths around the tiles (32 and 64 columns, slices of 32),
widths that are not multiples of 4, ragged chunks, more taps than the shared-memory chunk table holds, grouped weights.

Tolerance: fp32 operands and sums; an element sums at most a few thousand products of size one with relative
rounding 2^-24 each, so the relative Frobenius error stays below 1e-6 * 4."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

CASES = [  # n_out, n_in, K, T, G, C, M
    (1, 1, 1, 1, 1, 1, 1),
    (300, 200, 27, 3000, 1, 32, 32),
    (300, 200, 27, 3000, 1, 33, 65),
    (129, 128, 8, 1025, 1, 6, 20),
    (200, 200, 27, 2500, 1, 300, 128),
    (100, 90, 27, 900, 3, 5, 36),
    (50, 50, 1500, 4000, 1, 8, 12),
    (70, 60, 3, 700, 2, 64, 96),
]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(str(v) for v in c))
def test_cuda_core_engines(case, dtype):
    from pointelligence_b200 import _cabi

    n_out, n_in, K, T, G, C, M = case
    g = torch.Generator(device=DEV).manual_seed(7)
    k = torch.sort(torch.randint(0, K, (T,), device=DEV, generator=g)).values
    i = torch.randint(0, n_out, (T,), device=DEV, generator=g).int()
    j = torch.randint(0, n_in, (T,), device=DEV, generator=g).int()
    seg = torch.searchsorted(k, torch.arange(K + 1, device=DEV)).to(torch.int64)
    w = torch.randn(K, G, C, M, device=DEV, generator=g).to(dtype)
    x = torch.randn(n_in, G * C, device=DEV, generator=g).to(dtype)
    go = torch.randn(n_out, G * M, device=DEV, generator=g).to(dtype)
    core = _cabi.ENGINE_CUDA_CORE
    y = _cabi.mvmr(w, x, j, i, seg, None, n_out, False, core).double().view(n_out, G, M)
    gx = _cabi.mvmr(w, go, i, j, seg, None, n_in, True, core).double().view(n_in, G, C)
    gw = _cabi.vvor(x.view(n_in, G, C), j, go.view(n_out, G, M), i, seg, None, K, core).double()
    xd, gd, wd = x.double().view(n_in, G, C), go.double().view(n_out, G, M), w.double()
    il, jl = i.long(), j.long()
    y_ref = torch.zeros_like(y).index_add_(0, il, torch.einsum("tgc,tgcm->tgm", xd[jl], wd[k]))
    gx_ref = torch.zeros_like(gx).index_add_(0, jl, torch.einsum("tgm,tgcm->tgc", gd[il], wd[k]))
    gw_ref = torch.zeros_like(gw).index_add_(0, k, torch.einsum("tgc,tgm->tgcm", xd[jl], gd[il]))
    tol = 4e-6 if dtype == torch.float32 else 2.9e-3      # bf16: one rounding of the result, 2^-9 at most
    for a, b in ((y, y_ref), (gx, gx_ref), (gw, gw_ref)):
        assert float((a - b).norm() / b.norm().clamp_min(1e-30)) < tol
