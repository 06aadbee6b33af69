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
