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
