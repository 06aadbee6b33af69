"""The segmentation backbone without gradients: the weights of a pass are those its layers have when they run."""
import copy

import pytest
import torch
from torch.nn.utils import prune

pytestmark = pytest.mark.gpu

CLASSES = 20


@pytest.fixture(scope="module")
def scene():
    from pointelligence_b200.synthetic import indoor_scene, ragged_batch

    pts, inds, sizes = (torch.from_numpy(a).cuda() for a in ragged_batch([indoor_scene(3000, 1), indoor_scene(2000, 2)]))
    feat = torch.randn(pts.shape[0], 3, device="cuda", generator=torch.Generator(device="cuda").manual_seed(0))
    return feat, pts, inds, sizes, 0.02


def _model(seed=0):
    from pointelligence_b200.backbone import ResUNet

    torch.manual_seed(seed)
    return ResUNet(in_channels=3, num_classes=CLASSES, layers=(1,) * 8).cuda()


def _same(got, want):
    # forty bf16 layers in a row, whose fp32 sums may be added in another order: far below a change of any weight
    return float((got.float() - want.float()).norm() / want.float().norm()) < 3e-2


def _bias_alone(model, logits):
    return torch.equal(logits, model.final_conv.bias.detach().bfloat16().expand_as(logits))


def test_same_with_and_without_gradients(scene):
    model = _model()
    with torch.no_grad():
        got = model(*scene)
    assert _same(got, model(*scene).detach())


def test_pruned_network_after_loading_weights(scene):
    model = _model()
    for conv in (model.conv1, model.block1[0].conv1, model.enc_block2[0].conv2, model.upsample3.conv, model.final_conv):
        prune.random_unstructured(conv, "weight", amount=0.3)
    with torch.no_grad():
        before = model(*scene)
    other = copy.deepcopy(model.state_dict())
    for name in other:
        if name.endswith("weight_orig"):
            other[name].mul_(-2.0)
    model.load_state_dict(other)
    with torch.no_grad():
        got = model(*scene)
    want = model(*scene).detach()
    assert _same(got, want) and not _same(before, want)
    model.final_conv.weight_orig.data.zero_()
    with torch.no_grad():
        assert _bias_alone(model, model(*scene))


@pytest.mark.parametrize("change", ["data", "in place", "new storage", "new parameter"])
@pytest.mark.parametrize("kind", ["pre", "post", "global"])
def test_hook_that_changes_the_weight_of_a_later_layer(scene, change, kind):
    model = _model()
    with torch.no_grad():
        torch.nn.init.normal_(model.final_conv.bias)

    def hook(module, *_):
        if module is not model.block1[0]:
            return
        conv = model.final_conv
        if change == "data":
            conv.weight.data.zero_()
        elif change == "in place":
            conv.weight.zero_()
        elif change == "new storage":
            conv.weight.data = torch.zeros_like(conv.weight)
        else:
            conv.weight = torch.nn.Parameter(torch.zeros_like(conv.weight))

    handle = (model.block1[0].register_forward_pre_hook(hook) if kind == "pre" else
              model.block1[0].register_forward_hook(hook) if kind == "post" else
              torch.nn.modules.module.register_module_forward_pre_hook(hook))
    try:
        with torch.no_grad():
            assert _bias_alone(model, model(*scene))
    finally:
        handle.remove()


def test_layer_that_changes_the_weight_of_a_later_one(scene):
    """No hook: a layer put into the network does it, in each of the ways that leave a trace on the tensor."""
    for change in (lambda conv: conv.weight.zero_(), lambda conv: setattr(conv.weight, "data", torch.zeros_like(conv.weight)),
                   lambda conv: setattr(conv, "weight", torch.nn.Parameter(torch.zeros_like(conv.weight)))):
        model = _model()

        class Block(type(model.block1[0])):
            def forward(self, x, m):
                change(model.final_conv)
                return super().forward(x, m)

        model.block1[0].__class__ = Block
        with torch.no_grad():
            torch.nn.init.normal_(model.final_conv.bias)
            assert _bias_alone(model, model(*scene))


def test_weights_computed_on_use_and_networks_inside_networks(scene):
    from torch.nn.utils import parametrize

    class Scaled(torch.nn.Module):
        factor = 1.0

        def forward(self, w):
            return w * self.factor

    inner = _model()
    scaled = Scaled()
    parametrize.register_parametrization(inner.final_conv, "weight", scaled)

    class Outer(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.first, self.second = _model(1), inner

        def forward(self, *args):
            a = self.first(*args)
            scaled.factor = 0.0
            return a, self.second(*args)

    net = Outer()
    with torch.no_grad():
        a, b = net(*scene)
        assert _bias_alone(inner, b)
    assert _same(a, net.first(*scene).detach())
    # weights of another type or address than the joined cast takes, and a single one
    net.first.conv1.weight.data = net.first.conv1.weight.data.bfloat16()
    with torch.inference_mode():
        got = net.first(*scene)
    assert _same(got, net.first(*scene).detach())


def _kernels(call):
    from pointelligence_b200 import _cabi

    _cabi.profile_enable(True)
    out = call()
    torch.cuda.synchronize()
    names = [n for n, _ in _cabi.profile_records()]
    _cabi.profile_enable(False)
    return out, names


@pytest.mark.parametrize("C,M,n,grid,per_row,thin", [
    (24, 40, 6000, 0.0362, (13, 26), False), (40, 24, 6000, 0.0362, (13, 26), False), (40, 40, 6000, 0.0362, (13, 26), False),
    (3, 24, 6000, 0.0362, (13, 26), True), (24, 6, 6000, 0.0362, (13, 26), True), (3, 64, 60000, 0.0165, (13, 26), True),
    (64, 6, 60000, 0.0165, (13, 26), True), (3, 64, 60000, 0.023, (28, 60), False)])
def test_padded_widths_choose_their_kernels_like_others(C, M, n, grid, per_row, thin):
    """Dense rulebooks of 27 taps: the output-stationary kernel, which a layer of the next multiples of 16 takes in both
    directions; contractions of up to eight channels take the kernel of thin layers on fewer than a triplet for a row and a tap."""
    from pointelligence_b200.backbone import Bf16PointConv3d
    from pointelligence_b200.layers import MetaData, PointConv3d
    from pointelligence_b200.layers.triplets import handle_stride_and_build_triplets

    g = torch.Generator(device="cuda").manual_seed(C + M)
    pts = torch.rand(n, 3, device="cuda", generator=g)
    m = MetaData(points=pts, sample_inds=torch.zeros(n, dtype=torch.int64, device="cuda"),
                 sample_sizes=torch.tensor([n], device="cuda"), grid_size=grid)
    m = handle_stride_and_build_triplets(m, 1.0, (3, 3, 3), 2.5)
    assert per_row[0] < m.i.numel() / n < per_row[1]
    conv = Bf16PointConv3d(C, M, 3, device="cuda")
    x = torch.randn(n, C, device="cuda", generator=g).bfloat16().requires_grad_()
    go = torch.randn(n, M, device="cuda", generator=g).bfloat16()
    y, forward = _kernels(lambda: conv(x, m.i, m.j, m.k, n, contract=m.contract, seg_offs=m.seg_offs))
    (gx, gw), backward = _kernels(lambda: torch.autograd.grad(y, (x, conv.weight), go))
    convolutions = lambda names: [n.split("(")[0] for n in names if n.startswith(("bucket_sum", "mvmr_"))]
    assert convolutions(forward) == (["mvmr_thin_kernel"] if thin and C <= 8 else ["bucket_sum_kernel", "mvmr_os_kernel"])
    assert convolutions(backward) == (["mvmr_thin_kernel"] if thin and M <= 8 else ["bucket_sum_kernel", "mvmr_os_kernel"])
    w64, x64 = conv.weight.detach().bfloat16().double()[:, 0], x.detach().double()
    ref, gref, wref = torch.zeros(n, M, device="cuda").double(), torch.zeros(n, C, device="cuda").double(), torch.zeros_like(w64)
    for t in range(27):
        s = slice(int(m.seg_offs[t]), int(m.seg_offs[t + 1]))
        ref.index_add_(0, m.i[s].long(), x64[m.j[s].long()] @ w64[t])
        gref.index_add_(0, m.j[s].long(), go[m.i[s].long()].double() @ w64[t].t())
        wref[t] = x64[m.j[s].long()].t() @ go[m.i[s].long()].double()
    # sums of a (row, tap) rounded to bf16, their products summed in fp32, rounded: two roundings of 2^-9
    for a, r in ((y.detach() - conv.bias.detach().bfloat16(), ref), (gx, gref), (gw[:, 0], wref)):
        assert a.shape == r.shape and float((a.double() - r).norm() / r.norm()) < 1.5 * 2.0 ** -8
    # other layers of such widths keep exact operands
    plain = PointConv3d(C, M, 3, device="cuda", dtype=torch.bfloat16)
    _, names = _kernels(lambda: plain(x, m.i, m.j, m.k, n, contract=m.contract, seg_offs=m.seg_offs))
    assert "mvmr_os_kernel" not in convolutions(names)


def test_network_of_padded_widths(scene):
    from pointelligence_b200.backbone import ResUNet

    torch.manual_seed(0)
    model = ResUNet(in_channels=5, num_classes=13, base_channels=24, channels=(24, 40, 40, 72), tr_channels=(24, 40, 56, 72), layers=(1,) * 8).cuda()
    feat = torch.randn(scene[0].shape[0], 5, device="cuda")
    with torch.no_grad():
        got, names = _kernels(lambda: model(feat, *scene[1:4], 0.1))
    assert any(n.startswith("mvmr_os_kernel") for n in names)
    logits = model(feat, *scene[1:4], 0.1)
    assert logits.shape == (feat.shape[0], 13) and _same(got, logits.detach())
    logits.float().square().mean().backward()
    assert all(p.grad is not None and bool(p.grad.isfinite().all()) for p in model.parameters())
