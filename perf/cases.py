"""Performance cases of the point-convolution framework: what its users run, at the sizes they run it.

A case is one call (or one training step) through the public entry points:

``conv``      ``PointConv3d`` over a rulebook the program keeps: a layer of a network, forward only
              (inference) or forward and backward (training)
``rulebook``  the tap-segmented triplets of a cloud, or of its down-sampled cloud: the geometry of one level
``strided``   ``conv_with_stride``: down-sampling, rulebook, convolution and its backward pass
``norm``      ``RaggedLayerNorm`` / ``RaggedGroupNorm`` over a ragged batch, forward and backward
``unet``      the residual U-Net of ``pointelligence_b200.backbone``: logits of a scene, or one training step

Clouds are indoor scenes (points on the surfaces of a furnished room, one per 2 cm voxel) or spinning
64-beam LiDAR sweeps, generated on the GPU from the seed.  ``density`` is points per square metre of
surface: about 670 for a sparsely scanned room, 2500 where every 2 cm voxel of a surface holds a point.
"""
import math

import torch

from pointelligence_b200.backbone import ResUNet
from pointelligence_b200.layers import MetaData, PointConv3d
from pointelligence_b200.layers.conv import conv_with_stride
from pointelligence_b200.layers.norm import RaggedGroupNorm, RaggedLayerNorm
from pointelligence_b200.layers.triplets import handle_stride_and_build_triplets, radius_scaler_for_kernel_size

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
BYTES = {"bf16": 2, "fp16": 2, "fp32": 4}
RFS = 2.5           # receptive field of the networks' convolutions: 5 cm on a 2 cm grid
INDOOR_GRID, LIDAR_GRID = 0.02, 0.05
LIDAR_POINTS = 106_000   # hits of one 64 x 2048 sweep after 10 % dropout
CLASSES = 20


def listed():
    return [
        # one deep layer of a network at serving time: a thousand points, wide rows; latency is what counts
        dict(name="conv_infer_deep", kind="conv", cloud="indoor", points=1000, scenes=1, density=2500.0, kernel=3,
             c_in=256, c_out=256, groups=1, dtype="bf16", train=False),
        # the deepest stage in training: 942 points and 512 channels, fp16, the smallest clouds of a network
        dict(name="conv_train_c512", kind="conv", cloud="indoor", points=942, scenes=1, density=2500.0, kernel=3,
             c_in=512, c_out=512, groups=1, dtype="fp16", train=True),
        # a single fp32 layer on a small uniform cloud: full-precision users, first experiments
        dict(name="conv_train_fp32_20k", kind="conv", cloud="uniform", points=20000, scenes=1, density=0.0, kernel=3,
             c_in=32, c_out=32, groups=1, dtype="fp32", train=True),
        # the stem: few input channels and 125 taps, a ragged batch of two rooms, inference
        dict(name="conv_infer_stem", kind="conv", cloud="indoor", points=80001, scenes=2, density=1500.0, kernel=5,
             c_in=6, c_out=32, groups=1, dtype="bf16", train=False),
        # the benchmark's layer: 150 000 points, 64 channels
        dict(name="conv_train_150k_c64", kind="conv", cloud="indoor", points=150000, scenes=1, density=670.0,
             kernel=3, c_in=64, c_out=64, groups=1, dtype="bf16", train=True),
        # a wide layer on a fully scanned room: bound by the matrix units
        dict(name="conv_train_200k_c256", kind="conv", cloud="indoor", points=200000, scenes=1, density=2500.0,
             kernel=3, c_in=256, c_out=256, groups=1, dtype="bf16", train=True),
        # geometry alone, as every new input pays it: one room, and the first strided level of a batch
        dict(name="rulebook_150k", kind="rulebook", cloud="indoor", points=150000, scenes=1, density=670.0, kernel=3,
             stride=1.0),
        dict(name="rulebook_stride2_1m", kind="rulebook", cloud="indoor", points=1000000, scenes=8, density=1500.0,
             kernel=3, stride=2.0),
        # a strided layer on outdoor sweeps, training
        dict(name="strided_train_lidar", kind="strided", cloud="lidar", points=4 * LIDAR_POINTS, scenes=4,
             density=0.0, kernel=3, stride=2.0, c_in=32, c_out=64, dtype="bf16"),
        # the norm behind every convolution, on a training batch
        dict(name="norm_train_1m_c64", kind="norm", norm="layer", points=1100003, scenes=8, c_in=64, dtype="bf16"),
        # serving: the logits of one small scene, geometry included
        dict(name="unet_infer_40k", kind="unet", points=40000, scenes=1, density=1500.0, train=False),
        # one training step of the network on a batch of eight rooms, geometry included
        dict(name="unet_train_8x130k", kind="unet", points=1040000, scenes=8, density=1500.0, train=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["conv", "rulebook", "strided", "norm", "unet"], [10, 3, 2, 2, 2])[0]
    density = round(math.exp(rng.uniform(math.log(600), math.log(2600))), 1)
    if kind == "conv":
        train = rng.random() < 0.65
        dtype = rng.choices(["bf16", "fp16", "fp32"], [6, 2, 2])[0]
        kernel = rng.choices([3, 5, 1], [8, 1, 1])[0]
        wide = [16, 20, 32, 48, 64, 96, 128, 192, 256]
        c_in, c_out = rng.choice([3, 6] + wide + [384, 512]), rng.choice(wide + [512])
        groups = 2 if c_in % 2 == 0 and c_out % 2 == 0 and rng.random() < 0.08 else 1
        # wide layers sit deep in a network, on few points; fp32 is for the smaller ones
        most = 3e9 / (c_in * c_out) * (0.1 if dtype == "fp32" else 1.0) * (0.3 if kernel == 5 else 1.0)
        points = _log(rng, 500, max(1500, min(500_000, most)))
        return dict(kind=kind, cloud="indoor", points=points, scenes=rng.choice([1, 1, 2, 4]), density=density,
                    kernel=kernel, c_in=c_in, c_out=c_out, groups=groups, dtype=dtype, train=train)
    if kind == "rulebook":
        return dict(kind=kind, cloud="indoor", points=_log(rng, 2000, 1_000_000), scenes=rng.choice([1, 2, 8]),
                    density=density, kernel=rng.choice([3, 3, 5]), stride=rng.choice([1.0, 2.0]))
    if kind == "strided":
        lidar = rng.random() < 0.4
        scenes = rng.randint(1, 4)
        points = scenes * _log(rng, 20_000, LIDAR_POINTS) if lidar else _log(rng, 4000, 400_000)
        return dict(kind=kind, cloud="lidar" if lidar else "indoor", points=points, scenes=scenes,
                    density=0.0 if lidar else density, kernel=3, stride=2.0, c_in=rng.choice([32, 64, 96]),
                    c_out=rng.choice([64, 96, 128]), dtype=rng.choice(["bf16", "bf16", "fp16"]))
    if kind == "norm":
        return dict(kind=kind, norm=rng.choice(["layer", "layer", "group"]), points=_log(rng, 2000, 1_100_000),
                    scenes=rng.choice([1, 4, 8]), c_in=rng.choice([32, 64, 96, 128, 256]),
                    dtype=rng.choice(["bf16", "bf16", "fp32"]))
    if rng.random() < 0.4:
        # training batches; single small scenes are not trained on (their bf16 gradients are mostly rounding)
        return dict(kind=kind, points=_log(rng, 400_000, 1_000_000), scenes=rng.choice([4, 8]),
                    density=max(1500.0, density), train=True)
    return dict(kind=kind, points=_log(rng, 8000, 500_000), scenes=rng.choice([1, 1, 2, 4]), density=density,
                train=False)


# ------------------------------------------------------------------ clouds ----
def _shares(total, scenes):
    """Ragged sizes: between 0.6 and 1.4 times the mean, the same for every seed."""
    w = [0.6 + 0.8 * ((b * 0.618) % 1.0) for b in range(scenes)]
    sizes = [int(total * v / sum(w)) for v in w]
    sizes[0] += total - sum(sizes)
    return sizes


def _first_per_voxel(pts, voxel):
    cell = torch.floor(pts / voxel).to(torch.int64)
    cell -= cell.amin(0)
    ext = cell.amax(0) + 1
    key, order = torch.sort((cell[:, 0] * ext[1] + cell[:, 1]) * ext[2] + cell[:, 2], stable=True)
    head = torch.ones_like(key, dtype=torch.bool)
    head[1:] = key[1:] != key[:-1]
    return pts[order[head]]


def _room(n, density, gen):
    """``n`` points on the surfaces of a furnished room, 5 mm noise, one point per 2 cm voxel."""
    dev = gen.device
    side = math.sqrt(n / density / 25.0)              # room 2s x 2s x s and its furniture: about 25 s^2 of surface
    lo, hi = [[0.0, 0.0, 0.0]], [[2 * side, 2 * side, side]]
    u = torch.rand(20, 5, generator=gen, device=dev).tolist()
    for a, b, c, x, y in u:
        size = [side / 3 * (0.3 + 1.2 * v) for v in (a, b, c)]
        corner = [x * (2 * side - size[0]), y * (2 * side - size[1]), 0.0]
        lo.append(corner)
        hi.append([p + s for p, s in zip(corner, size)])
    lo, hi = torch.tensor(lo, device=dev), torch.tensor(hi, device=dev)
    d = hi - lo
    # faces: (box, axis, side); the furniture stands on the floor
    area = torch.stack([d[:, 1] * d[:, 2], d[:, 0] * d[:, 2], d[:, 0] * d[:, 1]], 1)
    area = torch.stack([area, area], 2)
    area[1:, 2, 0] = 0.0
    cdf = torch.cumsum(area.flatten().double(), 0)
    kept, ask = None, 2 * n
    for _ in range(12):
        f = torch.searchsorted(cdf, torch.rand(ask, generator=gen, device=dev, dtype=torch.float64) * cdf[-1])
        f = f.clamp_(max=cdf.numel() - 1)
        box, axis, top = f // 6, (f // 2) % 3, (f % 2).float()
        p = torch.rand(ask, 3, generator=gen, device=dev)
        p.scatter_(1, axis[:, None], top[:, None])
        p = lo[box] + p * d[box] + 0.005 * torch.randn(ask, 3, generator=gen, device=dev)
        kept = _first_per_voxel(p if kept is None else torch.cat([kept, p]), INDOOR_GRID)
        if kept.shape[0] >= n:
            break
    pick = torch.randperm(kept.shape[0], generator=gen, device=dev)[:n]
    return kept[pick].contiguous()


def _sweep(keep, gen):
    """Hits of a 64-beam sweep over a plane with 40 boxes, of which a share is kept; sensor 1.73 m above the ground."""
    dev = gen.device
    elev = torch.deg2rad(torch.linspace(-25.0, 3.0, 64, device=dev))
    azim = torch.arange(2048, device=dev) * (2 * math.pi / 2048)
    ce, se = torch.cos(elev)[:, None], torch.sin(elev)[:, None].expand(64, 2048)
    rays = torch.stack([ce * torch.cos(azim), ce * torch.sin(azim), se], -1).reshape(-1, 1, 3)
    sensor = torch.tensor([0.0, 0.0, 1.73], device=dev)
    u = torch.rand(40, 5, generator=gen, device=dev)
    r = torch.sqrt(9.0 + u[:, 0] * (2500.0 - 9.0))
    th = 2 * math.pi * u[:, 1]
    size = torch.stack([1 + 4 * u[:, 2], 1 + 2 * u[:, 3], 1 + 2 * u[:, 4]], 1)
    lo = torch.stack([r * torch.cos(th) - size[:, 0] / 2, r * torch.sin(th) - size[:, 1] / 2, 0 * r], 1)
    t1, t2 = (lo - sensor) / rays, (lo + size - sensor) / rays
    near, far = torch.minimum(t1, t2).amax(-1), torch.maximum(t1, t2).amin(-1)
    hit = torch.where((near <= far) & (near > 0), near, torch.full_like(near, float("inf"))).amin(1)
    down = rays[:, 0, 2]
    t = torch.minimum(hit, torch.where(down < 0, -sensor[2] / down, torch.full_like(down, float("inf"))))
    ok = (t <= 80.0) & (torch.rand(t.shape[0], generator=gen, device=dev) < keep)
    return (sensor + rays[ok, 0] * t[ok, None]).contiguous()


def _cloud(case, gen):
    dev = gen.device
    if case["cloud"] == "lidar":
        keep = 0.9 * case["points"] / (case["scenes"] * LIDAR_POINTS)
        clouds = [_sweep(keep, gen) for _ in range(case["scenes"])]
    elif case["cloud"] == "uniform":
        clouds = [torch.rand(case["points"], 3, generator=gen, device=dev)]
    else:
        clouds = [_room(n, case["density"], gen) for n in _shares(case["points"], case["scenes"])]
    sizes = torch.tensor([c.shape[0] for c in clouds], device=dev)
    inds = torch.repeat_interleave(torch.arange(len(clouds), device=dev), sizes)
    return torch.cat(clouds), inds, sizes


def _grid_and_field(case):
    if case["cloud"] == "lidar":
        return LIDAR_GRID, RFS
    if case["cloud"] == "uniform":
        # cell 0.05 and radius 0.075 at kernel size 3
        return 0.05, 4 * math.pi / 3 * 1.5 ** 3 / 27
    return INDOOR_GRID, RFS


# ----------------------------------------------------------------- prepare ----
def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    torch.manual_seed(int(seed))     # parameters of the modules
    return {"conv": _prepare_conv, "rulebook": _prepare_cloud, "strided": _prepare_strided, "norm": _prepare_norm,
            "unet": _prepare_unet}[case["kind"]](case, gen)


def _features(n, width, dtype, gen, grad):
    x = torch.randn(n, width, generator=gen, device=gen.device).to(dtype)
    return x.requires_grad_(grad)


def _prepare_conv(case, gen):
    points, inds, sizes = _cloud(case, gen)
    grid, field = _grid_and_field(case)
    m = MetaData(points=points, sample_inds=inds, sample_sizes=sizes, grid_size=grid, kernel_size=(case["kernel"],) * 3,
                 receptive_field_scaler=field)
    dtype, n = DTYPES[case["dtype"]], points.shape[0]
    conv = PointConv3d(case["c_in"], case["c_out"], case["kernel"], groups=case["groups"], device=gen.device, dtype=dtype)
    return dict(case=case, m=m, conv=conv, x=_features(n, case["c_in"], dtype, gen, case["train"]),
                go=_features(n, case["c_out"], dtype, gen, False))


def _prepare_cloud(case, gen):
    # how many triplets and down-sampled points there are depends on the cloud: it is the case's own, and
    # the seed gives the order in which the scanner delivers its points
    points, inds, sizes = _cloud(case, torch.Generator(device=gen.device).manual_seed(20))
    order = _shuffled(points, inds, 2 * _grid_and_field(case)[0], gen)
    return dict(case=case, points=points[order].contiguous(), inds=inds, sizes=sizes)


def _shuffled(points, inds, cell_size, gen):
    """A random order that stays inside each sample and keeps the points of one cell in sequence, so that
    a tie between two points of a cell falls the same way in every order."""
    n = points.shape[0]
    cell = torch.floor(points / cell_size).to(torch.int64)
    cell -= cell.amin(0)
    ext = cell.amax(0) + 1
    key = ((inds * ext[0] + cell[:, 0]) * ext[1] + cell[:, 1]) * ext[2] + cell[:, 2]
    order = torch.randperm(n, generator=gen, device=gen.device)
    order = order[torch.sort(inds[order], stable=True)[1]]
    places = torch.sort(key[order], stable=True)[1]          # the places of every cell, ascending
    order[places] = torch.sort(key, stable=True)[1]          # ... and its points, as they came
    return order


def _prepare_strided(case, gen):
    s = _prepare_cloud(case, gen)
    dtype = DTYPES[case["dtype"]]
    s["conv"] = PointConv3d(case["c_in"], case["c_out"], case["kernel"], device=gen.device, dtype=dtype)
    s["x"] = _features(s["points"].shape[0], case["c_in"], dtype, gen, True)
    s["go"] = _features(s["points"].shape[0], case["c_out"], dtype, gen, False)
    return s


def _prepare_norm(case, gen):
    dev, dtype, width = gen.device, DTYPES[case["dtype"]], case["c_in"]
    norm = RaggedLayerNorm(width) if case["norm"] == "layer" else RaggedGroupNorm(8, width)
    norm = norm.to(dev)
    with torch.no_grad():
        norm.weight.uniform_(0.5, 1.5)
        norm.bias.uniform_(-0.5, 0.5)
    sizes = torch.tensor(_shares(case["points"], case["scenes"]), device=dev)
    return dict(case=case, norm=norm, sizes=sizes, x=_features(case["points"], width, dtype, gen, True),
                go=_features(case["points"], width, dtype, gen, False))


def _prepare_unet(case, gen):
    points, inds, sizes = _cloud(dict(case, cloud="indoor"), gen)
    with torch.device(gen.device):
        net = ResUNet(in_channels=3, num_classes=CLASSES)
    n = points.shape[0]
    s = dict(case=case, net=net, points=points, inds=inds, sizes=sizes, feat=_features(n, 3, torch.float32, gen, False))
    if case["train"]:
        s["labels"] = torch.randint(0, CLASSES, (n,), generator=gen, device=gen.device)
        # gradients live in one flat buffer, as they do for a bucketed all-reduce
        params = [p for p in net.parameters()]
        s["grads"] = torch.zeros(sum(p.numel() for p in params), device=gen.device)
        at = 0
        for p in params:
            p.grad = s["grads"][at:at + p.numel()].view_as(p)
            at += p.numel()
    return s


# --------------------------------------------------------------------- run ----
def run(s):
    return {"conv": _run_conv, "rulebook": _run_rulebook, "strided": _run_strided, "norm": _run_norm,
            "unet": _run_unet}[s["case"]["kind"]](s)


def _run_conv(s):
    m, conv = s["m"], s["conv"]
    if not s["case"]["train"]:
        with torch.no_grad():
            return conv(s["x"], m.i, m.j, m.k, m.num_points(), contract=m.contract, seg_offs=m.seg_offs)
    y = conv(s["x"], m.i, m.j, m.k, m.num_points(), contract=m.contract, seg_offs=m.seg_offs)
    return (y,) + torch.autograd.grad(y, (s["x"], conv.weight, conv.bias), s["go"])


def _run_rulebook(s):
    case = s["case"]
    grid, field = _grid_and_field(case)
    m = MetaData(points=s["points"], sample_inds=s["inds"], sample_sizes=s["sizes"], grid_size=grid)
    m = handle_stride_and_build_triplets(m, case["stride"], (case["kernel"],) * 3, field)
    return m.points, m.sample_inds, m.sample_sizes, m.i, m.j, m.k, m.seg_offs


def _run_strided(s):
    case, conv = s["case"], s["conv"]
    grid, field = _grid_and_field(case)
    m = MetaData(points=s["points"], sample_inds=s["inds"], sample_sizes=s["sizes"], grid_size=grid)
    y, m = conv_with_stride(conv, s["x"], m, case["stride"], field)
    grads = torch.autograd.grad(y, (s["x"], conv.weight, conv.bias), s["go"][:y.shape[0]])
    return (y, m.points, m.downsample_indices) + grads


def _run_norm(s):
    norm = s["norm"]
    y = norm(s["x"], s["sizes"])
    return (y,) + torch.autograd.grad(y, (s["x"], norm.weight, norm.bias), s["go"])


def _run_unet(s):
    if not s["case"]["train"]:
        with torch.no_grad():
            return s["net"](s["feat"], s["points"], s["inds"], s["sizes"], INDOOR_GRID)
    s["grads"].zero_()
    logits = s["net"](s["feat"], s["points"], s["inds"], s["sizes"], INDOOR_GRID)
    loss = torch.nn.functional.cross_entropy(logits.float(), s["labels"])
    loss.backward()
    return logits.detach(), loss.detach(), s["grads"]


# -------------------------------------------------------------------- work ----
def _neighbours(cloud, points, density, radius):
    """Points within ``radius`` of one: a disc of the surface (more in small rooms, where walls meet), or
    what the LiDAR and uniform clouds measure."""
    if cloud == "lidar":
        return 9.2
    if cloud == "uniform":
        return 33.4
    return 1.0 + density * math.pi * radius * radius * (1.05 + 1.8 * radius / math.sqrt(points / density / 25.0))


def _levels(points, density, grid, count):
    """(points, density, grid) of every level of a pyramid of stride-2 centre-nearest down-sampling."""
    out = [(points, density, grid)]
    for _ in range(count - 1):
        grid *= 2
        kept = min(density, 1.4 / (grid * grid))      # about 1.4 occupied cells per cell face of a noisy surface
        points, density = points * kept / density, kept
        out.append((points, density, grid))
    return out


def work(case):
    kind, n = case["kind"], case["points"]
    if kind == "norm":
        # forward: x in, y out; backward: gradient and x in, gradient out
        return {"bytes": 5.0 * n * case["c_in"] * BYTES[case["dtype"]], "flops": 16.0 * n * case["c_in"]}
    if kind == "unet":
        lv = _levels(n, case["density"], INDOOR_GRID, 4)
        radius = radius_scaler_for_kernel_size(3, RFS)
        room = n / case["scenes"]
        t = [p * _neighbours("indoor", p / case["scenes"], d, g * radius) for p, d, g in lv]
        t5 = n * _neighbours("indoor", room, case["density"], INDOOR_GRID * radius_scaler_for_kernel_size(5, RFS))
        convs = [(t5, 3, 32), (t[0], 32, 32, 4)]
        convs += [(t[0] * lv[1][0] / n, 32, 64), (t[1], 64, 64, 3), (t[1] * lv[2][0] / lv[1][0], 64, 128),
                  (t[2], 128, 128, 3), (t[2] * lv[3][0] / lv[2][0], 128, 256), (t[3], 256, 256, 3)]
        up = [p[0] * _neighbours("indoor", q[0] / case["scenes"], q[1], q[2] * radius) for p, q in zip(lv, lv[1:])]
        convs += [(up[2], 256, 256), (t[2], 256, 256, 4), (up[1], 384, 128), (t[1], 128, 128, 4), (up[0], 192, 96),
                  (t[0], 96, 96, 4), (t[0], 128, 96), (n, 96, CLASSES)]
        flops = sum(2.0 * c[0] * c[1] * c[2] * (c[3] if len(c) > 3 else 1) for c in convs)
        passes = 3 if case["train"] else 1
        rows = sum(p * w for (p, _, _), w in zip(lv, (32 * 5 + 96 * 5, 64 * 4 + 128 * 5, 128 * 4 + 256 * 5, 256 * 4)))
        index = 12.0 * (t5 + sum(t) + sum(up) + t[0] * lv[1][0] / n + n)
        return {"bytes": rows * 4.0 * passes + index + 22.8e6 * (8 if case["train"] else 4), "flops": flops * passes}
    grid, field = _grid_and_field(case)
    radius = grid * radius_scaler_for_kernel_size(case["kernel"], field)
    per_point = _neighbours(case["cloud"], n / case["scenes"], case["density"], radius)
    n_out = n
    if case.get("stride", 1.0) != 1.0:
        n_out = 0.39 * n if case["cloud"] == "lidar" else _levels(n, case["density"], grid, 2)[1][0]
    t, taps = n_out * per_point, case["kernel"] ** 3
    geometry = 20.0 * n + (28.0 * n_out if n_out != n else 0.0) + 12.0 * t + 8.0 * (taps + 1)
    if kind == "rulebook":
        return {"bytes": geometry, "flops": 8.0 * t}
    e, c_in, c_out = BYTES[case["dtype"]], case["c_in"], case["c_out"]
    weight = taps * c_in * c_out / case.get("groups", 1)
    flops = 2.0 * t * c_in * c_out / case.get("groups", 1)
    moved = (n * c_in + n_out * c_out + weight) * e
    if kind == "strided":
        return {"bytes": geometry + 2 * moved, "flops": 3 * flops}
    return {"bytes": 8.0 * t + (2 if case["train"] else 1) * moved, "flops": (3 if case["train"] else 1) * flops}


def tolerance(case):
    if case["kind"] == "rulebook":
        return "exact"
    if case["kind"] == "unet":
        # some forty roundings to bf16 in a row, and the gradients' way back
        return {"rel": 2e-2, "max": 0.6}
    return {"rel": {"bf16": 1e-2, "fp16": 2e-3, "fp32": 1e-5}[case["dtype"]]}
