"""The work that the performance of this framework is measured on: what a user's program
has it do, through the public entry points, over the sizes and types that are in use.

    voxelize   raw points of one or more scans -> sorted unique voxels, their mean features
               and, for a loader that maps predictions back, the voxel of every point
    maps       output coordinates and kernel maps of a new input (a cold KernelMapCache)
    conv       one sparse convolution, forward, its map already in the cache
    conv_step  one sparse convolution, forward and backward (training), map in the cache
    unet       inference of the sparse UNet on a new input: all maps, all layers
    unet_step  one training step of the sparse UNet on a new input up to its gradients

Clouds are drawn on the GPU with the geometry of ``minuet_b200.synth``: uniform voxels in
a cube, outdoor scans (noisy ground plane, boxes, range-dependent dropout) and indoor rooms
(walls, boxes, spheres).  Smaller clouds come from coarser voxels, so that the voxels keep
about the same number of neighbours.
"""
import math
import random

import torch

import minuet_b200 as minuet
from minuet_b200.nn import functional as F
from minuet_b200.unet import SparseUNet

DEVICE = "cuda:0"
DTYPES = {"float32": torch.float32, "float16": torch.float16, "bfloat16": torch.bfloat16}
FULL_WIDTH = (32, 64, 128, 256)
HALF_WIDTH = (16, 32, 64, 128)

# Of a cloud's voxels: the share that is left at strides 1, 2, 4, 8, 16, and the 3x3x3
# neighbours of a voxel (itself among them) there; the neighbours in a 3x3x3 window with
# stride 2; the voxels that a scan's points fill, per point.
ROWS = {"outdoor": (1.0, 0.97, 0.87, 0.62, 0.24), "indoor": (1.0, 0.72, 0.28, 0.065, 0.013),
        "uniform": (1.0, 0.99, 0.91, 0.52, 0.09)}
NEIGHBOURS = {"outdoor": (1.15, 1.65, 3.6, 10.0, 16.5), "indoor": (3.0, 7.0, 12.0, 14.0, 15.0),
              "uniform": (1.07, 1.6, 5.2, 19.5, 24.0)}
STRIDED3 = {"outdoor": 1.1, "indoor": 1.85, "uniform": 1.05}
FILLED = {"outdoor": 0.96, "indoor": 0.88}


def listed():
    return [
        # one sweep of an outdoor scanner as it arrives: xyz + intensity
        {"name": "voxelize_sweep", "call": "voxelize", "scene": "outdoor", "clouds": 1,
         "voxels": 120_000, "channels": 4, "inverse": False, "dtype": "float32"},
        # a loader's batch of indoor scans with colour; predictions go back to the points
        {"name": "voxelize_rooms", "call": "voxelize", "scene": "indoor", "clouds": 8,
         "voxels": 250_001, "channels": 6, "inverse": True, "dtype": "float32"},
        # the smallest map in use: one small cloud, where launches and host time count
        {"name": "maps_small", "call": "maps", "scene": "uniform", "clouds": 1,
         "voxels": 3_001, "geometry": "submanifold", "int64": False},
        # the map benchmark: four outdoor clouds, (3,s1) (2,s1) (3,s2) (2,s2)
        {"name": "maps_four_scans", "call": "maps", "scene": "outdoor", "clouds": 4,
         "voxels": 120_000, "geometry": "four", "int64": False},
        # the maps of a large batch: 3x3x3 at stride 1 and the way down to stride 2
        {"name": "maps_batch", "call": "maps", "scene": "outdoor", "clouds": 64,
         "voxels": 120_000, "geometry": "level", "int64": False},
        # the single-layer configuration: 50 000 uniform voxels, 32 -> 32, fp32
        {"name": "conv_fp32", "call": "conv", "scene": "uniform", "clouds": 1,
         "voxels": 50_000, "dtype": "float32", "c_in": 32, "c_out": 32, "kernel": 3,
         "stride": 1, "transposed": False, "epilogue": False},
        # a middle layer of inference in half precision, BatchNorm, skip and ReLU folded in
        {"name": "conv_fp16", "call": "conv", "scene": "outdoor", "clouds": 4,
         "voxels": 120_000, "dtype": "float16", "c_in": 64, "c_out": 64, "kernel": 3,
         "stride": 1, "transposed": False, "epilogue": True},
        # a downsampling layer on a ragged indoor batch in bf16
        {"name": "conv_down_bf16", "call": "conv", "scene": "indoor", "clouds": 3,
         "voxels": 77_777, "dtype": "bfloat16", "c_in": 64, "c_out": 128, "kernel": 2,
         "stride": 2, "transposed": False, "epilogue": False},
        # a layer in mixed-precision training
        {"name": "conv_step_fp16", "call": "conv_step", "scene": "indoor", "clouds": 2,
         "voxels": 100_003, "dtype": "float16", "c_in": 64, "c_out": 64, "kernel": 3,
         "stride": 1, "transposed": False},
        # inference on one scan as it arrives: latency counts
        {"name": "unet_scan", "call": "unet", "scene": "outdoor", "clouds": 1,
         "voxels": 120_000, "dtype": "float16", "width": "full", "fused": True},
        # inference on a large batch: throughput counts
        {"name": "unet_batch", "call": "unet", "scene": "outdoor", "clouds": 64,
         "voxels": 120_000, "dtype": "float16", "width": "full", "fused": True},
        # training in the precision that modules have by default
        {"name": "unet_step", "call": "unet_step", "scene": "indoor", "clouds": 2,
         "voxels": 30_011, "dtype": "float32", "width": "full"},
    ]


def draw(rng):
    def sizes(low, high, most_clouds, total):
        voxels = int(math.exp(rng.uniform(math.log(low), math.log(high))))
        clouds = int(round(math.exp(rng.uniform(0.0, math.log(most_clouds)))))
        return {"clouds": max(1, min(clouds, total // voxels)), "voxels": voxels}

    def layer(kernel_stride):
        channels = (16, 32, 48, 64, 96, 128, 192, 256)
        kernel, stride = kernel_stride
        c_in = rng.choice(channels)
        return {"c_in": c_in, "c_out": rng.choice([c for c in channels if c_in // 4 <= c <= c_in * 4]),
                "kernel": kernel, "stride": stride, "transposed": stride > 1 and rng.random() < 0.5}

    call = rng.choice(("voxelize", "maps", "conv", "conv", "conv_step", "unet", "unet_step"))
    scene = rng.choice(("outdoor", "indoor"))
    geometries = ((3, 1), (3, 1), (3, 1), (2, 2), (3, 2))
    if call == "voxelize":
        return {"call": call, "scene": scene, **sizes(2_000, 250_000, 32, 4_000_000),
                "channels": rng.choice((1, 3, 4, 6, 9)), "inverse": rng.random() < 0.5,
                "dtype": rng.choice(("float32", "float32", "float16"))}
    if call == "maps":
        return {"call": call, "scene": rng.choice(("outdoor", "indoor", "uniform")),
                **sizes(1_000, 250_000, 64, 7_000_000),
                "geometry": rng.choice(("submanifold", "four", "level", "encoder")),
                "int64": rng.random() < 0.2}
    if call == "conv":
        return {"call": call, "scene": rng.choice(("outdoor", "indoor", "uniform")),
                **sizes(1_000, 200_000, 16, 1_000_000),
                "dtype": rng.choice(("float32", "float16", "float16", "bfloat16")),
                **layer(rng.choice(geometries)), "epilogue": rng.random() < 0.5}
    if call == "conv_step":
        return {"call": call, "scene": scene, **sizes(1_000, 100_000, 8, 300_000),
                "dtype": rng.choice(("float32", "float16", "bfloat16")),
                **layer(rng.choice(geometries))}
    if call == "unet":
        dtype = rng.choice(("float16", "float16", "float16", "float32"))
        return {"call": call, "scene": scene,
                **sizes(2_000, 200_000, 64, 4_000_000 if dtype == "float16" else 200_000),
                "dtype": dtype, "width": rng.choice(("full", "full", "half")),
                "fused": rng.random() < 0.75}
    return {"call": call, "scene": scene, **sizes(1_000, 60_000, 4, 60_000), "dtype": "float32",
            "width": rng.choice(("full", "half"))}


# ---------------------------------------------------------------------------
# clouds: what a scene looks like follows from its size and its place in the batch, and the
# seed poses it (heading, mirror, place on the grid, order of clouds and points, place of a
# point inside its voxel), so that different inputs of one case have equally many voxels at
# every stride
# ---------------------------------------------------------------------------

def _rand(gen, *shape):
    return torch.rand(*shape, generator=gen, device=DEVICE)


def _cloud_sizes(case):
    """Voxels (or points) of every cloud: up to a tenth fewer than the case says."""
    n = case["voxels"]
    return [n - (37 * i % 11) * n // 100 for i in range(case["clouds"])]


def _surfaces(gen, centres, sides, count):
    """``count`` points on the surfaces of axis-aligned boxes, even in area."""
    sx, sy, sz = sides.unbind(1)
    areas = torch.stack([sy * sz, sx * sz, sx * sy], 1)
    which = torch.multinomial(areas.reshape(-1), count, replacement=True, generator=gen)
    box, axis = which // 3, which % 3
    p = _rand(gen, count, 3) - 0.5
    side = (_rand(gen, count) < 0.5).float() - 0.5
    p.scatter_(1, axis[:, None], side[:, None])
    return p * sides[box] + centres[box]


def _outdoor_points(gen, count):
    ground = torch.cat([_rand(gen, int(4.5 * count), 2) * 100.0 - 50.0,
                        torch.randn(int(4.5 * count), 1, generator=gen, device=DEVICE) * 0.1], 1)
    sides = _rand(gen, 200, 3) * 9.0 + 1.0
    sides[:, 2].clamp_(max=3.5)
    centres = torch.cat([_rand(gen, 200, 2) * 100.0 - 50.0, sides[:, 2:] / 2 - 0.5], 1)
    points = torch.cat([ground, _surfaces(gen, centres, sides, 8 * count)])
    reach = points[:, 0].hypot(points[:, 1])
    keep = (_rand(gen, len(points)) >= (reach / 60.0).clamp(max=0.9)) & \
        (points[:, :2].abs().amax(1) < 50.0)
    points = points[keep]
    points[:, 2].clamp_(-3.0, 1.0 - 1e-6)
    return points


def _indoor_points(gen, count):
    room = torch.tensor([8.0, 8.0, 3.0], device=DEVICE)
    walls = _surfaces(gen, room[None] / 2, room[None], int(2.2 * count))
    sides = _rand(gen, 15, 3) * 1.7 + 0.3
    at = _rand(gen, 30, 2) * 7.0 + 0.5
    boxes = _surfaces(gen, torch.cat([at[:15], sides[:, 2:] / 2], 1), sides, int(1.3 * count))
    radius = _rand(gen, 15, 1) * 0.85 + 0.15
    which = torch.multinomial(radius.square()[:, 0], int(1.5 * count), replacement=True, generator=gen)
    way = torch.randn(len(which), 3, generator=gen, device=DEVICE)
    way = way / way.norm(dim=1, keepdim=True).clamp(min=1e-6)
    balls = torch.cat([at[15:], radius], 1)[which] + way * radius[which]
    return torch.minimum(torch.cat([walls, boxes, balls]).clamp(min=0.0), room - 1e-6)


def _voxel_size(scene, count):
    if scene == "outdoor":
        return 0.05 * math.sqrt(max(1.0, 120_000 / count))
    return 0.02 * math.sqrt(max(1.0, 200_000 / count))


def _sorted_rows(cells):
    """Unique rows of int64 cells in lexicographic order (each within +-8192)."""
    c = cells + 8192
    keys = torch.unique((c[:, 0] << 28) + (c[:, 1] << 14) + c[:, 2])
    return torch.stack([keys >> 28, keys >> 14 & 16383, keys & 16383], 1) - 8192


def _cells(scene, count, i, unique):
    """The cells of cloud ``i``: ``count`` distinct ones, or those of ``count`` points."""
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(1000 * count + i)
    if scene == "uniform":
        extent = round(256 * (count / 50_000) ** (1 / 3)) + 1
        keys = torch.randperm(extent ** 3, generator=gen, device=DEVICE)[:count]
        return torch.stack([keys // (extent * extent), keys // extent % extent, keys % extent], 1)
    points = (_outdoor_points if scene == "outdoor" else _indoor_points)(gen, count)
    cells = torch.floor(points / _voxel_size(scene, count)).to(torch.int64)
    if unique:
        cells = _sorted_rows(cells)
    return cells[torch.randperm(len(cells), generator=gen, device=DEVICE)[:count]]


def _posed(cells, rng):
    """The same cloud with another heading, mirrored or not, elsewhere on the grid."""
    x, y, z = cells.unbind(1)
    x, y = (x, y) if rng.random() < 0.5 else (y, x)
    x, y = (-1 - v if rng.random() < 0.5 else v for v in (x, y))
    return torch.stack([x + 16 * rng.randint(-64, 64), y + 16 * rng.randint(-64, 64), z], 1)


def _clouds(case, seed, unique):
    rng = random.Random(seed)
    sizes = _cloud_sizes(case)
    clouds = [_posed(_cells(case["scene"], n, i, unique), rng) for i, n in enumerate(sizes)]
    rng.shuffle(clouds)
    return clouds


def _batch(clouds):
    """Clouds one after the other and their bounds (None for a single one)."""
    bounds = [0]
    for c in clouds:
        bounds.append(bounds[-1] + len(c))
    return torch.cat(clouds), (torch.tensor(bounds, device=DEVICE) if len(clouds) > 1 else None)


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------

class _State:
    pass


def _new_cache(int64=False):
    return minuet.nn.KernelMapCache(ndim=3, dtype=torch.int64 if int64 else torch.int32, device=DEVICE)


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    torch.manual_seed(seed)          # the modules' own initialisation
    call, scene = case["call"], case["scene"]
    s = _State()
    s.case = case
    dtype = DTYPES[case.get("dtype", "float32")]
    if call == "voxelize":
        s.voxel = _voxel_size(scene, case["voxels"])
        clouds = [(c + 0.05 + 0.9 * _rand(gen, *c.shape))[torch.randperm(
            len(c), generator=gen, device=DEVICE)] for c in _clouds(case, seed, unique=False)]
        s.points, s.bounds = _batch([(c * s.voxel).float() for c in clouds])
        s.features = _rand(gen, len(s.points), case["channels"]).to(dtype)
        return s

    coords, s.bounds = _batch([_sorted_rows(c) for c in _clouds(case, seed, unique=True)])
    s.coords = coords if case.get("int64") else coords.to(torch.int32)
    s.cache = _new_cache(case.get("int64", False))
    if call == "maps":
        return s

    if call in ("conv", "conv_step"):
        kernel, stride, c_in, c_out = case["kernel"], case["stride"], case["c_in"], case["c_out"]
        down = minuet.nn.SparseConv3d(c_in, c_out, kernel, stride=stride, dtype=dtype, device=DEVICE)
        minuet.set_kernel_map_cache(down, s.cache)
        at, at_stride, at_bounds = s.coords, 1, s.bounds
        if case["transposed"]:
            # the layer that a decoder has: back to the voxels of its downsampling twin
            at, at_stride, at_bounds = down.prepare(s.coords, 1, s.bounds)
            s.layer = minuet.nn.SparseConv(3, c_in, c_out, kernel, stride=stride, transposed=True,
                                           dtype=dtype, device=DEVICE)
            minuet.set_kernel_map_cache(s.layer, s.cache)
        else:
            s.layer = down
        out_coords, _, _ = s.layer.prepare(at, at_stride, at_bounds)
        features = torch.randn(len(at), c_in, generator=gen, device=DEVICE).to(dtype)
        if call == "conv":
            s.layer.eval()
            s.scale = s.shift = s.skip = None
            if case["epilogue"]:
                s.scale, s.shift = _rand(gen, c_out) + 0.5, _rand(gen, c_out) - 0.5
                s.skip = torch.randn(len(out_coords), c_out, generator=gen, device=DEVICE).to(dtype)
        else:
            features.requires_grad_()
            s.grad = torch.randn(len(out_coords), c_out, generator=gen, device=DEVICE).to(dtype)
        s.x = minuet.SparseTensor(features, at, stride=at_stride, batch_dims=at_bounds)
        return s

    # the networks: position and intensity outdoors, colour indoors
    n = len(s.coords)
    features = _rand(gen, n, 4 if scene == "outdoor" else 3)
    if scene == "outdoor":
        features[:, :3] = s.coords * (_voxel_size(scene, case["voxels"]) / 50.0)
    net = SparseUNet(features.shape[1], num_classes=20,
                     channels=FULL_WIDTH if case["width"] == "full" else HALF_WIDTH,
                     stem_channels=32 if case["width"] == "full" else 16).to(DEVICE)
    for m in net.modules():
        if isinstance(m, minuet.nn.BatchNorm):
            m.running_mean.uniform_(-0.2, 0.2)
            m.running_var.uniform_(0.5, 1.5)
            torch.nn.init.uniform_(m.weight, 0.5, 1.5)
            torch.nn.init.uniform_(m.bias, -0.2, 0.2)
    minuet.set_kernel_map_cache(net, s.cache)
    s.net = net.to(dtype)
    if call == "unet":
        s.net.eval()
        if case["fused"]:
            s.net.fuse()
    else:
        s.net.train()
        s.labels = torch.randint(0, 20, (n,), generator=gen, device=DEVICE)
    s.x = minuet.SparseTensor(features.to(dtype), s.coords, batch_dims=s.bounds)
    return s


def _run_maps(s):
    """(kernel, stride) maps, each level's output coordinates found on the way."""
    s.cache.reset()
    out = []

    def one(coords, stride, bounds, kernel, kernel_stride):
        to, to_stride, to_bounds = s.cache.get_target_coordinates(coords, bounds, stride, kernel_stride)
        out.append(s.cache.get_kernel_map(coords, stride, bounds, to, to_stride, to_bounds, kernel, 1))
        if kernel_stride != 1:
            out.append((to, to_bounds))
        return to, to_stride, to_bounds

    at = (s.coords, 1, s.bounds)
    geometry = s.case["geometry"]
    if geometry == "four":
        for kernel, stride in ((3, 1), (2, 1), (3, 2), (2, 2)):
            one(*at, kernel, stride)
        return out
    one(*at, 3, 1)
    for _ in range({"submanifold": 0, "level": 1, "encoder": 4}[geometry]):
        at = one(*at, 2, 2)
        if geometry == "encoder":
            one(*at, 3, 1)
    return out


def run(s):
    call = s.case["call"]
    if call == "voxelize":
        return F.voxelize(s.points, s.voxel, batch_dims=s.bounds, return_inverse=s.case["inverse"],
                          features=s.features)
    if call == "maps":
        return _run_maps(s)
    if call == "conv":
        with torch.no_grad():
            if s.case["epilogue"]:
                return s.layer.forward_fused(s.x, scale=s.scale, shift=s.shift, residual=s.skip,
                                             relu=True).F
            return s.layer(s.x).F
    if call == "conv_step":
        out = s.layer(s.x).F
        return (out.detach(), *torch.autograd.grad(out, (s.x.F, s.layer.kernel), s.grad))
    if call == "unet":
        s.cache.reset()
        with torch.no_grad():
            return s.net(s.x).F
    s.cache.reset()
    out = s.net(s.x).F
    loss = torch.nn.functional.cross_entropy(out, s.labels)
    # one vector of all gradients, as a data-parallel program reduces them
    grads = torch.autograd.grad(loss, tuple(s.net.parameters()))
    return loss.detach(), out.detach(), torch.nn.utils.parameters_to_vector(grads)


# ---------------------------------------------------------------------------
# what the calls cannot do without
# ---------------------------------------------------------------------------

def _map_work(sources, targets, offsets, coord_bytes=4):
    """Both coordinate sets read, both masks, the sizes and the order written."""
    return 3 * coord_bytes * (sources + targets) + 4 * offsets * (sources + targets + 2)


def _layer_work(sources, targets, pairs, offsets, c_in, c_out, size):
    """Features, weights and the pairs' rows read once, the output written once."""
    return (size * (sources * c_in + targets * c_out + offsets * c_in * c_out) + 4 * pairs,
            2.0 * pairs * c_in * c_out)


def _unet_layers(case, n):
    """(sources, targets, pairs, offsets, c_in, c_out) of every convolution of the UNet."""
    rows = [n * r for r in ROWS[case["scene"]]]
    near = [a * b for a, b in zip(rows, NEIGHBOURS[case["scene"]])]
    widths = FULL_WIDTH if case["width"] == "full" else HALF_WIDTH
    stem = widths[0]
    layers = [(n, n, near[0], 27, 4 if case["scene"] == "outdoor" else 3, stem)]
    prev = stem
    for level, c in enumerate(widths):
        layers.append((rows[level], rows[level + 1], rows[level], 8, prev, c))
        layers += 4 * [(rows[level + 1], rows[level + 1], near[level + 1], 27, c, c)]
        prev = c
    for level, c in reversed(list(enumerate((stem,) + widths[:-1]))):
        r = rows[level]
        layers.append((rows[level + 1], r, r, 8, prev, c))
        layers.append((r, r, near[level], 27, 2 * c, c))
        layers += 3 * [(r, r, near[level], 27, c, c)]
        layers.append((r, r, r, 1, 2 * c, c))
        prev = c
    layers.append((n, n, n, 1, prev, 20))
    return layers


def work(case):
    call, scene = case["call"], case["scene"]
    n = float(sum(_cloud_sizes(case)))
    size = 4 if case.get("dtype", "float32") == "float32" else 2
    if call == "voxelize":
        filled = FILLED[scene] * n
        return {"bytes": n * (12 + size * case["channels"] + (8 if case["inverse"] else 0)) +
                filled * (12 + size * case["channels"]), "flops": n * (6 + case["channels"])}
    rows = [n * r for r in ROWS[scene]]
    if call == "maps":
        size = 8 if case["int64"] else 4
        if case["geometry"] == "four":
            parts = [(n, n, 27), (n, n, 8), (n, rows[1], 27), (n, rows[1], 8)]
        else:
            parts = [(n, n, 27)]
            for level in range({"submanifold": 0, "level": 1, "encoder": 4}[case["geometry"]]):
                parts.append((rows[level], rows[level + 1], 8))
                if case["geometry"] == "encoder":
                    parts.append((rows[level + 1], rows[level + 1], 27))
        return {"bytes": sum(_map_work(*p, size) for p in parts), "flops": 0.0}
    if call in ("conv", "conv_step"):
        offsets = case["kernel"] ** 3
        sources, targets = n, n if case["stride"] == 1 else rows[1]
        pairs = n * NEIGHBOURS[scene][0] if case["stride"] == 1 else \
            n if case["kernel"] == 2 else n * STRIDED3[scene]
        if case["transposed"]:
            sources, targets = targets, sources
        c_in, c_out = case["c_in"], case["c_out"]
        moved, flops = _layer_work(sources, targets, pairs, offsets, c_in, c_out, size)
        if call == "conv":
            return {"bytes": moved + (size * targets * c_out if case["epilogue"] else 0), "flops": flops}
        # backward: the output's gradient, the features and the weights read, the gradients of
        # features and weights written
        back = size * (targets * c_out + 2 * sources * c_in + 2 * offsets * c_in * c_out) + 4 * pairs
        return {"bytes": moved + back, "flops": 3 * flops}
    # a network: every layer's features once in each direction, its maps once
    layers = _unet_layers(case, n)
    moved = flops = 0.0
    for layer in layers:
        b, f = _layer_work(*layer, size)
        moved, flops = moved + b, flops + f
    maps = sum(12 * (s + t) + 4 * e for s, t, e in {layer[:3] for layer in layers if layer[3] > 1})
    if call == "unet_step":
        moved, flops = 3 * moved, 3 * flops
    return {"bytes": moved + maps, "flops": flops}


def tolerance(case):
    call, dtype = case["call"], case.get("dtype", "float32")
    if call == "maps":
        return "exact"
    if call == "voxelize":
        # whole numbers the same, means within the rounding of the feature type
        return {"rel": 1e-5 if dtype == "float32" else 1e-3, "differ": 0.0}
    if call in ("conv", "conv_step"):
        return {"rel": {"float32": 1e-5, "float16": 2e-3, "bfloat16": 1e-2}[dtype]}
    if call == "unet_step":
        # some eighty layers there and back, each with sums of 32 bits
        return {"rel": 1e-4, "max": 2e-2}
    return {"rel": 1e-4 if dtype == "float32" else 1e-2}
