"""The workloads that this library's speed is judged by: what a program that
trains or renders 3D Gaussian scenes calls, over the sizes it calls it with.

listed() names them, draw() gives more of the same ranges, prepare() makes what
such a program holds before the call, run() is one call, work() what the call
cannot do without, and exact() the same outputs from plain torch in 64 bits.

Every input comes from the seed alone and is drawn on the GPU. Two kinds of
scene stand for real ones, with the distributions of diorama_gb300/scenes.py:
Gaussians on planes and boxes seen from a ring of cameras (a captured scene),
and Gaussians filling a box seen from a sphere (a dense random one).
"""

from __future__ import annotations

import math
import random
from dataclasses import replace

import numpy as np
import torch

from diorama_gb300 import (DEFAULT_SETTINGS, CameraData, DensifyMLP, Device, GaussianRenderer, PrefixSum, RadixSort,
                           RawGaussians, Trainer, TrainingLoss, TrainingView, meanNeighborDistance2Buffers)
from diorama_gb300.mat4 import lookAt, perspective

SH_C0 = 0.28209479177387814
VIEWS = 8  # photos of a training case
EXTENT = 4.0  # training's scene extent


# ------------------------------------------------------------------ the cases

def listed() -> list[dict]:
    return [
        # A training step of a full captured scene at the photos' size, every SH degree in use: the
        # steady state after densification, where most of a training run's time goes.
        {"name": "train_1100k_980x545", "kind": "train", "count": 1_100_000, "width": 980, "height": 545, "degree": 3},
        # A training step near the start of a run: the first 100,000 points, SH degree 1.
        {"name": "train_100k_980x545", "kind": "train", "count": 100_000, "width": 980, "height": 545, "degree": 1},
        # A training step of a small object at a ragged photo size (a preview, a test): launches count.
        {"name": "train_5k_251x187", "kind": "train", "count": 5_003, "width": 251, "height": 187, "degree": 2},
        # One frame of a dense scene at the viewer's full size: 26M (tile, splat) pairs.
        {"name": "frame_1100k_1960x1090", "kind": "frame", "count": 1_100_000, "width": 1960, "height": 1090,
         "degree": 3},
        # One frame of a small scene: interactive viewing, latency.
        {"name": "frame_16k_256x256", "kind": "frame", "count": 16_384, "width": 256, "height": 256, "degree": 3},
        # Render, loss and all gradients for a caller with its own optimizer, at a ragged size.
        {"name": "gradients_201k_489x273", "kind": "gradients", "count": 201_003, "width": 489, "height": 273,
         "degree": 2},
        # The held-out views of a scene in one batched call.
        {"name": "views_12x300k_490x272", "kind": "views", "count": 300_000, "width": 490, "height": 272, "degree": 3,
         "views": 12},
        # The training loss and its gradient alone, at a large photo size.
        {"name": "loss_1957x1091", "kind": "loss", "width": 1957, "height": 1091},
        # The stable sort of (tile, depth) keys, as a tile rasterizer of one's own would call it.
        {"name": "sort_4200k_48bit", "kind": "sort", "count": 4_200_000, "high_bits": 16},
        # The prefix sum of per-splat tile counts.
        {"name": "scan_1100k", "kind": "scan", "count": 1_100_000},
        # Neighbour distances of a structure-from-motion cloud: training's starting sizes.
        {"name": "neighbours_180k", "kind": "neighbours", "count": 180_000},
        # The learned densification's scores for the candidates of one densification.
        {"name": "scores_300k", "kind": "scores", "count": 300_007},
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    """An integer of [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _size(rng: random.Random, lo: int, hi_width: int, hi_height: int) -> dict:
    """A photo size between lo pixels and the largest each way, ragged ones mostly."""
    width = _log_int(rng, lo, hi_width)
    return {"width": width, "height": max(lo // 2, min(hi_height, round(width * rng.uniform(0.5, 1.0))))}


def draw(rng: random.Random) -> dict:
    # Training and rendering are most of what a program does.
    kind = rng.choice(["train", "train", "train", "frame", "frame", "gradients", "views", "loss", "sort", "scan",
                       "neighbours", "scores"])
    if kind == "train":
        return {"kind": kind, "count": _log_int(rng, 2_000, 1_100_000), **_size(rng, 128, 980, 545),
                "degree": rng.randint(0, 3)}
    if kind == "frame":
        return {"kind": kind, "count": _log_int(rng, 4_000, 1_100_000), **_size(rng, 192, 1960, 1090),
                "degree": rng.randint(0, 3)}
    if kind == "gradients":
        return {"kind": kind, "count": _log_int(rng, 4_000, 600_000), **_size(rng, 128, 980, 545),
                "degree": rng.randint(0, 3)}
    if kind == "views":
        return {"kind": kind, "count": _log_int(rng, 10_000, 300_000), **_size(rng, 128, 490, 272),
                "degree": rng.randint(0, 3), "views": rng.randint(2, 12)}
    if kind == "loss":
        return {"kind": kind, **_size(rng, 96, 1957, 1091)}
    if kind == "sort":
        return {"kind": kind, "count": _log_int(rng, 20_000, 4_200_000), "high_bits": rng.choice([0, 16])}
    if kind == "scan":
        return {"kind": kind, "count": _log_int(rng, 20_000, 12_000_000)}
    if kind == "neighbours":
        return {"kind": kind, "count": _log_int(rng, 10_000, 1_100_000)}
    return {"kind": "scores", "count": _log_int(rng, 5_000, 1_100_000)}


# ------------------------------------------------------------------ inputs

def _gpu() -> torch.device:
    return torch.device("cuda")


def _generator(seed: int, stream: int = 0) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(1_000_003 * seed + stream)


def _normal(gen, shape, mean=0.0, std=1.0):
    return torch.randn(shape, generator=gen, device="cuda") * std + mean


def _uniform(gen, shape, lo=0.0, hi=1.0):
    return torch.rand(shape, generator=gen, device="cuda") * (hi - lo) + lo


def _rotations(q):
    """Rotation matrices of unit quaternions (w, x, y, z)."""
    w, x, y, z = q.unbind(-1)
    return torch.stack([
        1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
        2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
        2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], -1).reshape(*q.shape[:-1], 3, 3)


def _unit(v):
    return v / v.square().sum(-1, keepdim=True).sqrt()


def _surface_scene(count: int, seed: int):
    """Raw parameters (count x 16) and SH (count x 45) of Gaussians on 40 planes and boxes."""
    gen, shapes = _generator(seed, 1), 40
    kinds = _uniform(gen, (shapes,)) < 0.5
    centers = _uniform(gen, (shapes, 3), -1.2, 1.2)
    sizes = _uniform(gen, (shapes, 3), 0.15, 0.6)
    rot = _rotations(_unit(_normal(gen, (shapes, 4))))
    palette = _normal(gen, (shapes, 3), 0.0, 0.8)
    which = torch.randint(0, shapes, (count,), generator=gen, device="cuda")
    local = _uniform(gen, (count, 3), -1.0, 1.0) * sizes[which]
    face = torch.randint(0, 3, (count, 1), generator=gen, device="cuda")
    sign = torch.where(_uniform(gen, (count, 1)) < 0.5, -1.0, 1.0)
    box = kinds[which]
    on_face = local.scatter(1, face, sign * sizes[which].gather(1, face))
    on_plane = local.clone()
    on_plane[:, 2] = 0.0
    local = torch.where(box[:, None], on_face, on_plane)
    raw = torch.zeros((count, 16), device="cuda")
    raw[:, 0:3] = (rot[which] * local[:, None, :]).sum(-1) + centers[which]
    raw[:, 3] = _normal(gen, (count,), 1.0, 1.0)
    raw[:, 4:7] = _normal(gen, (count, 3), -4.2, 0.4)
    raw[:, 8:12] = _unit(_normal(gen, (count, 4)))
    raw[:, 12:15] = palette[which] + _normal(gen, (count, 3), 0.0, 0.15)
    return raw, _normal(gen, (count, 45), 0.0, 0.05)


def _random_scene(count: int, seed: int, half_extent: float):
    """Raw parameters and SH of Gaussians filling a box."""
    gen = _generator(seed, 2)
    raw = torch.zeros((count, 16), device="cuda")
    raw[:, 0:3] = _uniform(gen, (count, 3), -half_extent, half_extent)
    raw[:, 3] = _normal(gen, (count,))
    raw[:, 4:7] = _normal(gen, (count, 3), -3.5, 0.5)
    raw[:, 8:12] = _unit(_normal(gen, (count, 4)))
    raw[:, 12:15] = _normal(gen, (count, 3), 0.0, 0.5)
    return raw, _normal(gen, (count, 45), 0.0, 0.05)


def _activate(raw):
    """Raw parameters as the renderer takes them, rounded to float32 from 64 bits."""
    r = raw.double()
    out = torch.zeros_like(r)
    out[:, 0:3] = r[:, 0:3]
    out[:, 3] = torch.sigmoid(r[:, 3])
    out[:, 4:7] = torch.exp(r[:, 4:7])
    out[:, 8:12] = r[:, 8:12]
    out[:, 12:15] = 0.5 + SH_C0 * r[:, 12:15]
    return out.float()


def _ring_cameras(count: int, seed: int, width: int, height: int) -> list[CameraData]:
    """Cameras on a jittered ellipse ring of radius 3 to 5 around the origin."""
    rng = random.Random(9_176 + seed)
    cams = []
    for i in range(count):
        angle = 2 * math.pi * i / count + rng.gauss(0, 0.05)
        r = 15.0 / math.sqrt((3.0 * math.cos(angle)) ** 2 + (5.0 * math.sin(angle)) ** 2) * (1 + rng.gauss(0, 0.03))
        eye = [r * math.cos(angle), rng.uniform(0.3, 1.5), r * math.sin(angle)]
        view = lookAt(eye, [rng.gauss(0, 0.1) for _ in range(3)], [0.0, 1.0, 0.0])
        cams.append(CameraData(view, perspective(math.radians(55.0), width / height, 0.01, 100.0), (width, height)))
    return cams


def _sphere_camera(seed: int, width: int, height: int) -> CameraData:
    rng = random.Random(77 + seed)
    z, angle = rng.uniform(-0.9, 0.9), rng.uniform(0, 2 * math.pi)
    s = 4.0 * math.sqrt(1 - z * z)
    view = lookAt([s * math.cos(angle), 4.0 * z, s * math.sin(angle)], [0.0, 0.0, 0.0], [0.0, 1.0, 0.0])
    return CameraData(view, perspective(math.radians(60.0), width / height, 0.01, 100.0), (width, height))


def _photo(points, colors, cam: CameraData):
    """A photo (height x width x 4 bytes) of coloured points: the nearer ones weigh more, gaps take
    the colour of a coarser grid. Integer sums, so the bytes depend on the inputs alone."""
    width, height = (int(v) for v in cam.viewport)
    v, p = cam.view, cam.proj
    t = [sum(v[4 * c + r] * points[:, c] for c in range(3)) + v[12 + r] for r in range(3)]
    depth = -t[2]
    x = torch.floor((p[0] * t[0] / depth * 0.5 + 0.5) * width)
    y = torch.floor((p[5] * t[1] / depth * -0.5 + 0.5) * height)
    seen = (depth > 0.2) & (x >= 0) & (y >= 0) & (x < width) & (y < height)
    x, y, near, c = x[seen].long(), y[seen].long(), depth[seen], colors[seen]
    weight = torch.exp2(torch.clamp(18.0 - 6.0 * near, -4.0, 12.0))
    values = torch.cat([weight[:, None], weight[:, None] * c], 1).mul(1024.0).long()
    out = torch.zeros((height, width, 3), device="cuda")
    empty = torch.ones((height, width), dtype=torch.bool, device="cuda")
    rows, cols = torch.arange(height, device="cuda"), torch.arange(width, device="cuda")
    for level in range(6):
        cells_x = (width >> level) + 1
        sums = torch.zeros(((height >> level) + 1) * cells_x, 4, dtype=torch.int64, device="cuda")
        sums.index_add_(0, (y >> level) * cells_x + (x >> level), values)
        cell = sums[((rows >> level) * cells_x)[:, None] + (cols >> level)[None, :]]
        fill = empty & (cell[..., 0] > 0)
        mean = cell[..., 1:].double() / cell[..., :1].clamp(min=1).double()
        out = torch.where(fill[..., None], mean.float(), out)
        empty &= ~fill
    rgba = torch.full((height, width, 4), 255, dtype=torch.uint8, device="cuda")
    rgba[..., :3] = (out.clamp(0, 1) * 255).round().to(torch.uint8)
    return rgba


def _training_inputs(case: dict, seed: int):
    """A scene to train, its cameras, and photos of the scene it should become."""
    truth, sh = _surface_scene(case["count"], seed)
    gen = _generator(seed, 3)
    raw = truth.clone()
    raw[:, 0:3] += _normal(gen, (case["count"], 3), 0.0, 0.005)
    raw[:, 12:15] += _normal(gen, (case["count"], 3), 0.0, 0.1)
    cams = _ring_cameras(VIEWS if case["kind"] == "train" else 1, seed, case["width"], case["height"])
    colors = (0.5 + SH_C0 * truth[:, 12:15]).clamp(0, 1)
    return raw, sh, cams, [_photo(truth[:, 0:3], colors, cam) for cam in cams]


def _loss_inputs(case: dict, seed: int):
    """A render (vec4 per pixel) and the photo it is compared with: smooth pictures that differ by noise."""
    gen, w, h = _generator(seed, 4), case["width"], case["height"]
    y = torch.linspace(0, 1, h, device="cuda")[:, None, None]
    x = torch.linspace(0, 1, w, device="cuda")[None, :, None]
    f = _uniform(gen, (4, 3), 2.0, 40.0)
    picture = 0.5 + 0.2 * torch.sin(f[0] * x + f[1] * y) + 0.2 * torch.cos(f[2] * x * y + f[3] * y)
    photo = torch.full((h, w, 4), 255, dtype=torch.uint8, device="cuda")
    photo[..., :3] = ((picture + _normal(gen, (h, w, 3), 0.0, 0.02)).clamp(0, 1) * 255).round().to(torch.uint8)
    rendered = torch.zeros((h, w, 4), device="cuda")
    rendered[..., :3] = picture + _normal(gen, (h, w, 3), 0.0, 0.05)
    return rendered, photo


def _sort_inputs(case: dict, seed: int):
    """Keys as u32 words (depth bits, and the tile above them for 64-bit keys) and values."""
    gen, n = _generator(seed, 5), case["count"]
    depth = _uniform(gen, (n,), 0.5, 12.0).view(torch.int32)
    values = torch.arange(n, dtype=torch.int32, device="cuda")
    if not case["high_bits"]:
        return depth, values
    tile = torch.randint(0, 8_000, (n,), generator=gen, device="cuda", dtype=torch.int32)
    return torch.stack([depth, tile], 1).reshape(-1).contiguous(), values


def _scan_inputs(case: dict, seed: int):
    return torch.randint(0, 40, (case["count"],), generator=_generator(seed, 6), device="cuda", dtype=torch.int32)


def _cloud(case: dict, seed: int):
    """A structure-from-motion-like cloud (count x 4, xyz and padding): clusters, a plane, far outliers."""
    gen, n = _generator(seed, 7), case["count"]
    clusters = max(1, n // 2_000)
    centres, sizes = _uniform(gen, (clusters, 3), -5, 5), _uniform(gen, (clusters,), 0.01, 0.5)
    n_cluster, n_plane = int(n * 0.8), int(n * 0.15)
    which = torch.randint(0, clusters, (n_cluster,), generator=gen, device="cuda")
    plane = _uniform(gen, (n_plane, 3), -4, 4)
    plane[:, 1] = -1.5
    points = torch.zeros((n, 4), device="cuda")
    points[:, :3] = torch.cat([centres[which] + _normal(gen, (n_cluster, 3)) * sizes[which][:, None], plane,
                               _normal(gen, (n - n_cluster - n_plane, 3), 0.0, 60.0)])
    return points[torch.randperm(n, generator=gen, device="cuda")].contiguous()


def _score_inputs(case: dict, seed: int):
    """Candidates' features, and the model's weights with its normalization."""
    gen = _generator(seed, 8)
    mean, dev = _uniform(gen, (12,), -1, 1), _uniform(gen, (12,), 0.5, 2.0)
    features = _normal(gen, (case["count"], 12)) * dev + mean
    parts = [_normal(gen, (12, 64), 0.0, (2 / 12) ** 0.5), _normal(gen, (64,), 0.0, 0.1),
             _normal(gen, (64, 64), 0.0, (2 / 64) ** 0.5), _normal(gen, (64,), 0.0, 0.1),
             _normal(gen, (64, 2), 0.0, (1 / 64) ** 0.5), _normal(gen, (2,), 0.0, 0.1), mean, 1 / dev]
    return features.contiguous(), parts


# ------------------------------------------------------------------ states

_device: Device | None = None


def _dg() -> Device:
    global _device
    if _device is None:
        torch.zeros(1, device="cuda")
        _device = Device(torch.cuda.current_device())
    return _device


class _Objects:
    """Library objects, destroyed together once neither a state nor an output needs them."""

    def __init__(self):
        self.items = []

    def add(self, item):
        self.items.append(item)
        return item

    def __del__(self):
        for item in reversed(self.items):
            item.destroy()


class _Memory:
    """A library buffer as torch sees it; keeps the object that owns it alive."""

    def __init__(self, buffer, shape, typestr, objects):
        self.objects = objects
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": typestr, "version": 3,
                                         "data": (buffer.device_pointer, False)}


class _State:
    """What a program holds between calls. `call` makes one pass; `outputs` names the buffers it
    leaves its results in, looked up after the first pass (which may create them)."""

    def __init__(self, objects):
        self.objects, self.call, self.outputs, self.tensors = objects, None, None, None

    def tensor(self, buffer, shape, typestr="<f4"):
        return torch.as_tensor(_Memory(buffer, shape, typestr, self.objects), device="cuda")


def _host(t) -> np.ndarray:
    return t.cpu().numpy()


def prepare(case: dict, seed: int) -> _State:
    state = _PREPARE[case["kind"]](case, seed, _State(_Objects()))
    _dg().synchronize()
    return state


def run(state: _State):
    state.call()
    if state.tensors is None:
        state.tensors = state.outputs()
    return state.tensors


def _prepare_train(case, seed, s):
    raw, sh, cams, photos = _training_inputs(case, seed)
    dev, w, h, n = _dg(), case["width"], case["height"], case["count"]
    views = []
    for k, (cam, photo) in enumerate(zip(cams, photos)):
        texture = s.objects.add(dev.createTexture(w, h))
        texture.write(_host(photo))
        views.append(TrainingView(f"view {k}", cam, texture))
    # Densification past, the learning rates of the defaults; the scene's SH degree is set on the renderer.
    settings = replace(DEFAULT_SETTINGS, extent=EXTENT, shDegreeInterval=10**9, densifyUntil=0)
    trainer = s.objects.add(Trainer(dev, RawGaussians(_host(raw).reshape(-1), _host(sh).reshape(-1)), views, settings))
    trainer.renderer.setShDegree(case["degree"])
    trainer.setGraph(True)
    s.call = trainer.step

    def outputs():
        b, r = trainer.buffers, trainer.renderer
        return {"image": s.tensor(r.pixelBuffer, (h, w, 4)), "params": s.tensor(b["params"], (n, 16)),
                "moments": s.tensor(b["moments"], (n * 61, 2)), "stats": s.tensor(b["stats"], (n, 4)),
                "gaussians": s.tensor(r.gaussianBuffer, (n, 16)), "sh": s.tensor(r.shBuffer, (n, 45))}

    s.outputs = outputs
    return s


def _renderer(case, objects, raw, sh, pairs_per_gaussian):
    r = objects.add(GaussianRenderer(_dg(), {"initialPairCapacity": max(1 << 16, case["count"] * pairs_per_gaussian)}))
    r.setGaussians(_host(_activate(raw)).reshape(-1), {"rest": _host(sh).reshape(-1), "degree": case["degree"]})
    return r


def _frame_inputs(case, seed):
    # The box grows with the scene, as in the reference scenes of 16,384 and 1.1M Gaussians.
    raw, sh = _random_scene(case["count"], seed, 1.0 if case["count"] < 100_000 else 3.0)
    return raw, sh, _sphere_camera(seed, case["width"], case["height"])


def _prepare_frame(case, seed, s):
    raw, sh, cam = _frame_inputs(case, seed)
    dev, w, h = _dg(), case["width"], case["height"]
    r = _renderer(case, s.objects, raw, sh, 40)
    target = s.objects.add(dev.createTexture(w, h))

    def call():
        r.encode(None, target, cam, (0.0, 0.0, 0.0))
        r.afterSubmit(wait=False)

    s.call = call
    s.outputs = lambda: {"colors": s.tensor(r.pixelBuffer, (h, w, 4)),
                         "image": s.tensor(target.buffer, (h, w, 4), "|u1")}
    return s


def _prepare_gradients(case, seed, s):
    raw, sh, (cam,), (photo,) = _training_inputs(case, seed)
    dev, w, h, n = _dg(), case["width"], case["height"], case["count"]
    r = _renderer(case, s.objects, raw, sh, 16)
    loss = s.objects.add(TrainingLoss(dev, w, h))
    texture = s.objects.add(dev.createTexture(w, h))
    texture.write(_host(photo))

    def call():
        r.encode(None, None, cam, (0.1, 0.2, 0.3))
        loss.encode(None, r.pixelBuffer, texture)
        r.encodeBackward(None, loss.pixelGrads)
        r.afterSubmit(wait=False)

    s.call = call
    s.outputs = lambda: {"colors": s.tensor(r.pixelBuffer, (h, w, 4)), "loss": s.tensor(loss.pixelLoss, (h, w)),
                         "gaussians": s.tensor(r.gradients["gaussians"], (n, 16)),
                         "sh": s.tensor(r.gradients["sh"], (n, 45))}
    return s


def _prepare_views(case, seed, s):
    raw, sh = _surface_scene(case["count"], seed)
    dev, w, h, k = _dg(), case["width"], case["height"], case["views"]
    cams = _ring_cameras(k, seed, w, h)
    r = _renderer(case, s.objects, raw, sh, 8)
    targets = s.objects.add(dev.createBuffer(k * w * h * 4))
    colors = s.objects.add(dev.createBuffer(k * w * h * 16))
    s.call = lambda: r.renderViews(cams, (0.0, 0.0, 0.0), targets, colors)
    s.outputs = lambda: {"colors": s.tensor(colors, (k, h, w, 4)), "images": s.tensor(targets, (k, h, w, 4), "|u1")}
    return s


def _prepare_loss(case, seed, s):
    rendered, photo = _loss_inputs(case, seed)
    dev, w, h = _dg(), case["width"], case["height"]
    loss = s.objects.add(TrainingLoss(dev, w, h))
    buffer = s.objects.add(dev.upload(_host(rendered)))
    texture = s.objects.add(dev.createTexture(w, h))
    texture.write(_host(photo))
    s.call = lambda: loss.encode(None, buffer, texture)
    s.outputs = lambda: {"grads": s.tensor(loss.pixelGrads, (h, w, 4)), "loss": s.tensor(loss.pixelLoss, (h, w))}
    return s


def _prepare_sort(case, seed, s):
    keys, values = _sort_inputs(case, seed)
    dev, n = _dg(), case["count"]
    sort = s.objects.add(RadixSort(dev, n, case["high_bits"]))
    k, v = s.objects.add(dev.upload(_host(keys))), s.objects.add(dev.upload(_host(values)))
    encoder = dev.createCommandEncoder()

    def call():  # the sort is in place: new keys are copied in before each call
        encoder.copyBufferToBuffer(k, 0, sort.keys, 0, k.size)
        encoder.copyBufferToBuffer(v, 0, sort.values, 0, v.size)
        sort.encode()

    s.call = call
    s.outputs = lambda: {"keys": s.tensor(sort.keys, (keys.numel(),), "<i4"),
                         "values": s.tensor(sort.values, (n,), "<i4")}
    return s


def _prepare_scan(case, seed, s):
    counts = _scan_inputs(case, seed)
    dev, n = _dg(), case["count"]
    source, data = s.objects.add(dev.upload(_host(counts))), s.objects.add(dev.createBuffer(4 * n))
    scan = s.objects.add(PrefixSum(dev, data, n))
    encoder = dev.createCommandEncoder()

    def call():  # in place, like the sort
        encoder.copyBufferToBuffer(source, 0, data, 0, 4 * n)
        scan.encode()

    s.call = call
    s.outputs = lambda: {"offsets": s.tensor(data, (n,), "<i4"), "total": s.tensor(scan.total, (1,), "<i4")}
    return s


def _prepare_neighbours(case, seed, s):
    dev, n = _dg(), case["count"]
    points = s.objects.add(dev.upload(_host(_cloud(case, seed))))
    out = s.objects.add(dev.createBuffer(4 * n))
    s.call = lambda: meanNeighborDistance2Buffers(dev, points, n, out)
    s.outputs = lambda: {"distance2": s.tensor(out, (n,))}
    return s


def _prepare_scores(case, seed, s):
    features, parts = _score_inputs(case, seed)
    dev, n = _dg(), case["count"]
    mlp = s.objects.add(DensifyMLP(dev))
    mlp.setWeights(np.concatenate([_host(p).reshape(-1) for p in parts]))
    source, out = s.objects.add(dev.upload(_host(features))), s.objects.add(dev.createBuffer(4 * n))
    s.call = lambda: mlp.predict(source, n, out)
    s.outputs = lambda: {"survive": s.tensor(out, (n,))}
    return s


_PREPARE = {"train": _prepare_train, "frame": _prepare_frame, "gradients": _prepare_gradients,
            "views": _prepare_views, "loss": _prepare_loss, "sort": _prepare_sort, "scan": _prepare_scan,
            "neighbours": _prepare_neighbours, "scores": _prepare_scores}


# ------------------------------------------------------------------ work

def _blends(case: dict) -> float:
    """(pixel, splat) pairs to blend, about: each Gaussian's 3-sigma ellipse, and at most the 250 a
    pixel blends before it is opaque."""
    if case["kind"] == "frame":
        sigma, focal = math.exp(-3.5) * 1.13, case["height"] / 2 / math.tan(math.radians(30.0))
    else:
        sigma, focal = math.exp(-4.2) * 1.08, case["height"] / 2 / math.tan(math.radians(27.5))
    area = math.pi * (3.0 * sigma * focal / 4.0) ** 2
    return min(case["count"] * area, 250.0 * case["width"] * case["height"])


def work(case: dict) -> dict:
    kind, n = case["kind"], case.get("count", 0)
    pixels = case.get("width", 0) * case.get("height", 0)
    loss_bytes, loss_flops = pixels * (16 + 4 + 16 + 4), pixels * 3 * (8 * 22 * 2 + 80)
    if kind == "train":
        # Per Gaussian: its raw and activated parameters, SH, and Adam's moments in and out, its
        # statistics; the photo in, the image and its gradient out.
        return {"bytes": n * (2 * (59 * 4 + 59 * 8) + 14 * 4 + 2 * 24) + pixels * (4 + 16),
                "flops": n * (500 + 1_500 + 59 * 15) + _blends(case) * (20 + 45) + loss_flops}
    if kind == "frame":
        return {"bytes": n * (64 + 180) + pixels * 20, "flops": n * 500 + _blends(case) * 20}
    if kind == "gradients":
        return {"bytes": 2 * n * (64 + 180) + pixels * 24,
                "flops": n * 2_000 + _blends(case) * (20 + 45) + loss_flops}
    if kind == "views":
        return {"bytes": n * (64 + 180) + case["views"] * pixels * 20,
                "flops": case["views"] * (n * 500 + _blends(case) * 20)}
    if kind == "loss":
        return {"bytes": loss_bytes, "flops": loss_flops}
    if kind == "sort":
        return {"bytes": 2 * n * ((8 if case["high_bits"] else 4) + 4), "flops": 0}
    if kind == "scan":
        return {"bytes": 8 * n, "flops": n}
    if kind == "neighbours":
        return {"bytes": 20 * n, "flops": 8 * 50 * n}
    return {"bytes": 52 * n, "flops": 2 * n * (12 * 64 + 64 * 64 + 64 * 2)}


# ------------------------------------------------------------------ the same in 64 bits

def exact(case: dict, seed: int):
    return _EXACT[case["kind"]](case, seed)


_C2 = (1.0925484305920792, -1.0925484305920792, 0.31539156525252005, -1.0925484305920792, 0.5462742152789498)
_C3 = (-0.5900435899266435, 2.890611442640554, -0.4570457994644658, 0.3731763325901154, -0.4570457994644658,
       1.445305721320277, -0.5900435899266435)


def _sh_basis(d):
    x, y, z = d.unbind(-1)
    xx, yy, zz = x * x, y * y, z * z
    c1 = 0.4886025119029199
    return torch.stack([
        -c1 * y, c1 * z, -c1 * x, _C2[0] * x * y, _C2[1] * y * z, _C2[2] * (2 * zz - xx - yy), _C2[3] * x * z,
        _C2[4] * (xx - yy), _C3[0] * y * (3 * xx - yy), _C3[1] * x * y * z, _C3[2] * y * (4 * zz - xx - yy),
        _C3[3] * z * (2 * zz - 3 * xx - 3 * yy), _C3[4] * x * (4 * zz - xx - yy), _C3[5] * z * (xx - yy),
        _C3[6] * x * (xx - 3 * yy)], -1)


def _project(g, sh, degree, cam):
    """Activated Gaussians as 2D splats: (mean, conic, opacity, colour), and depth, radius, and which are drawn."""
    w, h = cam.viewport
    view = torch.tensor(cam.view, dtype=torch.float32, device="cuda").double().reshape(4, 4).T
    proj = torch.tensor(cam.proj, dtype=torch.float32, device="cuda").double().reshape(4, 4).T
    t = g[:, 0:3] @ view[:3, :3].T + view[:3, 3]
    depth = -t[:, 2]
    safe = torch.where(depth > 0.2, depth, torch.ones_like(depth))
    m = _rotations(_unit(g[:, 8:12])) * g[:, None, 4:7]
    cov = m @ m.transpose(1, 2)
    fx, fy = float(proj[0, 0]) * w * 0.5, float(proj[1, 1]) * h * 0.5
    lx, ly = 1.3 * w * 0.5 / fx, 1.3 * h * 0.5 / fy
    tx, ty = (t[:, 0] / safe).clamp(-lx, lx) * safe, (t[:, 1] / safe).clamp(-ly, ly) * safe
    zero = torch.zeros_like(safe)
    j = torch.stack([fx / safe, zero, fx * tx / safe**2, zero, -fy / safe, -fy * ty / safe**2], -1).reshape(-1, 2, 3)
    jw = j @ view[:3, :3]
    cov2 = jw @ cov @ jw.transpose(1, 2)
    a, b, c = cov2[:, 0, 0] + 0.3, cov2[:, 0, 1], cov2[:, 1, 1] + 0.3
    det = a * c - b * b
    mid = 0.5 * (a + c)
    radius = torch.ceil(3 * torch.sqrt(mid + torch.sqrt((mid * mid - det).clamp(min=0.1)))).detach()
    clip = torch.cat([t, torch.ones_like(t[:, :1])], 1) @ proj.T
    cw = torch.where(depth > 0.2, clip[:, 3], torch.ones_like(depth))
    mean = torch.stack([(clip[:, 0] / cw * 0.5 + 0.5) * w, (clip[:, 1] / cw * -0.5 + 0.5) * h], -1)
    drawn = (depth > 0.2) & (det > 0) & (mean[:, 0] + radius >= 0) & (mean[:, 1] + radius >= 0)
    drawn = drawn & (mean[:, 0] - radius <= w) & (mean[:, 1] - radius <= h)
    color = g[:, 12:15]
    terms = (degree + 1) ** 2 - 1
    if terms:
        eye = -(view[:3, :3].T @ view[:3, 3])
        basis = _sh_basis(_unit(g[:, 0:3] - eye))[:, :terms]
        color = color + (basis[:, :, None] * sh.reshape(-1, 15, 3)[:, :terms]).sum(1)
    conic = torch.stack([c / det, -b / det, a / det], -1)
    return (mean, conic, g[:, 3], color.clamp(min=0)), depth.detach(), radius, drawn.detach()


def _tile_lists(mean, depth, radius, drawn, w, h):
    """The splats of each 16x16 tile, nearest first: splat indices, and each tile's run of them."""
    tx, ty = (w + 15) // 16, (h + 15) // 16
    lo = torch.floor((mean - radius[:, None]) / 16)
    hi = torch.floor((mean + radius[:, None]) / 16) + 1
    x0, x1 = lo[:, 0].clamp(0, tx).long(), hi[:, 0].clamp(0, tx).long()
    y0, y1 = lo[:, 1].clamp(0, ty).long(), hi[:, 1].clamp(0, ty).long()
    order = torch.argsort(torch.where(drawn, depth.float(), torch.inf), stable=True)
    order = order[drawn[order]]
    x0, x1, y0, y1 = x0[order], x1[order], y0[order], y1[order]
    counts = (x1 - x0) * (y1 - y0)
    owner = torch.repeat_interleave(torch.arange(order.numel(), device="cuda"), counts)
    local = torch.arange(owner.numel(), device="cuda") - (counts.cumsum(0) - counts)[owner]
    width = (x1 - x0)[owner]
    tile = (y0[owner] + local // width.clamp(min=1)) * tx + x0[owner] + local % width.clamp(min=1)
    tile, by = torch.sort(tile, stable=True)
    starts = torch.searchsorted(tile, torch.arange(tx * ty + 1, device="cuda"))
    return order[owner[by]], starts.tolist(), tx, ty


def _blend_tile(splats, index, px, py, bg):
    """Colours and final transmittance of the pixels (px, py) over the splats `index`, nearest first."""
    mean, conic, opacity, color = (v[index] for v in splats)
    dx, dy = px[None] - mean[:, 0:1], py[None] - mean[:, 1:2]
    power = -0.5 * (conic[:, 0:1] * dx * dx + conic[:, 2:3] * dy * dy) - conic[:, 1:2] * dx * dy
    a = opacity[:, None] * torch.exp(power.clamp(max=0))
    a = a + (a.clamp(max=0.99) - a).detach()  # the cap passes the gradient on, as training does
    a = torch.where((power <= 0) & (a >= 1 / 255), a, 0.0)
    log_t = torch.cumsum(torch.log1p(-a), 0)
    kept = torch.where(log_t.detach() >= math.log(1e-4), a, 0.0)
    t = torch.cat([torch.ones_like(px)[None], torch.exp(torch.cumsum(torch.log1p(-kept), 0))])
    out = (kept * t[:-1]).T @ color + t[-1][:, None] * bg
    return torch.cat([out, t[-1:].T], 1)


def _tiles64(splats, depth, radius, drawn, cam, bg, use):
    """Calls use(pixels, colours of those pixels) for every tile of the image."""
    w, h = cam.viewport
    lists, starts, tx, ty = _tile_lists(splats[0].detach(), depth, radius, drawn, w, h)
    bg = torch.tensor(bg, dtype=torch.float32, device="cuda").double()
    for k in range(tx * ty):
        xs = torch.arange(k % tx * 16, min(k % tx * 16 + 16, w), device="cuda")
        ys = torch.arange(k // tx * 16, min(k // tx * 16 + 16, h), device="cuda")
        py, px = (v.reshape(-1) for v in torch.meshgrid(ys, xs, indexing="ij"))
        use(py * w + px, _blend_tile(splats, lists[starts[k]:starts[k + 1]], px.double() + 0.5, py.double() + 0.5, bg))


def _image64(projected, cam, bg):
    w, h = cam.viewport
    image = torch.zeros((h * w, 4), dtype=torch.float64, device="cuda")

    def use(pixels, colors):
        image[pixels] = colors

    with torch.no_grad():
        _tiles64(*projected, cam, bg, use)
    return image


def _loss64(rendered, photo):
    """Each pixel's share of 0.8 L1 + 0.2 (1 - SSIM), less the constant, and its gradient per pixel."""
    h, w = photo.shape[:2]
    x = rendered.reshape(h, w, -1)[..., :3].permute(2, 0, 1)[:, None].detach().requires_grad_()
    y = (photo[..., :3].double() / 255).permute(2, 0, 1)[:, None]
    k = torch.exp(-torch.arange(-5, 6, dtype=torch.float64, device="cuda") ** 2 / (2 * 1.5**2))
    k = k / k.sum()

    def blur(v):
        rows = torch.nn.functional.pad(v, (5, 5, 0, 0))
        v = sum(k[i] * rows[..., i:i + w] for i in range(11))
        cols = torch.nn.functional.pad(v, (0, 0, 5, 5))
        return sum(k[i] * cols[..., i:i + h, :] for i in range(11))

    mx, my = blur(x), blur(y)
    vx, vy, cxy = blur(x * x) - mx * mx, blur(y * y) - my * my, blur(x * y) - mx * my
    ssim = (2 * mx * my + 1e-4) * (2 * cxy + 9e-4) / ((mx * mx + my * my + 1e-4) * (vx + vy + 9e-4))
    share = (0.8 * (x - y).abs() - 0.2 * ssim).sum(0)[0] / (3 * w * h)
    grad, = torch.autograd.grad(share.sum(), x)
    return share.detach(), torch.cat([grad[:, 0].permute(1, 2, 0), torch.zeros_like(grad[0, 0])[..., None]], -1)


def _gradients64(g, sh, degree, cam, photo, bg):
    """The image, loss shares, gradients of g and sh, the mean's gradient per splat, and the splats' radii."""
    g, sh = g.detach().requires_grad_(), sh.detach().requires_grad_()
    splats, depth, radius, drawn = _project(g, sh, degree, cam)
    leaves = tuple(v.detach().requires_grad_() for v in splats)
    image = _image64((leaves, depth, radius, drawn), cam, bg)
    share, pixel_grads = _loss64(image, photo)
    flat = pixel_grads.reshape(-1, 4)[:, :3]
    totals = [torch.zeros_like(v) for v in leaves]

    def use(pixels, colors):
        if colors.requires_grad:
            for total, got in zip(totals, torch.autograd.grad(colors[:, :3], leaves, flat[pixels])):
                total += got

    _tiles64(leaves, depth, radius, drawn, cam, bg, use)
    totals = [torch.where(drawn.reshape(-1, *[1] * (v.dim() - 1)), v, 0.0) for v in totals]
    gg, gsh = torch.autograd.grad(splats, (g, sh), totals, allow_unused=True)
    gsh = torch.zeros_like(sh) if gsh is None else gsh
    return image, share, torch.nan_to_num(gg), torch.nan_to_num(gsh), totals[0], torch.where(drawn, radius, 0.0)


def _first_view(views: int) -> int:
    """The view the first training step takes: the last of a mulberry32(1) Fisher-Yates shuffle."""
    queue, state = list(range(views)), 1
    for i in range(views - 1, 0, -1):
        state = (state + 0x6D2B79F5) & 0xFFFFFFFF
        t = state
        t = ((t ^ (t >> 15)) * (t | 1)) & 0xFFFFFFFF
        t ^= (t + (((t ^ (t >> 7)) * (t | 61)) & 0xFFFFFFFF)) & 0xFFFFFFFF
        j = int((t ^ (t >> 14)) / 4294967296.0 * (i + 1))
        queue[i], queue[j] = queue[j], queue[i]
    return queue[-1]


def _exact_train(case, seed):
    raw, sh, cams, photos = _training_inputs(case, seed)
    k = _first_view(len(cams))
    active = _activate(raw).double()
    image, _, gg, gsh, gmean, radius = _gradients64(active, sh.double(), case["degree"], cams[k], photos[k], (0, 0, 0))
    r = raw.double()
    sig = torch.sigmoid(r[:, 3:4])
    grad = torch.zeros_like(r)
    grad[:, 0:3], grad[:, 3:4] = gg[:, 0:3], gg[:, 3:4] * sig * (1 - sig)
    grad[:, 4:7], grad[:, 8:12], grad[:, 12:15] = gg[:, 4:7] * torch.exp(r[:, 4:7]), gg[:, 8:12], gg[:, 12:15] * SH_C0
    progress = 1 / 30_000
    rate = torch.zeros(16, dtype=torch.float64, device="cuda")
    rate[0:3] = math.exp(math.log(0.00016) * (1 - progress) + math.log(0.0000016) * progress) * EXTENT
    rate[3], rate[4:7], rate[8:12], rate[12:15] = 0.025, 0.005, 0.001, 0.0025
    params = r - rate * grad / (grad.abs() + 1e-15)
    new = torch.zeros_like(r)
    new[:, 0:3], new[:, 8:12] = params[:, 0:3], params[:, 8:12]
    new[:, 3], new[:, 4:7] = torch.sigmoid(params[:, 3]), torch.exp(params[:, 4:7])
    new[:, 12:15] = 0.5 + SH_C0 * params[:, 12:15]
    both = torch.cat([grad.reshape(-1), gsh.reshape(-1)])
    w, h = cams[k].viewport
    length = torch.sqrt((gmean[:, 0] * w * 0.5) ** 2 + (gmean[:, 1] * h * 0.5) ** 2)
    drawn = (radius > 0).double()
    return {"image": image.reshape(h, w, 4), "params": params,
            "moments": torch.stack([0.1 * both, 0.001 * both * both], 1),
            "stats": torch.stack([length * drawn, drawn, radius, torch.zeros_like(radius)], 1),
            "gaussians": new, "sh": sh.double() - 0.0025 / 20 * gsh / (gsh.abs() + 1e-15)}


def _exact_frame(case, seed):
    raw, sh, cam = _frame_inputs(case, seed)
    with torch.no_grad():
        projected = _project(_activate(raw).double(), sh.double(), case["degree"], cam)
    image = _image64(projected, cam, (0.0, 0.0, 0.0))
    return {"colors": image.reshape(case["height"], case["width"], 4), "image": None}


def _exact_gradients(case, seed):
    raw, sh, (cam,), (photo,) = _training_inputs(case, seed)
    image, share, gg, gsh, _, _ = _gradients64(_activate(raw).double(), sh.double(), case["degree"], cam, photo,
                                               (0.1, 0.2, 0.3))
    return {"colors": image.reshape(case["height"], case["width"], 4), "loss": share, "gaussians": gg, "sh": gsh}


def _exact_views(case, seed):
    raw, sh = _surface_scene(case["count"], seed)
    g, images = _activate(raw).double(), []
    for cam in _ring_cameras(case["views"], seed, case["width"], case["height"]):
        with torch.no_grad():
            projected = _project(g, sh.double(), case["degree"], cam)
        images.append(_image64(projected, cam, (0.0, 0.0, 0.0)).reshape(case["height"], case["width"], 4))
    return {"colors": torch.stack(images), "images": None}


def _exact_loss(case, seed):
    rendered, photo = _loss_inputs(case, seed)
    share, grads = _loss64(rendered.double(), photo)
    return {"grads": grads, "loss": share}


def _exact_neighbours(case, seed):
    if case["count"] > 250_000:
        return None  # all distances of more points take too long
    p = _cloud(case, seed)[:, :3].double()
    out = []
    for first in range(0, p.shape[0], 2_048):
        q = p[first:first + 2_048]
        d = sum((q[:, k, None] - p[None, :, k]) ** 2 for k in range(3))
        d[torch.arange(q.shape[0]), torch.arange(first, first + q.shape[0])] = torch.inf
        out.append(torch.topk(d, 3, dim=1, largest=False).values.mean(1))
    return {"distance2": torch.cat(out)}


def _exact_scores(case, seed):
    features, parts = _score_inputs(case, seed)
    w1, b1, w2, b2, w3, b3, mean, inverse = (p.double() for p in parts)
    x = (features.double() - mean) * inverse
    x = torch.nn.functional.gelu(x @ w1 + b1)
    x = torch.nn.functional.gelu(x @ w2 + b2)
    return {"survive": torch.softmax(x @ w3 + b3, 1)[:, 1]}


_EXACT = {"train": _exact_train, "frame": _exact_frame, "gradients": _exact_gradients, "views": _exact_views,
          "loss": _exact_loss, "neighbours": _exact_neighbours, "scores": _exact_scores,
          # Whole numbers have no rounding to compare.
          "sort": lambda case, seed: None, "scan": lambda case, seed: None}
