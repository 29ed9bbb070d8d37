"""What a user of this framework has it do, as measurable cases.

Seven kinds of work, each through the public entry points:

``layer``     one 3x3x3 ``SparseConv3d`` in inference, on a tensor whose kernel map an earlier layer of the
              network has built (a network runs tens of layers per map);
``resample``  the strided / transposed 2x2x2 pair between two levels of a U-Net, in inference;
``grad``      one 3x3x3 ``SparseConv3d`` in training: forward, input, weight and bias gradients;
``pool``      2x2x2 pooling and un-pooling in training;
``maps``      coordinates only: hash table, strided coordinates and the compact kernel maps of a batch of
              scenes in the order a scanner delivered them;
``infer``     MinkUNet-34 inference over a batch of scenes: Morton sort, all kernel maps, all layers, logits in
              the caller's row order;
``train``     one training step of two levels of such a network over a batch of scenes: Morton sort, kernel
              maps, forward under autocast, cross entropy, backward, SGD.

Scenes are synthetic, made on the GPU: rooms (floor, walls and 40 boxes rasterised at 1, 2 or 5 cm, cropped
around the centre), spinning-LiDAR sweeps (ground and boxes, 5 cm) and random cells.  They are what
``warpconvnet_b200.datasets.synthetic`` makes on the host, at the same densities.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from warpconvnet_b200 import SparseConv3d, Voxels, cat, generate_kernel_map, sparse_reduce, sparse_unpool, stride_coords
from warpconvnet_b200.examples.mink_unet import BasicBlock, ConvBlock, ConvTrBlock, MinkUNet34, randomize_batchnorm_

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
DEV = "cuda"
CLASSES = 20


def listed():
    return [
        # the smallest problem of the repository's configurations: one fp32 layer over 20 000 random cells
        {"name": "layer_20k_c32_f32", "kind": "layer", "scene": "cells", "voxels": 20000, "c_in": 32, "c_out": 32, "dtype": "f32"},
        # the layer sweep at 500 000 voxels of a 1 cm room: a narrow layer ...
        {"name": "layer_500k_c64_f16", "kind": "layer", "scene": "room", "voxels": 500000, "c_in": 64, "c_out": 64, "dtype": "f16"},
        # ... and the widest one
        {"name": "layer_500k_c256_bf16", "kind": "layer", "scene": "room", "voxels": 500000, "c_in": 256, "c_out": 256, "dtype": "bf16"},
        # an outdoor scene: few neighbours per voxel, an odd row count, unequal widths
        {"name": "layer_lidar_777k_bf16", "kind": "layer", "scene": "lidar", "voxels": 777777, "c_in": 128, "c_out": 96, "dtype": "bf16"},
        # down and up again between two levels of a decoder-sized feature map
        {"name": "resample_300k_c96_f16", "kind": "resample", "scene": "room", "voxels": 300001, "c_in": 96, "c_out": 96, "dtype": "f16"},
        # a layer trained without autocast: everything in fp32
        {"name": "grad_60k_c64_f32", "kind": "grad", "scene": "room", "voxels": 60000, "c_in": 64, "c_out": 64, "dtype": "f32"},
        # pooling network stage in training
        {"name": "pool_250k_c64_f16", "kind": "pool", "scene": "room", "voxels": 250007, "c_in": 64, "c_out": 64, "dtype": "f16", "reduction": "max"},
        # kernel maps of four rooms of 250 000 voxels
        {"name": "maps_4x250k", "kind": "maps", "scene": "room", "scenes": 4, "voxels": 1000000},
        # one small scan, as an interactive application sends it: latency
        {"name": "infer_1x20k_f16", "kind": "infer", "scenes": 1, "voxels": 20000, "dtype": "f16"},
        # one room
        {"name": "infer_1x150k_f16", "kind": "infer", "scenes": 1, "voxels": 150000, "dtype": "f16"},
        # the benchmark's batch: eight rooms
        {"name": "infer_8x150k_f16", "kind": "infer", "scenes": 8, "voxels": 1200000, "dtype": "f16"},
        # a training step over a batch of four scans
        {"name": "train_4x60k_bf16", "kind": "train", "scenes": 4, "voxels": 240000, "dtype": "bf16"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["layer", "layer", "resample", "grad", "pool", "maps", "infer", "infer", "train"])
    widths = [32, 48, 64, 96, 128, 160, 192, 256]
    if kind == "layer":
        dtype = rng.choice(["f16", "bf16", "f16", "bf16", "f32"])
        # fp32 layers are the small ones: large networks run in 16 bits
        voxels = _log_int(rng, 2000, 100000 if dtype == "f32" else 800000)
        scene = rng.choice(["room", "lidar", "cells"] if voxels <= 200000 else ["room", "lidar"])
        some = [c for c in widths if c <= 128] if dtype == "f32" else widths
        c_in = rng.choice(some)
        c_out = c_in if rng.random() < 0.6 else rng.choice(some)
        return {"kind": kind, "scene": scene, "voxels": voxels, "c_in": c_in, "c_out": c_out, "dtype": dtype}
    if kind == "resample":
        c_in = rng.choice(widths)
        return {"kind": kind, "scene": rng.choice(["room", "lidar"]), "voxels": _log_int(rng, 5000, 800000), "c_in": c_in,
                "c_out": c_in if rng.random() < 0.6 else rng.choice(widths), "dtype": rng.choice(["f16", "bf16"])}
    if kind == "grad":
        dtype = rng.choice(["f32", "f16", "bf16"])
        some = [c for c in widths if c <= 128] if dtype == "f32" else widths
        return {"kind": kind, "scene": rng.choice(["room", "lidar"]),
                "voxels": _log_int(rng, 4000, 80000 if dtype == "f32" else 300000), "c_in": rng.choice(some),
                "c_out": rng.choice(some), "dtype": dtype}
    if kind == "pool":
        c = rng.choice([16, 32, 64, 96, 128])
        return {"kind": kind, "scene": rng.choice(["room", "lidar"]), "voxels": _log_int(rng, 5000, 400000), "c_in": c,
                "c_out": c, "dtype": rng.choice(["f32", "f16", "bf16"]), "reduction": rng.choice(["max", "mean"])}
    if kind == "maps":
        scenes = rng.randint(1, 6)
        return {"kind": kind, "scene": "room", "scenes": scenes, "voxels": scenes * _log_int(rng, 5000, 160000) + rng.randint(0, 99)}
    scenes = rng.randint(1, 8 if kind == "infer" else 4)
    if kind == "infer":
        return {"kind": kind, "scenes": scenes, "voxels": scenes * _log_int(rng, 10000, 150000) - rng.randint(0, 99),
                "dtype": rng.choice(["f16", "f16", "bf16"])}
    return {"kind": kind, "scenes": scenes, "voxels": scenes * _log_int(rng, 8000, 100000) - rng.randint(0, 99),
            "dtype": rng.choice(["f16", "bf16"])}


# --------------------------------------------------------------------------- scenes


def _generator(seed, device):
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    return g


def _distinct(c):
    """Distinct rows of int64 ``[N, 3]`` in key order."""
    lo = c.min(dim=0).values
    span = c.max(dim=0).values - lo + 1
    d = c - lo
    key = torch.unique((d[:, 0] * span[1] + d[:, 1]) * span[2] + d[:, 2])
    return torch.stack([key // (span[1] * span[2]), key // span[2] % span[1], key % span[2]], dim=1) + lo


def _room(n, seed):
    """``n`` distinct voxels of a 10 x 10 x 3 m room, the ones nearest to its centre, in random order."""
    size = torch.tensor([10.0, 10.0, 3.0], dtype=torch.float64)
    voxel = 0.05 if n <= 40000 else 0.02 if n <= 300000 else 0.01
    g = _generator(seed, "cpu")
    side = torch.rand(40, 3, generator=g, dtype=torch.float64) * 1.8 + 0.2
    box_lo = torch.rand(40, 3, generator=g, dtype=torch.float64) * (size - side)
    faces = []  # fixed axis, its cell, first cells and cell counts along the other two axes

    def add(axis, at, lo, hi):
        a, b = [x for x in range(3) if x != axis]
        f = [int(math.floor(float(v) / voxel)) for v in (at, lo[a], lo[b], hi[a] - 1e-9, hi[b] - 1e-9)]
        faces.append((axis, f[0], f[1], f[3] - f[1] + 1, f[2], f[4] - f[2] + 1))

    zero = torch.zeros(3, dtype=torch.float64)
    add(2, 0.0, zero, size)
    for axis in (0, 1):
        add(axis, 0.0, zero, size)
        add(axis, float(size[axis]) - 1e-6, zero, size)
    for i in range(40):
        lo, hi = box_lo[i].tolist(), (box_lo[i] + side[i]).tolist()
        for axis in range(3):
            add(axis, lo[axis], lo, hi)
            add(axis, hi[axis], lo, hi)
    t = torch.tensor(faces, dtype=torch.int64)
    counts = t[:, 3] * t[:, 5]
    total = int(counts.sum())
    start = torch.cumsum(counts, 0) - counts
    face = torch.repeat_interleave(torch.arange(len(t), device=DEV), counts.to(DEV), output_size=total)
    t, start = t.to(DEV), start.to(DEV)
    local = torch.arange(total, device=DEV) - start[face]
    t = t[face]
    u, v = t[:, 2] + local // t[:, 5], t[:, 4] + local % t[:, 5]
    axis = t[:, 0]
    x = torch.where(axis == 0, t[:, 1], u)
    y = torch.where(axis == 0, u, torch.where(axis == 1, t[:, 1], v))
    z = torch.where(axis == 2, t[:, 1], v)
    c = _distinct(torch.stack([x, y, z], dim=1))
    half = (size / 2).to(DEV)
    away = (((c.double() + 0.5) * voxel - half).abs() / half).max(dim=1).values
    c = c[torch.sort(away, stable=True).indices[:n]]
    assert c.shape[0] == n, f"the room has {c.shape[0]} voxels, {n} were asked for"
    return c[torch.randperm(n, generator=_generator(seed, DEV), device=DEV)].int()


def _lidar(n, seed):
    """``n`` distinct 5 cm voxels hit by a 64-beam spinning sensor that drives past 300 boxes."""
    voxel, rays_per_beam, boxes = 0.05, 2048, 300
    g, gd = _generator(seed, "cpu"), _generator(seed, DEV)
    foot = torch.rand(boxes, 2, generator=g) * 5 + 1
    height = torch.rand(boxes, generator=g) * 3 + 1
    r, th = 80 * torch.sqrt(torch.rand(boxes, generator=g) * 0.99 + 0.01), torch.rand(boxes, generator=g) * (2 * math.pi)
    centre = torch.stack([r * torch.cos(th), r * torch.sin(th)], 1)
    lo = torch.cat([centre - foot / 2, torch.full((boxes, 1), -1.7)], 1).to(DEV)
    hi = torch.cat([centre + foot / 2, (height - 1.7)[:, None]], 1).to(DEV)
    el = torch.deg2rad(torch.linspace(-25.0, 3.0, 64, device=DEV))[:, None]
    az = (torch.arange(rays_per_beam, device=DEV) * (2 * math.pi / rays_per_beam))[None, :]
    dirs = torch.stack([torch.cos(el) * torch.cos(az), torch.cos(el) * torch.sin(az), torch.sin(el).expand(-1, rays_per_beam)], -1).reshape(-1, 3)
    pos, yaw = torch.zeros(3), 0.0
    hits = torch.empty((0, 3), dtype=torch.int64, device=DEV)
    while hits.shape[0] < n:
        new = []
        for _ in range(8):
            c, s = math.cos(yaw), math.sin(yaw)
            d = torch.stack([c * dirs[:, 0] - s * dirs[:, 1], s * dirs[:, 0] + c * dirs[:, 1], dirs[:, 2]], 1)
            p = pos.to(DEV)
            t = torch.where(d[:, 2] < -1e-6, (-1.7 - p[2]) / d[:, 2], torch.full_like(d[:, 2], math.inf))
            inv = 1.0 / torch.where(d.abs() < 1e-12, torch.full_like(d, 1e-12), d)
            for b in range(0, boxes, 100):
                near = torch.full((d.shape[0], 100), 0.0, device=DEV)
                far = torch.full((d.shape[0], 100), math.inf, device=DEV)
                for a in range(3):
                    t0, t1 = (lo[None, b:b + 100, a] - p[a]) * inv[:, a:a + 1], (hi[None, b:b + 100, a] - p[a]) * inv[:, a:a + 1]
                    near = torch.maximum(near, torch.minimum(t0, t1))
                    far = torch.minimum(far, torch.maximum(t0, t1))
                t = torch.minimum(t, torch.where(far >= near, near, torch.full_like(near, math.inf)).min(dim=1).values)
            t = t * (1 + 0.005 * torch.randn(t.shape[0], generator=gd, device=DEV))
            good = torch.isfinite(t) & (t <= 80) & (t > 0.5)
            new.append(torch.floor((p + d[good] * t[good, None]) / voxel).long())
            pos = pos + torch.tensor([c, s, 0.0]) * (float(torch.rand(1, generator=g)) * 1.5 + 0.5)
            yaw += math.radians(5 * float(torch.randn(1, generator=g)))
        hits = _distinct(torch.cat([hits] + new))
    return hits[torch.randperm(hits.shape[0], generator=gd, device=DEV)[:n]].int()


def _cells(n, seed):
    """``n`` cells of a cube, a thirteenth of it (20 000 of 64^3)."""
    e = max(4, round((n * 64 ** 3 / 20000) ** (1 / 3)))
    i = torch.randperm(e ** 3, generator=_generator(seed, DEV), device=DEV)[:n]
    return torch.stack([i // (e * e), i // e % e, i % e], dim=1).int()


_SCENES = {"room": _room, "lidar": _lidar, "cells": _cells}


def _sizes(case, seed):
    """Row counts of the scenes of a batch: ragged, their sum is the case's."""
    scenes, total = case.get("scenes", 1), case["voxels"]
    w = torch.rand(scenes, generator=_generator(seed, "cpu")) * 0.5 + 0.75
    cut = [int(round(total * float(v))) for v in torch.cumsum(w / w.sum(), 0)]
    cut[-1] = total
    return [b - a for a, b in zip([0] + cut[:-1], cut)]


def _placed(c, seed):
    """A scene seen from elsewhere: axes exchanged and mirrored, moved by a multiple of 16, rows in another order.
    Its number of strided coordinates and of neighbour pairs stays."""
    g = _generator(seed, "cpu")
    c = c[:, torch.randperm(3, generator=g).tolist()]
    flip = torch.randint(0, 2, (3,), generator=g).bool().to(DEV)
    move = (torch.randint(-50, 50, (3,), generator=g) * 16).int().to(DEV)
    c = torch.where(flip, -1 - c, c) + move
    return c[torch.randperm(c.shape[0], generator=_generator(seed, DEV), device=DEV)].contiguous()


def _batch(case, seed):
    """(coords [N, 3] int32, offsets [B + 1] on the host) in the order the scenes were delivered in.  Where results
    are as many as the scenes have coarse voxels or neighbours, the scenes are the case's own and the seed places them."""
    make = _SCENES[case.get("scene", "room")]
    own = case["kind"] in ("resample", "pool", "maps")
    which = case["voxels"] if own else seed
    sizes = _sizes(case, which)
    scenes = [make(n, which * 16 + i) for i, n in enumerate(sizes)]
    if own:
        scenes = [_placed(c, seed * 16 + i) for i, c in enumerate(scenes)]
    return torch.cat(scenes), torch.tensor([0] + sizes).cumsum(0)


def _randn(shape, seed, dtype):
    return torch.randn(shape, generator=_generator(seed, DEV), device=DEV).to(dtype)


# --------------------------------------------------------------------------- states


class TwoLevelUNet(torch.nn.Module):
    """Stem, one stride-2 level and back, with the blocks of the example network.  (A whole MinkUNet in training
    mode is no case: its gradients at random weights differ by a quarter when its inputs differ by 3e-4, so that
    two correct implementations could not be told from two that differ.)"""

    def __init__(self):
        super().__init__()
        self.stem = ConvBlock(3, 32, kernel_size=3)
        self.down = ConvBlock(32, 32, kernel_size=2, stride=2)
        self.enc = BasicBlock(32, 64)
        self.up = ConvTrBlock(64, 64, kernel_size=2, stride=2)
        self.dec = BasicBlock(96, 64)
        self.head = SparseConv3d(64, CLASSES, kernel_size=1)

    def forward(self, x):
        fine = self.stem(x)
        coarse = self.enc(self.down(fine))
        return self.head(self.dec(cat(self.up(coarse, fine), fine)))


def _flatten(tensors):
    """One buffer behind many tensors, as flat-parameter optimisers and gradient buckets keep them; each
    starts at a multiple of 64 elements.  Returns the buffer and its views."""
    at, views = 0, []
    for t in tensors:
        views.append((at, t))
        at += -(-t.numel() // 64) * 64
    flat = torch.zeros(at, dtype=tensors[0].dtype, device=DEV)
    out = []
    for a, t in views:
        v = flat.data[a:a + t.numel()].view(t.shape)
        v.copy_(t)
        out.append(v)
    return flat, out


def prepare(case, seed):
    torch.manual_seed(seed)
    kind = case["kind"]
    dtype = DTYPES.get(case.get("dtype"), torch.float32)
    coords, offsets = _batch(case, seed)
    n = case["voxels"]
    if kind == "maps":
        batch = torch.repeat_interleave(torch.arange(len(offsets) - 1, device=DEV, dtype=torch.int32), torch.diff(offsets).to(DEV))
        return {"kind": kind, "coords": torch.cat([batch[:, None], coords], dim=1).contiguous()}
    if kind in ("infer", "train"):
        feats = torch.rand((n, 3), generator=_generator(seed, DEV), device=DEV)
        state = {"kind": kind, "coords": coords, "offsets": offsets, "dtype": dtype}
        with torch.device(DEV):
            model = MinkUNet34(3, CLASSES) if kind == "infer" else TwoLevelUNet()
        if kind == "infer":
            randomize_batchnorm_(model, seed)
            state.update(feats=feats.to(dtype), model=model.to(dtype).eval())
            return state
        model.train()
        params = list(model.parameters())
        flat_p, views = _flatten([p.data for p in params])
        flat_g, grads = _flatten([torch.zeros_like(p.data) for p in params])
        for p, v, g in zip(params, views, grads):
            p.data, p.grad = v, g
        owners = [(m, name) for m in model.modules() for name in ("running_mean", "running_var") if name in m._buffers]
        flat_s, stats = _flatten([m._buffers[name] for m, name in owners])
        for (m, name), v in zip(owners, stats):
            m._buffers[name] = v
        height = coords[:, 2].long() - coords[:, 2].min()
        state.update(feats=feats, model=model, labels=height * CLASSES // (height.max() + 1), params=flat_p, grads=flat_g,
                     stats=flat_s, scale=65536.0 if dtype == torch.float16 else 1.0,
                     optimizer=torch.optim.SGD(params, lr=1e-3, momentum=0.9))
        return state

    x = _randn((n, case["c_in"]), seed, dtype)
    voxels = Voxels(coords, x, offsets=offsets)
    if case["scene"] != "cells":
        voxels = voxels.sort()  # as every scan enters a network here
    state = {"kind": kind, "voxels": voxels}
    with torch.device(DEV):
        if kind in ("layer", "grad"):
            state["conv"] = SparseConv3d(case["c_in"], case["c_out"], 3, bias=kind == "grad").to(dtype)
        elif kind == "resample":
            state["down"] = SparseConv3d(case["c_in"], case["c_out"], 2, stride=2, bias=False).to(dtype)
            state["up"] = SparseConv3d(case["c_out"], case["c_in"], 2, stride=2, bias=False, transposed=True).to(dtype)
    if kind in ("grad", "pool"):
        state["x"] = voxels.feature_tensor.detach().requires_grad_(True)
        state["dy"] = _randn((n, case["c_out"]), seed + 1, dtype)
    # the first use of the coordinates leaves their kernel map in the tensor's cache, where later layers find it
    with torch.no_grad():
        if kind == "resample":
            _run_resample(state)
        elif kind == "pool":
            state["reduction"] = case["reduction"]
            sparse_reduce(voxels, 2, 2, reduction=case["reduction"])
        else:
            state["conv"](voxels)
    return state


# --------------------------------------------------------------------------- one pass


def run(state):
    return _RUN[state["kind"]](state)


@torch.no_grad()
def _run_layer(s):
    return s["conv"](s["voxels"]).feature_tensor


@torch.no_grad()
def _run_resample(s):
    down = s["down"](s["voxels"])
    return [down.feature_tensor, s["up"](down, s["voxels"]).feature_tensor]


def _run_grad(s):
    conv = s["conv"]
    y = conv(s["voxels"].replace(batched_features=s["x"])).feature_tensor
    return [y.detach(), *torch.autograd.grad(y, [s["x"], conv.weight, conv.bias], s["dy"])]


def _run_pool(s):
    v = s["voxels"].replace(batched_features=s["x"])
    pooled = sparse_reduce(v, 2, 2, reduction=s["reduction"])
    up = sparse_unpool(pooled, v, 2, 2).feature_tensor
    return [pooled.feature_tensor.detach(), up.detach(), *torch.autograd.grad(up, [s["x"]], s["dy"])]


def _run_maps(s):
    fine = s["coords"]
    coarse, offsets = stride_coords(fine, (2, 2, 2))
    same = generate_kernel_map(fine, fine, (1, 1, 1), (3, 3, 3))
    down = generate_kernel_map(fine, coarse, (2, 2, 2), (2, 2, 2))
    out = [coarse, offsets]
    for m in (same, down):
        out += [m.in_maps, m.out_maps, m.offsets]
    return out


@torch.no_grad()
def _run_infer(s):
    v = Voxels(s["coords"], s["feats"], offsets=s["offsets"]).sort()
    return s["model"](v, restore_order=True)


def _run_train(s):
    v = Voxels(s["coords"], s["feats"], offsets=s["offsets"]).sort()
    s["grads"].zero_()
    with torch.autocast(DEV, dtype=s["dtype"]):
        out = s["model"](v).feature_tensor
        loss = F.cross_entropy(out.float(), s["labels"][v.extra_attributes["perm"]])
    if s["scale"] == 1.0:
        loss.backward()
    else:  # fp16: a fixed loss scale
        (loss * s["scale"]).backward()
        s["grads"].mul_(1.0 / s["scale"])
    s["optimizer"].step()
    return [out.detach(), loss.detach(), s["grads"], s["params"], s["stats"]]


_RUN = {"layer": _run_layer, "resample": _run_resample, "grad": _run_grad, "pool": _run_pool, "maps": _run_maps,
        "infer": _run_infer, "train": _run_train}


# --------------------------------------------------------------------------- work and tolerance


def _density(scene, n):
    """(neighbours per voxel in a 3x3x3 window, coarse voxels per voxel at stride 2), as measured on these scenes."""
    if scene == "cells":
        return 2.9, 0.77
    if scene == "lidar":  # sweeps accumulate: more voxels are denser ones
        return max(1.1, 1.34 * (n / 20000) ** 0.567), min(0.97, 0.965 - 0.096 * math.log2(n / 20000))
    return 9.8, 0.25


class _Sum:
    """Bytes and operations of layers in 16 bits: every layer reads its input and its table and writes its output
    once; weights once."""

    def __init__(self):
        self.bytes = self.flops = 0.0

    def conv(self, m_in, m_out, c_in, c_out, offsets, pairs):
        self.bytes += 2 * (m_in * c_in + m_out * c_out + offsets * c_in * c_out) + (4 * offsets * m_out if offsets > 1 else 0)
        self.flops += 2.0 * pairs * m_out * c_in * c_out

    def stage(self, m, c_in, c_out, blocks=1):
        for b in range(blocks):
            c = c_in if b == 0 else c_out
            self.conv(m, m, c, c_out, 27, 10)
            self.conv(m, m, c_out, c_out, 27, 10)
            if c != c_out:
                self.conv(m, m, c, c_out, 1, 1)


def _infer_work(n):
    s, layers, planes = _Sum(), (2, 3, 4, 6, 2, 2, 2, 2), (32, 64, 128, 256, 256, 128, 96, 96)
    rows = [n * 0.25 ** i for i in range(5)]
    c = 32
    s.conv(n, n, 3, c, 1, 1)
    for i in range(4):
        s.conv(rows[i], rows[i + 1], c, c, 8, 4)
        s.stage(rows[i + 1], c, planes[i], layers[i])
        c = planes[i]
    skips = (32,) + planes[:3]
    for i in range(4):
        s.conv(rows[4 - i], rows[3 - i], c, planes[4 + i], 8, 1)
        s.stage(rows[3 - i], planes[4 + i] + skips[3 - i], planes[4 + i], layers[4 + i])
        c = planes[4 + i]
    s.conv(n, n, c, CLASSES, 1, 1)
    return {"bytes": s.bytes + 16.0 * n, "flops": s.flops}


def _train_work(n):
    s, m = _Sum(), n / 4
    s.conv(n, n, 3, 32, 27, 10)
    s.conv(n, m, 32, 32, 8, 4)
    s.stage(m, 32, 64)
    s.conv(m, n, 64, 64, 8, 1)
    s.stage(n, 96, 64)
    s.conv(n, n, 64, CLASSES, 1, 1)
    # backward: each layer reads its output gradient and its input again and writes two gradients
    return {"bytes": 3 * s.bytes + 16.0 * n, "flops": 3 * s.flops}


def work(case):
    n, kind = case["voxels"], case["kind"]
    if kind == "infer":
        return _infer_work(n)
    if kind == "train":
        return _train_work(n)
    pairs, m = (v * n for v in _density(case["scene"], n))
    if kind == "maps":
        # coordinates in, coarse coordinates out, (in, out) pairs of both maps
        return {"bytes": 16.0 * n + 16.0 * m + 8.0 * pairs + 8.0 * n, "flops": 0.0}
    e = 4 if case["dtype"] == "f32" else 2
    ci, co = case["c_in"], case["c_out"]
    if kind == "layer":
        return {"bytes": e * (n * (ci + co) + 27.0 * ci * co) + 4 * 27.0 * n, "flops": 2.0 * pairs * ci * co}
    if kind == "grad":
        return {"bytes": e * (n * (2 * ci + 2 * co) + 2 * 27.0 * ci * co) + 4 * 27.0 * n, "flops": 6.0 * pairs * ci * co}
    if kind == "resample":
        return {"bytes": e * (2 * n * ci + 2 * m * co + 16.0 * ci * co) + 2 * 32.0 * m, "flops": 4.0 * n * ci * co}
    return {"bytes": e * ci * (4.0 * n + m) + 32.0 * m, "flops": 4.0 * n * ci}  # pool


def tolerance(case):
    kind, dtype = case["kind"], case.get("dtype")
    if kind == "maps":
        return "exact"
    if kind == "train":  # a rounding that falls on the other side moves activations across the ReLU and back
        return {"rel": 0.02 if dtype == "f16" else 0.03, "max": 0.5}
    if kind == "infer":  # some sixty layers
        return {"rel": 0.01 if dtype == "f16" else 0.03, "max": 0.3}
    return {"rel": {"f32": 1e-5, "f16": 2e-3, "bf16": 1e-2}[dtype]}
