"""The work that users of this library have it do, as cases that can be timed and whose outputs can be compared.

A case is one pass through the public entry points: an operator call as a caller of ``FGMS.backend`` makes it, a
training step of a layer through ``fgms_b200.nn``, an inference call, a step of the encoder-decoder stack, or the
construction of a scene's kernel maps.  The listed cases are the layer shapes of the configurations in
``fgms_b200/workloads.py`` and their neighbours; ``draw`` gives others of the same ranges.

``kind`` says what a pass is:

* ``call``    forward alone through ``backend.fgms_fusion_fwd_cuda`` into a zeroed output (inference);
* ``seq``     forward through ``backend.fgms_fwd_cuda`` with the centre offset separate (the form in which the
              reference's data files come: the map omits the centre);
* ``drop_in`` forward and backward through the ``FGMS.backend`` functions, outputs and gradients zeroed by the caller;
* ``layer``   forward and backward through ``nn.sparse_conv`` and autograd;
* ``infer``   ``nn.sparse_conv_inference`` with bias and ReLU;
* ``step``    one training step of the stack with ``unet.UNetStep``;
* ``module``  one training step of the stack as ``nn.SparseUNet`` with autograd;
* ``maps``    all kernel maps of a scene, ``unet.build_unet_maps``.

``map`` is ``subm`` (3x3x3), ``down`` (2x2x2 stride 2) or ``up`` (its transpose); ``mode`` is ``fp16``, ``tf32``
(fp32 storage) or ``fp32`` (exact).  Clouds: ``uniform``, ``surface`` (planes and boxes), ``lidar`` (a rotating scanner),
``full`` (every voxel of a block occupied).
"""
from __future__ import annotations

import math

import torch

from fgms_b200 import backend, gpu_maps, nn, unet

# surface scenes of a batch lie this far apart along x, so that they share no voxel neighbourhood
SCENE_PITCH = 4096
ELEM = {"fp16": 2, "tf32": 4, "fp32": 4}


def _case(name, kind, **kw):
    c = {"kind": kind, "cloud": "surface", "voxels": 0, "scenes": 1, "map": "subm", "mode": "fp16", "c_in": 0, "c_out": 0}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a serving call on a crop of a scene: a few hundred voxels, all latency
        _case("call_fp16_crop", "call", voxels=301, c_in=32, c_out=32),
        # the reference's CPU-checkable layer: exact fp32, nothing but launches and latency
        _case("dropin_fp32_8k", "drop_in", cloud="uniform", voxels=8000, mode="fp32", c_in=16, c_out=16),
        # a ragged exact-fp32 layer of a middle size: channel counts that no tile divides
        _case("layer_fp32_ragged", "layer", voxels=40009, mode="fp32", c_in=20, c_out=36),
        # an ordinary training layer of an indoor scene
        _case("layer_fp16_indoor", "layer", voxels=100000, c_in=64, c_out=64),
        # the stride-2 convolution between two resolutions, fp32 storage on the tensor cores
        _case("layer_tf32_down", "layer", voxels=200000, map="down", mode="tf32", c_in=32, c_out=64),
        # a wide layer of a LiDAR sweep, called as the reference's caller does
        _case("dropin_fp16_lidar", "drop_in", cloud="lidar", voxels=146000, c_in=128, c_out=128),
        # the per-offset forward with a separate centre, as the reference's data files have it; odd row count, odd widths
        _case("seq_fp16_ragged", "seq", voxels=37013, c_in=96, c_out=160),
        # reproducible inference with bias and ReLU on a fully occupied block
        _case("infer_fp16_block", "infer", cloud="full", voxels=110592, c_in=64, c_out=64),
        # the finest level of the stack for a batch of scenes: short rows, the most pairs
        _case("layer_fp16_batch", "layer", voxels=120000, scenes=8, c_in=32, c_out=32),
        # one training step of the 25-layer stack, one scene per GPU
        _case("step_fp16_scene", "step", voxels=120000),
        # the same stack as a module with autograd on a small scan: many short launches
        _case("module_fp16_small", "module", voxels=8009),
        # the kernel maps of a scene, paid for once per scene
        _case("maps_scene", "maps", voxels=120000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _widths(rng, mode):
    wide = [16, 32, 32, 48, 64, 64, 96, 128, 128, 160, 256]
    a = rng.choice(wide)
    return a, rng.choice(wide if mode == "fp16" or a <= 128 else wide[:9])


def draw(rng):
    kind = rng.choice(["call", "drop_in", "drop_in", "layer", "layer", "layer", "seq", "infer", "step", "module", "maps"])
    if kind == "step":
        return _case(None, kind, voxels=_log(rng, 20_000, 150_000))
    if kind == "module":
        return _case(None, kind, voxels=_log(rng, 3_000, 60_000))
    if kind == "maps":
        return _case(None, kind, cloud=rng.choice(["surface", "lidar"]), voxels=_log(rng, 10_000, 250_000))
    if kind == "infer":
        cloud = rng.choice(["full", "full", "surface"])
        mode = rng.choice(["fp16", "fp16", "tf32"])
        n = _log(rng, 1_000, 110_000)
        if cloud == "full":
            n = max(8, round(n ** (1 / 3))) ** 3
        return _case(None, kind, cloud=cloud, voxels=n, mode=mode, c_in=rng.choice([16, 32, 48, 64, 96, 128]),
                     c_out=rng.choice([16, 32, 48, 64, 96, 128]))
    if kind == "call":
        return _case(None, kind, voxels=_log(rng, 150, 20_000), mode=rng.choice(["fp16", "fp16", "tf32", "fp32"]),
                     c_in=rng.choice([16, 32, 48, 64, 96, 128]), c_out=rng.choice([16, 32, 48, 64, 96, 128]))
    if kind == "seq":
        mode = rng.choice(["fp16", "tf32"])
        a, b = _widths(rng, mode)
        return _case(None, kind, voxels=_log(rng, 5_000, 80_000), mode=mode, c_in=a, c_out=b)
    mode = rng.choice(["fp16", "fp16", "fp16", "tf32", "tf32", "fp32"])
    which = rng.choice(["subm", "subm", "subm", "down", "up"])
    if mode == "fp32":
        return _case(None, kind, cloud=rng.choice(["uniform", "surface"]), voxels=_log(rng, 3_000, 60_000), map=which, mode=mode,
                     c_in=rng.choice([3, 4, 16, 17, 24, 32, 40, 64]), c_out=rng.choice([16, 20, 24, 32, 33, 48, 64]))
    a, b = _widths(rng, mode)
    # the largest layers stay below the batch of scenes: fewer voxels where the rows are long
    top = 250_000 if a * b <= 64 * 64 else (150_000 if a * b <= 128 * 128 else 50_000)
    return _case(None, kind, cloud=rng.choice(["surface", "surface", "lidar", "uniform"]), voxels=_log(rng, 4_000, top), map=which,
                 mode=mode, c_in=a, c_out=b)


# ---- clouds (made on the GPU; int32 [n, 3], no voxel twice, ascending) ------------------------------
def _unique(p):
    key = (p[:, 0].long() << 42) | (p[:, 1].long() << 21) | p[:, 2].long()
    key = torch.unique(key)
    return torch.stack([key >> 42, (key >> 21) & 0x1FFFFF, key & 0x1FFFFF], 1).to(torch.int32)


def _thin(c, n, gen):
    if c.size(0) <= n:
        return c.contiguous()
    keep = torch.randperm(c.size(0), generator=gen, device="cuda")[:n].sort().values
    return c[keep].contiguous()


def _rand(gen, *shape):
    return torch.rand(shape, generator=gen, device="cuda")


def _surface(n, gen):
    """Points of 12 random planes and the faces of 20 random boxes, at unit voxel size, at a scale that gives n voxels."""
    grid = max(24.0, 0.8 * math.sqrt(n))
    nrm = torch.nn.functional.normalize(torch.randn((12, 3), generator=gen, device="cuda"), dim=1)
    ref = torch.zeros_like(nrm)
    ref[torch.arange(12, device="cuda"), nrm.abs().argmin(1)] = 1.0
    u = torch.nn.functional.normalize(torch.linalg.cross(nrm, ref), dim=1)
    v = torch.linalg.cross(nrm, u)
    pc, ext = 0.3 + 0.4 * _rand(gen, 12, 3), 0.5 + 0.5 * _rand(gen, 12)
    size, bc = 0.3 + 0.7 * _rand(gen, 20, 3), 0.2 + 0.6 * _rand(gen, 20, 3)
    plane_area = 4 * ext * ext
    box_area = 2 * (size[:, 0] * size[:, 1] + size[:, 1] * size[:, 2] + size[:, 0] * size[:, 2])
    weight = torch.cat([plane_area, box_area])
    scale = math.sqrt(1.1 * n / float(weight.sum()))
    for _ in range(40):
        m = int(6 * scale * scale * float(weight.sum())) + 64
        which = torch.multinomial(weight, m, replacement=True, generator=gen)
        r = _rand(gen, m, 3)
        pl, bx = which.clamp(max=11), (which - 12).clamp(min=0)
        e = (ext[pl] * scale)[:, None]
        on_plane = pc[pl] * grid + (2 * r[:, :1] - 1) * e * u[pl] + (2 * r[:, 1:2] - 1) * e * v[pl]
        sz = size[bx] * scale
        face = torch.randint(0, 6, (m,), generator=gen, device="cuda")
        side = torch.nn.functional.one_hot(face % 3, 3).bool()
        r = torch.where(side, (face // 3).float()[:, None].expand(m, 3), r)
        on_box = bc[bx] * grid + (r - 0.5) * sz
        p = torch.where((which < 12)[:, None], on_plane, on_box)
        p = p[((p >= 0) & (p < grid)).all(1)]
        c = _unique(p.floor())
        if c.size(0) >= n:
            break
        scale *= 1.05
    return _thin(c, n, gen)


def _lidar(n, gen):
    """Sweeps of a 64-beam scanner over a ground plane, log-normal ranges, voxels of 5 cm, thinned to n voxels."""
    elev = torch.deg2rad(torch.linspace(-25.0, 3.0, 64, device="cuda"))[:, None]
    steps, parts, c = 2048, [], None
    for _ in range(8):
        az = (torch.arange(steps, device="cuda") + _rand(gen, 1))[None, :] * (2 * math.pi / steps)
        r = torch.exp(math.log(15.0) + 0.6 * torch.randn((64, steps), generator=gen, device="cuda")).clamp(1.0, 80.0)
        r = torch.minimum(r, torch.where(elev < 0, -1.7 / torch.sin(elev), torch.full_like(elev, 1e9)))
        p = torch.stack([r * torch.cos(elev) * torch.cos(az), r * torch.cos(elev) * torch.sin(az), r * torch.sin(elev)], -1)
        p = p.reshape(-1, 3) + torch.tensor([50.0, 50.0, 3.0], device="cuda")
        p = p[((p >= 0) & (p < torch.tensor([100.0, 100.0, 4.0], device="cuda"))).all(1)]
        parts.append((p / 0.05).floor())
        c = _unique(torch.cat(parts))
        if c.size(0) >= n:
            break
    return _thin(c, n, gen)


def _uniform(n, gen):
    side = max(8, round((n * 32.8) ** (1 / 3)))  # 8 000 voxels in 64^3
    cells = torch.randperm(side ** 3, generator=gen, device="cuda")[:n].sort().values
    return torch.stack([cells // (side * side), cells // side % side, cells % side], 1).to(torch.int32).contiguous()


def _full(n, gen):
    side = round(n ** (1 / 3))
    i = torch.arange(side ** 3, device="cuda")
    return torch.stack([i // (side * side), i // side % side, i % side], 1).to(torch.int32).contiguous()


CLOUDS = {"surface": _surface, "lidar": _lidar, "uniform": _uniform, "full": _full}


def _in_frame(c, gen):
    """The scene in another frame: axes exchanged, some of them reversed, moved by whole voxels of the coarsest level,
    rows ascending again.  Every map of every level changes, the numbers of voxels and pairs do not."""
    axes = torch.randperm(3, generator=gen, device="cuda")
    flip = torch.randint(0, 2, (3,), generator=gen, device="cuda", dtype=torch.int32)
    move = 16 * torch.randint(0, 32, (3,), generator=gen, device="cuda", dtype=torch.int32)
    c = c[:, axes]
    side = (c.max(0).values // 16 + 1) * 16
    return _unique(torch.where(flip.bool(), side - 1 - c, c) + move)


def _cloud(case, gen):
    """The case's scenes are the same for every seed; the frame they are seen in comes from ``gen``."""
    shape = torch.Generator(device="cuda")
    shape.manual_seed(case["voxels"])
    parts = []
    for s in range(case["scenes"]):
        c = _in_frame(CLOUDS[case["cloud"]](case["voxels"], shape), gen)
        c[:, 0] += SCENE_PITCH * s
        parts.append(c)
    return torch.cat(parts).contiguous()


# ---- maps ----------------------------------------------------------------------------------------------------------
def _map(case, coords):
    if case["map"] == "subm":
        return gpu_maps.build_submanifold_map(coords, 3)
    down = gpu_maps.build_strided_map(coords, 2)
    return down if case["map"] == "down" else gpu_maps.transpose_map(down, coords)


def _without_centre(km):
    """The map without its centre offset's pairs, and the host counts per offset."""
    kpos = km.kpos.cpu()
    a, b = int(kpos[13]), int(kpos[14])
    keep = torch.cat([torch.arange(0, a), torch.arange(b, int(kpos[27]))]).cuda()
    nnz = kpos.diff()
    nnz[13] = 0
    new = torch.zeros_like(kpos)
    new[1:] = nnz.cumsum(0)
    return (gpu_maps.DeviceKernelMap(km.n_in, km.n_out, 27, new.cuda(), km.imap[keep].contiguous(), km.omap[keep].contiguous()),
            nnz.to(torch.int32))


# ---- a pass ----------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) * 7919 + 17)
    kind = case["kind"]
    coords = _cloud(case, gen)
    s = {"kind": kind, "coords": coords}
    if kind == "maps":
        return s

    def normal(rows, cols, dtype, gain=1.0):
        return (gain * torch.randn((rows, cols), generator=gen, device="cuda")).to(dtype)

    if kind in ("step", "module"):
        spec = unet.minkunet_spec()
        umaps = unet.build_unet_maps(coords)
        weights = []
        for l in spec:  # uniform with the bound that keeps the features' variance about constant through the stack
            km = umaps.of(l)
            bound = math.sqrt(3.0 / (l.c_in * max(km.pairs / km.n_out, 1.0))) * (2 ** -0.5 if l.skip else 1.0)
            weights.append(((2 * _rand(gen, l.k_vol, l.c_in, l.c_out) - 1) * bound).half())
        feats = normal(coords.size(0), spec[0].c_in, torch.float16)
        grad = normal(coords.size(0), spec[-1].c_out, torch.float16, 0.25)
        s.update(umaps=umaps, feats=feats, grad=grad)
        if kind == "step":
            s["step"] = unet.UNetStep(spec, umaps, weights, feats, grad)
        else:
            s["net"] = nn.SparseUNet(spec)
            s["net"].load_weights(weights)
            s["params"] = list(s["net"].parameters())
        return s

    dtype = torch.float16 if case["mode"] == "fp16" else torch.float32
    km = _map(case, coords)
    c_in, c_out = case["c_in"], case["c_out"]
    bound = 1.0 / math.sqrt(c_in * km.k_vol)  # kaiming-uniform
    s["arch80"] = case["mode"] != "fp32"
    s["feats"] = normal(km.n_in, c_in, dtype)
    s["weight"] = ((2 * _rand(gen, km.k_vol, c_in, c_out) - 1) * bound).to(dtype)
    if kind == "seq":
        km, s["nnz"] = _without_centre(km)
    s["km"], s["pairs"] = km, km.pairs
    if kind == "infer":
        s["bias"] = (0.1 * torch.randn(c_out, generator=gen, device="cuda")).to(dtype)
    elif kind in ("call", "seq", "drop_in"):
        s["out"] = torch.empty((km.n_out, c_out), dtype=dtype, device="cuda")
    if kind in ("drop_in", "layer"):
        s["grad"] = normal(km.n_out, c_out, dtype)
    if kind == "drop_in":
        s["feats_grad"], s["weight_grad"] = torch.empty_like(s["feats"]), torch.empty_like(s["weight"])
    if kind == "layer":
        s["feats"].requires_grad_()
        s["weight"].requires_grad_()
    return s


def run(s):
    kind = s["kind"]
    if kind == "maps":
        m = unet.build_unet_maps(s["coords"])
        return [[k.kpos, k.imap, k.omap] for k in m.subm + m.down + m.up] + [d.out_coords for d in m.down]
    if kind == "step":
        s["step"].run()
        return {"out": s["step"].val[s["step"].out_name], "weight_grad": s["step"].w_grad}
    if kind == "module":
        out = s["net"](s["feats"], s["umaps"])
        return {"out": out.detach(), "weight_grad": torch.autograd.grad(out, s["params"], s["grad"])}
    km, arch80 = s["km"], s["arch80"]
    if kind == "infer":
        return nn.sparse_conv_inference(s["feats"], s["weight"], km, bias=s["bias"], relu=True, arch80=arch80)
    if kind == "layer":
        out = nn.sparse_conv(s["feats"], s["weight"], km, arch80)
        feats_grad, weight_grad = torch.autograd.grad(out, (s["feats"], s["weight"]), s["grad"])
        return {"out": out.detach(), "feats_grad": feats_grad, "weight_grad": weight_grad}
    out = s["out"]
    out.zero_()
    if kind == "seq":
        backend.fgms_fwd_cuda(s["feats"], s["weight"], s["pairs"], out, s["nnz"], km.kpos, km.imap, km.omap, True, arch80)
        return out
    backend.fgms_fusion_fwd_cuda(s["feats"], s["weight"], s["pairs"], out, km.kpos, None, km.imap, km.omap, False, arch80)
    if kind == "call":
        return out
    s["feats_grad"].zero_()
    s["weight_grad"].zero_()
    backend.fgms_bwd_cuda(s["grad"], s["feats"], s["weight"], s["pairs"], s["feats_grad"], s["weight_grad"], km.kpos, None,
                          km.imap, km.omap, False, arch80)
    return {"out": out, "feats_grad": s["feats_grad"], "weight_grad": s["weight_grad"]}


# ---- what a pass cannot do without -------------------------------------------------------------------------------------
# Typical counts of the clouds above: pairs per voxel of a 3x3x3 map, and voxels of the next coarser level per voxel.
PAIRS = {"surface": 9.5, "lidar": 2.1, "uniform": 1.8, "full": 25.0}
COARSER = {"surface": 0.28, "lidar": 0.75, "uniform": 0.9, "full": 0.125}


def work(case):
    kind, n = case["kind"], case["voxels"] * case["scenes"]
    es = ELEM[case["mode"]]
    ppv, coarser = PAIRS[case["cloud"]], COARSER[case["cloud"]]
    if kind == "maps":  # coordinates in, every level's maps and coordinates out
        total = 12.0 * n
        for level in range(5):
            total += 8 * ppv * n
            if level < 4:
                total += 16 * n + 12 * coarser * n
            n *= coarser
        return {"bytes": total, "flops": 0.0}
    if kind in ("step", "module"):
        total = flops = 0.0
        level = [n * coarser ** r for r in range(5)]
        for i, l in enumerate(unet.minkunet_spec()):
            pairs = ppv * level[l.res_in] if l.kind == "subm" else level[min(l.res_in, l.res_out)]
            rows_in, rows_out = level[l.res_in] * l.c_in, level[l.res_out] * l.c_out
            # forward: input, output; backward: input and output gradient again, input gradient; maps and weights both ways
            total += 2 * (2 * rows_in + 2 * rows_out + (rows_in if i else 0)) + 16 * pairs + 2 * 3 * l.k_vol * l.c_in * l.c_out
            flops += 2.0 * pairs * l.c_in * l.c_out * (3 if i else 2)
        return {"bytes": total, "flops": flops}
    a, b = case["c_in"], case["c_out"]
    k_vol = 27 if case["map"] == "subm" else 8
    n_in, n_out, pairs = n, n, ppv * n
    if case["map"] != "subm":
        n_in, n_out, pairs = (n, coarser * n, n) if case["map"] == "down" else (coarser * n, n, n)
    passes = 3 if kind in ("drop_in", "layer") else 1
    rows = n_in * a + n_out * b
    # features, output, weights and map; with a backward also the output gradient, both gradients
    return {"bytes": (1 if passes == 1 else 2) * es * (rows + k_vol * a * b) + 8.0 * pairs, "flops": 2.0 * pairs * a * b * passes}


def tolerance(case):
    if case["kind"] == "maps":
        return "exact"
    if case["kind"] in ("step", "module"):
        return {"rel": 2e-2}  # 25 layers of fp16 activations
    # fp16 storage adds up to 27 partial results per row in fp16, a weight gradient those of many blocks; tf32 rounds
    # its inputs to 11 bits; exact fp32 sums up to about 1e5 products
    return {"fp16": {"rel": 1e-2}, "tf32": {"rel": 1e-3}, "fp32": {"rel": 1e-5}}[case["mode"]]
