"""What this package is measured on: whole frames of one groom, a batched
frame of many grooms, the learned shading passes, and the surrogate's
inference, training and sample generation, each through the public entry
points (``HairRenderer``, ``HairBatch``, ``Surrogate``) as a renderer or the
training command calls them.

``listed()`` holds the cases, ``draw`` makes more of the same ranges,
``prepare`` builds what a program holds before the call (grooms uploaded,
targets sized, weights set), ``run`` is one pass, ``work`` the bytes and
operations a pass cannot do without, ``exact`` the same outputs in 64 bits
where they are plain numbers.
"""
import functools
import math

import numpy as np
import torch

from bevy_hair_gb300 import abi, configs, envmap, groom, host
from bevy_hair_gb300 import surrogate as S
from bevy_hair_gb300.pipeline import HairBatch, HairRenderer, Light, pack_lights

F = np.float32


def listed():
    return [
        # A preview thumbnail: a tuft in a small window, where launches and latency are the cost.
        dict(name="frame_thumbnail", kind="frame", strands=300, segments=16, style="straight", width=96, height=64,
             dom=32, lod=True, filter=True, lights=1, probe=False, distance=1000.0, lam=3.0),
        # The 512x512 benchmark frame: 10k straight strands, LOD off, one key light.
        dict(name="frame_512", kind="frame", strands=10_000, segments=32, style="straight", width=512, height=512,
             dom=256, lod=False, filter=True, lights=1, probe=False, distance=1000.0, lam=3.0),
        # The headline frame: 100k wavy strands at 1080p, 1024^2 opacity map, 9 lights, light probe.
        dict(name="frame_1080p", kind="frame", strands=100_000, segments=64, style="wavy", width=1920, height=1080,
             dom=1024, lod=True, filter=True, lights=9, probe=True, distance=900.0, lam=3.0),
        # The largest frame: 200k curly strands at 3840x2160, 2048^2 opacity map, 16 lights, several LOD levels.
        dict(name="frame_2160p", kind="frame", strands=200_000, segments=128, style="curly", width=3840, height=2160,
             dom=2048, lod=True, filter=True, lights=16, probe=False, distance=1400.0, lam=1.5),
        # A window of odd size over a scene with its own depth buffer, without opacity map or filter
        # (the reference's cheaper settings): strands are generated in the camera raster itself.
        dict(name="frame_odd_nomap", kind="frame", strands=30_011, segments=48, style="curly", width=1283, height=717,
             dom=0, lod=True, filter=False, lights=5, probe=False, distance=700.0, lam=3.0),
        # A crowd: grooms of uneven size, each with its own view and 512^2 map, one graph replay.
        dict(name="batch_24", kind="batch", items=24, strands=20_000, side=1024, dom=512, lights=3),
        # The compact learned BSDF in the shade pass (1080p groom, 9 lights, light probe).
        dict(name="shade_compact_1080p", kind="shade", model=3, strands=100_000, segments=64, style="wavy", width=1920,
             height=1080, dom=1024, lod=True, filter=True, lights=9, probe=True, distance=900.0, lam=3.0),
        # The accurate learned lobes (4 x 64 network) in the same pass.
        dict(name="shade_deep_1080p", kind="shade", model=1, strands=100_000, segments=64, style="wavy", width=1920,
             height=1080, dom=1024, lod=True, filter=True, lights=9, probe=True, distance=900.0, lam=3.0),
        # Network evaluation on its own, a ragged million of rows.
        dict(name="infer_deep_1m", kind="infer", arch=0, tc=True, rows=1_000_003),
        # Training as the package's own command does it: batches of 16,384, Adam, weights read back at the end.
        dict(name="train_deep", kind="train", arch=0, batch=16_384, steps=16),
        dict(name="train_compact", kind="train", arch=1, batch=16_384, steps=16),
        # The FP64-integrated samples the training set is made of.
        dict(name="samples_256k", kind="samples", rows=262_144),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("frame", "frame", "frame", "batch", "shade", "infer", "train", "samples"))
    if kind in ("frame", "shade"):
        width = _log(rng, 64, 3840)
        c = dict(kind=kind, strands=_log(rng, 64, 120_000), segments=_log(rng, 16, 128),
                 style=rng.choice(("straight", "wavy", "curly")), width=width,
                 height=max(48, int(width * rng.uniform(0.5, 0.58))), dom=_log(rng, 32, 1500), lod=rng.random() < 0.8,
                 filter=rng.random() < 0.8, lights=rng.randint(1, 16), probe=rng.random() < 0.3,
                 distance=rng.uniform(600.0, 1600.0), lam=rng.choice((1.5, 3.0)))
        if kind == "shade":
            c["model"] = rng.choice((1, 2, 3))
        elif rng.random() < 0.25:
            c["dom"] = 0
        return c
    if kind == "batch":
        return dict(kind=kind, items=rng.randint(2, 16), strands=_log(rng, 2_000, 20_000), side=_log(rng, 300, 1024),
                    dom=_log(rng, 64, 512), lights=rng.randint(1, 6))
    if kind == "infer":
        arch = rng.randint(0, 1)
        return dict(kind=kind, arch=arch, tc=arch == 0 and rng.random() < 0.5, rows=_log(rng, 100, 1_000_000))
    if kind == "train":
        return dict(kind=kind, arch=rng.randint(0, 1), batch=_log(rng, 1_000, 16_384), steps=rng.randint(4, 16))
    return dict(kind=kind, rows=_log(rng, 1_000, 250_000))


# ---------------------------------------------------------------- scenes


@functools.lru_cache(maxsize=64)
def _groom(strands, segments, style, seed):
    """One baked groom; the baker is not what is measured."""
    return groom.bake(groom.synthetic_strands(strands, segments, style, configs.SEED_BASE + seed))


def _varied(mesh, rng):
    """The groom with other curl and occlusion per lock, as an artist's pass over it leaves it."""
    n = mesh.bundle_count
    style = (mesh.style.reshape(n, -1) * rng.uniform(0.7, 1.2, (n, 1)).astype(F)).reshape(-1, 4)
    layers = mesh.layers.copy()
    layers["pos_ao"].reshape(n, -1, 4)[..., 3] *= rng.uniform(0.8, 1.0, (n, 1)).astype(F)
    return groom.HairMesh(mesh.bundles, layers, style, mesh.bounds_min, mesh.bounds_max)


def _camera(rng, width, height, distance):
    azimuth, elevation = rng.uniform(0.0, 2.0 * math.pi), rng.uniform(-0.05, 0.35)
    target = np.array([0.0, -10.0, 0.0], dtype=F)
    away = np.array([math.sin(azimuth) * math.cos(elevation), math.sin(elevation),
                     math.cos(azimuth) * math.cos(elevation)], dtype=F)
    return host.View(host.looking_at(target + away * F(distance), target),
                     host.perspective_infinite_reverse_rh(math.pi / 4.0, width / height, 0.1), width, height)


def _lights(rng, count, spots):
    """A shadowing key light, then point lights around the groom, spots and a rectangle among them if asked for."""
    sun = host.normalize_or(host.v3(*(np.array([0.35, 0.82, 0.45]) + rng.uniform(-0.15, 0.15, 3))), (0, 1, 0))
    out = [Light(kind=abi.LIGHT_DIRECTIONAL, color=tuple(rng.uniform(2.0, 3.5, 3).tolist()),
                 direction=tuple(sun.tolist()), casts_shadows=True)]
    for i in range(1, count):
        a = 2.0 * math.pi * (i + rng.uniform(0.2, 0.8)) / count
        kind = (abi.LIGHT_SPOT if i % 3 == 1 else abi.LIGHT_RECT if i % 3 == 2 else abi.LIGHT_POINT) if spots \
            else abi.LIGHT_POINT
        out.append(Light(kind=kind, color=tuple((rng.uniform(0.6, 1.0, 3) * 6.0e4).tolist()),
                         position=(500.0 * math.cos(a), 50.0 + 60.0 * math.sin(3 * a), 500.0 * math.sin(a)),
                         direction=(-math.cos(a), 0.0, -math.sin(a)), range=1250.0, spot_scale=2.5, spot_offset=-1.2,
                         right=(-math.sin(a), 0.0, math.cos(a)), up=(0.0, 1.0, 0.0), width=80.0, height=40.0))
    return out, [host.Directional(sun, True)]


def _scene(rng, mesh, width, height, dom, distance, lights, directionals, *, lod, use_filter, lam):
    yaw = rng.uniform(-0.5, 0.5)
    model = np.eye(4, dtype=F)
    model[0, 0] = model[2, 2] = F(math.cos(yaw))
    model[0, 2], model[2, 0] = F(math.sin(yaw)), F(-math.sin(yaw))
    g = host.HairGroom(world_from_model=model, lam=lam, albedo=tuple(rng.uniform(0.05, 0.4, 3).tolist()),
                       roughness=float(rng.uniform(0.25, 0.4)), lod=lod, filter=use_filter, deep_opacity=dom > 0,
                       ambient_occlusion=True)
    view = _camera(rng, width, height, distance * rng.uniform(0.9, 1.1))
    return configs.Scene("scene", mesh, g, view, (max(dom, 1), max(dom, 1)), lights, directionals)


@functools.lru_cache(maxsize=1)
def _sky():
    return envmap.procedural()


@functools.lru_cache(maxsize=1)
def _stream():
    """One stream for every renderer of the program, as an application's render thread has one."""
    return torch.cuda.Stream()


class _Device:
    """A library buffer as a tensor (the memory stays the library's)."""

    def __init__(self, owner, where, typestr):
        address, nbytes = where
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (nbytes // int(typestr[2:]),), "typestr": typestr, "version": 2,
                                         "data": (address, False)}


def _view(owner, where, typestr):
    return torch.as_tensor(_Device(owner, where, typestr), device="cuda")


class _Owner:
    """A renderer and its grooms; given back when neither a state nor a tensor over their memory is left."""

    def __init__(self):
        self.renderer = HairRenderer(torch.cuda.current_device(), _stream().cuda_stream)
        self.grooms = []

    def __del__(self):
        torch.cuda.synchronize()
        for s in list(getattr(self.renderer, "_batches", ())):
            s.close()
        for g in self.grooms:
            g.close()
        self.renderer.close()


class _State:
    """What a program keeps between passes."""

    def __init__(self):
        self.owner = _Owner()
        self.renderer = self.owner.renderer

    def upload(self, mesh):
        self.owner.grooms.append(self.renderer.upload(mesh))
        return self.owner.grooms[-1]


def _buffers(owner, names):
    """The context's targets; words and counters as integers."""
    kinds = {"center": (abi.BUF_CENTER, "<i8"), "conservative": (abi.BUF_CONSERVATIVE, "<i8"),
             "beta": (abi.BUF_BETA, "<i4"), "dom": (abi.BUF_DOM, "<i4"), "shaded": (abi.BUF_SHADED, "<f4"),
             "shaded_depth": (abi.BUF_SHADED_DEPTH, "<f4"), "color": (abi.BUF_COLOR, "<f4"),
             "depth": (abi.BUF_DEPTH, "<f4")}
    return {k: _view(owner, owner.renderer.buffer(kinds[k][0]), kinds[k][1]) for k in names}


def _prepare_frame(case, seed):
    rng = np.random.default_rng(seed)
    s = _State()
    r = s.renderer
    mesh = _varied(_groom(case["strands"], case["segments"], case["style"], 1), rng)
    lights, directionals = _lights(rng, case["lights"], spots=not case["dom"])
    sc = _scene(rng, mesh, case["width"], case["height"], case["dom"], case["distance"], lights, directionals,
                lod=case["lod"], use_filter=case["filter"], lam=case["lam"])
    r.ensure_targets(case["width"], case["height"], case["dom"], case["dom"])
    if case["probe"]:
        sky = _sky()
        angle = rng.uniform(0.0, math.pi)
        r.set_environment(envmap.Environment(sky.specular, sky.diffuse, (0.0, math.sin(angle), 0.0, math.cos(angle)),
                                             float(rng.uniform(0.5, 1.5))))
    s.mesh = s.upload(mesh)
    s.camera, dom = sc.params()
    s.dom = dom if case["dom"] else None
    s.lights = sc.light_array()
    s.scene_depth = None
    if not case["dom"]:  # a wall that cuts through the groom, in the camera's reverse-Z depth
        x = torch.linspace(0.0, 1.0, case["width"], device="cuda")[None, :].expand(case["height"], -1)
        s.scene_depth = (0.1 / (case["distance"] * (0.85 + 0.5 * x))).contiguous()
    s.outputs = None
    if case["kind"] == "frame":
        s.outputs = _buffers(s.owner, ["center", "conservative", "beta", "shaded", "shaded_depth", "color", "depth"] +
                             (["dom"] if case["dom"] else []))
        return s
    # the learned shade pass: the frame up to shading is there, the network bound
    arch = abi.MLP_ARCH_COMPACT if case["model"] == 3 else abi.MLP_ARCH_DEEP
    r.render_groom(s.mesh, s.camera, s.dom, s.lights)
    s.network = S.Surrogate(r, S.load_params(arch), arch)
    r.bind_surrogate(s.network)
    s.outputs = _buffers(s.owner, ["shaded", "shaded_depth"])
    return s


def _prepare_batch(case, seed):
    rng, sizes = np.random.default_rng(seed), np.random.default_rng(7)
    s = _State()
    lights, directionals = _lights(rng, case["lights"], spots=False)
    scenes, shapes = [], []
    for k in range(case["items"]):
        # sizes are the case's, log-uniform; poses, looks and lights are the seed's
        n = int(round(math.exp(sizes.uniform(math.log(1_000), math.log(case["strands"])))))
        segments = int(round(math.exp(sizes.uniform(math.log(16), math.log(128)))))
        side = int(round(math.exp(sizes.uniform(math.log(256), math.log(case["side"])))))
        mesh = _varied(_groom(n, segments, ("straight", "wavy", "curly")[k % 3], 400 + k), rng)
        scenes.append(_scene(rng, mesh, side, side, case["dom"], rng.uniform(700.0, 1100.0), lights, directionals,
                             lod=True, use_filter=True, lam=3.0))
        shapes.append((side, side, case["dom"], case["dom"]))
    s.batch = HairBatch(s.renderer, [s.upload(sc.mesh) for sc in scenes], shapes)
    s.params = [sc.params() for sc in scenes]
    s.lights = pack_lights(lights)
    kinds = {"color": (abi.BUF_COLOR, "<f4"), "center": (abi.BUF_CENTER, "<i8")}
    if case["items"] <= 16:
        kinds |= {"depth": (abi.BUF_DEPTH, "<f4"), "dom": (abi.BUF_DOM, "<i4")}
    s.outputs = {"%s_%d" % (n, k): _view(s.owner, s.batch.buffer(k, b), t)
                 for k in range(case["items"]) for n, (b, t) in kinds.items()}
    return s


# ---------------------------------------------------------------- the surrogate


def _rows(rows, seed, lobes=False):
    """Network inputs of the training distribution (and smooth stand-in lobes, log-transformed), from torch alone."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = torch.rand((rows, 8), generator=g, device="cuda", dtype=torch.float64)
    phi = math.pi * u[:, 2]
    sigma = torch.exp(math.log(0.02) + math.log(400.0) * u[:, 3:6])
    beta_m, beta_n = 0.03 + 0.27 * u[:, 6], 0.2 + 0.6 * u[:, 7]
    x = torch.cat([2.0 * u[:, :2] - 1.0, torch.cos(phi)[:, None], torch.sin(phi)[:, None], sigma, beta_m[:, None],
                   beta_n[:, None], torch.full((rows, 1), 1.55, device="cuda", dtype=torch.float64)], dim=1)
    if not lobes:
        return x.float(), None
    half = torch.asin(x[:, 0]) + torch.asin(x[:, 1])
    out = []
    for p, (shift, width, exit_at) in enumerate(((0.08, 1.0, 0.0), (-0.04, 0.5, math.pi), (-0.12, 2.0, 0.0),
                                                 (0.0, 2.0, math.pi))):
        b = width * beta_m
        m = torch.exp(-0.5 * ((half - shift) / b) ** 2) / (math.sqrt(2.0 * math.pi) * b)
        n = torch.exp(-0.5 * ((phi - exit_at) / (2.0 * beta_n)) ** 2)
        out.append(0.25 * (m * n)[:, None] * torch.exp(-float(p) * sigma))
    return x.float(), torch.log1p(torch.cat(out, dim=1) / 1e-3).float()


def _train_data(case, seed):
    x, y = _rows(case["batch"] * case["steps"], seed, lobes=True)
    rates = [3e-3 * (k + 1) / case["steps"] for k in range(case["steps"])]
    return x, y, rates


def _start_params(case):
    """Where training goes on from: the shipped weights, moved a little so that gradients are those of training."""
    p = S.load_params(case["arch"])
    rng = np.random.default_rng(11)
    return (p * rng.uniform(0.9, 1.1, p.shape)).astype(F)


def _prepare_network(case, seed):
    s = _State()
    if case["kind"] == "samples":
        n = case["rows"]
        s.seed = S.SAMPLE_SEED + seed
        s.outputs = dict(inputs=torch.empty((n, 10), device="cuda"), targets=torch.empty((n, 12), device="cuda"),
                         lobes=torch.empty((n, 12), dtype=torch.float64, device="cuda"))
    elif case["kind"] == "infer":
        s.network = S.Surrogate(s.renderer, S.load_params(case["arch"]), case["arch"])
        s.inputs, _ = _rows(case["rows"], seed)
        s.outputs = torch.empty((case["rows"], s.network.n_out), device="cuda")
    else:
        s.params = _start_params(case)
        s.network = S.Surrogate(s.renderer, s.params, case["arch"])
        x, y, rates = _train_data(case, seed)
        b = case["batch"]
        s.losses = torch.zeros(case["steps"], device="cuda")
        s.steps = [(x[k * b:(k + 1) * b], y[k * b:(k + 1) * b], b, rates[k], s.losses[k:k + 1])
                   for k in range(case["steps"])]
    return s


def prepare(case, seed):
    kind = case["kind"]
    s = (_prepare_frame if kind in ("frame", "shade") else _prepare_batch if kind == "batch" else _prepare_network)(
        case, seed)
    s.case = case
    torch.cuda.synchronize()
    return s


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "frame":
        s.renderer.render_groom(s.mesh, s.camera, s.dom, s.lights,
                                scene_depth_ptr=None if s.scene_depth is None else s.scene_depth.data_ptr())
    elif kind == "shade":
        s.renderer.shade(s.camera, s.lights, model=case["model"])
    elif kind == "batch":
        for k, (camera, dom) in enumerate(s.params):
            s.batch.set_params(k, camera, dom)
        s.batch.frame(s.lights)
    elif kind == "infer":
        (s.network.infer_tc if case["tc"] else s.network.infer)(s.inputs, case["rows"], s.outputs)
    elif kind == "samples":
        o = s.outputs
        S.samples(s.renderer, s.seed, 0, case["rows"], o["inputs"], o["targets"], o["lobes"])
    else:
        s.network.set_params(s.params)
        for step in s.steps:
            s.network.train_step(*step)
        return {"params": s.network.get_params(), "losses": s.losses}
    return s.outputs


# ---------------------------------------------------------------- what a pass cannot do without


def _groom_bytes(strands):
    # bundles the baker makes of so many strands, about; 64 cage corners and 1,024 style texels each
    return min(strands, 20.0 * strands ** 0.53) * (16 + 64 * 32 + 1024 * 16)


def work(case):
    kind = case["kind"]
    params = {0: abi.MLP_PARAMS, 1: abi.MLP_COMPACT_PARAMS}
    flops = {0: 2 * (10 * 64 + 3 * 64 * 64 + 64 * 12), 1: 2 * (10 * 32 + 32 * 32 + 32 * 3)}
    if kind == "frame":
        px, texels = case["width"] * case["height"], case["dom"] ** 2
        per_px = 8 + 8 + 4 + 16 + 4 + 16 + 4 + (20 if case["filter"] else 0) + (0 if case["dom"] else 4)
        # ~150 operations per control point, ~400 per light and covered pixel (about a third of the image)
        return {"bytes": _groom_bytes(case["strands"]) + per_px * px + 68 * texels,
                "flops": 150.0 * 65 * case["strands"] + 400.0 * case["lights"] * px / 3}
    if kind == "batch":
        items, top = case["items"], case["strands"]
        strands = items * (top - 1_000) / math.log(top / 1_000)
        side = case["side"]
        px = items * (side ** 2 - 256 ** 2) / (2 * math.log(side / 256))
        return {"bytes": items * _groom_bytes(strands / items) + 80 * px + 68 * items * case["dom"] ** 2,
                "flops": 150.0 * 65 * strands + 400.0 * case["lights"] * px / 3}
    if kind == "shade":
        px = case["width"] * case["height"]
        return {"bytes": 32.0 * px + 4 * case["dom"] ** 2, "flops": flops[int(case["model"] == 3)] * case["lights"] * px / 4}
    if kind == "infer":
        return {"bytes": case["rows"] * 4.0 * (10 + (3 if case["arch"] else 12)) + 4 * params[case["arch"]],
                "flops": float(case["rows"] * flops[case["arch"]])}
    if kind == "train":
        rows = case["batch"] * case["steps"]
        return {"bytes": rows * 88.0 + case["steps"] * 28.0 * params[case["arch"]], "flops": 3.0 * rows * flops[case["arch"]]}
    # samples: 64 nodes x 2 integrals; transcendental functions counted as ~20 operations each
    return {"bytes": case["rows"] * (40.0 + 48.0 + 96.0), "flops": case["rows"] * 64.0 * 2 * 20 * 20}


# ---------------------------------------------------------------- 64 bits


def _network64(case, flat):
    """The layers (W, b) of a flat parameter vector, as float64 tensors."""
    shapes = ((32, 16), (32, 32), (16, 32)) if case["arch"] else ((64, 16), (64, 64), (64, 64), (64, 64), (16, 64))
    out, at = [], 0
    for rows, cols in shapes:
        w = flat[at:at + rows * cols].reshape(rows, cols)
        at += rows * cols
        out += [w, flat[at:at + rows]]
        at += rows
    return out


def _forward64(net, x, n_out):
    x = x.double()
    log_mid = math.log(0.4)
    h = torch.cat([x[:, :4], (torch.log(x[:, 4:7].clamp_min(1e-6)) - log_mid) / math.log(20.0),
                   (x[:, 7:8] - 0.165) / 0.135, (x[:, 8:9] - 0.5) / 0.3, (x[:, 9:10] - 1.55) * 10.0,
                   torch.zeros((len(x), 6), dtype=torch.float64, device=x.device)], dim=1)
    for k in range(0, len(net), 2):
        h = h @ net[k].T + net[k + 1]
        if k + 2 < len(net):
            h = torch.relu(h)
    return h[:, :n_out]


def _train64(case, seed):
    n_out = 3 if case["arch"] else 12
    x, y, rates = _train_data(case, seed)
    y = y.double()
    if case["arch"]:
        lobes = 1e-3 * torch.expm1(y)
        y = torch.log1p((lobes[:, 0:3] + lobes[:, 3:6] + lobes[:, 6:9] + 0.7 * lobes[:, 9:12]) / 1e-3)
    p = torch.from_numpy(_start_params(case)).cuda().double().requires_grad_(True)
    m, v, losses = torch.zeros_like(p), torch.zeros_like(p), []
    b = case["batch"]
    for k, rate in enumerate(rates):
        rows = slice(k * b, (k + 1) * b)
        loss = ((_forward64(_network64(case, p), x[rows], n_out) - y[rows]) ** 2).sum()
        (g,) = torch.autograd.grad(loss, p)
        losses.append(loss.detach())
        with torch.no_grad():
            g = g / (b * n_out)
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g * g
            p -= rate * (m / (1.0 - 0.9 ** (k + 1))) / (torch.sqrt(v / (1.0 - 0.999 ** (k + 1))) + 1e-8)
    return {"params": p.detach(), "losses": torch.stack(losses)}


def _hash64(z):
    """SplitMix64 on int64 tensors."""
    def shifted(a, k):
        return (a >> k) & ((1 << (64 - k)) - 1)

    def signed(c):
        return c - (1 << 64) if c >= 1 << 63 else c

    z = z + signed(0x9E3779B97F4A7C15)
    z = (z ^ shifted(z, 30)) * signed(0xBF58476D1CE4E5B9)
    z = (z ^ shifted(z, 27)) * signed(0x94D049BB133111EB)
    return z ^ shifted(z, 31)


def _samples64(rows, seed, tilt=float(F(0.08))):
    """The lobes of a dielectric cylinder (Marschner et al. 2003, d'Eon et al. 2011) and the dual-scattering
    back lobe (Zinke et al. 2008), 64-point Gauss-Legendre over the entry angle."""
    index = torch.arange(rows, device="cuda", dtype=torch.int64)

    def unit(dim):
        return ((_hash64(seed ^ _hash64(index * 16 + dim)) >> 40) & 0xFFFFFF).float() * 2.0 ** -24

    def affine(lo, span, dim):  # of float32 constants, rounded once
        return (float(F(lo)) + float(F(span)) * unit(dim).double()).float()

    phi = math.pi * unit(2).double()
    x = torch.stack([2.0 * unit(0) - 1.0, 2.0 * unit(1) - 1.0, torch.cos(phi).float(), torch.sin(phi).float()] +
                    [torch.exp(math.log(0.02) + math.log(400.0) * unit(3 + c).double()).float() for c in range(3)] +
                    [affine(0.03, 0.27, 6), affine(0.2, 0.6, 7), torch.full((rows,), 1.55, device="cuda")], dim=1)
    z = x.double()
    sin_o = z[:, 1]
    th_i, th_o = torch.asin(z[:, 0]), torch.asin(sin_o)
    th_h, phi, eta = th_i + th_o, torch.atan2(z[:, 3], z[:, 2]), z[:, 9]
    beta_m, beta_n, sigma = z[:, 7], z[:, 8], z[:, 4:7]
    alpha, beta = (tilt, -0.5 * tilt, -1.5 * tilt), (beta_m, 0.5 * beta_m, 2.0 * beta_m)
    nodes, weights = np.polynomial.legendre.leggauss(64)
    nodes = 0.5 * math.pi * nodes
    weights = 0.5 * math.pi * weights * np.cos(nodes)

    def gauss(b, d):
        b = torch.clamp_min(b, 1e-3)
        return torch.exp(-0.5 * (d / b) ** 2) / (math.sqrt(2.0 * math.pi) * b)

    def terms(u, cos_t, eta_p, cos_tt):
        gt = torch.asin(math.sin(u) / eta_p)
        c = torch.clamp(cos_t * math.cos(u), 0.0, 1.0)
        st2 = (1.0 - c * c) / (eta * eta)
        ct = torch.sqrt(torch.clamp_min(1.0 - st2, 0.0))
        f = 0.5 * (((c - eta * ct) / (c + eta * ct)) ** 2 + ((eta * c - ct) / (eta * c + ct)) ** 2)
        f = torch.where(st2 >= 1.0, torch.ones_like(f), f)
        tr = torch.exp(-sigma * (2.0 * torch.cos(gt) / cos_tt)[:, None])
        g = (1.0 - f) ** 2
        return gt, (f[:, None].expand(-1, 3), g[:, None] * tr, (g * f)[:, None] * tr * tr)

    def wrapped(a):
        return a - 2.0 * math.pi * torch.round(a / (2.0 * math.pi))

    td = 0.5 * (th_o - th_i)
    cos_td, sin_td = torch.clamp_min(torch.cos(td), 1e-3), torch.sin(td)
    eta_p, cos_tt = torch.sqrt(eta * eta - sin_td ** 2) / cos_td, torch.sqrt(1.0 - (sin_td / eta) ** 2)
    single = [torch.zeros_like(sigma) for _ in range(3)]
    for u, w in zip(nodes, weights):
        gt, att = terms(u, cos_td, eta_p, cos_tt)
        for p in range(3):
            d = wrapped(phi - (2.0 * p * gt - 2.0 * u + p * math.pi))
            dens = sum(torch.exp(-0.5 * ((d + k * 2.0 * math.pi) / beta_n) ** 2) for k in (-1, 0, 1))
            single[p] = single[p] + (w * dens / (math.sqrt(2.0 * math.pi) * beta_n))[:, None] * att[p]
    out = [gauss(beta[p], th_h - alpha[p])[:, None] * 0.5 * single[p] for p in range(3)]

    cos_to = torch.clamp_min(torch.sqrt(torch.clamp_min(1.0 - sin_o ** 2, 1e-6)), 1e-3)
    sin_to = torch.sqrt(torch.clamp_min(1.0 - cos_to ** 2, 0.0))
    eta_p, cos_tt = torch.sqrt(eta * eta - sin_to ** 2) / cos_to, torch.sqrt(1.0 - (sin_to / eta) ** 2)
    fwd, back = [torch.zeros_like(sigma) for _ in range(3)], [torch.zeros_like(sigma) for _ in range(3)]
    r = 1.0 / (beta_n * math.sqrt(2.0))
    for u, w in zip(nodes, weights):
        gt, att = terms(u, cos_to, eta_p, cos_tt)
        for p in range(3):
            c0 = wrapped(2.0 * p * gt - 2.0 * u + p * math.pi)
            e = [torch.erf((0.5 * math.pi + (j - 5) * math.pi - c0) * r) for j in range(11)]
            mb = 0.5 * ((e[9] - e[8]) + (e[7] - e[6]) + (e[5] - e[4]) + (e[3] - e[2]) + (e[1] - e[0]))
            mf = 0.5 * ((e[10] - e[9]) + (e[8] - e[7]) + (e[6] - e[5]) + (e[4] - e[3]) + (e[2] - e[1]))
            back[p] = back[p] + (w * mb)[:, None] * att[p]
            fwd[p] = fwd[p] + (w * mf)[:, None] * att[p]
    f, b = [0.5 * v for v in fwd], [0.5 * v for v in back]
    b2 = [(v * v)[:, None] for v in beta]
    a_f, a_b = torch.clamp_max(f[0] + f[1] + f[2], 0.95), b[0] + b[1] + b[2]
    tf, tb = torch.clamp_min(a_f, 1e-5), torch.clamp_min(a_b, 1e-5)
    beta_f2 = (f[0] * b2[0] + f[1] * b2[1] + f[2] * b2[2]) / tf
    alpha_b = (b[0] * alpha[0] + b[1] * alpha[1] + b[2] * alpha[2]) / tb
    beta_b2 = (b[0] * b2[0] + b[1] * b2[1] + b[2] * b2[2]) / tb
    af2 = a_f * a_f
    rest, ab2, ab3 = 1.0 - af2, a_b * a_b, a_b ** 3
    a_back = a_b * af2 / rest + ab3 * af2 / rest ** 3
    delta_b = alpha_b * (1.0 - 2.0 * ab2 / rest ** 2) + alpha_b * (2.0 * rest ** 2 + 4.0 * af2 * ab2) / rest ** 3
    sigma_b = (1.0 + 0.7 * af2) * (a_b * torch.sqrt(2.0 * beta_f2 + beta_b2) + ab3 * torch.sqrt(2.0 * beta_f2 + 3.0 * beta_b2)) \
        / torch.clamp_min(a_b + ab3 * (2.0 * torch.sqrt(beta_f2) + 3.0 * torch.sqrt(beta_b2)), 1e-5)
    out.append(2.0 * a_back * gauss(sigma_b, th_h[:, None] - delta_b) / math.pi)
    lobes = torch.cat(out, dim=1)
    return {"inputs": x, "targets": torch.log1p(lobes / 1e-3), "lobes": lobes}


def exact(case, seed):
    kind = case["kind"]
    if kind == "infer":
        net = [torch.from_numpy(v.copy()).cuda().double() for v in _network64(case, S.load_params(case["arch"]))]
        x, _ = _rows(case["rows"], seed)
        return 1e-3 * torch.expm1(torch.relu(_forward64(net, x, 3 if case["arch"] else 12)))
    if kind == "train":
        return _train64(case, seed)
    if kind == "samples":
        return _samples64(case["rows"], S.SAMPLE_SEED + seed)
    return None  # frames and shade passes: what is drawn rests on rounded coordinates and 24-bit depths
