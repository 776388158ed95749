"""The work that programs have this library do, as cases to be timed.

A case is a dict of plain values; ``listed`` names the standard ones and
``draw`` gives more of the same ranges.  ``prepare`` builds what a program has
in hand before the call (scene, accelerator, tracer, pool, network, device
inputs), ``run`` makes one call through the public entry points and returns
its outputs, ``exact`` the same outputs in 64-bit arithmetic where there is
such a value, ``work`` what a pass has to read, write and compute at least and
``tolerance`` how far two correct implementations may differ.

The kinds:

* ``hit``       closest hits of rays in device memory (GPUScene.hit)
* ``build``     a scene's accelerator built again, and its first hits
* ``frame``     one progressive frame of the plain tracer, its image read back
* ``guided``    the same of the path-guiding tracer, from a cold octree on
* ``pool``      a batch of render jobs of several scenes through one pool
* ``splat``     samples at any image coordinates through a filter
* ``forward``   the guiding network's inference
* ``backward``  its loss and gradients
"""
from __future__ import annotations

import ctypes
import functools
import math
import random

import numpy as np
import torch

import meturay_b200 as mrb
from meturay_b200 import learned, pool, scenes

CLUSTER_TRIANGLES = 1000  # triangles of one Gaussian cluster
MISS_T = 1000.0           # tMax of the rays given to hit, as the cameras' far plane


def _log(rng: random.Random, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _hit(scene, triangles, rays):
    return {"kind": "hit", "scene": scene, "triangles": triangles, "rays": rays}


def _build(scene, triangles, rays):
    return {"kind": "build", "scene": scene, "triangles": triangles, "rays": rays}


def _frame(scene, triangles, width, height, samples, depth, nee=1, mis=0, mixed=0,
           recon="Tent", radius=1.0):
    return {"kind": "frame", "scene": scene, "triangles": triangles, "width": width,
            "height": height, "samples": samples, "depth": depth, "nee": nee, "mis": mis,
            "mixed": mixed, "filter": recon, "radius": radius}


def _guided(scene, triangles, width, height, samples, depth, level, nee=1, product=1, mixed=0):
    return {"kind": "guided", "scene": scene, "triangles": triangles, "width": width,
            "height": height, "samples": samples, "depth": depth, "nee": nee, "mis": 0,
            "mixed": mixed, "filter": "Tent", "radius": 1.0, "level": level, "product": product}


def _pool(scene_count, triangles, jobs, frames, depth, capacity):
    return {"kind": "pool", "scenes": scene_count, "triangles": triangles, "jobs": jobs,
            "frames": frames, "depth": depth, "capacity": capacity}


def _splat(samples, width, height, channels, recon, radius):
    return {"kind": "splat", "samples": samples, "width": width, "height": height,
            "channels": channels, "filter": recon, "radius": radius}


def _network(kind, samples):
    return {"kind": kind, "samples": samples}


def _named(name, case):
    return dict(case, name=name)


def listed():
    return [
        # a picking or visibility query of an interactive program: few rays,
        # a small scene, so the launch and the longest ray count
        _named("hit_small", _hit("cornell", 7692, 2000)),
        # bounce rays of a host's own integrator: incoherent, 1M triangles
        _named("hit_1m", _hit("clusters", 1_000_000, 1_000_000)),
        # geometry was edited: the accelerator again, then the first rays
        _named("build_1m", _build("clusters", 1_000_000, 65_536)),
        # the preview: 128 x 128, 4 samples per pixel, a small closed scene;
        # many short launches
        _named("frame_preview", _frame("cornell", 7692, 128, 128, 2, 5)),
        # the headline frame: 1M triangles in the open, most rays leave early
        _named("frame_open", _frame("clusters", 1_000_000, 1920, 1080, 1, 8)),
        # a room at full resolution: every ray hits, most paths go all the
        # way; every material, light samples weighted against the BxDF
        _named("frame_closed", _frame("cornell", 7692, 1920, 1080, 2, 5, mis=1, mixed=1)),
        # guiding where paths are few and the octree's cells many
        _named("guided_preview", _guided("cornell", 7692, 128, 128, 2, 5, 10, nee=0)),
        # guiding at full resolution on the 1M-triangle scene
        _named("guided_open", _guided("clusters", 1_000_000, 1920, 1080, 1, 8, 10)),
        # batch of small jobs: product thumbnails, data sets
        _named("pool_batch", _pool(6, 64_000, 24, 4, 6, 1 << 20)),
        # samples of a host's own renderer onto a full-HD image
        _named("splat_1m", _splat(1_000_000, 1920, 1080, 4, "Tent", 1.0)),
        # inference for one wavefront of the guided preview
        _named("network_forward", _network("forward", 65_536)),
        # one training batch of the guided tracer
        _named("network_backward", _network("backward", 16_384)),
    ]


def _drawn_scene(rng):
    """(scene, triangles): a closed room or an open field of clusters."""
    if rng.random() < 0.5:
        return "cornell", _log(rng, 1000, 200_000)
    return "clusters", CLUSTER_TRIANGLES * _log(rng, 5, 1000)


def _drawn_filter(rng):
    """No filter, or one of the four with a radius that configurations use."""
    kind = rng.choice(["", "Box", "Tent", "Gaussian", "Mitchell"])
    return kind, (rng.choice([0.5, 1.0]) if kind == "Box" else round(rng.uniform(0.75, 2.0), 2))


def draw(rng: random.Random):
    kind = rng.choice(["hit", "hit", "build", "frame", "frame", "frame", "guided", "pool",
                       "splat", "forward", "backward"])
    if kind == "hit":
        scene, tris = _drawn_scene(rng)
        return _hit(scene, tris, _log(rng, 100, 2_000_000))
    if kind == "build":
        scene, tris = _drawn_scene(rng)
        return _build(scene, tris, _log(rng, 1000, 200_000))
    if kind == "frame":
        scene, tris = _drawn_scene(rng)
        samples = rng.choice([1, 1, 2])
        width = _log(rng, 61, 1280 if samples == 1 else 800)
        height = max(33, int(width * rng.uniform(0.4, 1.2)))
        recon, radius = _drawn_filter(rng)
        nee = rng.choice([0, 1, 1])
        return _frame(scene, tris, width, height, samples, rng.randint(2, 9), nee,
                      nee * rng.choice([0, 1]), scene == "cornell" and rng.choice([0, 1]),
                      recon, radius)
    if kind == "guided":
        scene, tris = _drawn_scene(rng)
        width = _log(rng, 61, 640)
        return _guided(scene, tris, width, max(33, int(width * rng.uniform(0.4, 1.0))), 1,
                       rng.randint(2, 6), rng.randint(7, 10), rng.choice([0, 1]),
                       rng.choice([0, 1, 1]), scene == "cornell" and rng.choice([0, 1]))
    if kind == "pool":
        return _pool(rng.randint(1, 6), _log(rng, 2000, 64_000), _log(rng, 2, 24),
                     rng.randint(1, 4), rng.randint(2, 6), 1 << rng.randint(18, 21))
    if kind == "splat":
        recon, radius = _drawn_filter(rng)
        if not recon:
            recon, radius = "Box", 0.0
        return _splat(_log(rng, 1000, 2_000_000), _log(rng, 33, 1920), _log(rng, 33, 1080),
                      rng.choice([1, 4]), recon, radius)
    return _network(kind, _log(rng, 100, 300_000))


# ---------------------------------------------------------------------------
# what a program holds before the call
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=1)
def _system():
    return mrb.TracerSystem(0)


@functools.lru_cache(maxsize=12)
def _host_scene(kind, triangles, mixed, seed):
    if kind == "clusters":
        return scenes.clusters(seed=seed, n_clusters=triangles // CLUSTER_TRIANGLES,
                               tris_per_cluster=CLUSTER_TRIANGLES)
    return scenes.cornell(seed=seed, triangles=triangles, mixed=bool(mixed))


def _scene(case, seed):
    """The case's geometry: one of four scenes, by the seed."""
    g = mrb.GPUScene(_system(), _host_scene(case["scene"], case["triangles"],
                                            case.get("mixed", 0), 1 + seed % 4))
    g.construct_accelerators()
    return g


def _rays(case, seed):
    """Origins uniform in the scene's box, directions uniform on the sphere."""
    n, size = case["rays"], 100.0 if case["scene"] == "clusters" else 1.0
    gen = torch.Generator(device="cuda").manual_seed(seed)
    o = torch.rand((n, 4), generator=gen, device="cuda") * size
    d = torch.randn((n, 4), generator=gen, device="cuda")
    d[:, :3] /= d[:, :3].norm(dim=1, keepdim=True)
    o[:, 3] = 0.0
    d[:, 3] = MISS_T
    return o, d


def _hit_buffers(n):
    return {"key": torch.zeros(n, dtype=torch.int32, device="cuda"),
            "prim": torch.zeros(n, dtype=torch.int32, device="cuda"),
            "t": torch.zeros(n, device="cuda"), "bary": torch.zeros((n, 2), device="cuda")}


def _camera(scene, case, seed):
    """The scene's camera for the case's image, moved a little by the seed."""
    cam = dict(scene.camera)
    size = 100.0 if case["scene"] == "clusters" else 1.0
    rng = random.Random(seed)
    cam["position"] = [p + size * rng.uniform(-0.05, 0.05) for p in cam["position"]]
    fx = cam["fov"][0]
    cam["fov"] = [fx, 2.0 * math.atan(math.tan(fx / 2.0) * case["height"] / case["width"])]
    return cam


def _recon_filter(kind, radius):
    options = {"Gaussian": {"alpha": 1.5}, "Mitchell": {"b": 1 / 3, "c": 1 / 3}}.get(kind, {})
    return mrb.ReconFilter(kind, radius, options)


def _tracer(case, seed, name):
    g = _scene(case, seed)
    t = _system().generate_tracer(g, name, {
        "Samples": case["samples"], "MaxDepth": case["depth"],
        "NextEventEstimation": case["nee"], "DirectLightMIS": case["mis"],
        "RussianRouletteStart": 3, "Seed": seed % (1 << 31)})
    t.set_resolution(case["width"], case["height"])
    if case["filter"]:
        t.attach_recon_filter(_recon_filter(case["filter"], case["radius"]))
    image = torch.zeros((case["height"], case["width"], 4)).pin_memory()
    return {"tracer": t, "camera": _camera(g.scene, case, seed), "image": image}


def _pool_state(case, seed):
    """Scenes and image sizes belong to the case; the seed draws the samples."""
    rng, held = random.Random(case["jobs"]), []
    for i in range(case["scenes"]):
        held.append(mrb.GPUScene(_system(), _host_scene(
            "cornell", _log(rng, 1000, case["triangles"]), i % 2, 10 + i)))
        held[-1].construct_accelerators()
    jobs = []
    for i in range(case["jobs"]):
        side = rng.choice([64, 128, 256, 500])
        jobs.append(mrb.Job(held[i % len(held)], side, side, frames=case["frames"],
                            max_depth=case["depth"], seed=1000 * (seed % (1 << 31)) + i))
    return {"pool": mrb.WavefrontPool(_system(), case["capacity"], case["depth"]), "jobs": jobs}


class _Device:
    """Device memory of the library as an array for torch, which keeps its
    owner alive as long as the array."""

    def __init__(self, owner, pointer, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (pointer, False), "shape": shape,
                                         "typestr": "<f4", "version": 3}


def _splat_inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = case["samples"]
    coords = torch.rand((n, 2), generator=gen, device="cuda")
    coords *= torch.tensor([float(case["width"]), float(case["height"])], device="cuda")
    # radiance: mostly small, some bright
    values = torch.rand((n, case["channels"]), generator=gen, device="cuda").pow(4) * 10.0
    return coords, values


def _splat_state(case, seed):
    coords, values = _splat_inputs(case, seed)
    w, h, c = case["width"], case["height"], case["channels"]
    image = mrb.ImageMemory(w, h, c)
    pixels, counts = image.device_pointers()
    return {"filter": _recon_filter(case["filter"], case["radius"]), "image": image,
            "values": values if c > 1 else values[:, 0].contiguous(), "coords": coords,
            "pixels": torch.as_tensor(_Device(image, pixels, (h, w, c)), device="cuda"),
            "counts": torch.as_tensor(_Device(image, counts, (h, w)), device="cuda")}


# The network: 80 features (78 used) -> 64 -> 64 -> 64 -> 40 (8 lobes of 5);
# per layer the weights (in x 64) and 64 biases, unused rows and columns zero
_LAYER_IN = (80, 64, 64, 64)


def _layers(flat):
    at, out = 0, []
    for k in _LAYER_IN:
        out.append((flat[at:at + k * 64].view(k, 64), flat[at + k * 64:at + (k + 1) * 64]))
        at += (k + 1) * 64
    return out


def _network_params(seed):
    p = torch.zeros(learned.PARAM_COUNT)
    gen = torch.Generator().manual_seed(seed)
    for i, (w, b) in enumerate(_layers(p)):
        limit = math.sqrt((6.0 if i < 3 else 3.0) / w.shape[0])
        w[:] = (torch.rand(w.shape, generator=gen) * 2.0 - 1.0) * limit
        b[:] = torch.randn(64, generator=gen) * 0.1
        if i == 0:
            w[78:] = 0.0
        if i == 3:
            w[:, 40:] = 0.0
            b[40:] = 0.0
    return p


def _directions(n, gen):
    d = torch.randn((n, 3), generator=gen, device="cuda")
    return d / d.norm(dim=1, keepdim=True)


def _network_inputs(case, seed):
    """Encoded path vertices, incident directions and their weights."""
    n = case["samples"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    pos = torch.rand((n, 3), generator=gen, device="cuda")
    features = torch.zeros((n, learned.N_IN), device="cuda")
    learned.GuideMLP.encode(pos, _directions(n, gen), _directions(n, gen), features)
    targets = torch.zeros((n, 4), device="cuda")
    targets[:, :3] = _directions(n, gen)
    weight = torch.rand(n, generator=gen, device="cuda")
    targets[:, 3] = torch.where(weight < 0.1, torch.zeros_like(weight), 2.0 * weight)
    return features, targets


def _network_state(case, seed):
    features, targets = _network_inputs(case, seed)
    net = learned.GuideMLP(_system(), _network_params(seed).numpy())
    if case["kind"] == "forward":
        return {"net": net, "x": features,
                "out": torch.zeros((case["samples"], learned.N_OUT), device="cuda")}
    return {"net": net, "x": features, "targets": targets,
            "grad": torch.zeros(learned.PARAM_COUNT, device="cuda"),
            "loss": torch.zeros(2, device="cuda")}


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("hit", "build"):
        state = {"scene": _scene(case, seed), "n": case["rays"], "out": _hit_buffers(case["rays"])}
        state["o"], state["d"] = _rays(case, seed)
    elif kind == "frame":
        state = _tracer(case, seed, "PathTracer")
    elif kind == "guided":
        state = _tracer(case, seed, "WFPGTracer")
        state["tracer"].set_options({
            "OctreeLevel": case["level"], "MinRayBinLevel": 5, "BinRayCount": 512,
            "DoProductPathGuiding": case["product"], "GuideBounceAmount": 512,
            "BXDF-GuideMISRatio": 0.5, "RFieldFilterAlpha": 0.6})
    elif kind == "pool":
        state = _pool_state(case, seed)
    elif kind == "splat":
        state = _splat_state(case, seed)
    else:
        state = _network_state(case, seed)
    state["kind"] = kind
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind in ("hit", "build"):
        if kind == "build":
            state["scene"].construct_accelerators()
        out = state["out"]
        state["scene"].hit(state["o"].data_ptr(), state["d"].data_ptr(), state["n"],
                           out["key"].data_ptr(), out["prim"].data_ptr(), out["t"].data_ptr(),
                           out["bary"].data_ptr())
        return out
    if kind in ("frame", "guided"):
        # a viewer's loop: this frame's camera up, its image on the way down
        # while the next frame renders
        tracer = state["tracer"]
        tracer.set_camera(state["camera"])
        tracer.render_frame()
        tracer.image_into_async(ctypes.c_void_p(state["image"].data_ptr()))
        return state["image"]
    if kind == "pool":
        return state["pool"].run(state["jobs"])
    if kind == "splat":
        image = state["image"]
        image.reset()
        state["filter"].filter_to_img(image, state["values"], state["coords"],
                                      state["coords"].shape[0])
        return {"pixels": state["pixels"], "counts": state["counts"]}
    if kind == "forward":
        state["net"].forward(state["x"], state["out"])
        return state["out"]
    state["grad"].zero_()
    state["loss"].zero_()
    state["net"].gradients(state["x"], state["targets"], state["grad"], state["loss"])
    return {"grad": state["grad"], "loss": state["loss"]}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("hit", "build"):
        # rays in (32 B), hits out (20 B), the triangles once
        return {"bytes": 52 * case["rays"] + 36 * case["triangles"], "flops": 0}
    if kind in ("frame", "guided"):
        return {"bytes": 16 * case["width"] * case["height"] + 36 * case["triangles"], "flops": 0}
    if kind == "pool":
        # mean image of the four sizes, the scenes at their mean size
        pixels = (64 ** 2 + 128 ** 2 + 256 ** 2 + 500 ** 2) / 4
        return {"bytes": 16 * pixels * case["jobs"] + 36 * case["scenes"] * case["triangles"] / 4,
                "flops": 0}
    if kind == "splat":
        c = case["channels"]
        return {"bytes": case["samples"] * 4 * (2 + c) +
                case["width"] * case["height"] * 4 * (c + 1), "flops": 0}
    n, weights = case["samples"], 80 * 64 + 3 * 64 * 64
    if kind == "forward":
        return {"bytes": 4 * (n * (80 + 40) + learned.PARAM_COUNT), "flops": 2.0 * weights * n}
    # forward, weight gradients, and input gradients of the last three layers
    return {"bytes": 4 * (n * (80 + 4) + 2 * learned.PARAM_COUNT),
            "flops": 2.0 * (2 * weights + 3 * 64 * 64) * n}


def tolerance(case):
    kind = case["kind"]
    if kind in ("hit", "build"):
        # distances in 32 bits; two triangles may share a distance, and
        # either may be reported
        return {"rel": 1e-5, "max": 0.9, "differ": 1e-3}
    if kind in ("frame", "guided", "pool"):
        # the samples' sums are added in no fixed order
        return {"rel": 1e-4, "max": 0.9}
    if kind == "splat":
        return {"rel": 1e-5, "max": 1e-4}
    # 16-bit operands, 32-bit sums
    return {"rel": 1e-2, "max": 0.2}


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------
def _exact_hit(case, seed):
    """Every ray against every triangle (Moeller and Trumbore 1997)."""
    if case["rays"] * case["triangles"] > 4e9:
        return None
    scene = _host_scene(case["scene"], case["triangles"], 0, 1 + seed % 4)
    pos = torch.from_numpy(scene.positions).cuda().double()
    idx = torch.from_numpy(scene.indices.astype(np.int64)).cuda()
    v0, v1, v2 = (pos[idx[:, k]] for k in range(3))
    e0, e1 = v1 - v0, v2 - v0
    o, d = (x.double() for x in _rays(case, seed))
    t_out = torch.full((case["rays"],), MISS_T, dtype=torch.float64, device="cuda")
    bary = torch.zeros((case["rays"], 2), dtype=torch.float64, device="cuda")
    step = max(1, 20_000_000 // idx.shape[0])

    def dot(a, b):
        return (a * b).sum(-1)

    for b in range(0, case["rays"], step):
        ro, rd = o[b:b + step, None, :3], d[b:b + step, None, :3]
        p = torch.linalg.cross(rd.expand(-1, idx.shape[0], -1), e1.expand(ro.shape[0], -1, -1))
        det = dot(e0, p)
        tv = ro - v0
        u = dot(tv, p) / det
        q = torch.linalg.cross(tv, e0.expand(ro.shape[0], -1, -1))
        v = dot(rd, q) / det
        t = dot(e1, q) / det
        ok = (det.abs() >= 1e-7) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (t > 1e-7)
        t = torch.where(ok & (t < MISS_T), t, torch.full_like(t, math.inf))
        near, at = t.min(dim=1)
        found = near < MISS_T
        uu, vv = u.gather(1, at[:, None])[:, 0], v.gather(1, at[:, None])[:, 0]
        t_out[b:b + step] = torch.where(found, near, t_out[b:b + step])
        bary[b:b + step] = torch.where(found[:, None], torch.stack([1 - uu - vv, uu], 1),
                                       bary[b:b + step])
    return {"key": None, "prim": None, "t": t_out, "bary": bary}


def _weight(case, dx, dy):
    r, kind = case["radius"], case["filter"]
    if kind == "Box":
        return ((dx < r) & (dy < r)).double() if r > 0 else torch.ones_like(dx)
    if kind == "Tent":
        return (1 - dx / r).clamp(min=0) * (1 - dy / r).clamp(min=0)
    if kind == "Gaussian":
        edge = math.exp(-1.5 * r * r)
        return ((-1.5 * dx * dx).exp() - edge).clamp(min=0) * \
            ((-1.5 * dy * dy).exp() - edge).clamp(min=0)

    def cubic(x):  # Mitchell and Netravali 1988, B = C = 1/3
        b = c = 1 / 3
        # the constant term carries + 2 b, as the MRay reference writes it
        near = (12 - 9 * b - 6 * c) * x ** 3 + (-18 + 12 * b + 6 * c) * x ** 2 + (6 + 2 * b)
        far = (-b - 6 * c) * x ** 3 + (6 * b + 30 * c) * x ** 2 + (-12 * b - 48 * c) * x + \
            (8 * b + 24 * c)
        zero = torch.zeros_like(x)
        return torch.where(x < 1, near, torch.where(x < 2, far, zero)) / 6
    return cubic(2 * dx / r) * cubic(2 * dy / r)


def _exact_splat(case, seed):
    """Which pixels a sample reaches is decided in 32 bits, as the library
    states it; weights and sums are in 64."""
    coords, values = _splat_inputs(case, seed)
    w, h, c = case["width"], case["height"], case["channels"]
    wh = mrb.filter_pixel_wh(case["radius"])
    pixels = torch.zeros((h * w, c), dtype=torch.float64, device="cuda")
    counts = torch.zeros(h * w, dtype=torch.float64, device="cuda")
    whole = coords.trunc()
    first = torch.full_like(coords, -((wh - 1) // 2))
    if wh % 2 == 0:
        first -= (coords - whole < 0.5).float()
    r2 = torch.tensor(case["radius"], dtype=torch.float32).square().item()
    for y in range(wh):
        for x in range(wh):
            at = whole + first + torch.tensor([float(x), float(y)], device="cuda")
            gap = coords - (at + 0.5)
            ok = torch.full((len(at),), True, device="cuda") if wh == 1 else \
                (gap * gap).sum(1) <= r2
            ok &= (at >= 0).all(1) & (at[:, 0] < w) & (at[:, 1] < h)
            exact_gap = (coords[ok].double() - (at[ok].double() + 0.5)).abs()
            weight = _weight(case, exact_gap[:, 0], exact_gap[:, 1])
            pixel = at[ok, 1].long() * w + at[ok, 0].long()
            pixels.index_add_(0, pixel, values[ok].double() * weight[:, None])
            counts.index_add_(0, pixel, weight)
    return {"pixels": pixels.view(h, w, c), "counts": counts.view(h, w)}


def _exact_forward(params, x):
    for i, (w, b) in enumerate(_layers(params)):
        x = x @ w + b
        x = x.relu() if i < 3 else x[:, :learned.N_OUT]
    return x


def _exact_network(case, seed):
    features, targets = _network_inputs(case, seed)
    params = _network_params(seed).cuda().double().requires_grad_(True)
    raw = _exact_forward(params, features.double())
    if case["kind"] == "forward":
        return raw.detach()
    lobes = raw.view(-1, 8, 5)
    mu = lobes[..., :3] / (lobes[..., :3].square().sum(-1, keepdim=True) + 1e-12).sqrt()
    log_kappa = lobes[..., 3].clamp(-10.0, 8.0)
    kappa = log_kappa.exp()
    norm = log_kappa - math.log(2 * math.pi) - (-torch.expm1(-2 * kappa)).log()
    direction, weight = targets[:, None, :3].double(), targets[:, 3].double()
    each = lobes[..., 4].log_softmax(-1) + norm + kappa * ((mu * direction).sum(-1) - 1)
    loss = -(weight * each.logsumexp(-1)).sum()
    loss.backward()
    return {"grad": params.grad, "loss": torch.stack([loss.detach(), weight.sum()])}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("hit", "build"):
        return _exact_hit(case, seed)
    if kind == "splat":
        return _exact_splat(case, seed)
    if kind in ("forward", "backward"):
        return _exact_network(case, seed)
    return None  # paths in other arithmetic are other paths
