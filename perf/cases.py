"""What is timed: the calls that a program built on muon_gb300 makes.

Frames of every integrator family (path tracer with its sampling options, ray
tracer, previews), from a thumbnail to the full-size dense mesh, into host and
device films; opening a scene; batched ray queries; a batch of small scenes;
and learned guiding (a guided frame, the training gradients). Each case goes
through the package's public entry points with the settings of the
repository's own scenes (muon_gb300/scenes.py).

A case is a dict of plain values; `kind` names the call, `scene` the scene.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import muon_gb300 as m
from muon_gb300 import native, scenes


def listed():
    return [
        # The smallest call: the look a user takes at a scene while editing it
        # (one sample per pixel of the normals integrator, film to the host).
        dict(name="look_normals_128", kind="frame", scene="feature_mix", width=128, height=128, spp=1,
             integrator="normals", film="host"),
        # The Cornell box of the benchmark, as the CLI renders it.
        dict(name="cornell_256x16", kind="frame", scene="cornell", width=256, height=256, spp=16, depth=5,
             film="host"),
        # Unbounded depth with Russian roulette, stratified light samples,
        # three lights, every material and primitive, an odd film.
        dict(name="mix_rr_317x211x12", kind="frame", scene="feature_mix", width=317, height=211, spp=12, depth=-1,
             rr=1, light_samples=4, stratify=1, film="host"),
        # The sphere field of the benchmark: shallow tree, mixed materials.
        dict(name="spheres_512x64", kind="frame", scene="sphere_field", width=512, height=512, spp=64, depth=8,
             film="device"),
        # The dense mesh of the benchmark (1,320,756 triangles): the largest
        # frame, several wavefronts, a quarter of its samples.
        dict(name="dense_1024x64", kind="frame", scene="dense_mesh", level=8, width=1024, height=1024, spp=64,
             depth=10, film="device"),
        # A medium mesh in the fast intersection mode, light sampling without
        # MIS, a wide film.
        dict(name="mesh_fast_960x540x16", kind="frame", scene="dense_mesh", level=6, width=960, height=540, spp=16,
             depth=6, mode="fast", nee="on", film="device"),
        # The ray tracer with point, directional and quad lights.
        dict(name="whitted_640x480x4", kind="frame", scene="whitted", width=640, height=480, spp=4, depth=5,
             integrator="raytracer", film="host"),
        # Opening a model and showing it: scene creation (upload, records,
        # BVH), one preview frame, and closing it again.
        dict(name="open_mesh_87k", kind="open", scene="dense_mesh", level=6, width=512, height=384),
        # Ray queries of a host program (picking, visibility, baking).
        dict(name="queries_mesh_1000003", kind="queries", scene="dense_mesh", level=6, rays=1000003),
        # Many small scenes of uneven size rendered as one batch.
        dict(name="batch_8", kind="batch", count=8, max_tris=50000, spp=16),
        # A frame guided by the learned mixture, as each training pass renders.
        dict(name="guided_320x240x16", kind="guided", scene="slit_room", level=6, width=320, height=240, spp=16,
             depth=6),
        # The gradients of one training batch.
        dict(name="guide_gradients_65536", kind="gradients", batch=65536),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "open", "queries", "batch", "guided", "gradients"])
    width, height = _log(rng, 64, 1024), _log(rng, 64, 1024)
    if kind == "frame":
        scene = rng.choice(["cornell", "feature_mix", "sphere_field", "dense_mesh", "dense_mesh", "whitted"])
        spp = max(1, min(_log(rng, 1, 64), (1 << 24) // (width * height)))
        case = dict(kind=kind, scene=scene, width=width, height=height, spp=spp, film=rng.choice(["host", "device"]),
                    mode=rng.choice(["exact", "exact", "fast"]))
        if scene == "dense_mesh":
            case["level"] = rng.randint(4, 7)
        if scene == "whitted":
            return dict(case, integrator=rng.choice(["raytracer", "analyticdirect"]), depth=rng.randint(2, 6),
                        spp=min(spp, 16))
        if rng.random() < 0.2:
            return dict(case, integrator=rng.choice(["normals", "albedo", "depth"]), spp=min(spp, 4))
        if rng.random() < 0.25:
            case.update(depth=-1, rr=1)
        else:
            case["depth"] = rng.randint(2, 10)
        case["nee"] = rng.choice(["mis", "mis", "on", "off"])
        if rng.random() < 0.3:
            case.update(light_samples=4, stratify=rng.randint(0, 1))
        return case
    if kind == "open":
        return dict(kind=kind, scene="dense_mesh", level=rng.randint(3, 7), width=width, height=height)
    if kind == "queries":
        return dict(kind=kind, scene=rng.choice(["dense_mesh", "sphere_field", "feature_mix"]),
                    level=rng.randint(4, 7), rays=_log(rng, 1000, 1500000))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(3, 12), max_tris=_log(rng, 2000, 100000), spp=rng.randint(4, 16))
    if kind == "guided":
        return dict(kind=kind, scene="slit_room", level=rng.randint(4, 6), width=min(width, 640),
                    height=min(height, 480), spp=rng.randint(1, 16), depth=rng.randint(2, 8))
    return dict(kind=kind, batch=_log(rng, 1000, 1 << 18))


# ---- scenes ----------------------------------------------------------------------

def _text(case, geometry_seed):
    """The .muon text of a case's scene; the geometry differs with the seed
    where the scene has random parts."""
    w, h, spp = case.get("width", 64), case.get("height", 64), case.get("spp", 1)
    depth = case.get("depth", 5)
    name = case["scene"]
    if name == "cornell":
        return scenes.cornell(w, h, spp, depth, 1)
    if name == "feature_mix":
        return scenes.feature_mix(w, h, spp, "pathtracer", "mis", depth)
    if name == "sphere_field":
        return scenes.sphere_field(w, h, spp, depth, 512, geometry_seed)
    if name == "dense_mesh":
        return scenes.dense_mesh(w, h, spp, depth, case["level"], _clutter(case["level"]), geometry_seed)
    if name == "slit_room":
        return scenes.slit_room(w, h, spp, depth, case["level"], _clutter(case["level"]), geometry_seed)
    return scenes.whitted(w, h, spp, depth, geometry_seed)


def _clutter(level):
    return 10000 if level >= 8 else 5000 if level >= 6 else 1000


@functools.lru_cache(maxsize=4)
def _parsed_large(items):
    return m.parse_string(_text(dict(items), 1))


def _parse(case, seed):
    """The parsed scene a program holds, its camera moved a little by the seed.

    Meshes of level 7 and 8 (0.3 and 1.3 million triangles, seconds of text)
    are one model file, looked at from another place; smaller scenes have
    geometry of their own for each seed."""
    if case.get("level", 0) >= 7:
        key = tuple(sorted((k, v) for k, v in case.items() if k in ("scene", "level", "width", "height", "spp", "depth")))
        parsed = _parsed_large(key)
    else:
        parsed = m.parse_string(_text(case, 1 + seed % 1000))
    rng = np.random.default_rng(seed)
    if not hasattr(parsed, "eye0"):
        parsed.eye0 = list(parsed.desc.camera.eye)
    for k in range(3):
        parsed.desc.camera.eye[k] = parsed.eye0[k] + 0.02 * float(rng.uniform(-1, 1))
    return parsed


def _params(case, scene, seed):
    over = dict(integrator=case.get("integrator", "pathtracer"), pixel_samples=case.get("spp", 1), seed=seed,
                intersect_mode=case.get("mode", "exact"))
    if "depth" in case:
        over["max_depth"] = case["depth"]
    if "nee" in case:
        over["next_event_estimation"] = case["nee"]
    if "rr" in case:
        over["russian_roulette"] = case["rr"]
    if "light_samples" in case:
        over.update(light_samples=case["light_samples"], light_stratify=case["stratify"])
    return scene.params(**over)


def _device_film(scene):
    h, w = scene.height, scene.width
    return dict(sum=torch.zeros(h, w, 3, dtype=torch.float64, device="cuda"),
                sum_sq=torch.zeros(h, w, 3, dtype=torch.float64, device="cuda"),
                count=torch.zeros(h, w, dtype=torch.int32, device="cuda"))


def _film(film):
    return dict(sum=film.sum, sum_sq=film.sum_sq, count=film.count)


# ---- guiding network ---------------------------------------------------------------

_LAYERS = [(256, 64), (64, 64), (64, 64), (64, 64), (64, 64)]


def _network(rng):
    """Weights as a network some way into training has them: He-uniform, with
    biases off zero; weights [in][out] then biases, layer by layer."""
    parts = []
    for fan_in, fan_out in _LAYERS:
        lim = math.sqrt(6.0 / fan_in)
        parts += [rng.uniform(-lim, lim, fan_in * fan_out), rng.uniform(-0.1, 0.1, fan_out)]
    return np.concatenate(parts).astype(np.float32)


def _train_batch(n, rng):
    """Features in [0, 1], unit directions, and heavy-tailed weights of mean 1
    (a tenth of them zero), as the sample pool holds them."""
    f = rng.uniform(0.0, 1.0, (n, 8)).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    w = np.exp(rng.normal(0.0, 1.0, n)) * (rng.uniform(size=n) > 0.1)
    return f, d, (w / w.mean()).astype(np.float32)


# ---- the cases ---------------------------------------------------------------------

class _State:
    """What the program holds; closed with the last reference to it."""

    def __init__(self, **kw):
        self.__dict__.update(kw)


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng([seed, 7])
    if kind == "frame":
        scene = m.Scene(_parse(case, seed))
        return _State(kind=kind, scene=scene, params=_params(case, scene, seed),
                      film=_device_film(scene) if case["film"] == "device" else None)
    if kind == "open":
        return _State(kind=kind, parsed=_parse(case, seed))
    if kind == "queries":
        scene = m.Scene(_parse(case, seed))
        n = case["rays"]
        size = 10.0 if case["scene"] == "sphere_field" else 0.9
        lift = 0.0 if case["scene"] == "sphere_field" else 1.0
        o = rng.uniform(-size, size, (n, 3)).astype(np.float32) + np.float32([0, lift, 0])
        d = rng.normal(size=(n, 3))
        d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
        return _State(kind=kind, scene=scene, o=o, d=d, far=rng.uniform(0.1 * size, 2 * size, n).astype(np.float32))
    if kind == "batch":
        made = [m.Scene.from_string(scenes.batch_scene(i, seed=1 + seed % 1000, max_tris=case["max_tris"],
                                                       resolutions=((64, 256, 128)[i % 3],),
                                                       spp_range=(4, case["spp"])))
                for i in range(case["count"])]
        return _State(kind=kind, scenes=made, batch=m.Batch(made), params=[s.params() for s in made])
    if kind == "guided":
        scene = m.Scene(_parse(case, seed))
        guide = m.Guide(scene, seed=seed, wave_paths=1 << 21)
        guide.set_params(_network(rng))
        return _State(kind=kind, scene=scene, guide=guide, params=_params(case, scene, seed), film=_device_film(scene))
    scene = m.Scene.from_string(scenes.cornell(64, 64, 1, 5, 1))
    guide = m.Guide(scene, seed=seed, batch=case["batch"], wave_paths=1 << 16, pool_capacity=1 << 16)
    guide.set_params(_network(rng))
    f, d, w = _train_batch(case["batch"], rng)
    return _State(kind=kind, scene=scene, guide=guide, f=f, d=d, w=w)


def run(state):
    kind = state.kind
    if kind == "frame":
        if state.film is None:
            return _film(state.scene.render(state.params))
        f = state.film
        state.scene.render_device(state.params, f["sum"].data_ptr(), f["sum_sq"].data_ptr(), f["count"].data_ptr())
        return f
    if kind == "open":
        scene = m.Scene(state.parsed)
        film = scene.render(integrator="normals", pixel_samples=1)
        scene.close()
        return _film(film)
    if kind == "queries":
        distance, prim, position, normal = state.scene.intersect(state.o, state.d)
        blocked = state.scene.occluded(state.o, state.d, state.far)
        return dict(distance=distance, prim=prim, position=position, normal=normal, blocked=blocked)
    if kind == "batch":
        return [_film(f) for f in state.batch.render(state.params)]
    if kind == "guided":
        f = state.film
        state.guide.render_device(state.params, f["sum"].data_ptr(), f["sum_sq"].data_ptr(), f["count"].data_ptr())
        return dict(f, samples=state.guide.samples())
    grad, loss = state.guide.gradients(state.f, state.d, state.w)
    return dict(grad=grad, loss=loss)


# ---- what the work cannot do without ---------------------------------------------

def _prims(case):
    if case["scene"] in ("dense_mesh", "slit_room"):
        return 20 * 4 ** case["level"] + _clutter(case["level"]) + 36
    return {"cornell": 36, "feature_mix": 400, "sphere_field": 516, "whitted": 28}[case["scene"]]


def _ray_flops(prims):
    """One ray down a balanced binary tree of leaves of four: two box tests (24
    operations each) per level, four primitive tests (50 each)."""
    return 48.0 * max(1.0, math.log2(max(prims, 2) / 4.0)) + 200.0


def _frame_work(prims, pixels, spp, depth, path):
    """Scene records in (64 bytes a primitive and as much of tree), the film out
    (52 bytes a pixel); per path vertex a closest-hit ray, a shadow ray and
    about 300 operations of shading, with seven in ten paths going on."""
    d = min(depth, 12) if depth >= 0 else 12
    vertices = sum(0.7 ** k for k in range(max(1, d))) if path else 1.0
    flops = pixels * spp * vertices * ((2.0 if path else 1.0) * _ray_flops(prims) + (300.0 if path else 20.0))
    return {"bytes": 128.0 * prims + 52.0 * pixels, "flops": flops}


def work(case):
    kind = case["kind"]
    if kind == "frame" or kind == "guided":
        preview = case.get("integrator", "pathtracer") in ("normals", "albedo", "depth")
        w = _frame_work(_prims(case), case["width"] * case["height"], case["spp"], case.get("depth", 5), not preview)
        if kind == "guided":  # the network (33,024 multiply-adds) at the first vertices of every path
            w["flops"] += 2.0 * 33024 * case["width"] * case["height"] * case["spp"] * 1.7
        return w
    if kind == "open":
        w = _frame_work(_prims(case), case["width"] * case["height"], 1, 1, False)
        w["bytes"] += 100.0 * _prims(case)  # the triangles' descriptions
        w["flops"] += 200.0 * _prims(case) * math.log2(_prims(case))
        return w
    if kind == "queries":
        n = case["rays"]
        return {"bytes": n * (2 * 24.0 + 4.0 + 32.0 + 1.0) + 128.0 * _prims(case),
                "flops": 2.0 * n * _ray_flops(_prims(case))}
    if kind == "batch":
        pixels, prims = case["count"] * 150 * 150, case["count"] * math.sqrt(1000.0 * case["max_tris"])
        return _frame_work(prims, pixels, (4 + case["spp"]) / 2, 7, True)
    # forward, data and weight gradients of the 33,024 weights per sample
    return {"bytes": 48.0 * case["batch"] + 4.0 * 33088 * 2, "flops": 3 * 2.0 * 33024 * case["batch"]}


# ---- 64-bit values ------------------------------------------------------------------

def exact(case, seed):
    """The training gradients in 64 bits. The other kinds have no plain
    restatement that takes seconds: films follow the rounding of every path."""
    if case["kind"] != "gradients":
        return None
    rng = np.random.default_rng([seed, 7])
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    net = torch.tensor(_network(rng), dtype=torch.float64, device=dev, requires_grad=True)
    f, d, w = (torch.tensor(x, dtype=torch.float64, device=dev) for x in _train_batch(case["batch"], rng))
    centres = (torch.arange(32, dtype=torch.float64, device=dev) + 0.5) / 32.0
    total = 0.0
    for k in range(0, len(f), 16384):
        fk, dk, wk = f[k:k + 16384], d[k:k + 16384], w[k:k + 16384]
        x = torch.exp(-0.5 * (32.0 * (fk[:, :, None] - centres)) ** 2).reshape(len(fk), 256)
        at = 0
        for l, (fan_in, fan_out) in enumerate(_LAYERS):
            weight = net[at:at + fan_in * fan_out].reshape(fan_in, fan_out)
            bias = net[at + fan_in * fan_out:at + fan_in * fan_out + fan_out]
            at += fan_in * fan_out + fan_out
            x = x @ weight + bias
            if l + 1 < len(_LAYERS):
                x = torch.relu(x)
        r = x.reshape(-1, 8, 8)
        log_pi = torch.log_softmax(r[:, :, 0], dim=1)
        mu = r[:, :, 1:4] / torch.linalg.norm(r[:, :, 1:4], dim=2, keepdim=True)
        c = (mu * dk[:, None, :]).sum(2)
        on = c > 1e-4
        cc = torch.where(on, c, torch.ones_like(c))
        b = torch.clamp(r[:, :, 4], -3.0, 8.0)
        s = torch.exp(b)
        u = r[:, :, 5:8]
        pu = u - (u * mu).sum(2, keepdim=True) * mu
        v = dk[:, None, :] / cc[:, :, None] - mu
        p2, v2, dv = (pu * pu).sum(2), (v * v).sum(2), (pu * v).sum(2)
        log_p = 0.5 * b + 0.5 * torch.log(s + p2) - math.log(2 * math.pi) - 0.5 * (s * v2 + dv * dv) - 3 * torch.log(cc)
        lobes = torch.where(on, math.log(0.98) + log_pi + log_p, torch.full_like(c, -torch.inf))
        flat = torch.full((len(fk), 1), math.log(0.02 / (4 * math.pi)), dtype=torch.float64, device=dev)
        loss = -(wk * torch.logsumexp(torch.cat([lobes, flat], 1), 1)).sum() / len(f)
        loss.backward()
        total += float(loss.detach())
    return dict(grad=net.grad.cpu().numpy(), loss=total)
