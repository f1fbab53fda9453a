"""Performance cases of the framework: what a user has it do, over the range of sizes it is used at.

Kinds of case (each goes through :class:`radiantium_gb300.device.Device`, the public binding):

* ``rays``      closest-hit (and, from host arrays, any-hit) queries: picking and visibility tests from a
                host program in small batches, incoherent device-resident batches of a baker in large ones;
* ``path``      a film of the ``path`` integrator: interactive previews (1 spp), final frames, progressive
                passes; methods, light strategies, the opt-in traversal and light sampling;
* ``volume``    a film of ``vol_path`` through a participating medium;
* ``particles`` a film of the ``adjoint_particle`` light tracer;
* ``batch``     many scenes rendered by one call (dataset generation);
* ``adjoint``   the gradient of an image loss w.r.t. an albedo texture and GGX alphas (an optimiser's step);
* ``upload``    a new or edited scene: upload (tree construction included), then its first query.

Scenes are the repository's procedural ones.  Meshes and environment maps are assets, as a user's files on
disk are; the camera, the random streams, the rays, the placement of geometry and the loss come from the seed.
"""
import copy
import functools
import math

import numpy as np
import torch

from radiantium_gb300 import native as N
from radiantium_gb300 import procedural
from radiantium_gb300.device import Device
from radiantium_gb300.scene import Camera, Mat4

# closest-hit and any-hit rays per camera sample (or particle) of each scene, from the benchmark's ray counters
RAYS_PER_SAMPLE = {"box": 6.2, "instances": 4.2, "zoo": 5.0, "volume": 5.1, "batch": 3.3, "adjoint": 3.5,
                   "particles": 12.4}


def listed():
    return [
        # a picking / visibility query of an interactive host program: 1,000 rays, host arrays, both forms
        {"name": "rays_box_small", "kind": "rays", "scene": "box", "n": 1000, "host": True, "any": True},
        # a baker's incoherent rays over the instanced scene, device resident
        {"name": "rays_instances", "kind": "rays", "scene": "instances", "n": 2_000_003, "host": False, "any": False},
        # one frame of an interactive preview: the smallest film call, bound by latency and launches
        {"name": "path_box_preview", "kind": "path", "scene": "box", "w": 256, "h": 256, "spp": 1, "depth": 5,
         "method": "mis", "strategy": "uniform", "wide": False, "alias": False},
        # the Cornell box at its benchmark settings (256 x 256, 64 spp, depth 5)
        {"name": "path_box_frame", "kind": "path", "scene": "box", "w": 256, "h": 256, "spp": 64, "depth": 5,
         "method": "mis", "strategy": "uniform", "wide": False, "alias": False},
        # every material and light type, All light strategy, odd film size
        {"name": "path_zoo_all_lights", "kind": "path", "scene": "zoo", "w": 333, "h": 217, "spp": 16, "depth": 6,
         "method": "mis", "strategy": "all", "wide": False, "alias": False},
        # the instanced benchmark: one progressive 16-spp pass at 1024 x 1024 (12.8 M instanced triangles)
        {"name": "path_instances_pass", "kind": "path", "scene": "instances", "w": 1024, "h": 1024, "spp": 16,
         "depth": 8, "method": "mis", "strategy": "uniform", "wide": False, "alias": False},
        # the same scene with the opt-in fast modes, a smaller film
        {"name": "path_instances_wide", "kind": "path", "scene": "instances", "w": 640, "h": 360, "spp": 8,
         "depth": 8, "method": "mis", "strategy": "uniform", "wide": True, "alias": True},
        # the participating-media benchmark: one 16-spp pass at 512 x 512, depth 32
        {"name": "volume_pass", "kind": "volume", "w": 512, "h": 512, "spp": 16, "depth": 32},
        # the light-tracer benchmark's film, 4 Mi particles
        {"name": "particles_box", "kind": "particles", "scene": "box", "w": 800, "h": 600, "count": 4 << 20},
        # twelve scenes in one call
        {"name": "batch_12", "kind": "batch", "scenes": 12, "spp": 6},
        # one optimiser step of the inverse-rendering benchmark (786,496 parameters), 16 spp
        {"name": "adjoint_step", "kind": "adjoint", "w": 256, "h": 256, "spp": 16, "depth": 6},
        # a new 199,692-triangle scene: upload with tree construction, then its first 16,384 rays
        {"name": "upload_sphere", "kind": "upload", "sphere_n": 129, "n": 16_384},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rays", "rays", "path", "path", "path", "volume", "particles", "batch", "adjoint", "upload"])
    if kind == "rays":
        host = rng.random() < 0.5
        return {"kind": "rays", "scene": rng.choice(["box", "zoo", "instances"]),
                "n": _log(rng, 64, 200_000 if host else 3_000_000), "host": host, "any": host}
    if kind == "path":
        scene = rng.choice(["box", "zoo", "instances"])
        w, h = _log(rng, 64, 1024), _log(rng, 64, 1024)
        spp = max(1, min(_log(rng, 1, 64), 8_000_000 // (w * h)))
        method = rng.choice(["mis", "mis", "mis", "nee", "bxdf"])
        wide = rng.random() < 0.25
        return {"kind": "path", "scene": scene, "w": w, "h": h, "spp": spp, "depth": rng.randint(3, 8),
                "method": method, "strategy": "all" if method != "bxdf" and scene == "zoo" and rng.random() < 0.5
                else "uniform", "wide": wide, "alias": wide and rng.random() < 0.5}
    if kind == "volume":
        w, h = _log(rng, 64, 512), _log(rng, 64, 512)
        return {"kind": "volume", "w": w, "h": h, "spp": max(1, min(_log(rng, 1, 32), 4_000_000 // (w * h))),
                "depth": rng.randint(4, 32)}
    if kind == "particles":
        return {"kind": "particles", "scene": rng.choice(["box", "zoo"]), "w": _log(rng, 64, 1024),
                "h": _log(rng, 64, 1024), "count": _log(rng, 1 << 12, 1 << 23)}
    if kind == "batch":
        return {"kind": "batch", "scenes": rng.randint(2, 12), "spp": rng.randint(1, 6)}
    if kind == "adjoint":
        return {"kind": "adjoint", "w": _log(rng, 48, 256), "h": _log(rng, 48, 256), "spp": _log(rng, 1, 32),
                "depth": rng.randint(3, 8)}
    return {"kind": "upload", "sphere_n": _log(rng, 8, 160), "n": _log(rng, 64, 20_000)}


# ------------------------------------------------------------------ scenes ----
@functools.lru_cache(maxsize=None)
def _asset(name, arg=0):
    """(scene, settings, params) of a procedural scene: geometry and maps, shared by every seed."""
    if name == "box":
        return (*procedural.cornell_box(256, 256), None)
    if name == "instances":
        return (*procedural.instanced_spheres(256, 256), None)
    if name == "zoo":
        return (*procedural.material_zoo(64, 64), None)
    if name == "volume":
        return (*procedural.volume_sphere(256, 256), None)
    if name == "adjoint":
        return procedural.adjoint_patches(256, 256)
    if name == "sphere":
        return procedural.displaced_sphere(arg, 7), None, None
    if name == "batch":
        return (*procedural.batch_scene(arg), None)
    raise ValueError(name)


VIEW = {"box": (40.0, (0.5, 0.5, 2.3), (0.5, 0.5, 0.0)), "instances": (40.0, (0.0, 13.0, 21.0), (0.0, 0.0, 0.0)),
        "zoo": (50.0, (0.0, 1.4, 4.2), (0.0, 0.6, 0.0)), "volume": (45.0, (0.0, 1.6, 5.0), (0.0, 1.0, 0.0)),
        "adjoint": (35.0, (0.0, 0.9, 3.6), (0.0, 0.0, 0.0)), "batch": (40.0, (0.0, 1.8, 4.2), (0.0, 0.9, 0.0))}


def _scene(name, w, h, rng, arg=0):
    """The asset under a camera of this seed, a little off the scene's usual view."""
    scene, st, params = _asset(name, arg)
    fov, origin, target = VIEW[name]
    dist = math.sqrt(sum((a - b) ** 2 for a, b in zip(origin, target)))
    origin = tuple(float(o + rng.uniform(-0.02, 0.02) * dist) for o in origin)
    scene = copy.copy(scene)
    scene.camera = Camera.look_at(w, h, fov, origin, target)
    return scene, st, params


# batch_scene indices of 10 k to 200 k triangles, so that twelve upload quickly
def _batch_ids(count):
    ids = []
    i = 0
    while len(ids) < count:
        tris = math.exp(np.random.default_rng(11 * 1000 + i).uniform(math.log(1e4), math.log(2e6)))
        if tris <= 2e5:
            ids.append(i)
        i += 1
    return ids


def _batch_films(case):
    """(scene index, width, height, spp) of each item: the scenes' own resolutions, spp rising with the index."""
    out = []
    for k, i in enumerate(_batch_ids(case["scenes"])):
        cam = _asset("batch", i)[0].camera
        out.append((i, cam.width, cam.height, 1 + (case["spp"] * (k % 3 + 1)) // 3))
    return out


# -------------------------------------------------------------------- rays ----
def _rays(name, n, rng):
    """Secondary-like rays: origins spread through the scene, directions uniform (in the box: towards its
    back, so that every ray meets a wall)."""
    rays = np.zeros(n, dtype=N.ray_dtype())
    lo, hi = {"box": ((0.02, 0.02, 0.02), (0.98, 0.98, 0.98)), "zoo": ((-3, 0.05, -1.9), (3, 2.7, 3)),
              "instances": ((-11, 0.0, -11), (11, 3.5, 11)), "sphere": ((-3, -3, -3), (3, 3, 3))}[name]
    rays["o"] = rng.uniform(lo, hi, (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3))
    if name == "box":
        d[:, 2] = -np.abs(d[:, 2]) - 1e-3
    if name == "sphere":
        d = rng.uniform(-1, 1, (n, 3)) - rays["o"]
    rays["d"] = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    rays["min_t"] = 1e-4
    rays["max_t"] = np.finfo(np.float32).max
    return rays


def _hit_fields(hits):
    """A device hit buffer (n x 6 words) as its float and its integer fields."""
    return {"tuv": hits[:, :3].view(torch.float32), "ids": hits[:, 3:]}


# ------------------------------------------------------------------- cases ----
METHOD = {"bxdf": N.METHOD_BXDF, "nee": N.METHOD_NEE, "mis": N.METHOD_MIS}
STRATEGY = {"uniform": N.STRATEGY_UNIFORM, "all": N.STRATEGY_ALL}


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    s = {"case": case, "dev": Device(0)}
    dev = s["dev"]
    if kind == "rays":
        scene, _, _ = _scene(case["scene"], 64, 64, rng)
        dev.upload(scene)
        rays = _rays(case["scene"], case["n"], rng)
        if case["host"]:
            s["rays"] = rays
            s["shadow"] = rays.copy()
            s["shadow"]["max_t"] = rng.uniform(0.1, 2.0, case["n"]).astype(np.float32)
        else:
            s["rays"] = torch.from_numpy(rays.view(np.float32).reshape(case["n"], 8)).cuda()
            s["hits"] = torch.empty((case["n"], 6), dtype=torch.int32, device="cuda")
        return s
    if kind in ("path", "volume", "particles"):
        scene, st, _ = _scene(case.get("scene", "volume"), case["w"], case["h"], rng)
        dev.upload(scene)
        s["film"] = torch.empty((case["w"], case["h"], 3), dtype=torch.float32, device="cuda")
        if kind == "path":
            s["settings"] = st.replace(method=METHOD[case["method"]], strategy=STRATEGY[case["strategy"]],
                                       spp=case["spp"], max_depth=case["depth"], seed=seed)
            if case["wide"]:
                dev.set_traversal(N.TRAVERSAL_WIDE)
            if case["alias"]:
                dev.set_light_sampling(N.LIGHT_SAMPLING_ALIAS)
        elif kind == "volume":
            s["settings"] = st.replace(spp=case["spp"], max_depth=case["depth"], seed=seed)
        else:                       # the reference's particle example: min_depth 7, unbounded depth, roulette 0.99
            s["settings"] = st.replace(integrator=N.INTEGRATOR_PARTICLE, max_depth=-1, min_depth=7,
                                       rr_threshold=0.99, seed=seed)
        return s
    if kind == "batch":
        s["items"], s["films"] = [], []
        for i, w, h, spp in _batch_films(case):
            scene, st, _ = _scene("batch", w, h, rng, i)
            d = Device(0)
            d.upload(scene)
            s["items"].append((d, st.replace(spp=spp, seed=seed + i)))
            s["films"].append(torch.empty((w, h, 3), dtype=torch.float32, device="cuda"))
        return s
    if kind == "adjoint":
        scene, st, params = _scene("adjoint", case["w"], case["h"], rng)
        dev.upload(scene)
        s["settings"] = st.replace(spp=case["spp"], max_depth=case["depth"], seed=seed)
        s["params"] = params
        # dL/dI of an L2 loss: twice the residual of a film against its target
        s["dldi"] = rng.normal(scale=0.05, size=(case["w"], case["h"], 3)).astype(np.float32)
        return s
    # upload: the sphere mesh under a transform of this seed
    scene, _, _ = _asset("box")
    scene = copy.copy(scene)
    scale = float(rng.uniform(0.9, 1.1))
    m = Mat4.scale((scale, scale, scale)) * Mat4.from_axis_angle((0, 1, 0), float(rng.uniform(0, 2 * math.pi)))
    scene.meshes = [_asset("sphere", case["sphere_n"])[0].transformed(m)]
    group = copy.copy(scene.groups[0])
    group.ref = 0
    scene.groups = [group]
    scene.camera = Camera.look_at(256, 256, 40.0, (0.0, 0.0, 4.0), (0.0, 0.0, 0.0))
    s["scene"] = scene
    s["rays"] = _rays("sphere", case["n"], rng)
    return s


def run(s):
    case, dev = s["case"], s["dev"]
    kind = case["kind"]
    if kind == "rays":
        if case["host"]:
            h = dev.trace_closest(s["rays"])
            return {"t": h["t"], "u": h["u"], "v": h["v"], "prim": h["prim"], "sub": h["sub"],
                    "flags": h["flags"].astype(np.int64), "occluded": dev.trace_any(s["shadow"])}
        dev.trace_closest_device(s["rays"].data_ptr(), case["n"], s["hits"].data_ptr())
        return _hit_fields(s["hits"])
    if kind in ("path", "volume"):
        dev.render_device(s["settings"], s["film"].data_ptr())
        return s["film"]
    if kind == "particles":
        dev.render_particles_device(s["settings"], case["count"], s["film"].data_ptr())
        return s["film"]
    if kind == "batch":
        dev.render_batch_device(s["items"], [f.data_ptr() for f in s["films"]])
        return s["films"]
    if kind == "adjoint":
        p = s["params"]
        g_albedo, g_alpha = dev.adjoint_backward(s["settings"], s["dldi"], p["albedo_texture"], p["alpha_materials"])
        return {"albedo": g_albedo, "alpha": g_alpha}
    dev.upload(s["scene"])
    h = dev.trace_closest(s["rays"])
    return {"t": h["t"], "u": h["u"], "v": h["v"], "prim": h["prim"]}


def work(case):
    """Bytes: the rays / parameters / film in and out, and the part of the scene that the rays can touch, once.
    Flops: for each ray the box tests of one root-to-leaf descent of a balanced binary tree (two 25-flop slab
    tests a level) and one 45-flop triangle test."""
    kind = case["kind"]
    tris = {"box": 36, "zoo": 448, "instances": 199_692 + 64, "volume": 499_392 + 4, "adjoint": 199_692,
            "batch": 60_000, "upload": 12 * case.get("sphere_n", 1) ** 2}
    name = case.get("scene", kind)
    t = tris[name]
    per_ray = math.ceil(math.log2(t)) * 2 * 25 + 45
    scene_bytes = t * (12 * 2 + 48)               # vertices and indices, one 48-byte test record a triangle
    if kind in ("rays", "upload"):
        n = case["n"]
        rays = n * (2 if case.get("any") else 1)
        out = n * 24 + (n if case.get("any") else 0)
        b = rays * 32 + out + (scene_bytes if kind == "upload" else min(scene_bytes, rays * 48))
        # upload: a tree over t primitives sorts them into 12 buckets a level
        build = t * math.ceil(math.log2(t)) * 30 if kind == "upload" else 0
        return {"bytes": b, "flops": rays * per_ray + build}
    if kind == "batch":
        films = [(w * h, spp) for _, w, h, spp in _batch_films(case)]
        samples, pixels = sum(p * s for p, s in films), sum(p for p, _ in films)
        scene_bytes *= case["scenes"]
    elif kind == "particles":
        samples, pixels = case["count"], case["w"] * case["h"]
    else:
        pixels = case["w"] * case["h"]
        samples = pixels * case["spp"]
    rays = samples * RAYS_PER_SAMPLE["particles" if kind == "particles" else name]
    b = min(scene_bytes, rays * 48) + pixels * 12
    if kind == "adjoint":
        rays *= 2                                  # forward and replay
        b += pixels * 12 + 2 * 512 * 512 * 12
    return {"bytes": b, "flops": rays * per_ray}


def exact(case, seed):
    """Ray queries of the box: the closest distance by testing every triangle in 64 bits.  The barycentrics of
    rays that meet two coplanar triangles at once depend on the order of the tests and have no one value; films,
    gradients and hits of the large scenes would need the whole renderer again."""
    if case["kind"] != "rays" or case["scene"] != "box" or not case["host"]:
        return None
    rng = np.random.default_rng(seed)
    scene, _, _ = _scene("box", 64, 64, rng)
    rays = _rays("box", case["n"], rng)
    tri = np.concatenate([scene.meshes[g.ref].positions[scene.meshes[g.ref].indices] for g in scene.groups])
    tri = tri.astype(np.float64)
    o, d = rays["o"].astype(np.float64), rays["d"].astype(np.float64)
    best = np.full(case["n"], np.inf)
    for a, b, c in tri:
        e1, e2 = b - a, c - a
        p = np.cross(d, e2)
        det = p @ e1
        with np.errstate(divide="ignore", invalid="ignore"):
            inv = 1.0 / det
            tv = o - a
            u = (tv * p).sum(1) * inv
            q = np.cross(tv, e1)
            v = (d * q).sum(1) * inv
            t = (q @ e2) * inv
        ok = (det != 0) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (t >= rays["min_t"].astype(np.float64))
        best = np.where(ok & (t < best), t, best)
    best = np.where(np.isinf(best), np.finfo(np.float32).max, best)
    return {"t": best, "u": None, "v": None, "prim": None, "sub": None, "flags": None, "occluded": None}
