"""Workloads of the transport loop, each one pass of what a program that uses it does.

The kinds, all through the public entry points (``CudaEngine``, ``Batch``, ``ptr_trace_closest``):

* ``view``     a frame of an interactive view: a few 1-spp ``render_frame`` calls that
  accumulate, then the picture read back (precompiled kernels: no compile while editing);
* ``frame``    one picture at its full samples per pixel, with the kernels compiled for the
  scene, read back;
* ``tiles``    a tiled production render with first-hit pictures and variance;
* ``batch``    many scenes of uneven size in one batched wavefront, every picture read back;
* ``adjoint``  gradients of every material parameter (path-replay adjoint);
* ``inverse``  a whole optimiser step: parameters pushed, picture, loss, gradients;
* ``open``     a scene with a mesh uploaded (BVHs built on the GPU) and its first frame;
* ``trace``    nearest-hit queries of the host's own rays (picking, visibility, baking).

Scenes are the package's synthetic ones (``pathtracerglsl_b200.scenes``): a case fixes their
structure and sizes; the seed draws materials, placements, cameras and the random stream.
"""
import ctypes
import math

import numpy as np
import torch

from pathtracerglsl_b200 import abi, adjoint, scenes
from pathtracerglsl_b200.compiler import Compiler
from pathtracerglsl_b200.engine import CudaEngine


def listed():
    return [
        # a viewport while the camera is dragged: the smallest call, launches and latency
        {"name": "view_128", "kind": "view", "scene": "cornell", "w": 128, "h": 128, "frames": 1, "depth": 8},
        # the plain Cornell box of the benchmark: 256 x 256, 64 spp, MIS
        {"name": "cornell_256", "kind": "frame", "scene": "cornell", "w": 256, "h": 256, "spp": 64, "depth": 8,
         "special": True},
        # the mesh workload of the benchmark: 1.31 M triangles x 16 instances under a sky, full HD, MIS;
        # device-built trees, the autotuner's recorded pick for it
        {"name": "mesh_1080p", "kind": "frame", "scene": "mesh", "w": 1920, "h": 1080, "spp": 16, "depth": 12,
         "level": 8, "instances": 16, "accel": "cwbvh", "build": "device", "special": True, "sort": 8, "ray_sort": 1,
         "capacity": 1 << 25},
        # an ordinary mesh preview at ragged size: host-built binary BVH, precompiled kernels, default tuning
        {"name": "mesh_bvh_517", "kind": "frame", "scene": "mesh", "w": 517, "h": 389, "spp": 4, "depth": 6,
         "level": 5, "instances": 9, "accel": "bvh", "build": "host", "special": False, "sort": 1, "ray_sort": 0,
         "capacity": 0},
        # the media + spectral workload of the benchmark: chromatic media, equiangular NEE, depth 64
        {"name": "media_1024", "kind": "frame", "scene": "media", "w": 1024, "h": 1024, "spp": 16, "depth": 64,
         "special": True},
        # hundreds of lamps in thin fog under the light tree, precompiled kernels
        {"name": "lights_512", "kind": "frame", "scene": "lights", "w": 512, "h": 384, "spp": 8, "depth": 6,
         "lamps": 256, "special": False},
        # a production render in tiles (ragged last column and row) of a heterogeneous fog, four pictures
        {"name": "tiles_fog", "kind": "tiles", "scene": "het", "w": 600, "h": 340, "spp": 4, "depth": 12, "tile": 256},
        # a page of thumbnails: 16 small scenes in one wavefront, precompiled kernels
        {"name": "batch_thumbs", "kind": "batch", "jobs": 16, "mix": 5, "spheres": 40, "res": 128, "spp": 4,
         "special": False},
        # the benchmark's 64-job mix (1-200 spheres, 128..1024 squared, depth 4-32) at up to 16 spp
        {"name": "batch_mix", "kind": "batch", "jobs": 64, "mix": 0, "spheres": 200, "res": 1024, "spp": 16,
         "special": True},
        # the inverse-rendering workload: 64 spheres and a medium, 252 parameters, 256 x 256, 16 spp
        {"name": "adjoint_256", "kind": "adjoint", "scene": "spheres", "w": 256, "h": 256, "spp": 16, "depth": 8,
         "spheres": 64, "special": True},
        # a scene opened: a 327,680-triangle mesh uploaded with device-built trees, and its first frame
        {"name": "open_mesh", "kind": "open", "scene": "mesh", "w": 640, "h": 360, "spp": 1, "depth": 4,
         "level": 7, "instances": 16, "accel": "cwbvh"},
        # the caller's own rays against instanced meshes
        {"name": "trace_200k", "kind": "trace", "level": 5, "instances": 4, "accel": "cwbvh", "rays": 200003},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["view", "frame", "mesh", "mesh", "media", "lights", "tiles", "batch", "batch", "adjoint",
                       "inverse", "open", "trace"])
    if kind == "view":
        return {"kind": "view", "scene": rng.choice(["cornell", "rough", "lights"]), "w": _log(rng, 64, 900),
                "h": _log(rng, 64, 700), "frames": rng.randint(1, 4), "depth": rng.randint(4, 12), "lamps": _log(rng, 8, 600)}
    if kind == "frame":
        w, h = _log(rng, 64, 1024), _log(rng, 64, 1024)
        return {"kind": "frame", "scene": rng.choice(["cornell", "rough", "het"]), "w": w, "h": h,
                "spp": max(1, min(_log(rng, 2, 128), (1 << 24) // (w * h))), "depth": rng.randint(4, 16),
                "special": rng.random() < 0.5}
    if kind == "mesh":
        w = _log(rng, 200, 1600)
        return {"kind": "frame", "scene": "mesh", "w": w, "h": _log(rng, 150, 1000), "spp": _log(rng, 1, 8),
                "depth": rng.randint(3, 12), "level": rng.randint(4, 8), "instances": _log(rng, 1, 40),
                "accel": rng.choice(["bvh", "cwbvh", "cwbvh"]), "build": "device", "special": rng.random() < 0.5,
                "sort": rng.choice([1, 8]), "ray_sort": rng.choice([0, 1]), "capacity": rng.choice([0, 1 << 25])}
    if kind == "media":
        return {"kind": "frame", "scene": "media", "w": _log(rng, 100, 1024), "h": _log(rng, 100, 1024),
                "spp": _log(rng, 1, 16), "depth": rng.randint(8, 64), "special": rng.random() < 0.7}
    if kind == "lights":
        return {"kind": "frame", "scene": "lights", "w": _log(rng, 100, 800), "h": _log(rng, 100, 600),
                "spp": _log(rng, 1, 16), "depth": rng.randint(3, 8), "lamps": _log(rng, 8, 2000),
                "special": rng.random() < 0.3}
    if kind == "tiles":
        return {"kind": "tiles", "scene": rng.choice(["het", "rough", "cornell"]), "w": _log(rng, 200, 1600),
                "h": _log(rng, 150, 1000), "spp": _log(rng, 1, 8), "depth": rng.randint(4, 12),
                "tile": rng.choice([128, 256, 512, 1000])}
    if kind == "batch":
        return {"kind": "batch", "jobs": _log(rng, 2, 64), "mix": rng.randint(1, 999), "spheres": _log(rng, 3, 200),
                "res": _log(rng, 64, 1024), "spp": _log(rng, 1, 12), "special": rng.random() < 0.5}
    if kind in ("adjoint", "inverse"):
        return {"kind": kind, "scene": rng.choice(["spheres", "spheres", "box"]), "w": _log(rng, 40, 400), "h": _log(rng, 40, 400),
                "spp": _log(rng, 1, 16), "depth": rng.randint(3, 8), "spheres": _log(rng, 4, 64),
                "special": rng.random() < 0.5}
    if kind == "open":
        return {"kind": "open", "scene": "mesh", "w": _log(rng, 100, 900), "h": _log(rng, 100, 600), "spp": 1,
                "depth": rng.randint(2, 6), "level": rng.randint(4, 8), "instances": _log(rng, 1, 40),
                "accel": rng.choice(["bvh", "cwbvh"])}
    return {"kind": "trace", "level": rng.randint(3, 7), "instances": _log(rng, 1, 16),
            "accel": rng.choice(["bvh", "cwbvh"]), "rays": _log(rng, 500, 2000000)}


# ------------------------------------------------------------------------------- scenes
def _jitter_materials(mats, rng):
    """The scene's materials with colours, roughness and IOR of their own."""
    out = {}
    for name, m in mats.items():
        m = dict(m)
        if m.get("model") == "lambert" and not m.get("emission"):
            m["albedo"] = [float(np.clip(a * rng.uniform(0.8, 1.15), 0.05, 0.92)) for a in m.get("albedo", [0.5] * 3)]
        elif m.get("model") == "ggx":
            m["roughness"] = float(np.clip(m.get("roughness", 0.5) * rng.uniform(0.8, 1.2), 0.1, 0.9))
        elif m.get("model") == "dielectric" and "medium" not in m:
            m["ior"] = float(np.clip(m.get("ior", 1.5) * rng.uniform(0.95, 1.1), 1.2, 1.9))
        out[name] = m
    return out


def _shrink_spheres(objects, rng):
    """Spheres a little smaller than placed (they stay disjoint)."""
    out = []
    for o in objects:
        if o.get("type") == "sphere":
            p = o["parameters"]
            o = dict(o, parameters=dict(p, radius=float(p["radius"] * rng.uniform(0.85, 1.0))))
        out.append(o)
    return out


def _camera(position, target, rng, by):
    """Camera parameters near the given ones."""
    return {"camera.position": [float(x + by * rng.uniform(-1, 1)) for x in position],
            "camera.target": [float(x + 0.5 * by * rng.uniform(-1, 1)) for x in target]}


_MESH = {}   # level -> a displaced icosphere (vertices, indices)


def _mesh(level):
    if level not in _MESH:
        v, f = scenes.icosphere(level)
        v = v * (1.0 + 0.05 * scenes.value_noise(v, 0))[:, None]
        _MESH[level] = (v.astype(np.float32), f.astype(np.uint32))
    return _MESH[level]


def _mesh_scene(case, rng):
    """scenes.mesh_scene's ground, sky and camera; the mesh itself scaled and instanced by the seed."""
    seed = int(rng.randint(1 << 30))
    sc, st, _ = scenes.mesh_scene(level=0, instances=case["instances"], seed=seed, max_depth=case.get("depth", 4),
                                  accel=case["accel"], env_size=(512, 256))
    v, f = _mesh(case["level"])
    proto = sc["objects"][1]["prototype"]
    proto["positions"] = (v * np.float32(rng.uniform(0.9, 1.1))).reshape(-1)
    proto["indices"] = f.reshape(-1)
    proto["triangleAlpha"] = rng.uniform(0.05, 0.5, len(f)).astype(np.float32)
    cam = st["measurement"]["camera"]
    return sc, st, _camera(cam["position"], cam["target"], rng, 0.3)


def _scene(case, rng):
    """(scene, strategy, live camera parameters) of a case."""
    name, depth = case["scene"], case["depth"]
    if name == "mesh":
        return _mesh_scene(case, rng)
    if name == "media":
        sc, st, _ = scenes.media_scene(max_depth=depth)
        objs = [dict(o) for o in sc["objects"]]
        for o in objs[1:]:
            c = o["parameters"]["center"]
            o["parameters"] = {"center": [float(c[0] + rng.uniform(-0.05, 0.05)), 1.0, float(rng.uniform(-0.2, 0.2))],
                               "radius": float(rng.uniform(0.9, 1.0))}
        lights = [dict(sc["lights"][0], position=[float(rng.uniform(-0.3, 0.3)), 2.4, 1.2]), sc["lights"][1]]
        cam = st["measurement"]["camera"]
        return dict(sc, objects=objs, lights=lights), st, _camera(cam["position"], cam["target"], rng, 0.2)
    if name == "spheres":
        sc, st, _ = scenes.adjoint_scene(case["spheres"], n_spheres=case["spheres"], max_depth=depth)
    elif name == "box":
        sc, st = scenes.adjoint_box_scene()
        st = dict(st, measurement=dict(st["measurement"], maxBounces=depth))
    elif name == "lights":
        sc, st = scenes.many_lights(n=2 * (case["lamps"] // 2), seed=int(rng.randint(1 << 30)), fog=True, max_depth=depth)
    elif name == "het":
        sc, st = scenes.het_fog(kind="ground", max_depth=depth)
    elif name == "rough":
        sc, st = scenes.cornell_rough(max_depth=depth)
    else:
        sc, st = scenes.cornell(max_depth=depth)
    sc = dict(sc, materials=_jitter_materials(sc["materials"], rng), objects=_shrink_spheres(sc["objects"], rng))
    return sc, st, _camera([0, 1, 4], [0, 1, 0], rng, 0.15)


class _State:
    """What a case's program holds; the engine is closed with it."""

    def __init__(self, case):
        self.case = case
        self.eng = CudaEngine(torch.cuda.current_device())

    def __del__(self):
        eng = getattr(self, "eng", None)
        if eng is not None:
            eng.close()


def _load(s, sc, st, params, rng):
    case, eng = s.case, s.eng
    s.renderer, s.packed = Compiler().compile(sc, st)
    eng.set_accel_build(case.get("build", "host"))
    if case.get("capacity") or case.get("sort", 1) != 1 or case.get("ray_sort"):
        eng.set_tuning(capacity=case.get("capacity", 0), sort_buckets=case.get("sort", 1), ray_sort=case.get("ray_sort", 0))
    eng.register_scene(s.packed)
    eng.load_renderer(s.renderer)
    eng.select_renderer(s.renderer.id)
    eng.params = dict(params)
    eng.pin_reset_salt(int(rng.randint(1 << 30)))
    if case.get("special"):
        eng.specialize()


def prepare(case, seed):
    rng = np.random.RandomState(seed % (1 << 32))
    s = _State(case)
    eng, kind = s.eng, case["kind"]
    if kind == "batch":
        items, s.frames = [], []
        for k, (sc, st, (w, _h, _spp)) in enumerate(scenes.batch_scenes(case["jobs"], case["mix"], case["spheres"])):
            sc = dict(sc, materials=_jitter_materials(sc["materials"], rng), objects=_shrink_spheres(sc["objects"], rng))
            items.append(Compiler().compile(sc, st))
            side = max(16, w * case["res"] // 1024) - k % 3
            s.frames.append((side, side, case["spp"], 0, int(rng.randint(1 << 30)), _camera([0, 1, 4], [0, 1, 0], rng, 0.15)))
        s.batch = eng.batch(items)
        if case["special"]:
            eng.set_tuning(block=128)     # the autotuner's recorded pick for the mix
            s.batch.specialize()
        return s
    if kind == "trace":
        sc, st, _ = _mesh_scene(case, rng)
        s.renderer, s.packed = Compiler().compile(sc, st)
        eng.register_scene(s.packed)
        s.rays = _rays(case, rng)
        return s
    if kind == "open":
        sc, st, params = _scene(case, rng)
        s.renderer, s.packed = Compiler().compile(sc, st)
        eng.set_accel_build("device")
        eng.load_renderer(s.renderer)
        eng.params = dict(params)
        eng.pin_reset_salt(int(rng.randint(1 << 30)))
        return s
    sc, st, params = _scene(case, rng)
    if kind == "tiles":
        st = dict(st, measurement=dict(st["measurement"], aovs=["albedo", "normal"]))
    _load(s, sc, st, params, rng)
    if kind == "adjoint":
        # the residual of a noisy picture against its target, as the L2 loss hands it over
        n = case["w"] * case["h"] * 3
        s.dl = (2.0 / n * rng.normal(0.0, 0.2, (case["h"], case["w"], 3))).astype(np.float32)
    elif kind == "inverse":
        s.target = rng.uniform(0.0, 1.0, (case["h"], case["w"], 3)).astype(np.float32)
        table = adjoint.param_table(s.packed)
        s.step = adjoint.with_params(s.packed, table * (1.0 + 0.02 * rng.uniform(-1, 1, table.shape)))
    return s


def _rays(case, rng):
    """Rays from a shell around the instances towards points among them."""
    n, grid = case["rays"], int(np.ceil(np.sqrt(case["instances"])))
    reach = 1.3 * grid
    o = rng.normal(size=(n, 3))
    o = o / np.linalg.norm(o, axis=1, keepdims=True) * (2.5 * reach)
    o[:, 1] = np.abs(o[:, 1]) + 0.1
    d = np.stack([rng.uniform(-reach, reach, n), rng.uniform(0.0, 2.0, n), rng.uniform(-reach, reach, n)], 1) - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.ascontiguousarray(np.concatenate([o, d], 1).astype(np.float32))


# --------------------------------------------------------------------------------- passes
def run(state):
    case, eng = state.case, state.eng
    kind = case["kind"]
    if kind == "batch":
        state.batch.render(state.frames)
        return [state.batch.read_export(j) for j in range(len(state.batch))]
    if kind == "trace":
        n = case["rays"]
        region, element, prim = (np.empty(n, np.int32) for _ in range(3))
        t = np.empty(n, np.float32)
        accel = abi.ACCEL_CWBVH if case["accel"] == "cwbvh" else abi.ACCEL_BVH
        eng._check(eng.lib.ptr_trace_closest(eng.ctx, eng.scene, accel, state.rays.ctypes.data, n, region.ctypes.data,
                                             element.ctypes.data, prim.ctypes.data, t.ctypes.data))
        return {"region": region, "element": element, "prim": prim, "t": t}
    w, h = case["w"], case["h"]
    if kind == "adjoint":
        return eng.backward(state.dl, w, h, case["spp"])
    if kind == "inverse":
        eng.update_params(state.step)
        eng.reset()
        eng.render_frame(w, h, case["spp"])
        image = eng.read_export("radiance")
        loss, dl = adjoint.l2_loss(image, state.target)
        return {"loss": loss, "image": image, "grad": eng.backward(dl, w, h, case["spp"])}
    if kind == "tiles":
        pictures = ("radiance", "variance", "albedo", "normal")
        return eng.render_tiled(w, h, case["spp"], tile_size=case["tile"], pictures=pictures)[0]
    if kind == "open":
        eng.register_scene(state.packed)
        eng.render_frame(w, h, case["spp"])
        return eng.read_export("radiance")
    eng.reset()
    for _ in range(case.get("frames", 1)):
        eng.render_frame(w, h, case.get("spp", 1))
    return eng.read_export("radiance")


# ----------------------------------------------------------------------------- what it takes
# Walk iterations (nearest-hit queries) and shadow queries per sample, about, of each scene,
# and the arithmetic of one region or triangle test, box test and shading event.
_WALK = {"cornell": (4.0, 3.0), "rough": (4.5, 3.0), "mesh": (2.2, 1.3), "media": (6.0, 3.0), "lights": (4.0, 3.5),
         "het": (6.0, 4.0), "spheres": (5.0, 4.0), "box": (5.0, 4.0), "batch": (5.0, 3.5)}
_TEST, _BOX, _SHADE = 30, 20, 400


def _per_sample(scene, case):
    """Operations of one sample: every query tests the regions (or the boxes and triangles
    that a tree leaves), every walk iteration shades."""
    walk, shadow = _WALK[scene]
    if scene == "mesh":
        query = 8 * 8 * _BOX + 6 * _TEST + _TEST
    else:
        regions = {"spheres": 6 + case.get("spheres", 0), "lights": 9 + 16, "box": 9, "media": 5}.get(scene, 8)
        query = regions * _TEST
    return (walk + shadow) * query + walk * _SHADE


def work(case):
    kind = case["kind"]
    if kind == "batch":
        flops = out = 0.0
        for k, (sc, _st, (w, _h, _spp)) in enumerate(scenes.batch_scenes(case["jobs"], case["mix"], case["spheres"])):
            side = max(16, w * case["res"] // 1024) - k % 3
            walk, shadow = _WALK["batch"]
            flops += side * side * case["spp"] * ((walk + shadow) * len(sc["objects"]) * _TEST + walk * _SHADE)
            out += 12.0 * side * side
        return {"bytes": out + 160 * case["jobs"], "flops": flops}
    tris = 20 * 4 ** case.get("level", 0)
    if kind == "trace":
        return {"bytes": case["rays"] * 40 + tris * 36, "flops": case["rays"] * (8 * 8 * _BOX + 6 * _TEST)}
    pixels = case["w"] * case["h"]
    samples = pixels * case.get("spp", 1) * case.get("frames", 1)
    flops = samples * _per_sample(case["scene"], case)
    byts = 12.0 * pixels + 160
    if case["scene"] == "mesh":
        byts += 20.0 * 512 * 256 + tris * 36          # the sky's table and CDFs, the triangles
    if kind == "tiles":
        byts = 4 * 12.0 * pixels
    elif kind in ("adjoint", "inverse"):
        flops *= 2.0 if kind == "adjoint" else 3.0    # the walk and its replay; a picture before them
        byts *= 2.0
    elif kind == "open":
        byts += tris * (12 * 0.5 + 12 + 4)            # vertices, indices and alphas once more: the trees' build
        flops += tris * 20 * _BOX
    return {"bytes": byts, "flops": flops}


# ------------------------------------------------------------------------------ exact values
def exact(case, seed):
    """Nearest distances by a float64 scan of every triangle.  A picture or a gradient has no
    such value: it is the mean of random walks whose branches follow the binary32 values."""
    tris = 20 * 4 ** case.get("level", 0) * case.get("instances", 0)
    if case["kind"] != "trace" or tris * case["rays"] > 3e10:
        return None
    rng = np.random.RandomState(seed % (1 << 32))
    sc, _st, _ = _mesh_scene(case, rng)
    rays = torch.from_numpy(_rays(case, rng)).cuda().double()
    o, d = rays[:, :3], rays[:, 3:]
    far = torch.full((len(rays),), 1000.0, dtype=torch.float64, device="cuda")
    t = torch.where(d[:, 1] < 0, -o[:, 1] / d[:, 1], far)          # the ground plane y = 0
    t = torch.where((t > 0) & (t < far), t, far)
    proto = sc["objects"][1]["prototype"]
    v = torch.from_numpy(proto["positions"].reshape(-1, 3)).cuda().double()
    f = torch.from_numpy(proto["indices"].reshape(-1, 3).astype(np.int64)).cuda()
    for p in sc["objects"][1]["placements"]:
        ax = torch.tensor(p["rotation"]["axis"], dtype=torch.float64, device="cuda")
        ax = ax / ax.norm()
        ang = p["rotation"]["angle"]
        k = torch.zeros(3, 3, dtype=torch.float64, device="cuda")
        k[0, 1], k[0, 2], k[1, 2] = -ax[2], ax[1], -ax[0]
        k = k - k.T
        rot = torch.eye(3, dtype=torch.float64, device="cuda") + math.sin(ang) * k + (1 - math.cos(ang)) * (k @ k)
        # the rays in the instance's frame: distances keep their scale
        lo = (o - torch.tensor(p["position"], dtype=torch.float64, device="cuda")) @ rot / p["scale"]
        ld = d @ rot / p["scale"]
        t = torch.minimum(t, _nearest(lo, ld, v[f[:, 0]], v[f[:, 1]], v[f[:, 2]]))
    return {"region": None, "element": None, "prim": None, "t": t}


def _nearest(o, d, a, b, c):
    e1, e2 = b - a, c - a
    n = torch.linalg.cross(e1, e2)
    an = (a * n).sum(1)
    ae1, ae2 = torch.linalg.cross(a, e1), torch.linalg.cross(a, e2)
    best = torch.full((len(o),), 1000.0, dtype=torch.float64, device=o.device)
    chunk = max(1, (1 << 25) // len(o))
    m = torch.linalg.cross(o, d)
    for i in range(0, len(a), chunk):
        j = slice(i, i + chunk)
        det = -(d @ n[j].T)
        t = (o @ n[j].T - an[j]) / det
        # u = e2 . ((o - a) x d) / det, v = -e1 . ((o - a) x d) / det, with a x d . e = d . (e x a)
        u = (m @ e2[j].T - d @ (-ae2[j]).T) / det
        w = -(m @ e1[j].T - d @ (-ae1[j]).T) / det
        ok = (u >= -1e-6) & (w >= -1e-6) & (1 - u - w >= -1e-6) & (t > 0) & (det.abs() >= 1e-12)
        best = torch.minimum(best, torch.where(ok, t, torch.full_like(t, 1000.0)).amin(1))
    return best
