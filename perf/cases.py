"""Performance cases of the ray queries and the renderers, through the framework's public entry points.

Each case is one kind of call with its sizes:

  query      lmgpu_accel_intersect_device / lmgpu_accel_occluded_device on rays that are on the GPU
  host       accel.intersect_batch on rays in host memory
  build      accel.build_triangles with the GPU builder, then a query: a scene that changes per call
  pt         renderer::pt, scheduler "sample"
  batch      BatchRenderer: many uneven renderer::pt jobs in one shared wavefront
  lt, bdpt   renderer::lt and renderer::bdpt, scheduler "sample"

Scenes are those of lightmetrica.synthetic: the closed box, random-triangle soups of 1k-200k
triangles, displaced spheres on a ground plane (up to the 3.8M triangles of the benchmark frame)
and instances of one mesh under affine transforms with an environment map. Scenes whose geometry
takes seconds to generate stay resident between preparations, as a program that renders many
frames of one scene keeps them; their rays and random streams come from the seed. Small scenes are
made and built from the seed each time.
"""
from __future__ import annotations

import ctypes
import itertools
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "lightmetrica-v3_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import lightmetrica as lm  # noqa: E402
from lightmetrica import _native as N  # noqa: E402
from lightmetrica import synthetic as syn  # noqa: E402
from lightmetrica.serving import BatchRenderer  # noqa: E402

lm.init()

# The largest renders and queries of the ranges, in paths and rays (the benchmark's probe and frame).
MAX_RAYS = 1 << 24
MAX_PATHS = 1920 * 1080 * 16


def listed():
    return [
        # a handful of picking rays into a small model: launch latency
        {"name": "query_tiny", "kind": "query", "scene": "soup", "tris": 1009, "pattern": "camera", "any": False, "rays": 257},
        # the benchmark's raycast probe: every direction from one point, 3.8M triangles
        {"name": "query_probe", "kind": "query", "scene": "spheres", "spheres": 40, "subdiv": 6, "pattern": "probe",
         "any": False, "rays": 1 << 24},
        # an ambient-occlusion bake: short any-hit rays off the surfaces, odd count
        {"name": "occlusion_bake", "kind": "query", "scene": "spheres", "spheres": 20, "subdiv": 5, "pattern": "bounce",
         "any": True, "rays": 3000007},
        # diffuse bounces inside a random-triangle soup (incoherent, many overlapping boxes)
        {"name": "query_soup", "kind": "query", "scene": "soup", "tris": 60000, "pattern": "bounce", "any": False, "rays": 1 << 20},
        # two-level tree: camera rays on 64 transformed instances of one mesh
        {"name": "query_instanced", "kind": "query", "scene": "instanced", "instances": 64, "lat": 200, "pattern": "camera",
         "any": False, "rays": 1920 * 1080},
        # rays and hits in pageable host memory, as a script's numpy arrays are
        {"name": "query_host", "kind": "host", "scene": "soup", "tris": 20011, "pattern": "probe", "rays": 200003},
        # dynamic geometry: GPU build from host triangles, then one frame's rays
        {"name": "build_and_query", "kind": "build", "scene": "soup", "tris": 200000, "pattern": "camera", "rays": 512 * 512},
        # a preview: the smallest resolution of the job mix, read back to the host
        {"name": "pt_preview", "kind": "pt", "scene": "box", "w": 64, "h": 64, "spp": 4, "max_verts": 9, "mode": "mis",
         "primary": "pixel", "read": True},
        # the benchmark frame at 16 of its 64 samples per pixel, left on the GPU
        {"name": "pt_frame", "kind": "pt", "scene": "spheres", "spheres": 40, "subdiv": 6, "w": 1920, "h": 1080, "spp": 16,
         "max_verts": 11, "mode": "mis", "primary": "pixel", "read": False},
        # sixteen jobs of the batched mix in one wavefront
        {"name": "batch_jobs", "kind": "batch", "jobs": 16, "mix": 2024, "max_tris": 200000},
        # light tracing and bidirectional path tracing of the benchmark scene
        {"name": "lt_frame", "kind": "lt", "scene": "spheres", "spheres": 40, "subdiv": 6, "w": 1920, "h": 1080,
         "samples": 1 << 22, "max_verts": 11},
        {"name": "bdpt_frame", "kind": "bdpt", "scene": "spheres", "spheres": 40, "subdiv": 6, "w": 1920, "h": 1080,
         "samples": 1 << 20, "max_verts": 11},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_scene(rng, kinds):
    scene = rng.choice(kinds)
    if scene == "soup":
        return {"scene": scene, "tris": _log_int(rng, 1000, 200000)}
    if scene == "spheres":
        return {"scene": scene, "spheres": rng.randint(4, 40), "subdiv": rng.randint(3, 5)}
    if scene == "instanced":
        return {"scene": scene, "instances": rng.randint(2, 64), "lat": rng.randint(16, 300)}
    return {"scene": scene}


def draw(rng):
    kind = rng.choice(["query", "query", "host", "build", "pt", "pt", "batch", "lt", "bdpt"])
    if kind == "query":
        c = _draw_scene(rng, ["soup", "spheres", "instanced"])
        patterns = ["camera", "probe"] if c["scene"] == "instanced" else ["camera", "probe", "bounce"]
        return dict(c, kind=kind, pattern=rng.choice(patterns), any=rng.random() < 0.4,
                    rays=_log_int(rng, 1, MAX_RAYS // 2))
    if kind == "host":
        c = _draw_scene(rng, ["soup", "spheres"])
        return dict(c, kind=kind, pattern=rng.choice(["camera", "probe"]), rays=_log_int(rng, 1, 1 << 20))
    if kind == "build":
        return {"kind": kind, "scene": "soup", "tris": _log_int(rng, 1000, 400000), "pattern": "camera",
                "rays": _log_int(rng, 256, 1 << 20)}
    if kind == "batch":
        return {"kind": kind, "jobs": rng.randint(2, 16), "mix": rng.randrange(1 << 20), "max_tris": _log_int(rng, 2000, 100000)}
    w = _log_int(rng, 48, 1920)
    h = max(1, int(w / rng.uniform(1.0, 2.0)))
    if kind == "pt":
        c = _draw_scene(rng, ["box", "soup", "spheres", "instanced"])
        return dict(c, kind=kind, w=w, h=h, spp=min(_log_int(rng, 1, 64), max(1, MAX_PATHS // (2 * w * h))),
                    max_verts=rng.randint(3, 13), mode=rng.choice(["mis", "mis", "nee", "naive"]),
                    primary=rng.choice(["pixel", "pixel", "image"]), read=rng.random() < 0.5)
    c = _draw_scene(rng, ["box", "soup", "spheres"])
    return dict(c, kind=kind, w=w, h=h, samples=_log_int(rng, 1 << 12, 1 << 22 if kind == "lt" else 1 << 20),
                max_verts=rng.randint(3, 11))


# ---------------------------------------------------------------------------------------------
# Scenes

# Loading an asset under a name that is taken releases the one before it. Preparations take turns on
# a few sets of names, so that several states live side by side and old ones give their memory back.
_turns, _turns_resident = itertools.count(), itertools.count()


def _prefix(kind):
    return f"perf_{kind}{next(_turns) % 64}_"


_resident = {}  # the last scenes whose geometry is slow to generate, oldest first


def _scene(case, seed, aspect=16 / 9):
    """The built scene of a case."""
    kind, w = case["scene"], round(aspect * 1024)
    if kind in ("spheres", "instanced"):
        key = (kind, case.get("spheres"), case.get("subdiv"), case.get("instances"), case.get("lat"), w)
        if key not in _resident:
            while len(_resident) >= 4:
                _resident.pop(next(iter(_resident)))
            at = next(_turns_resident) % 8
            if kind == "spheres":
                made = syn.spheres_scene(n_spheres=case["spheres"], subdiv=case["subdiv"], w=w, h=1024,
                                         ground_quads=_ground(case), prefix=f"perf_resident{at}_")
            else:
                made = syn.instanced_scene(n_instances=case["instances"], n_lat=case["lat"], n_lon=case["lat"], w=w, h=1024,
                                           env_w=512, env_h=256, prefix=f"perf_resident{at}_")
            made[0].build()
            _resident[key] = made[0]
        return _resident[key]
    if kind == "box":
        scene, _ = syn.box_scene(seed=seed, w=w, h=1024, prefix=_prefix("box"))
    else:
        scene, _ = syn.triangles_scene(seed, case["tris"], w, 1024, prefix=_prefix("soup"))
    scene.build()
    return scene


def _ground(case):
    return 512 if case["subdiv"] > 5 else 256


def _mix(case):
    """The job specs of a batch: sizes, samples (at most 16 per pixel) and path lengths."""
    return [dict(j, spp=min(j["spp"], 16)) for j in syn.batch_jobs(case["jobs"], seed=case["mix"], max_tris=case["max_tris"])]


def _soup(case, seed):
    rng = np.random.default_rng(seed)
    p, _ = syn.random_triangles(case["tris"], rng)
    return p.reshape(-1, 9)


# Eye, target, vertical field of view and the inner point of the probe, per scene.
_VIEWS = {"soup": ((0.5, 0.6, 2.3), (0.5, 0.5, 0.5), 40.0, (0.5, 0.5, 0.5)),
          "spheres": ((0.0, 4.0, 15.0), (0.0, 0.6, 0.0), 40.0, syn.RAYCAST_PROBE_ORIGIN),
          "instanced": ((0.0, 6.0, 22.0), (0.0, 1.0, 0.0), 40.0, (0.0, 2.0, 0.0))}


def _rays(case, seed, tri_p):
    """(n, 8) float32 rays (o, tmin, d, tmax) on the GPU."""
    n = case["rays"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = torch.rand((n, 4), generator=g, device="cuda", dtype=torch.float64)
    eye, at, fov, inner = _VIEWS[case["scene"]]
    out = torch.empty((n, 8), device="cuda", dtype=torch.float32)
    out[:, 3] = 1e-3
    out[:, 7] = 1e10
    if case["pattern"] == "camera":
        # one jittered ray per pixel of a 16:9 frame, in pixel order
        w = max(1, round(math.sqrt(n * 16 / 9)))
        h = -(-n // w)
        i = torch.arange(n, device="cuda")
        x = ((i % w).double() + u[:, 0]) / w * 2 - 1
        y = (torch.div(i, w, rounding_mode="floor").double() + u[:, 1]) / h * 2 - 1
        e, a = np.array(eye), np.array(at)
        z = (e - a) / np.linalg.norm(e - a)
        r = np.cross([0.0, 1.0, 0.0], z)
        r /= np.linalg.norm(r)
        up = np.cross(z, r)
        t = math.tan(math.radians(fov) / 2)
        cols = [torch.tensor(v, device="cuda", dtype=torch.float64) for v in (r * t * 16 / 9, up * t, z)]
        d = x[:, None] * cols[0] + y[:, None] * cols[1] - cols[2]
        out[:, :3] = torch.tensor(eye, device="cuda", dtype=torch.float32)
    elif case["pattern"] == "probe":
        z = 1 - 2 * u[:, 0]
        r = torch.sqrt((1 - z * z).clamp_min(0))
        d = torch.stack([r * torch.cos(2 * math.pi * u[:, 1]), r * torch.sin(2 * math.pi * u[:, 1]), z], 1)
        out[:, :3] = torch.tensor(inner, device="cuda", dtype=torch.float32)
    else:
        # cosine-distributed directions off uniformly chosen points of the surface (occlusion rays
        # end after a finite distance); 32 rays in a row leave one small neighbourhood
        p = torch.from_numpy(np.ascontiguousarray(tri_p)).cuda().reshape(-1, 3, 3)
        m = p.shape[0]
        k = torch.randint(0, m, (-(-n // 32),), generator=g, device="cuda").repeat_interleave(32)[:n]
        q = p[k].double()
        s = torch.sqrt(u[:, :1])
        v = u[:, 1:2]
        o = q[:, 0] * (1 - s) + q[:, 1] * (s * (1 - v)) + q[:, 2] * (s * v)
        nrm = torch.linalg.cross(q[:, 1] - q[:, 0], q[:, 2] - q[:, 0])
        nrm = nrm / nrm.norm(dim=1, keepdim=True).clamp_min(1e-30)
        z = 1 - 2 * u[:, 2]
        r = torch.sqrt((1 - z * z).clamp_min(0))
        d = nrm + 0.999 * torch.stack([r * torch.cos(2 * math.pi * u[:, 3]), r * torch.sin(2 * math.pi * u[:, 3]), z], 1)
        out[:, :3] = o.float()
        if case.get("any"):
            out[:, 7] = 0.25 if case["scene"] == "soup" else 4.0
    out[:, 4:7] = (d / d.norm(dim=1, keepdim=True)).float()
    return out


class _DeviceFilm:
    """The film's device pixels as a tensor (lmgpu_film_device_ptr), for a consumer on the GPU."""

    def __init__(self, film):
        ptr = ctypes.c_void_p()
        N.check(N.lib().lmgpu_film_device_ptr(film._h, ctypes.byref(ptr)))
        self.film = film
        self.__cuda_array_interface__ = {"shape": (film.h, film.w, 3), "typestr": "<f4", "data": (ptr.value, False), "version": 3}


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("query", "host", "build"):
        if case["scene"] == "soup":
            tri = _soup(case, seed)
            accel = lm.load_accel(_prefix("accel"), "sahbvh", builder="ploc" if kind == "build" else "sah")
            if kind != "build":
                accel.build_triangles(tri)
        else:
            scene = _scene(case, seed)
            accel, tri = scene.accel(), scene.flattened()["positions"]
        rays = _rays(case, seed, tri)
        if kind == "host":
            return {"kind": kind, "accel": accel, "rays": rays.cpu().numpy()}
        out = torch.empty((case["rays"], 4), device="cuda") if not case.get("any") else \
            torch.empty(case["rays"], device="cuda", dtype=torch.uint8)
        return {"kind": kind, "any": case.get("any", False), "accel": accel, "rays": rays, "out": out, "tri": tri}
    if kind == "batch":
        batch = BatchRenderer(queue_paths=1 << 22)
        jobs = []
        for i, j in enumerate(_mix(case)):
            scene, film = syn.triangles_scene(j["scene_seed"] ^ seed, j["tris"], j["res"], j["res"], prefix=_prefix(f"job{i}_"))
            scene.build()
            jobs.append({"scene": scene, "film": film, "spp": j["spp"], "max_verts": j["max_verts"], "seed": j["seed"] ^ seed})
        return {"kind": kind, "batch": batch, "jobs": jobs}
    scene = _scene(case, seed, case["w"] / case["h"])
    film = lm.load_film(_prefix("film"), "bitmap", w=case["w"], h=case["h"])
    prop = {"scene": scene, "output": film, "max_verts": case["max_verts"], "seed": seed, "scheduler": "sample"}
    if kind == "pt":
        prop.update(spp=case["spp"], sampling_mode=case["mode"], primary_ray_sampling_mode=case["primary"])
    else:
        prop["num_samples"] = case["samples"]
    renderer = lm.load_renderer(_prefix("renderer"), kind, **prop)
    read = case.get("read", False)
    return {"kind": kind, "renderer": renderer, "film": film, "view": None if read else torch.as_tensor(_DeviceFilm(film), device="cuda")}


def _hits(out):
    return {"t": out[:, 0], "u": out[:, 1], "v": out[:, 2], "prim": out.view(torch.int32)[:, 3]}


def run(state):
    kind = state["kind"]
    if kind == "host":
        h = state["accel"].intersect_batch(state["rays"])
        return {k: h[k] for k in ("t", "u", "v", "prim")}
    if kind in ("query", "build"):
        rays, out = state["rays"], state["out"]
        if kind == "build":
            state["accel"].build_triangles(state["tri"])
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        call = N.lib().lmgpu_accel_occluded_device if state["any"] else N.lib().lmgpu_accel_intersect_device
        N.check(call(state["accel"]._h, rays.data_ptr(), rays.shape[0], out.data_ptr(), stream))
        return out if state["any"] else _hits(out)
    if kind == "batch":
        state["batch"].reset()
        state["batch"].render(state["jobs"])
        return [j["film"].buffer_f32() for j in state["jobs"]]
    state["renderer"].render()
    return state["film"].buffer_f32() if state["view"] is None else state["view"]


# ---------------------------------------------------------------------------------------------

def _tris(case):
    if case.get("scene") == "soup":
        return case["tris"]
    if case.get("scene") == "spheres":
        return case["spheres"] * 20 * 4 ** case["subdiv"] + 2 * _ground(case) ** 2 + 12
    if case.get("scene") == "instanced":
        return 3 * 2 * case["lat"] * (case["lat"] - 1)
    return 56


# About what one ray takes through an 8-wide tree: a node per level (8 boxes of 6 planes, a multiply
# and an add each) and two triangle tests.
def _ray_flops(tris):
    return 96.0 * max(1.0, math.log(max(tris, 8), 8)) + 2 * 60.0


def work(case):
    kind = case["kind"]
    if kind == "batch":
        jobs = _mix(case)
        paths = [j["res"] ** 2 * j["spp"] for j in jobs]
        return {"bytes": sum(36.0 * j["tris"] + 12.0 * j["res"] ** 2 for j in jobs),
                "flops": sum(2 * n * (_ray_flops(j["tris"]) + 200) for n, j in zip(paths, jobs))}
    tris = _tris(case)
    if kind in ("query", "host", "build"):
        n = case["rays"]
        # a ray in, a hit out; the triangles once, as far as there are rays to read them
        return {"bytes": n * (33.0 if case.get("any") else 48.0) + 36.0 * (tris if kind == "build" else min(tris, 2 * n)),
                "flops": n * _ray_flops(tris)}
    paths = case["samples"] if kind != "pt" else case["w"] * case["h"] * case["spp"]
    # a path of two segments at least, each shaded once; bdpt: two subpaths
    seg = 2 * paths * (2 if kind == "bdpt" else 1)
    return {"bytes": 12.0 * case["w"] * case["h"] + 132.0 * min(tris, seg), "flops": seg * (_ray_flops(tris) + 200)}


def exact(case, seed):
    """Closest hits in 64 bits by testing every triangle, where rays x triangles allow it. Which of two
    equally near triangles is hit is no computed number, so `prim` has no value here. Renders are sums
    over random walks that only the renderers' own streams define: no value."""
    kind = case["kind"]
    if kind not in ("query", "host", "build") or case.get("any") or case["scene"] != "soup":
        return None
    if case["tris"] * case["rays"] > 20_000_000_000:
        return None
    tri = torch.from_numpy(_soup(case, seed)).cuda().double().reshape(-1, 3, 3)
    p1, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    rays = _rays(case, seed, _soup(case, seed)).double()
    out = torch.zeros((rays.shape[0], 3), dtype=torch.float64, device="cuda")
    step = max(1, 8_000_000 // tri.shape[0])
    for a in range(0, rays.shape[0], step):
        o, tmin, d, tmax = rays[a:a + step, None, 0:3], rays[a:a + step, None, 3], rays[a:a + step, None, 4:7], rays[a:a + step, None, 7]
        p = torch.linalg.cross(d, e2[None])
        tv = o - p1[None]
        q = torch.linalg.cross(tv, e1[None])
        det = (e1[None] * p).sum(-1)
        inv = 1.0 / det
        u, v, t = (tv * p).sum(-1) * inv, (d * q).sum(-1) * inv, (e2[None] * q).sum(-1) * inv
        ok = (det.abs() >= 1e-8) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= tmin) & (t <= tmax)
        best, k = torch.where(ok, t, torch.inf).min(dim=1)
        hit = torch.isfinite(best)
        got = torch.stack([best, u.gather(1, k[:, None])[:, 0], v.gather(1, k[:, None])[:, 0]], 1)
        out[a:a + step] = torch.where(hit[:, None], got, 0.0)
    return {"t": out[:, 0], "u": out[:, 1], "v": out[:, 2], "prim": None}
