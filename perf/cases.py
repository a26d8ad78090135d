"""The work a user of this framework has it do, as measurable cases.

Every case goes through the package's public entry points
(:class:`pathtracer_gb300.native.Renderer`): whole renders to a host or a
device film, a batch of jobs, ray / occlusion queries and radiance of given
rays, the finishing of a film, and the upload of a scene.  One renderer is
kept for the whole process, as a program keeps it; scenes are resident while
a case's state lives.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from pathtracer_gb300 import native as N
from pathtracer_gb300 import scene as S

OWEN, PERMUTE, STRATIFIED = N.SAMPLER_HALTON_OWEN, N.SAMPLER_HALTON_PERMUTE, N.SAMPLER_STRATIFIED
REF_NEE, NEE_MIS = N.EST_REF_NEE, N.EST_NEE_MIS


def _render(name, scene, subdiv, width, height, spp_x, spp_y, depth, rr, mis, sampler, film):
    return {"name": name, "kind": "render", "scene": scene, "subdiv": subdiv, "width": width, "height": height,
            "spp_x": spp_x, "spp_y": spp_y, "depth": depth, "rr": rr, "mis": mis, "sampler": sampler, "film": film}


def listed():
    return [
        # The smallest call: a thumbnail or the first preview of an editor.
        _render("preview_64", "cornell", 4, 64, 64, 2, 2, 8, -1, False, OWEN, "host"),
        # A whole frame of the plain scene (the benchmark's small configuration).
        _render("cornell_frame", "cornell", 4, 256, 256, 8, 8, 8, -1, False, OWEN, "host"),
        # The benchmark's headline step: 16 samples of every pixel of the
        # 1.3 M triangle glass scene, film kept on the device.
        _render("glass_16spp", "glass", 8, 1024, 1024, 4, 4, 16, 4, False, OWEN, "device"),
        # Progressive viewing: one sample per pixel and call, an odd window
        # size, light and BSDF sampling combined.
        _render("glass_progressive", "glass", 7, 801, 603, 1, 1, 16, 4, True, OWEN, "device"),
        # A frame of many materials in a medium, stratified sampler.
        _render("divergence_hd", "divergence", 5, 1920, 1080, 2, 2, 12, -1, False, STRATIFIED, "host"),
        # Hair: curve primitives and the hair BSDF.
        _render("hair_frame", "hair", 200, 400, 300, 4, 2, 8, 3, True, OWEN, "host"),
        # Many small jobs of three moving scenes with lens and shutter, as a
        # farm of thumbnails or a turntable sends them.
        {"name": "job_batch", "kind": "batch", "subdiv": 4, "jobs": 24, "res_min": 64, "res_max": 256, "spp_min": 4,
         "spp_max": 32},
        # Radiance along given rays (probe baking) in a textured scene, the
        # digit-permuted sampler.
        {"name": "probe_rays", "kind": "probes", "scene": "textured", "subdiv": 3, "n": 98_305, "depth": 6, "mis": False,
         "sampler": PERMUTE},
        # Closest hits of a scan from inside a closed scene (range images,
        # picking, physics).
        {"name": "scan_rays", "kind": "rays", "subdiv": 5, "n": 262_143},
        # Visibility between pairs of points.
        {"name": "visibility", "kind": "visibility", "subdiv": 6, "n": 1_500_007},
        # A frame's last step: blur and tone mapping to bytes.
        {"name": "finish_hd", "kind": "finish", "width": 1920, "height": 1080, "kernel": 5, "sigma": 1.2},
        # A new scene: upload of a large mesh (device builder) up to its first
        # hits, and its release.
        {"name": "scene_upload", "kind": "upload", "subdiv": 7, "n": 4096, "builder": N.BVH_BUILD_DEVICE},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render"] * 6 + ["batch", "probes", "rays", "visibility", "finish", "upload"])
    if kind == "render":
        scene = rng.choice(["cornell", "glass", "divergence", "hair", "textured"])
        subdiv = {"cornell": rng.randint(2, 5), "glass": rng.randint(5, 8), "divergence": rng.randint(3, 5),
                  "hair": rng.randint(50, 400), "textured": rng.randint(2, 4)}[scene]
        paths = _log(rng, 4096, {"glass": 12e6, "cornell": 8e6, "textured": 6e6, "divergence": 4e6, "hair": 1.5e6}[scene])
        sx, sy = rng.randint(1, 6), rng.randint(1, 6)
        pixels = max(256, paths // (sx * sy))
        width = max(8, min(2048, int(math.sqrt(pixels * rng.uniform(0.7, 1.8)))))
        height = max(8, min(2048, pixels // width))
        c = _render("", scene, subdiv, width, height, sx, sy, rng.randint(3, 16 if scene == "glass" else 10),
                    rng.choice([-1, 2, 4]), rng.random() < 0.5, rng.choice([OWEN, OWEN, PERMUTE, STRATIFIED]),
                    rng.choice(["host", "device"]))
        del c["name"]
        return c
    if kind == "batch":
        res = _log(rng, 48, 128)
        return {"kind": "batch", "subdiv": rng.randint(3, 5), "jobs": rng.randint(3, 32), "res_min": res,
                "res_max": 2 * res, "spp_min": rng.randint(1, 4), "spp_max": rng.randint(5, 24)}
    if kind == "probes":
        return {"kind": "probes", "scene": rng.choice(["textured", "cornell", "hair"]), "subdiv": rng.randint(2, 4),
                "n": _log(rng, 1000, 1e6), "depth": rng.randint(3, 8), "mis": rng.random() < 0.5,
                "sampler": rng.choice([OWEN, PERMUTE])}
    if kind in ("rays", "visibility"):
        return {"kind": kind, "subdiv": rng.randint(4, 7), "n": _log(rng, 1000, 2e6)}
    if kind == "finish":
        return {"kind": "finish", "width": _log(rng, 100, 3000), "height": _log(rng, 100, 2000),
                "kernel": rng.choice([3, 5, 7, 9]), "sigma": round(rng.uniform(0.5, 2.5), 2)}
    return {"kind": "upload", "subdiv": rng.randint(5, 8), "n": _log(rng, 500, 20000),
            "builder": rng.choice([N.BVH_BUILD_DEVICE, N.BVH_BUILD_DEVICE, N.BVH_BUILD_HOST])}


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=None)
def _renderer():
    return N.Renderer(0)


class _Resident:
    """Scenes of one state, released with it."""

    def __init__(self):
        self.r, self.ids = _renderer(), []

    def upload(self, scene, builder=N.BVH_BUILD_HOST):
        self.r.set_bvh_builder(builder)
        self.ids.append(self.r.upload(scene))
        return self.ids[-1]

    def __del__(self):
        for sid in self.ids:
            self.r.release(sid)


def _rotation(rng):
    q, r = np.linalg.qr(rng.normal(size=(3, 3)))
    return q * np.sign(np.diag(r)) * np.sign(np.linalg.det(q * np.sign(np.diag(r))))


@functools.lru_cache(maxsize=None)
def _glass_base(subdiv):
    sc, cam = S.rough_glass(subdiv, 8, 4, seed=0)
    return sc, cam


@functools.lru_cache(maxsize=None)
def _ball(subdiv, displace):
    m = S.sphere_mesh(subdiv, (0.0, 0.0, 0.0), 1.0, 0, displace=displace, seed=3)
    return m.positions, m.indices, m.normals


def _turned(mesh, rot):
    """The mesh turned about its origin: another mesh of the same kind."""
    r = rot.astype(np.float32)
    return S.Mesh(mesh.positions @ r.T, mesh.indices, None if mesh.normals is None else mesh.normals @ r.T, mesh.material)


def _scene(kind, subdiv, seed, aspect):
    rng = np.random.default_rng([seed, 11])
    if kind == "cornell":
        sc, cam = S.cornell_icosphere(subdiv)
    elif kind == "glass":
        base, cam = _glass_base(subdiv)
        sc = S.Scene(materials=base.materials, quads=base.quads, objects=base.objects,
                     meshes=[_turned(base.meshes[0], _rotation(rng))])
        sc.env = S.synthetic_hdri(1024, 512, seed=seed % 1000 + 1)
    elif kind == "divergence":
        sc, cam = S.material_divergence(subdiv, seed=seed % 100_000)
    elif kind == "hair":
        sc, cam = S.hair_curves(50 * subdiv if subdiv < 10 else subdiv, seed=seed % 100_000)
    else:
        sc, cam = S.textured_cornell(subdiv, seed=seed % 100_000)
    cam = dict(cam)
    cam["aspect"] = aspect
    cam["position"] = tuple(float(p + rng.uniform(-0.03, 0.03)) for p in cam["position"])
    return sc, cam


def _cave(subdiv, seed):
    """A closed rough cave around four boulders, in a box."""
    rng = np.random.default_rng([seed, 12])
    sc = S.Scene()
    mat = sc.add_material(N.LAMBERTIAN, [0.6, 0.6, 0.6])
    parts = [(subdiv, 4.0, (0.0, 0.0, 0.0))]
    parts += [(subdiv - 1, 0.7, (1.6 * math.cos(a), 0.0, 1.6 * math.sin(a))) for a in (0.0, 1.6, 3.1, 4.7)]
    for k, radius, center in parts:
        pos, idx, nrm = _ball(k, 0.05)
        m = _turned(S.Mesh(pos, idx, nrm, mat), _rotation(rng))
        sc.add_mesh(S.Mesh((m.positions * radius + np.asarray(center)).astype(np.float32), idx, m.normals, mat))
    sc.add_box((-6.0, -6.0, -6.0), (6.0, 6.0, 6.0), mat)
    return sc


def _directions(rng, n):
    d = rng.normal(size=(n, 3))
    return d / np.linalg.norm(d, axis=1, keepdims=True)


def _cave_rays(rng, n):
    """Rays from a few hundred places near the middle of the cave."""
    places = rng.uniform(-0.5, 0.5, size=(max(1, n // 1000), 3))
    o = places[np.sort(rng.integers(0, places.shape[0], n))]
    return np.concatenate([o, _directions(rng, n)], axis=1).astype(np.float32)


def prepare(case, seed):
    kind, rng = case["kind"], np.random.default_rng([seed, 13])
    st = {"case": case, "res": _Resident()}
    if kind == "render":
        sc, cam = _scene(case["scene"], case["subdiv"], seed, case["width"] / case["height"])
        env = N.ENV_ALIAS if case["mis"] else N.ENV_UNIFORM
        st["job"] = N.job_desc(st["res"].upload(sc), cam, case["width"], case["height"], case["spp_x"], case["spp_y"],
                               case["depth"], estimator=NEE_MIS if case["mis"] else REF_NEE, sampler=case["sampler"],
                               rr_start=case["rr"], env_sampling=env, seed=seed & 0x7fffffff,
                               sampler_seed=seed & 0xffff)
    elif kind == "batch":
        scenes = {}
        for name, focus in (("cornell", 2.0), ("rough_glass", 4.2), ("divergence", 11.0)):
            sc, cam = _scene({"rough_glass": "glass"}.get(name, name), case["subdiv"], seed, 1.0)
            S.with_motion(sc, seed=seed % 100_000)
            scenes[name] = (st["res"].upload(sc), cam, focus)
        # the mix of sizes, lenses and shutters is the case's own
        st["jobs"] = S.job_mix(scenes, case["jobs"], 7, res=(case["res_min"], case["res_max"]),
                               spp=(case["spp_min"], case["spp_max"]))
        for k, j in enumerate(st["jobs"]):
            j.seed = (seed + 1000 * k) & 0x7fffffff
    elif kind == "probes":
        sc, cam = _scene(case["scene"], case["subdiv"], seed, 1.0)
        n = case["n"]
        o = np.array([0.5, 0.5, 0.4]) + rng.uniform(-0.2, 0.2, size=(max(1, n // 64), 3))
        if case["scene"] == "hair":
            o = o * 2.0 + np.array([-1.0, 0.5, -1.0])
        o = np.repeat(o, -(-n // o.shape[0]), axis=0)[:n]
        st["rays"] = np.concatenate([o, _directions(rng, n)], axis=1).astype(np.float32)
        st["job"] = N.job_desc(st["res"].upload(sc), cam, 1, 1, 1, 1, case["depth"],
                               estimator=NEE_MIS if case["mis"] else REF_NEE, sampler=case["sampler"],
                               seed=seed & 0x7fffffff, sampler_seed=seed & 0xffff)
    elif kind == "rays":
        st["sid"] = st["res"].upload(_cave(case["subdiv"], seed))
        st["rays"] = _cave_rays(rng, case["n"])
    elif kind == "visibility":
        st["sid"] = st["res"].upload(_cave(case["subdiv"], seed))
        o, p = rng.uniform(-2.2, 2.2, size=(2, case["n"], 3))
        d = p - o
        dist = np.linalg.norm(d, axis=1)
        st["rays"] = np.concatenate([o, d / dist[:, None]], axis=1).astype(np.float32)
        st["tmax"] = (dist - 1e-3).astype(np.float32)
    elif kind == "finish":
        st["film"] = _film(case, seed)
    else:
        st["scene"] = _scene("glass", case["subdiv"], seed, 1.0)[0]
        o = np.array([0.0, 0.0, -4.0]) + rng.uniform(-0.2, 0.2, size=(case["n"], 3))
        d = rng.uniform(-0.8, 0.8, size=(case["n"], 3)) - o
        st["rays"] = np.concatenate([o, d / np.linalg.norm(d, axis=1, keepdims=True)], axis=1).astype(np.float32)
    return st


def _film(case, seed):
    """A rendered frame's values: smooth areas, noise and a few very bright pixels."""
    rng = np.random.default_rng([seed, 14])
    h, w = case["height"], case["width"]
    y, x = np.meshgrid(np.linspace(0, 1, h), np.linspace(0, 1, w), indexing="ij")
    base = 0.4 + 0.3 * np.sin(9 * x + seed % 7)[..., None] * np.cos(7 * y)[..., None] * np.array([1.0, 0.8, 0.6])
    f = base * rng.uniform(0.7, 1.3, size=(h, w, 1))
    f[rng.random((h, w)) < 1e-3] *= 40.0
    return f.astype(np.float32)


# -------------------------------------------------------------------- runs
def run(state):
    c, r = state["case"], state["res"].r
    kind = c["kind"]
    if kind == "render":
        if c["film"] == "host":
            return r.render(state["job"])
        film = torch.zeros((c["height"], c["width"], 3), device="cuda")
        torch.cuda.current_stream().synchronize()  # the renderer has a stream of its own
        r.render_device(state["job"], film.data_ptr(), sync=True)
        return film
    if kind == "batch":
        return r.render_batch(state["jobs"])
    if kind == "probes":
        return r.ray_color(state["job"], state["rays"])
    if kind == "rays":
        t, prim, uv = r.trace_closest(state["sid"], state["rays"], 1e-4, 1e5)
        return {"t": t, "prim": prim, "uv": uv}
    if kind == "visibility":
        return r.trace_any(state["sid"], state["rays"], state["tmax"], 1e-3)
    if kind == "finish":
        blurred = r.gaussian_blur(state["film"], c["kernel"], c["sigma"])
        return {"blurred": blurred, "rgb8": r.tonemap(blurred, 2.2)}
    r.set_bvh_builder(c["builder"])
    sid = r.upload(state["scene"])
    t, prim, uv = r.trace_closest(sid, state["rays"], 1e-4, 1e5)
    info = r.scene_info(sid)
    r.release(sid)
    return {"t": t, "prim": prim, "uv": uv, "info": info}


# -------------------------------------------------------------------- work
def _triangles(scene, subdiv):
    return {"cornell": 20 * 4 ** subdiv, "glass": 20 * 4 ** subdiv, "divergence": 64 * 20 * 4 ** subdiv,
            "textured": 20 * 4 ** subdiv, "hair": 8 * subdiv}[scene]


def _ray_flops(triangles):
    """A walk down a tree of four children per node and one leaf's tests."""
    return (math.log(max(4, triangles), 4) + 1) * 4 * 12 + 4 * 45


# closest and shadow rays, and shaded vertices, of one path
_PER_PATH = {"cornell": (16.0, 4.0), "glass": (5.0, 1.4), "divergence": (34.0, 9.0), "textured": (16.0, 4.0),
             "hair": (6.0, 1.5)}


def _path_flops(scene, subdiv, depth):
    rays, vertices = _PER_PATH[scene]
    part = min(1.0, depth / 8.0)
    return part * (rays * _ray_flops(_triangles(scene, subdiv)) + vertices * 1500)


def work(case):
    kind = case["kind"]
    if kind == "render":
        pixels = case["width"] * case["height"]
        paths = pixels * case["spp_x"] * case["spp_y"]
        return {"bytes": 12 * pixels + 100 * _triangles(case["scene"], case["subdiv"]),
                "flops": paths * _path_flops(case["scene"], case["subdiv"], case["depth"])}
    if kind == "batch":
        pixels = case["jobs"] * ((case["res_min"] + case["res_max"]) / 2) ** 2
        paths = pixels * (case["spp_min"] + case["spp_max"]) / 2
        k = [("cornell", 8), ("glass", 16), ("divergence", 12)]
        return {"bytes": 12 * pixels + 100 * sum(_triangles(s, case["subdiv"]) for s, _ in k),
                "flops": paths * sum(_path_flops(s, case["subdiv"], d) for s, d in k) / 3}
    if kind == "probes":
        return {"bytes": 36 * case["n"] + 100 * _triangles(case["scene"], case["subdiv"]),
                "flops": case["n"] * _path_flops(case["scene"], case["subdiv"], case["depth"])}
    if kind in ("rays", "visibility"):
        tris = 20 * 4 ** case["subdiv"] * 2
        return {"bytes": (40 if kind == "rays" else 29) * case["n"] + 60 * tris, "flops": case["n"] * _ray_flops(tris)}
    if kind == "finish":
        n = 3 * case["width"] * case["height"]
        return {"bytes": n * (4 + 4 + 1), "flops": n * (2 * case["kernel"] ** 2 + 10)}
    tris = 20 * 4 ** case["subdiv"]
    return {"bytes": tris * (12 + 12 + 12 + 48 + 64 + 30) + case["n"] * 40,
            "flops": tris * 20 * math.log2(tris) + case["n"] * _ray_flops(tris)}


# ------------------------------------------------------------------- exact
def exact(case, seed):
    """Renders are random walks that no plain formula gives: None."""
    if case["kind"] == "finish":
        return {"blurred": _blur64(case, seed), "rgb8": None}
    if case["kind"] == "rays" and case["n"] * 40 * 4.0 ** case["subdiv"] <= 3e10:
        return {"t": _closest64(case, seed), "prim": None, "uv": None}
    return None


def _blur64(case, seed):
    k, sigma = case["kernel"], case["sigma"]
    x = torch.arange(-(k // 2), k // 2 + 1, dtype=torch.float64)
    w = torch.exp(-(x[:, None] ** 2 + x[None, :] ** 2) / (2 * sigma * sigma))
    w = w / w.sum()
    f = torch.from_numpy(_film(case, seed)).double()
    h, wd = f.shape[:2]
    out = torch.zeros_like(f)
    rows, cols = torch.arange(h), torch.arange(wd)
    for i in range(k):
        fr = f[(rows + i - k // 2).clamp(0, h - 1)]
        for j in range(k):
            out += w[i, j] * fr[:, (cols + j - k // 2).clamp(0, wd - 1)]
    return out.numpy()


def _closest64(case, seed):
    """Every ray against every triangle (the cave is closed: each ray hits)."""
    sc = _cave(case["subdiv"], seed)
    rays = torch.from_numpy(_cave_rays(np.random.default_rng([seed, 13]), case["n"])).cuda().double()
    tri = torch.cat([torch.from_numpy(m.positions[m.indices]) for m in sc.meshes]).cuda().double()
    p0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    normal, best = torch.cross(e1, e2, dim=1), []
    # with M = d x o, the products of the ray and the edges are matrix products
    a1, a2 = torch.cross(p0, e1, dim=1), torch.cross(p0, e2, dim=1)
    for c in torch.split(rays, 1024):
        o, d = c[:, :3], c[:, 3:]
        m = torch.cross(d, o, dim=1)
        det = -(d @ normal.T)
        t = ((o @ normal.T) - (normal * p0).sum(1)) / det
        u = ((d @ a2.T) - (m @ e2.T)) / det       # (o - p0) . (d x e2)
        v = ((m @ e1.T) - (d @ a1.T)) / det       # d . ((o - p0) x e1)
        ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= 1e-4)
        best.append(torch.where(ok, t, torch.full_like(t, torch.finfo(torch.float32).max)).amin(dim=1))
    return torch.cat(best).cpu().numpy()
