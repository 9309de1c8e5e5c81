"""What a user of the light-probe baker has it do, as measurable passes through its public entry points.

A program keeps one context, its direction sets and its scenes, and calls: probe bakes (a preview, a level, a large volume,
the reference baker's own full-resolution run, a smooth mesh), a batch of uneven volumes, a service under a burst of
requests, skybox projections (one map, a batch, a panorama), the evaluation of a baked grid at shading points, and the
loading of a new scene up to its first preview.  Scenes are seeded rooms of boxes (the repository's benchmark geometry)
and tessellated terrains with spheres (generic smooth meshes)."""
import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path("vulkan-light-bakery_gb300").resolve())
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import vlb  # noqa: E402

PRECISIONS = {"fp32": vlb.PREC_FP32, "fused": vlb.PREC_FUSED, "mixed": vlb.PREC_MIXED, "bf16": vlb.PREC_BF16}
LAYOUTS = {"cube": vlb.SKY_CUBEMAP, "panorama": vlb.SKY_PANORAMA, "envmap": vlb.SKY_ENVMAP}
SUN_INTENSITY = 5.0


def listed():
    return [
        # an editor's preview: a handful of probes, host arrays in and out, waited for: latency and launches
        {"name": "bake_preview", "kind": "bake", "scene": "boxes", "size": 64, "nx": 4, "ny": 4, "nz": 4, "dirs": 64,
         "eq_w": 0, "eq_h": 0, "lmax": 2, "precision": "fp32", "phong": False, "accumulate": False, "sky": 32, "host": True},
        # an ordinary level: 16^3 probes of a small room, results stay on the GPU
        {"name": "bake_level", "kind": "bake", "scene": "boxes", "size": 64, "nx": 16, "ny": 16, "nz": 16, "dirs": 256,
         "eq_w": 0, "eq_h": 0, "lmax": 2, "precision": "fp32", "phong": False, "accumulate": False, "sky": 128, "host": False},
        # a smooth mesh with a ragged grid and direction count, the tile-free path, 16 coefficients
        {"name": "bake_terrain", "kind": "bake", "scene": "terrain", "size": 250, "nx": 21, "ny": 13, "nz": 17, "dirs": 515,
         "eq_w": 0, "eq_h": 0, "lmax": 3, "precision": "fused", "phong": False, "accumulate": False, "sky": 64, "host": True},
        # the benchmark's large volume: 64^3 probes x 1024 directions in 4096 boxes
        {"name": "bake_large", "kind": "bake", "scene": "boxes", "size": 4096, "nx": 64, "ny": 64, "nz": 64, "dirs": 1024,
         "eq_w": 0, "eq_h": 0, "lmax": 2, "precision": "fp32", "phong": False, "accumulate": False, "sky": 128, "host": False},
        # the reference baker's own run: 7^3 probes, its 3141 x 1000 sample set, its shading and running sums
        {"name": "bake_reference", "kind": "bake", "scene": "boxes", "size": 64, "nx": 7, "ny": 7, "nz": 7, "dirs": 0,
         "eq_w": 3141, "eq_h": 1000, "lmax": 3, "precision": "fp32", "phong": True, "accumulate": True, "sky": 0, "host": True},
        # a build farm's batch: many uneven volumes at once
        {"name": "batch_volumes", "kind": "batch", "jobs": 60, "shapes": 7, "max_boxes": 16384, "max_probes": 8192,
         "lmax": 2, "precision": "fp32"},
        # the service under a burst of requests, with relights of kept bakes
        {"name": "service_burst", "kind": "service", "bakes": 24, "relights": 8, "shapes": 3, "max_boxes": 4096,
         "max_probes": 4096, "lmax": 2, "precision": "mixed"},
        # one skybox: the smallest call
        {"name": "sky_single", "kind": "sky", "layout": "cube", "w": 128, "h": 128, "count": 1, "lmax": 3, "rgba8": False,
         "swap": False, "host": False},
        # every reflection capture of a world
        {"name": "sky_batch", "kind": "sky", "layout": "cube", "w": 128, "h": 128, "count": 1024, "lmax": 2, "rgba8": False,
         "swap": False, "host": False},
        # the reference's own skybox form: an 8-bit panorama with its swapped channels
        {"name": "sky_panorama", "kind": "sky", "layout": "panorama", "w": 2048, "h": 1024, "count": 1, "lmax": 3,
         "rgba8": True, "swap": True, "host": False},
        # the consumer side: a frame's shading points against a baked grid
        {"name": "probe_eval", "kind": "eval", "scene": "boxes", "size": 341, "nx": 7, "ny": 7, "nz": 7, "points": 1000000,
         "lmax": 3},
        # a new scene, up to its first preview
        {"name": "scene_load", "kind": "load", "scene": "terrain", "size": 310, "lmax": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bake", "bake", "bake", "batch", "service", "sky", "sky", "eval", "load"])
    scene = rng.choice(["boxes", "boxes", "terrain"])
    size = _log(rng, 16, 4096) if scene == "boxes" else _log(rng, 12, 300)
    lmax = rng.choice([2, 3])
    if kind == "bake":
        equirect = rng.random() < 0.2
        nx, ny, nz = (rng.randint(1, 6) if equirect else _log(rng, 1, 40) for _ in range(3))
        w = _log(rng, 64, 1024) if equirect else 0
        phong = rng.random() < 0.25
        # the carry-over sums belong to the reference's own form
        return {"kind": "bake", "scene": scene, "size": size, "nx": nx, "ny": ny, "nz": nz,
                "dirs": 0 if equirect else _log(rng, 64, 1024), "eq_w": w, "eq_h": w // 2, "lmax": lmax,
                "precision": rng.choice(["fp32", "fp32", "fused", "mixed", "bf16"]), "phong": phong,
                "accumulate": phong and rng.random() < 0.5, "sky": rng.choice([0, 32, 100, 128]),
                "host": rng.random() < 0.5}
    if kind == "batch":
        return {"kind": "batch", "jobs": _log(rng, 2, 60), "shapes": rng.randint(0, 1 << 20),
                "max_boxes": _log(rng, 64, 16384), "max_probes": _log(rng, 256, 8192), "lmax": lmax,
                "precision": rng.choice(["fp32", "fused", "mixed"])}
    if kind == "service":
        return {"kind": "service", "bakes": _log(rng, 2, 24), "relights": rng.randint(0, 8), "shapes": rng.randint(0, 1 << 20),
                "max_boxes": _log(rng, 64, 4096), "max_probes": _log(rng, 64, 4096), "lmax": lmax,
                "precision": rng.choice(["fp32", "fused", "mixed"])}
    if kind == "sky":
        layout = rng.choice(["cube", "cube", "panorama", "envmap"])
        w = _log(rng, 16, 512) if layout == "cube" else _log(rng, 64, 4096)
        h = w if layout == "cube" else _log(rng, max(32, w // 4), w)
        texels = 6 * w * w if layout == "cube" else w * h
        return {"kind": "sky", "layout": layout, "w": w, "h": h, "count": _log(rng, 1, max(1, min(1024, 100000000 // texels))),
                "lmax": lmax, "rgba8": rng.random() < 0.5, "swap": rng.random() < 0.3, "host": rng.random() < 0.2}
    if kind == "eval":
        return {"kind": "eval", "scene": scene, "size": size, "nx": rng.randint(1, 20), "ny": rng.randint(1, 20),
                "nz": rng.randint(1, 20), "points": _log(rng, 1000, 1000000), "lmax": lmax}
    return {"kind": "load", "scene": scene, "size": size, "lmax": lmax}


# ---- inputs ---------------------------------------------------------------------------------
def _boxes(rng, n):
    """A unit room open at +Y and n boxes in it: positions, indices, albedo (the benchmark's distributions)."""
    room = np.array([[0, 4, 5], [0, 5, 1], [0, 2, 6], [0, 6, 4], [1, 5, 7], [1, 7, 3], [0, 1, 3], [0, 3, 2], [4, 6, 7],
                     [4, 7, 5]])
    box = np.array([[0, 4, 5], [0, 5, 1], [2, 3, 7], [2, 7, 6], [0, 2, 6], [0, 6, 4], [1, 5, 7], [1, 7, 3], [0, 1, 3],
                    [0, 3, 2], [4, 6, 7], [4, 7, 5]])
    bits = np.array([[c & 1, c >> 1 & 1, c >> 2] for c in range(8)], np.float32)
    centre, edge = rng.uniform(0.1, 0.9, (n, 3)), rng.uniform(0.05, 0.2, (n, 3))
    corners = (centre[:, None] + (bits[None] - 0.5) * edge[:, None]).astype(np.float32)
    pos = np.concatenate([bits, corners.reshape(-1, 3)])
    idx = np.concatenate([room, (8 + 8 * np.arange(n)[:, None, None] + box[None]).reshape(-1, 3)])
    alb = np.concatenate([np.full((10, 3), 0.5), np.repeat(rng.uniform(0.2, 0.8, (n, 3)), 12, axis=0)])
    return pos, idx.astype(np.uint32), alb.astype(np.float32)


def _surface(p):
    """A (rows, cols) grid of points as triangles."""
    r, c = p.shape[:2]
    i = (np.arange(r - 1)[:, None] * c + np.arange(c - 1)[None]).reshape(-1, 1)
    return p.reshape(-1, 3), np.concatenate([i + [0, c, c + 1], i + [0, c + 1, 1]], axis=1).reshape(-1, 3)


def _terrain(rng, m):
    """An m x m quad height field over the unit square under six spheres, smooth normals varying everywhere."""
    g = np.linspace(0, 1, m + 1)
    x, z = np.meshgrid(g, g)
    y = 0.1 + 0.002 * rng.random(x.shape)
    for _ in range(6):
        f = rng.uniform(2, 14, 2)
        y = y + rng.uniform(0.005, 0.04) * np.sin(f[0] * x + f[1] * z + rng.uniform(0, 6.28))
    parts = [_surface(np.stack([x, y, z], -1))]
    k = max(8, m // 6)
    for _ in range(6):
        t, f = np.meshgrid(np.linspace(0.02, math.pi - 0.02, k), np.linspace(0, 2 * math.pi, 2 * k), indexing="ij")
        s = np.stack([np.sin(t) * np.cos(f), np.cos(t), np.sin(t) * np.sin(f)], -1)
        parts.append(_surface(s * rng.uniform(0.05, 0.12) + [rng.uniform(0.2, 0.8), rng.uniform(0.3, 0.7), rng.uniform(0.2, 0.8)]))
    pos, idx, at = [], [], 0
    for p, i in parts:
        pos.append(p)
        idx.append(i + at)
        at += len(p)
    idx = np.concatenate(idx)
    return np.concatenate(pos).astype(np.float32), idx.astype(np.uint32), rng.uniform(0.2, 0.8, (len(idx), 3)).astype(np.float32)


def _scene(rng, kind, size):
    return _boxes(rng, size) if kind == "boxes" else _terrain(rng, size)


def _sun(rng):
    d = rng.normal(size=3)
    d[1] = abs(d[1]) + 0.3
    return (d / np.linalg.norm(d)).astype(np.float32)


def _cube_dirs(n):
    """Unit directions of a cubemap's texels, (6, n, n, 3), FP64, and the faces' texel edges."""
    c = (torch.arange(n, dtype=torch.float64, device="cuda") + 0.5) * (2.0 / n) - 1.0
    v, u = torch.meshgrid(c, c, indexing="ij")
    one = torch.ones_like(u)
    d = torch.stack([torch.stack(f, -1) for f in ((one, -v, -u), (-one, -v, u), (u, one, v), (u, -one, -v), (u, -v, one),
                                                  (-u, -v, -one))])
    return d / d.norm(dim=-1, keepdim=True)


def _lobes(rng, d):
    """A sky: an ambient term and three sharp coloured lobes, at directions d (..., 3)."""
    out = torch.full_like(d, 0.3)
    for _ in range(3):
        mu = rng.normal(size=3)
        mu = torch.tensor(mu / np.linalg.norm(mu), dtype=d.dtype, device=d.device)
        col = torch.tensor(rng.uniform(1, 50, 3), dtype=d.dtype, device=d.device)
        out = out + col * torch.exp(rng.uniform(20, 200) * ((d * mu).sum(-1, keepdim=True) - 1.0))
    return out


def _sky_map(rng, n):
    return _lobes(rng, _cube_dirs(n).float()).contiguous() if n else None


def _grid(pos, nx, ny, nz, inset=0.0):
    """nx x ny x nz probes over the scene's bounds with the origin, as the baker places them."""
    lo, hi = np.minimum(pos.min(0), 0).astype(np.float64), np.maximum(pos.max(0), 0).astype(np.float64)
    ax = [np.linspace(lo[a] + inset, hi[a] - inset, n) if n > 1 else [(lo[a] + hi[a]) / 2] for a, n in enumerate((nx, ny, nz))]
    return np.stack(np.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3).astype(np.float32)


def _bake_inputs(case, seed):
    rng = np.random.default_rng([seed, 1])
    mesh = _scene(rng, case["scene"], case["size"])
    return {"mesh": mesh, "probes": _grid(mesh[0], case["nx"], case["ny"], case["nz"]), "sun": _sun(rng),
            "sky": _sky_map(rng, case["sky"])}


def _volumes(case, seed, sizes):
    """Uneven volumes: the shapes go by the case, the contents by the seed; a few scenes are shared."""
    shape, rng = np.random.default_rng([case["shapes"], 2]), np.random.default_rng([seed, 2])
    meshes = [_boxes(rng, int(np.exp(shape.uniform(np.log(16), np.log(case["max_boxes"]))))) for _ in range(min(6, sizes))]
    out = []
    for i in range(sizes):
        mesh = i % len(meshes)
        lo, hi = meshes[mesh][0].min(0), meshes[mesh][0].max(0)
        n = int(np.exp(shape.uniform(np.log(16), np.log(case["max_probes"]))))
        out.append({"mesh": mesh, "dirs": int(shape.choice([64, 256, 1024])), "sun": _sun(rng),
                    "probes": (lo + rng.random((n, 3)) * (hi - lo)).astype(np.float32)})
    return meshes, _sky_map(rng, 64), out


def _sky_inputs(case, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    faces = 6 if case["layout"] == "cube" else 1
    shape = (case["count"], faces, case["h"], case["w"])
    if case["rgba8"]:
        return torch.randint(0, 256, shape + (4,), generator=gen, device="cuda", dtype=torch.uint8)
    # log-normal texels: a high-dynamic-range image
    return torch.exp(torch.randn(shape + (3,), generator=gen, device="cuda"))


def _eval_inputs(case, seed):
    rng = np.random.default_rng([seed, 3])
    pos, idx, alb = _scene(rng, case["scene"], case["size"])
    # the grid stands just inside the scene's bounds: no probe in the plane of a wall
    lo, hi = pos.min(0), pos.max(0)
    lo, hi = lo + 0.002 * (hi - lo), hi - 0.002 * (hi - lo)
    counts = np.array([case["nx"], case["ny"], case["nz"]])
    step = ((hi - lo) / np.maximum(counts - 1, 1)).astype(np.float32)
    coeffs = rng.normal(size=(int(counts.prod()), (case["lmax"] + 1) ** 2, 3)).astype(np.float32)
    # shading points on the surfaces, as a renderer's primary hits are
    t = rng.integers(0, len(idx), case["points"])
    v = pos[idx[t]].astype(np.float64)
    a, b = rng.random((2, case["points"], 1))
    a, b = np.where(a + b > 1, 1 - a, a), np.where(a + b > 1, 1 - b, b)
    x = v[:, 0] + a * (v[:, 1] - v[:, 0]) + b * (v[:, 2] - v[:, 0])
    n = np.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
    return {"mesh": (pos, idx, alb), "origin": lo.astype(np.float32), "step": step, "counts": counts, "coeffs": coeffs,
            "points": x.astype(np.float32), "normals": (n / np.linalg.norm(n, axis=1, keepdims=True)).astype(np.float32)}


# ---- a program's own objects ------------------------------------------------------------------
_KEPT = {}


def _ctx():
    if "ctx" not in _KEPT:
        _KEPT["ctx"] = vlb.Context(0)
    return _KEPT["ctx"]


def _dirs(n, w=0, h=0):
    """Direction sets depend on their size alone: a program makes each once."""
    if (n, w, h) not in _KEPT:
        _KEPT[n, w, h] = _ctx().fibonacci(n) if n else _ctx().equirect(w, h)
    return _KEPT[n, w, h]


def _params(case, dirs, sun, sky):
    flags = vlb.BAKE_REF_ACCUMULATE if case.get("accumulate") else 0
    shading = vlb.SHADE_REF_PHONG if case.get("phong") else vlb.SHADE_LAMBERT_SUN
    return vlb.bake_params(dirs, case["lmax"], PRECISIONS[case.get("precision", "fp32")], sun, SUN_INTENSITY, sky,
                           shading=shading, flags=flags)


def prepare(case, seed):
    ctx, K = _ctx(), (case["lmax"] + 1) ** 2
    if case["kind"] == "bake":
        x = _bake_inputs(case, seed)
        sky = None if x["sky"] is None else ctx.sky(x["sky"], case["sky"])
        s = {"case": case, "scene": ctx.scene(*x["mesh"]), "probes": x["probes"],
             "params": _params(case, _dirs(case["dirs"], case["eq_w"], case["eq_h"]), x["sun"], sky)}
        if not case["host"]:
            s["probes"] = torch.from_numpy(x["probes"]).cuda()
            s["out"] = torch.empty((len(x["probes"]), K, 3), device="cuda")
    elif case["kind"] in ("batch", "service"):
        meshes, sky, volumes = _volumes(case, seed, case["jobs" if case["kind"] == "batch" else "bakes"])
        scenes, sky = [ctx.scene(*m) for m in meshes], ctx.sky(sky, 64)
        params = [_params(case, _dirs(v["dirs"]), v["sun"], sky) for v in volumes]
        s = {"case": case, "params": params}
        if case["kind"] == "batch":
            s["jobs"] = [(scenes[v["mesh"]], torch.from_numpy(v["probes"]).cuda(),
                          torch.empty((len(v["probes"]), K, 3), device="cuda"), p) for v, p in zip(volumes, params)]
        else:
            s["service"] = vlb.Service(ctx, lmax=case["lmax"], precision=PRECISIONS[case["precision"]])
            s["requests"] = [(scenes[v["mesh"]], v["probes"], p) for v, p in zip(volumes, params)]
            rng = np.random.default_rng([seed, 4])
            s["relights"] = [(i % len(volumes), _params(case, _dirs(volumes[i % len(volumes)]["dirs"]), _sun(rng), sky))
                             for i in range(case["relights"])]
    elif case["kind"] == "sky":
        t = _sky_inputs(case, seed)
        s = {"case": case, "texels": t.cpu().numpy() if case["host"] else t}
        if not case["host"]:
            s["out"] = torch.empty((case["count"], K, 3), device="cuda")
    elif case["kind"] == "eval":
        x = _eval_inputs(case, seed)
        s = {"case": case, "scene": ctx.scene(*x["mesh"]), "origin": x["origin"], "step": x["step"], "counts": x["counts"]}
        s |= {k: torch.from_numpy(x[k]).cuda() for k in ("coeffs", "points", "normals")}
    else:
        rng = np.random.default_rng([seed, 5])
        mesh = _scene(rng, case["scene"], case["size"])
        s = {"case": case, "mesh": mesh, "probes": _grid(mesh[0], 4, 4, 4, 0.05),
             "params": _params(case, _dirs(64), _sun(rng), None)}
    torch.cuda.synchronize()
    return s


def run(s):
    ctx, case = _ctx(), s["case"]
    if case["kind"] == "bake":
        if case["host"]:
            return ctx.bake(s["scene"], s["probes"], s["params"])
        ctx.bake_async(s["scene"], s["probes"], s["params"], s["out"])
        return s["out"]
    if case["kind"] == "batch":
        return ctx.bake_batch(s["jobs"], s["params"][0])
    if case["kind"] == "service":
        svc, kept = s["service"], {i for i, _ in s["relights"]}
        tickets = [svc.submit(scene, probes, p, keep_hits=i in kept) for i, (scene, probes, p) in enumerate(s["requests"])]
        again = [svc.submit(None, None, p, relight_of=tickets[i]) for i, p in s["relights"]]
        out = [svc.wait(t)[0] for t in tickets + again]
        for i in kept:
            svc.release(tickets[i])
        return out
    if case["kind"] == "sky":
        flags = vlb.SKY_REF_BGRA_SWAP if case["swap"] else 0
        return ctx.skybox_sh(s["texels"], LAYOUTS[case["layout"]], case["w"], case["h"], case["lmax"],
                             vlb.TEXEL_RGBA8 if case["rgba8"] else vlb.TEXEL_RGB32F, flags, case["count"], s.get("out"))
    if case["kind"] == "eval":
        return list(ctx.probe_eval(s["scene"], s["coeffs"], case["lmax"], s["origin"], s["step"], s["counts"], s["points"],
                                   s["normals"]))
    scene = ctx.scene(*s["mesh"])
    out = [scene.bounds(), ctx.bake(scene, s["probes"], s["params"])]
    scene.close()
    return out


# ---- what a pass cannot do without -----------------------------------------------------------
def _triangles(scene, size):
    if scene == "boxes":
        return 10 + 12 * size
    k = max(8, size // 6)
    return 2 * size * size + 12 * (k - 1) * (2 * k - 1)


def _bake_work(tris, probes, dirs, K, sky):
    # a ray: its hit's triangle test and shading (about 60 operations), its projection
    return {"bytes": 64.0 * tris + 12 * probes + 12 * K * probes + 80 * dirs + 72 * sky * sky,
            "flops": float(probes) * dirs * (60 + 6 * K)}


def work(case):
    K = (case["lmax"] + 1) ** 2
    if case["kind"] == "bake":
        return _bake_work(_triangles(case["scene"], case["size"]), case["nx"] * case["ny"] * case["nz"],
                          case["dirs"] or case["eq_w"] * case["eq_h"], K, case["sky"])
    if case["kind"] in ("batch", "service"):
        n = case["jobs" if case["kind"] == "batch" else "bakes"]
        shape = np.random.default_rng([case["shapes"], 2])
        tris = sum(10 + 12 * int(np.exp(shape.uniform(np.log(16), np.log(case["max_boxes"])))) for _ in range(min(6, n)))
        w = {"bytes": 64.0 * tris, "flops": 0.0}
        for _ in range(n):
            p = int(np.exp(shape.uniform(np.log(16), np.log(case["max_probes"]))))
            b = _bake_work(0, p, int(shape.choice([64, 256, 1024])), K, 0)
            w = {k: w[k] + b[k] for k in w}
        return w
    if case["kind"] == "sky":
        texels = case["count"] * case["w"] * case["h"] * (6 if case["layout"] == "cube" else 1)
        return {"bytes": texels * (4.0 if case["rgba8"] else 12.0) + case["count"] * K * 12, "flops": texels * 6.0 * K}
    if case["kind"] == "eval":
        # per point: position, normal, colour, mask; eight corners' rays and sums
        return {"bytes": 64.0 * _triangles(case["scene"], case["size"]) + 37.0 * case["points"]
                + 12.0 * K * case["nx"] * case["ny"] * case["nz"], "flops": case["points"] * 8.0 * (60 + 6 * K)}
    # the geometry in; nodes, triangles and colours out; the preview
    tris = _triangles(case["scene"], case["size"])
    w = _bake_work(tris, 64, 64, K, 0)
    return {"bytes": w["bytes"] + tris * (30.0 + 128), "flops": w["flops"] + 50.0 * tris}


# ---- the same in 64 bits ------------------------------------------------------------------------
_TESTS = 60e9  # ray-triangle tests that fit the time of one answer


def _basis(d, lmax):
    x, y, z = d.unbind(-1)
    b = [0.282095 + 0 * x, -0.488603 * y, 0.488603 * z, -0.488603 * x, 1.092548 * x * y, -1.092548 * y * z,
         0.315392 * (2 * z * z - x * x - y * y), -1.092548 * x * z, 0.546274 * (x * x - y * y)]
    if lmax == 3:
        b += [-0.590044 * y * (3 * x * x - y * y), 2.890611 * x * y * z, -0.457046 * y * (4 * z * z - x * x - y * y),
              0.373176 * z * (2 * z * z - 3 * x * x - 3 * y * y), -0.457046 * x * (4 * z * z - x * x - y * y),
              1.445306 * z * (x * x - y * y), -0.590044 * x * (x * x - 3 * y * y)]
    return torch.stack(b, -1)


def _fibonacci(n):
    i = np.arange(n, dtype=np.float64)
    z = 1.0 - (2.0 * i + 1.0) / n
    r, f = np.sqrt(np.maximum(0.0, 1.0 - z * z)), i * 0.6180339887498949
    phi = 6.283185307179586 * (f - np.floor(f))
    d = torch.from_numpy(np.stack([r * np.cos(phi), r * np.sin(phi), z], -1).astype(np.float32)).double().cuda()
    return d, d, torch.full((n,), 4 * math.pi / n, dtype=torch.float64, device="cuda")


def _equirect(w, h):
    pi = 3.1415926538
    th, phi = np.meshgrid(pi * (np.arange(h) + 0.5) / h, 2 * pi * (np.arange(w) + 0.5) / w, indexing="ij")
    v = np.stack([np.sin(th) * np.cos(phi), np.sin(th) * np.sin(phi), np.cos(th)], -1).reshape(-1, 3)
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    wt = (2 * pi / w) * (pi / h) * np.sin(th).reshape(-1)
    return (torch.from_numpy(v[:, [0, 2, 1]].astype(np.float32)).double().cuda(), torch.from_numpy(v).cuda(),
            torch.from_numpy(wt).cuda())


class _Rays:
    """Every ray against every triangle."""

    def __init__(self, mesh):
        pos, idx, alb = mesh
        p = torch.from_numpy(pos).double().cuda()[torch.from_numpy(idx.astype(np.int64)).cuda()]
        self.v0, self.e1, self.e2 = p[:, 0], p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
        self.albedo = torch.from_numpy(alb).double().cuda()
        n = torch.linalg.cross(self.e1, self.e2)
        self.normal = n / n.norm(dim=1, keepdim=True)

    def nearest(self, o, d, tmin, tmax):
        """(distance or inf, triangle) of each ray's nearest hit in (tmin, tmax); o, d (R, 3)."""
        T, at, best = len(self.v0), [], []
        step = max(1, (1 << 24) // T)
        for r in range(0, len(o), step):
            oo, dd = o[r:r + step, None], d[r:r + step, None]
            p = [dd[..., 1] * self.e2[:, 2] - dd[..., 2] * self.e2[:, 1], dd[..., 2] * self.e2[:, 0] - dd[..., 0] * self.e2[:, 2],
                 dd[..., 0] * self.e2[:, 1] - dd[..., 1] * self.e2[:, 0]]
            det = p[0] * self.e1[:, 0] + p[1] * self.e1[:, 1] + p[2] * self.e1[:, 2]
            s = [oo[..., a] - self.v0[:, a] for a in range(3)]
            u = (s[0] * p[0] + s[1] * p[1] + s[2] * p[2]) / det
            del p
            q = [s[1] * self.e1[:, 2] - s[2] * self.e1[:, 1], s[2] * self.e1[:, 0] - s[0] * self.e1[:, 2],
                 s[0] * self.e1[:, 1] - s[1] * self.e1[:, 0]]
            del s
            v = (dd[..., 0] * q[0] + dd[..., 1] * q[1] + dd[..., 2] * q[2]) / det
            t = (self.e2[:, 0] * q[0] + self.e2[:, 1] * q[1] + self.e2[:, 2] * q[2]) / det
            far = tmax if not isinstance(tmax, torch.Tensor) else tmax[r:r + step, None]
            ok = (det != 0) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t > tmin) & (t < far)
            t, k = torch.where(ok, t, math.inf).min(dim=1)
            at.append(t)
            best.append(k)
        return torch.cat(at), torch.cat(best)


def _cube_lookup(sky, d):
    n = sky.shape[1]
    a = d.abs()
    x, y, z = d.unbind(-1)
    fx, fy = (a[:, 0] >= a[:, 1]) & (a[:, 0] >= a[:, 2]), a[:, 1] >= a[:, 2]
    f = torch.where(fx, torch.where(x >= 0, 0, 1), torch.where(fy, torch.where(y >= 0, 2, 3), torch.where(z >= 0, 4, 5)))
    table = [(-z, -y, a[:, 0]), (z, -y, a[:, 0]), (x, z, a[:, 1]), (x, -z, a[:, 1]), (x, -y, a[:, 2]), (-x, -y, a[:, 2])]
    s, t, m = (torch.stack([row[c] for row in table], -1).gather(1, f[:, None])[:, 0] for c in range(3))
    i, j = (((q / m + 1) * 0.5 * n).floor().long().clamp(0, n - 1) for q in (s, t))
    return sky.double()[f, j, i]


def _exact_bake(rays, probes, dirs, basis_dirs, w, lmax, sun, sky):
    o = torch.from_numpy(probes).double().cuda()
    P, S = len(o), len(dirs)
    sun = torch.from_numpy(sun.astype(np.float64)).cuda()
    sun = sun / sun.norm()
    B = _basis(basis_dirs, lmax) * w[:, None]
    out = torch.zeros((P, B.shape[1], 3), dtype=torch.float64, device="cuda")
    step = max(1, (1 << 21) // S)
    for p in range(0, P, step):
        oo = o[p:p + step].repeat_interleave(S, 0)
        dd = dirs.repeat(len(oo) // S, 1)
        t, k = rays.nearest(oo, dd, 0.001, 10000.0)
        hit = torch.isfinite(t)
        L = torch.zeros_like(oo)
        if sky is not None:
            L[~hit] = _cube_lookup(sky, dd[~hit])
        n = rays.normal[k]
        n = torch.where(((n * dd).sum(1, keepdim=True) > 0), -n, n)
        ndl = (n * sun).sum(1)
        lit = (hit & (ndl > 0)).nonzero()[:, 0]
        ts, _ = rays.nearest(oo[lit] + t[lit, None] * dd[lit] + 0.005 * n[lit], sun.expand(len(lit), 3), 0.0, 10000.0)
        lit = lit[~torch.isfinite(ts)]
        L[lit] = rays.albedo[k[lit]] * (SUN_INTENSITY / math.pi * ndl[lit])[:, None]
        out[p:p + step] = torch.einsum("psc,sk->pkc", L.reshape(-1, S, 3), B)
    return out


def exact(case, seed):
    lmax = case["lmax"]
    if case["kind"] == "bake":
        S = case["dirs"] or case["eq_w"] * case["eq_h"]
        if case["phong"] or case["nx"] * case["ny"] * case["nz"] * S * 2.0 * _triangles(case["scene"], case["size"]) > _TESTS:
            return None
        x = _bake_inputs(case, seed)
        d, b, w = _fibonacci(case["dirs"]) if case["dirs"] else _equirect(case["eq_w"], case["eq_h"])
        return _exact_bake(_Rays(x["mesh"]), x["probes"], d, b, w, lmax, x["sun"], x["sky"])
    if case["kind"] in ("batch", "service"):
        meshes, sky, volumes = _volumes(case, seed, case["jobs" if case["kind"] == "batch" else "bakes"])
        out, left = [], _TESTS / 2
        for v in volumes:
            need = len(v["probes"]) * v["dirs"] * 2.0 * len(meshes[v["mesh"]][1])
            if need > left:
                out.append(None)
                continue
            left -= need
            d, b, w = _fibonacci(v["dirs"])
            out.append(_exact_bake(_Rays(meshes[v["mesh"]]), v["probes"], d, b, w, lmax, v["sun"], sky))
        return out + [None] * case.get("relights", 0)
    if case["kind"] == "sky":
        return _exact_sky(case, _sky_inputs(case, seed))
    if case["kind"] == "eval":
        x = _eval_inputs(case, seed)
        return None if case["points"] * 8.0 * len(x["mesh"][1]) > _TESTS else _exact_eval(case, x)
    rng = np.random.default_rng([seed, 5])
    mesh = _scene(rng, case["scene"], case["size"])
    d, b, w = _fibonacci(64)
    bounds = np.concatenate([np.minimum(mesh[0].min(0), 0), np.maximum(mesh[0].max(0), 0)]).astype(np.float64)
    return [bounds, _exact_bake(_Rays(mesh), _grid(mesh[0], 4, 4, 4, 0.05), d, b, w, lmax, _sun(rng), None)]


def _exact_sky(case, texels):
    w, h, lmax = case["w"], case["h"], case["lmax"]
    if case["layout"] == "cube":
        e = torch.arange(w + 1, dtype=torch.float64, device="cuda") * (2.0 / w) - 1.0
        v, u = torch.meshgrid(e, e, indexing="ij")
        A = torch.atan2(u * v, torch.sqrt(u * u + v * v + 1.0))
        omega = A[1:, 1:] - A[:-1, 1:] - A[1:, :-1] + A[:-1, :-1]
        B = _basis(_cube_dirs(w), lmax) * omega[None, :, :, None]
    else:
        pi = 3.1415926538
        th = pi * (torch.arange(h, dtype=torch.float64, device="cuda") + 0.5) / h
        phi = 2 * pi * (torch.arange(w, dtype=torch.float64, device="cuda") + 0.5) / w
        if case["layout"] == "panorama":
            phi = phi - pi / 2
        th, phi = torch.meshgrid(th, phi, indexing="ij")
        x, y, z = torch.sin(th) * torch.cos(phi), torch.sin(th) * torch.sin(phi), torch.cos(th)
        d = torch.stack([x, z, y] if case["layout"] == "panorama" else [x, y, z], -1)
        B = _basis(d, lmax) * ((2 * pi / w) * (pi / h) * torch.sin(th))[..., None]
    B = B.reshape(-1, B.shape[-1])
    out = []
    for m in texels.reshape(case["count"], -1, texels.shape[-1]):
        m = m.double()[:, :3] / 255.0 if case["rgba8"] else m.double()
        out.append(B.T @ m)
    out = torch.stack(out)
    if case["swap"]:
        out = out.flip(-1)
    return out[0] if case["host"] and case["count"] == 1 else out


def _exact_eval(case, x):
    rays, K = _Rays(x["mesh"]), (case["lmax"] + 1) ** 2
    org, step = (torch.from_numpy(x[k]).double().cuda() for k in ("origin", "step"))
    counts = torch.from_numpy(x["counts"]).cuda()
    c = torch.from_numpy(x["coeffs"]).double().cuda()
    p, n = (torch.from_numpy(x[k]).double().cuda() for k in ("points", "normals"))
    n = n / n.norm(dim=1, keepdim=True)
    cell = ((p - org) / step).floor().long()
    cell = torch.minimum(cell.clamp(min=0), (counts - 2).clamp(min=0))
    Y, far = _basis(n, case["lmax"])[:, :K], step.norm()
    total, weight = torch.zeros_like(p), torch.zeros_like(p[:, :1])
    mask = torch.zeros(len(p), dtype=torch.uint8, device="cuda")
    for corner in range(8):
        ijk = torch.minimum(cell + torch.tensor([corner >> 2 & 1, corner >> 1 & 1, corner & 1], device="cuda"), counts - 1)
        d = org + step * ijk - p
        t = d.norm(dim=1)
        at, _ = rays.nearest(p + 0.005 * n, d / t[:, None], 0.0, t)
        seen = ~torch.isfinite(at) | (t == 0)
        # breadth-first order of the baker's grid
        i, j, k = ijk.unbind(1)
        q = torch.where(j == 0, i, counts[0] + i * (counts[1] - 1) + (j - 1))
        q = torch.where(k == 0, q, counts[0] * counts[1] + q * (counts[2] - 1) + (k - 1))
        wc = torch.where(seen, far - t, 0.0)[:, None]
        for ch in range(3):
            total[:, ch] += wc[:, 0] * (c[q, :, ch] * Y).sum(1)
        weight += wc
        mask |= (seen.to(torch.uint8) << corner)
    return [torch.where(weight > 0, total / weight, 0.0), mask]
