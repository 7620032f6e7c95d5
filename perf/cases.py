"""The work that programs built on gpugi_gb300 have it do, as measurable cases.

Kinds of case, each through the package's public entry points:

  closest / any   ray queries on device arrays, on the context's stream
  streams         ray queries of independent batches on caller streams
  host            ray queries on host arrays (copies in and out included)
  render          one accumulation: clear, render a pass, read the image
  batch           many small render jobs in one call, then reading their images
  nrc_train       one training step of the radiance cache on device samples
  nrc_infer       radiance-cache lookups of device queries

Scenes are the package's seeded generators (gpugi_gb300/scenes.py) at the
sizes of its benchmark and tests. A scene's geometry is an asset, the same
for every seed; rays, light samples, iterations, weights and training data
come from the seed.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from gpugi_gb300 import bvh, cuda, nrc, render, scenes

RES = ("slot", "t", "u", "v")


# ------------------------------------------------------------------- scenes
@functools.lru_cache(maxsize=None)
def _context():
    return cuda.Context(0)


@functools.lru_cache(maxsize=None)
def _streams():
    return tuple(torch.cuda.Stream() for _ in range(4))


@functools.lru_cache(maxsize=24)
def _geometry(scene: str, tris: int):
    """The scene's arrays and the asked number of triangles' nearest generator setting."""
    if scene == "icosphere":
        return scenes.displaced_icosphere(tris, seed=1)
    if scene == "instanced":
        return scenes.instanced_scene(seed=1, num_triangles=tris)
    if scene == "terrain":  # fBm heightfield and boxes: 2 grid^2 + 6,000 triangles
        return scenes.heightfield_boxes(seed=1, grid=max(24, int(math.sqrt(max(tris - 6000, 1152) / 2))))
    if scene == "room":  # Cornell room: walls of grid^2 quads, 20 4^level triangles of spheres
        level = max(2, min(6, int(math.log(max(tris, 500) / 23.9, 4))))
        return scenes.cornell_room(seed=1, sphere_level=level, wall_grid=max(4, min(40, int(math.sqrt(tris / 60)))))
    raise ValueError(scene)


@functools.lru_cache(maxsize=24)
def _hierarchy(scene: str, tris: int, bounds: str):
    g = _geometry(scene, tris)
    return bvh.build_bvh(g["positions"], g["triangles"], method="sweep", fit=bounds)


def _upload(case, shading=False):
    """The scene on the device: bvhmake's hierarchy uploaded, or ("lbvh") built on the GPU."""
    g = _geometry(case["scene"], case["tris"])
    vi = cuda.vertex_info(g["normals"], g["texcoords"]) if shading else None
    mats = g["materials"] if shading else None
    if case["bounds"] == "lbvh":
        ds = _context().build_scene(g["positions"], g["triangles"], vi, mats)
    else:
        ds = _context().upload_scene(_hierarchy(case["scene"], case["tris"], case["bounds"]), g["positions"], vi, mats)
    if case.get("watertight"):
        ds.set_triangle_test(True)
    return ds


# --------------------------------------------------------------------- rays
def _rays(case, seed: int, n: int):
    """random: origins in twice the scene's box, any direction (most miss a small object);
    aimed: from outside at the object (most hit); inside: from points in the scene's box in any
    direction (diffuse bounces and ambient occlusion), tmax a share of its diagonal for any hit."""
    pos = _geometry(case["scene"], case["tris"])["positions"]
    rng = np.random.default_rng([17, seed])
    lo, hi = pos.min(0).astype(np.float64), pos.max(0).astype(np.float64)
    c, h = (lo + hi) / 2, (hi - lo) / 2
    d = rng.normal(size=(n, 3))
    if case["rays"] == "random":
        o = c + 2 * np.max(h) * rng.uniform(-2, 2, (n, 3))
    elif case["rays"] == "inside":
        o = c + h * rng.uniform(-1, 1, (n, 3))
    else:
        o = c + 1.5 * h * rng.uniform(-1, 1, (n, 3))
        d = lo + (hi - lo) * rng.uniform(size=(n, 3)) - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    tmax = math.inf if case["kind"] != "any" else 0.25 * 2 * float(np.linalg.norm(h))
    a = np.concatenate([o, d, np.full((n, 1), tmax)], 1).astype(np.float32).T
    return {k: np.ascontiguousarray(a[i]) for i, k in enumerate(cuda.RAY_KEYS)}


def _device_rays(rays):
    return {k: torch.from_numpy(v).cuda() for k, v in rays.items()}


def _result(n):
    return {k: torch.empty(n, dtype=torch.int32 if k == "slot" else torch.float32, device="cuda") for k in RES}


# -------------------------------------------------------------------- cases
def listed():
    return [
        # picking and single-object queries: a thousand rays, where a call's latency counts; the
        # watertight test is the one a picker wants
        dict(name="closest_small", kind="closest", scene="icosphere", tris=4096, bounds="aabox", rays="aimed",
             n=1000, watertight=True),
        # the benchmark's headline batch as one synchronous-style call on the context's stream
        dict(name="closest_icosphere", kind="closest", scene="icosphere", tris=65536, bounds="aabox", rays="random",
             n=1 << 20, watertight=False),
        # the headline as the benchmark runs it: independent batches over four caller streams
        dict(name="streams_icosphere", kind="streams", scene="icosphere", tris=65536, bounds="aabox", rays="random",
             n=1 << 20, batches=8, watertight=False),
        # shadow / ambient-occlusion rays in a large terrain whose hierarchy was built on the GPU; ragged size
        dict(name="any_terrain", kind="any", scene="terrain", tris=528242, bounds="lbvh", rays="inside",
             n=3_000_001, watertight=False),
        # diffuse-bounce rays through instanced geometry under fitted ellipsoid bounds
        dict(name="closest_ellipsoid", kind="closest", scene="instanced", tris=100_000, bounds="ellipsoid",
             rays="inside", n=500_000, watertight=False),
        # a batch from the host and back, as a program without device arrays calls it; ragged size
        dict(name="host_icosphere", kind="host", scene="icosphere", tris=65536, bounds="aabox", rays="aimed",
             n=300_001, watertight=False),
        # the path-tracing benchmark: Cornell room of 98k triangles, 512^2, 16 samples per pixel
        dict(name="pt_room", kind="render", scene="room", tris=97946, bounds="aabox", pass_="PT", width=512,
             height=512, samples=16, depth=8, rr=3),
        # an interactive preview frame: one sample per pixel at a low resolution
        dict(name="pt_preview", kind="render", scene="room", tris=97946, bounds="aabox", pass_="PT", width=320,
             height=180, samples=1, depth=8, rr=3),
        # light tracing in the same room (particles, camera connections, splats)
        dict(name="lt_room", kind="render", scene="room", tris=97946, bounds="aabox", pass_="LT", width=512,
             height=512, samples=8, depth=8, rr=3),
        # many thumbnails in one call: mixed passes and scenes
        dict(name="batch_small", kind="batch", jobs=24, tris=20_000, size=128, samples=4, depth=8),
        # one training step of the radiance cache on a frame's samples
        dict(name="nrc_train", kind="nrc_train", n=65536),
        # the cache lookups of one 1280 x 720 frame
        dict(name="nrc_infer", kind="nrc_infer", n=921600),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["closest", "closest", "any", "streams", "host", "render", "render", "batch", "nrc_train",
                       "nrc_infer"])
    if kind in ("nrc_train", "nrc_infer"):
        return dict(kind=kind, n=_log(rng, 2000, 65536) if kind == "nrc_train" else _log(rng, 5000, 921600))
    if kind == "batch":
        return dict(kind=kind, jobs=rng.randint(6, 24), tris=_log(rng, 5000, 20_000), size=rng.randint(60, 128),
                    samples=rng.randint(1, 4), depth=rng.randint(4, 8))
    if kind == "render":
        w = _log(rng, 160, 512)
        scene = rng.choice(["room", "terrain"])
        return dict(kind=kind, scene=scene, tris=_log(rng, 5000, 97946),
                    bounds=rng.choice(["aabox", "aabox", "lbvh"]),
                    pass_="PT" if scene == "terrain" else rng.choice(["PT", "LT"]), width=w,
                    height=max(90, int(w * rng.uniform(0.5, 1.0))), samples=_log(rng, 1, 8), depth=rng.randint(4, 8),
                    rr=rng.choice([0, 3]))
    scene = rng.choice(["icosphere", "instanced", "terrain", "room"])
    tris = _log(rng, 4096, 400_000) if scene in ("instanced", "terrain") else _log(rng, 2000, 65536)
    bounds = rng.choice(["aabox", "aabox", "lbvh"])
    if kind == "closest" and tris <= 60_000 and rng.random() < 0.25:
        bounds = "ellipsoid"
    c = dict(kind=kind, scene=scene, tris=tris, bounds=bounds, rays=rng.choice(["random", "aimed", "inside"]),
             n=_log(rng, 1000, 1 << 20 if kind != "host" else 400_000),
             watertight=bounds != "ellipsoid" and rng.random() < 0.2)
    if kind == "streams":
        c["batches"], c["n"] = rng.randint(2, 8), max(1000, c["n"] // 4)
    return c


# ------------------------------------------------------------------ prepare
def _queries(rng, n):
    """Cache queries: positions in the box, unit directions and normals, albedos."""
    q = np.concatenate([rng.uniform(-1, 1, (n, 3)), rng.normal(size=(n, 6)), rng.uniform(0.1, 0.9, (n, 3))], 1)
    q[:, 3:6] /= np.linalg.norm(q[:, 3:6], axis=1, keepdims=True)
    q[:, 6:9] /= np.linalg.norm(q[:, 6:9], axis=1, keepdims=True)
    return q.astype(np.float32)


def _weights(rng):
    """He-uniform weights of the 64-64x4-3 network (the output layer padded to 16)."""
    return np.concatenate([rng.uniform(-1, 1, i * o) * math.sqrt(6.0 / i) for i, o in nrc.LAYER_SHAPES]).astype(np.float32)


def _nrc_inputs(case, seed):
    rng = np.random.default_rng([29, seed])
    w, q = _weights(rng), _queries(rng, case["n"])
    if case["kind"] == "nrc_infer":
        return w, q
    # a smooth field with a sharp edge, as radiance is
    y = np.stack([0.5 + 0.5 * np.sin(3 * q[:, 0] + k) * q[:, 9 + k] + (q[:, 1] > 0.2) for k in range(3)], 1)
    return w, np.concatenate([q, y.astype(np.float32)], 1)


def _camera(case, w, h):
    return render.camera_lookat(*(scenes.HEIGHTFIELD_CAMERA if case["scene"] == "terrain" else scenes.CORNELL_CAMERA),
                                w, h)


def prepare(case, seed):
    ctx, kind = _context(), case["kind"]
    s = {"case": case, "ctx": ctx, "seed": seed}
    if kind in ("nrc_train", "nrc_infer"):
        w, x = _nrc_inputs(case, seed)
        s["cache"] = nrc.RadianceCache(ctx, (-1, -1, -1), (1, 1, 1), seed=1)
        s["cache"].set_weights(w)
        s["x"] = torch.from_numpy(x).cuda()
        return s
    if kind == "batch":
        s["jobs"], s["scenes"] = [], []
        for k in range(4):
            sub = dict(scene="instanced" if k % 2 else "room", tris=case["tris"] // (k + 1), bounds="aabox")
            s["scenes"].append((sub, _upload(sub, shading=True)))
        for k in range(case["jobs"]):
            sub, ds = s["scenes"][k % 4]
            cam = _camera(sub, case["size"], case["size"]) if k % 2 == 0 else render.camera_lookat(
                (0.0, 1.0, 7.0), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 45.0, case["size"], case["size"])
            s["jobs"].append(dict(scene=ds, camera=cam, image=render.Image(ctx, case["size"], case["size"]),
                                  pass_="LT" if k % 3 == 2 else "PT", samples=case["samples"],
                                  max_path_length=case["depth"], sky=(0.3, 0.3, 0.3), iteration=seed % 1000))
        return s
    if kind == "render":
        s["scene"] = _upload(case, shading=True)
        if case["scene"] == "terrain":
            render.add_directional_light(s["scene"], scenes.HEIGHTFIELD_SUN, (5.0, 5.0, 5.0))
        s["camera"] = _camera(case, case["width"], case["height"])
        s["image"] = render.Image(ctx, case["width"], case["height"])
        return s
    s["scene"] = _upload(case)
    n = case["n"]
    if kind == "streams":
        s["rays"] = [_device_rays(_rays(case, 100 * seed + b, n)) for b in range(case["batches"])]
        s["out"] = [_result(n) for _ in s["rays"]]
    elif kind == "host":
        s["rays"] = _rays(case, seed, n)
    else:
        s["rays"] = _device_rays(_rays(case, seed, n))
        s["out"] = torch.empty(n, dtype=torch.uint8, device="cuda") if kind == "any" else _result(n)
    return s


# ---------------------------------------------------------------------- run
def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "closest":
        cuda.trace_closest_device(ctx, s["scene"], s["rays"], s["out"])
        return s["out"]
    if kind == "any":
        cuda.trace_any_device(ctx, s["scene"], s["rays"], s["out"])
        return s["out"]
    if kind == "streams":
        st = _streams()
        for b, (r, o) in enumerate(zip(s["rays"], s["out"])):
            cuda.trace_closest_device_async(ctx, s["scene"], r, o, st[b % 4].cuda_stream)
        return s["out"]
    if kind == "host":
        return cuda.trace_closest(ctx, s["scene"], s["rays"])
    if kind == "render":
        s["image"].clear()
        render.render(ctx, s["scene"], s["camera"], s["image"], case["pass_"], max_path_length=case["depth"],
                      samples=case["samples"], iteration=s["seed"] % 1000, rr_start_depth=case["rr"],
                      sky=(0.5, 0.5, 0.5) if case["scene"] == "terrain" else (0.0, 0.0, 0.0),
                      rng_state=[1 + s["seed"]])
        return s["image"].read()
    if kind == "batch":
        for k, j in enumerate(s["jobs"]):
            j["image"].clear()
            j["rng_state"] = [1 + s["seed"] + k]
        render.render_batch(ctx, s["jobs"])
        return [j["image"].read() for j in s["jobs"]]
    if kind == "nrc_train":
        loss = s["cache"].train(s["x"])
        return {"loss": loss, "weights": s["cache"].weights()}
    return s["cache"].infer(s["x"])


# --------------------------------------------------------------------- work
def _trace_work(n, hits, tris, out_bytes, scene_bytes_per_tri):
    """Rays read, results written and the scene read once; per ray that enters the scene at least
    one box test per level of a binary tree of 8-triangle leaves and one triangle test."""
    levels = max(1.0, math.log2(max(2, tris / 8)))
    return {"bytes": n * (28 + out_bytes) + tris * scene_bytes_per_tri, "flops": hits * (18 * levels + 45)}


def work(case):
    kind = case["kind"]
    if kind == "nrc_infer":
        return {"bytes": case["n"] * 60 + 34816, "flops": 2.0 * case["n"] * 16576}
    if kind == "nrc_train":
        return {"bytes": case["n"] * 60 + 3 * 69632, "flops": 2.0 * case["n"] * (16576 + 12480 + 16576)}
    if kind == "batch":
        n = case["jobs"] * case["size"] ** 2 * case["samples"]
        w = _trace_work(2 * n, 2 * n, case["tris"], 0, 60)
        return {"bytes": case["jobs"] * case["size"] ** 2 * 16 + case["tris"] * 120, "flops": w["flops"]}
    if kind == "render":  # at least a camera (or light) ray and a shadow (or camera) connection per sample
        n = case["width"] * case["height"] * case["samples"]
        w = _trace_work(2 * n, 2 * n, case["tris"], 0, 60)
        return {"bytes": case["width"] * case["height"] * 16 + case["tris"] * 60, "flops": w["flops"]}
    n = case["n"] * case.get("batches", 1)
    share = 0.06 if case["rays"] == "random" else 1.0
    return _trace_work(n, n * share, case["tris"], 1 if kind == "any" else 16, 60)


# -------------------------------------------------------------------- exact
def _exact_closest(case, seed):
    """Nearest triangle of each ray by testing every one, in float64."""
    g = _geometry(case["scene"], case["tris"])
    r = {k: torch.from_numpy(v).cuda().double() for k, v in _rays(case, seed, case["n"]).items()}
    o, d = (torch.stack([r[k] for k in ks], 1) for ks in (("ox", "oy", "oz"), ("dx", "dy", "dz")))
    p = torch.from_numpy(np.asarray(g["positions"], np.float64)).cuda()
    tri = torch.from_numpy(np.asarray(g["triangles"])[:, :3].astype(np.int64)).cuda()
    p0, e1, e2 = p[tri[:, 0]], p[tri[:, 1]] - p[tri[:, 0]], p[tri[:, 2]] - p[tri[:, 0]]
    nrm = torch.linalg.cross(e1, e2)
    n, step = case["n"], max(1, 20_000_000 // len(tri))
    out = [torch.empty(n, dtype=torch.float64, device="cuda") for _ in range(3)]
    for a in range(0, n, step):
        oo, dd = o[a:a + step], d[a:a + step]
        det = dd @ nrm.T
        w = torch.linalg.cross(oo, dd)  # triple products by (a x b) . c = a . (b x c)
        tvec_n = (p0 * nrm).sum(1)[None] - oo @ nrm.T
        t = tvec_n / det
        q = lambda e: dd @ torch.linalg.cross(p0, e).T + w @ e.T  # noqa: E731  (d x (p0 - o)) . e
        u, v = -q(e2) / det, q(e1) / det
        ok = (t > 1e-4) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t < r["tmax"][a:a + step, None])
        t = torch.where(ok, t, math.inf)
        best, at = t.min(1)
        hit = torch.isfinite(best)
        z = torch.zeros_like(best)
        out[0][a:a + step] = torch.where(hit, best, r["tmax"][a:a + step])
        out[1][a:a + step] = torch.where(hit, u.gather(1, at[:, None])[:, 0], z)
        out[2][a:a + step] = torch.where(hit, v.gather(1, at[:, None])[:, 0], z)
    return {"slot": None, "t": out[0], "u": out[1], "v": out[2]}


# Real spherical harmonics of degree < 4: the square roots of the textbook constants.
_PI = math.pi
_SH = [math.sqrt(x / _PI) / y for x, y in ((1, 2), (3, 2), (15, 2), (5, 4), (15, 4), (17.5, 4), (105, 2), (10.5, 4),
                                           (7, 4), (105, 4))]


def _encode(q):
    p, cols = (q[:, 0:3] + 1) / 2, []
    for k in range(3):
        for o in range(6):
            cols += [torch.sin(_PI * 2 ** o * p[:, k]), torch.cos(_PI * 2 ** o * p[:, k])]
    x, y, z = q[:, 3], q[:, 4], q[:, 5]
    c, xx, yy, zz = _SH, x * x, y * y, z * z
    cols += [torch.full_like(x, c[0]), -c[1] * y, c[1] * z, -c[1] * x, c[2] * x * y, -c[2] * y * z,
             c[3] * (3 * zz - 1), -c[2] * x * z, c[4] * (xx - yy), c[5] * y * (yy - 3 * xx), c[6] * x * y * z,
             c[7] * y * (1 - 5 * zz), c[8] * z * (5 * zz - 3), c[7] * x * (1 - 5 * zz), c[9] * z * (xx - yy),
             c[5] * x * (3 * yy - xx)]
    cols += [q[:, k] for k in range(6, 12)] + [torch.ones_like(x)]
    return torch.nn.functional.pad(torch.stack(cols, 1), (0, 64 - len(cols)))


def exact(case, seed):
    kind = case["kind"]
    if kind == "closest" and case["n"] * _geometry(case["scene"], case["tris"])["triangles"].shape[0] <= 5_000_000_000:
        return _exact_closest(case, seed)
    if kind not in ("nrc_train", "nrc_infer"):
        return None  # images have no closed form; larger queries would take too long one by one
    w, x = _nrc_inputs(case, seed)
    W = [torch.from_numpy(w[at:at + i * o].reshape(i, o).astype(np.float64)).cuda()
         for at, (i, o) in zip(range(0, 5 * 4096, 4096), nrc.LAYER_SHAPES)]
    x = torch.from_numpy(x).cuda().double()
    if kind == "nrc_train":
        W = [m.requires_grad_() for m in W]
    h = _encode(x[:, :12])
    for m in W[:4]:
        h = torch.relu(h @ m)
    p = (h @ W[4])[:, :3]
    if kind == "nrc_infer":
        return torch.relu(p)  # radiance: lookups are clamped at 0
    loss = ((p - x[:, 12:]) ** 2 / (p.detach() ** 2 + 0.01)).mean()
    loss.backward()
    # the first step of Adam from zero moments: m / (1 - b1) = g, v / (1 - b2) = g^2
    new = [(m.detach() - 1e-2 * m.grad / (m.grad.abs() + 1e-8)).reshape(-1) for m in W]
    return {"loss": float(loss), "weights": torch.cat(new)}
