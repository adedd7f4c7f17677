"""Workloads that the framework's speed is measured on: one pass each through its public
entry points (Engine, Batch, Server, Hierarchy).

listed() names the standing cases, draw() gives more of the same ranges, prepare() makes
what a program holds before the call (the uploaded meshes, built grids, rays and output
buffers, all from a seed), run() is one pass, work() what a pass cannot do without, and
exact() the same results in 64 bits where the closest hits of all rays can be found by
brute force.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from happyray_b200 import GRID_TWO_LEVEL, GRID_UNIFORM, RENDER_AO, RENDER_PATH, RENDER_PRIMARY, Engine
from happyray_b200 import scenes as S

GRIDS = {"uniform": GRID_UNIFORM, "two_level": GRID_TWO_LEVEL}
MODES = {"primary": RENDER_PRIMARY, "ao": RENDER_AO, "path": RENDER_PATH}
SEED = 0x853C49E6748FEA9B
FLT_MAX = float(np.finfo(np.float32).max)


def listed():
    return [
        # picking in an editor: a handful of rays from host memory against a built grid;
        # all latency
        dict(name="query_pick", kind="query", mesh="heightfield", grid="two_level", tris=8192, rays=64),
        # the small animated terrain preview: uniform grid with exact insertion rebuilt every
        # frame, 256 x 256 camera rays
        dict(name="uniform_primary_256", kind="frame", mesh="heightfield", grid="uniform", mode="primary", tris=32768,
             keyframes=1, w=256, h=256, spp=1, frames=1, host=False, materials=False),
        # a mid-sized model on a uniform grid (past the single-launch build), odd image size
        dict(name="uniform_primary_mid", kind="frame", mesh="clusters", grid="uniform", mode="primary", tris=300_001,
             keyframes=1, w=801, h=601, spp=1, frames=1, host=False, materials=False),
        # the drop-in loop of an application that keeps its meshes and images in host memory:
        # upload two key frames, build, render AO, read the image back
        dict(name="dropin_ao", kind="frame", mesh="clusters", grid="two_level", mode="ao", tris=100_003, keyframes=2,
             w=641, h=479, spp=4, frames=1, host=True, materials=False),
        # the headline frame: 1M triangles rebuilt, AO 8 samples at 1080p, image left on the device
        dict(name="ao_1080p", kind="frame", mesh="clusters", grid="two_level", mode="ao", tris=1_048_576, keyframes=1,
             w=1920, h=1080, spp=8, frames=1, host=False, materials=False),
        # a progressive path-traced preview: four images accumulated over one grid, shading
        # normals, materials and two lights
        dict(name="path_preview", kind="frame", mesh="heightfield", grid="two_level", mode="path", tris=100_000,
             keyframes=1, w=320, h=200, spp=1, frames=4, host=False, materials=True),
        # a frame of a key-frame animation, path traced: 2M triangles interpolated and rebuilt, 720p
        dict(name="path_720p", kind="frame", mesh="clusters", grid="two_level", mode="path", tris=2_097_152,
             keyframes=4, w=1280, h=720, spp=1, frames=1, host=False, materials=False),
        # collision and line-of-sight queries against an animated mesh: the rebuild of 2M
        # triangles and a few thousand rays
        dict(name="rebuild_2m", kind="rebuild", mesh="clusters", grid="two_level", tris=2_097_152, keyframes=4,
             rays=4096),
        # a lighting bake: incoherent closest hits and shadow rays of the same number, device buffers
        dict(name="rays_bake", kind="rays", mesh="clusters", grid="two_level", tris=500_009, rays=1_000_003),
        # many scenes a step (data generation): all grids rebuilt, all images rendered and downloaded
        dict(name="batch_24", kind="batch", scenes=24, tris_lo=1000, tris_hi=200_000, px_lo=64, px_hi=512, spp=4),
        # a burst of requests to a server that holds four animated scenes
        dict(name="served_burst", kind="served", scenes=4, tris_lo=10_000, tris_hi=200_000, keyframes=4, requests=24,
             px_lo=128, px_hi=384),
        # a rigid-body frame of an instanced scene: new instances, instance grid, 1080p camera rays
        dict(name="hier_1080p", kind="hier", objects=64, instances=16_384, tri_lo=320, tri_hi=20_480, w=1920, h=1080),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "frame", "frame", "frame", "rebuild", "rays", "batch", "served", "hier"])
    mesh = rng.choice(["heightfield", "clusters"])
    grid = rng.choice(["two_level", "two_level", "uniform"])
    if kind == "query":
        return dict(kind=kind, mesh="heightfield", grid=grid, tris=_log_int(rng, 500, 200_000),
                    rays=_log_int(rng, 1, 20_000))
    if kind == "frame":
        mode = rng.choice(["primary", "ao", "path"])
        side = _log_int(rng, 64, 1000)
        return dict(kind=kind, mesh=mesh, grid=grid, mode=mode, tris=_log_int(rng, 1000, 1_000_000),
                    keyframes=rng.choice([1, 2, 4]), w=side, h=max(16, int(side * rng.uniform(0.5, 1.0))),
                    spp=rng.choice([1, 3, 4, 8]) if mode == "ao" else 1, frames=rng.choice([1, 1, 4]),
                    host=rng.random() < 0.3, materials=mode == "path" and rng.random() < 0.5)
    if kind == "rebuild":
        return dict(kind=kind, mesh=mesh, grid=grid, tris=_log_int(rng, 2000, 1_500_000), keyframes=rng.choice([2, 4]),
                    rays=_log_int(rng, 256, 8192))
    if kind == "rays":
        return dict(kind=kind, mesh=mesh, grid=grid, tris=_log_int(rng, 2000, 500_000),
                    rays=_log_int(rng, 1000, 500_000))
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(2, 24), tris_lo=500, tris_hi=_log_int(rng, 5000, 200_000), px_lo=32,
                    px_hi=_log_int(rng, 64, 400), spp=rng.choice([1, 4]))
    if kind == "served":
        return dict(kind=kind, scenes=rng.randint(1, 4), tris_lo=5000, tris_hi=_log_int(rng, 10_000, 200_000),
                    keyframes=rng.choice([1, 4]), requests=rng.randint(2, 24), px_lo=64, px_hi=_log_int(rng, 96, 384))
    side = _log_int(rng, 64, 1200)
    return dict(kind="hier", objects=rng.randint(2, 64), instances=_log_int(rng, 64, 16_384), tri_lo=320,
                tri_hi=_log_int(rng, 1000, 20_480), w=8 * max(1, side // 8), h=4 * max(1, side // 8))


# ---- inputs ------------------------------------------------------------------------


def _mesh(case, seed):
    if case["mesh"] == "heightfield":
        return S.heightfield_tris(case["tris"], seed)
    return S.clusters(case["tris"], seed=seed)


def _frames(case, seed):
    """Key frames (K, V, 3) and triangles."""
    v, f = _mesh(case, seed)
    k = case.get("keyframes", 1)
    if k == 1:
        return v[None], f
    if torch.cuda.is_available():
        return S.curl_keyframes_torch(v, k, seed=seed), f
    return S.curl_keyframes(v, k, seed=seed), f


def _frame_time(case, seed):
    k = case.get("keyframes", 1)
    return 0.0 if k == 1 else float(np.float32(np.random.default_rng(seed + 7).uniform(0.05, k - 1.05)))


def _query_rays(n, seed):
    """Rays from above the terrain of [0, 1]^2 down into its interior."""
    rng = np.random.default_rng(seed + 1)
    org = np.concatenate([rng.uniform(0.2, 0.8, (n, 2)), rng.uniform(0.5, 1.5, (n, 1))], axis=1)
    to = np.concatenate([rng.uniform(0.1, 0.9, (n, 2)), np.zeros((n, 1))], axis=1)
    d = to - org
    return org.astype(np.float32), (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)


def _scene_rays(v, n, seed):
    """Rays from points all over the scene's box in all directions."""
    rng = np.random.default_rng(seed + 1)
    lo, hi = v.min(0), v.max(0)
    org = rng.uniform(lo, hi, (n, 3))
    d = rng.normal(size=(n, 3))
    return org.astype(np.float32), (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _hits(n):
    return [torch.zeros(n, dtype=torch.int32, device="cuda")] + [torch.zeros(n, device="cuda") for _ in range(3)]


def _instances(objs, boxes, rng, n):
    """Random rotations, uniform scales and positions in [0, 1]^3, as scenes.instanced_scene."""
    rec = np.zeros(n, S.INSTANCE_DTYPE)
    obj = rng.integers(0, objs, n)
    q = rng.normal(size=(n, 4))
    a, b, c, d = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    R = np.stack([np.stack([a * a + b * b - c * c - d * d, 2 * (b * c - a * d), 2 * (b * d + a * c)], -1),
                  np.stack([2 * (b * c + a * d), a * a - b * b + c * c - d * d, 2 * (c * d - a * b)], -1),
                  np.stack([2 * (b * d - a * c), 2 * (c * d + a * b), a * a - b * b - c * c + d * d], -1)], 1)
    s = np.exp(rng.uniform(math.log(0.01), math.log(0.05), n))
    T = rng.uniform(0.0, 1.0, (n, 3))
    inv = R.transpose(0, 2, 1) / s[:, None, None]
    m = np.concatenate([inv, -np.einsum("nij,nj->ni", inv, T)[:, :, None]], axis=2)
    lo, hi = boxes[0][obj], boxes[1][obj]
    corners = np.stack([np.stack([(lo, hi)[i][:, 0], (lo, hi)[j][:, 1], (lo, hi)[k][:, 2]], -1)
                        for i in (0, 1) for j in (0, 1) for k in (0, 1)], 1)
    wc = np.einsum("nij,nkj->nki", R * s[:, None, None], corners) + T[:, None, :]
    span = np.abs(wc).max(axis=(1, 2))[:, None] + 1.0
    rec["obj"], rec["m"] = obj, m.reshape(n, 12)
    rec["bmin"], rec["bmax"] = wc.min(1) - 1e-5 * span, wc.max(1) + 1e-5 * span
    return rec


def _hier_scene(case, seed):
    rng = np.random.default_rng(seed)
    v, f, counts, _ = S.instanced_scene(case["objects"], 1, seed=seed, tri_range=(case["tri_lo"], case["tri_hi"]))
    first = np.concatenate([[0], np.cumsum(counts)[:-1]]).astype(np.int64)
    tv = v[f].reshape(len(f), 9).reshape(-1, 3, 3)
    boxes = (np.minimum.reduceat(tv.min(1), first), np.maximum.reduceat(tv.max(1), first))
    inst = _instances(len(counts), boxes, rng, case["instances"])
    lo, hi = inst["bmin"].min(0).astype(np.float64), inst["bmax"].max(0).astype(np.float64)
    pos = np.array([0.5, -0.8, 0.9]) * (hi - lo) + lo
    fwd = 0.5 * (lo + hi) - pos
    fwd /= np.linalg.norm(fwd)
    right = np.cross(fwd, [0.0, 0.0, 1.0])
    right /= np.linalg.norm(right)
    up = np.cross(right, fwd)
    w, h = case["w"], case["h"]
    th = math.tan(math.radians(30.0))
    xs = ((np.arange(w) + 0.5) / w * 2 - 1) * th * w / h
    ys = (1 - (np.arange(h) + 0.5) / h * 2) * th
    d = fwd + xs[None, :, None] * right + ys[:, None, None] * up
    d = (d / np.linalg.norm(d, axis=2, keepdims=True)).astype(np.float32)
    d = d.reshape(h // 4, 4, w // 8, 8, 3).transpose(0, 2, 1, 3, 4).reshape(-1, 3)   # 8 x 4 pixel tiles
    return v, f, counts, inst, np.broadcast_to(pos.astype(np.float32), d.shape), d


def _engine(case, seed):
    e = Engine(0)
    kf, f = _frames(case, seed)
    e.setGridDensities(0.0625, 2.0)
    if len(kf) == 1:
        e.upload(kf[0], kf[0], f, 1.0)
    else:
        e.set_keyframes(kf, f)
    return e, kf, f


def _shading(e, v, f, seed):
    """Smooth vertex normals, eight materials and two lights above the scene."""
    rng = np.random.default_rng(seed + 3)
    p = v[f].astype(np.float64)
    fn = np.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0])
    n = np.stack([np.bincount(f.reshape(-1), np.repeat(fn[:, k], 3), len(v)) for k in range(3)], 1)
    n[:, 2] += 1e-12
    e.set_normals((n / np.linalg.norm(n, axis=1, keepdims=True)).astype(np.float32), f)
    e.set_materials(rng.uniform(0.2, 0.9, 8).astype(np.float32), rng.integers(0, 8, len(f)).astype(np.uint32))
    e.setLights([[0.4, 0.4, 1.0], [0.0, 0.7, 0.8]], [[0.2, 0, 0], [0.1, 0, 0]], [[0, 0.2, 0], [0, 0.1, 0]], [20.0, 30.0])


# ---- states ------------------------------------------------------------------------


def prepare(case, seed):
    s = _PREPARE[case["kind"]](case, seed)
    s["kind"] = case["kind"]
    torch.cuda.synchronize()
    return s


def run(state):
    return _RUN[state["kind"]](state)


def _prepare_query(case, seed):
    e, _, _ = _engine(case, seed)
    e.build(GRIDS[case["grid"]])
    org, d = _query_rays(case["rays"], seed)
    return dict(e=e, org=org, d=d)


def _run_query(s):
    return s["e"].trace_rays(s["org"], s["d"])


def _prepare_frame(case, seed):
    e, kf, f = _engine(case, seed)
    cam = S.camera_at_bounds(kf[0], (case["w"], case["h"]))
    e.setCamera(cam["position"], cam["orientation"], cam["up"], cam["fov"], cam["res_x"], cam["res_y"])
    e.set_integrator(ao_samples=case["spp"], ao_radius=-0.1, pt_bounces=4, seed=SEED)
    if case["materials"]:
        _shading(e, kf[0], f, seed)
    n = case["w"] * case["h"]
    fb = np.zeros((n, 3), np.float32) if case["host"] else torch.zeros(n, 3, device="cuda")
    return dict(e=e, kf=kf, f=f, t=_frame_time(case, seed), grid=GRIDS[case["grid"]], mode=MODES[case["mode"]],
                frames=case["frames"], host=case["host"], fb=fb)


def _run_frame(s):
    e, t = s["e"], s["t"]
    if s["host"]:
        k = int(t)
        e.upload(s["kf"][k], s["kf"][(k + 1) % len(s["kf"])], s["f"], t - k)
    elif len(s["kf"]) > 1:
        e.set_frame_time(t)
    e.build(s["grid"])
    for i in range(s["frames"]):
        if s["host"]:
            e.renderFrame(s["fb"], i, s["mode"])
        else:
            e.render_device(s["fb"], i, s["mode"])
    return s["fb"]


def _prepare_rebuild(case, seed):
    e, kf, _ = _engine(case, seed)
    org, d = _scene_rays(kf[0], case["rays"], seed)
    return dict(e=e, t=_frame_time(case, seed), grid=GRIDS[case["grid"]], n=case["rays"], org=_dev(org), d=_dev(d),
                out=_hits(case["rays"]))


def _run_rebuild(s):
    e = s["e"]
    e.set_frame_time(s["t"])
    e.build(s["grid"])
    e.trace_rays_device(s["org"], s["d"], s["n"], *s["out"])
    return s["out"]


def _prepare_rays(case, seed):
    e, kf, f = _engine(case, seed)
    e.build(GRIDS[case["grid"]])
    v, n = kf[0], case["rays"]
    org, d = _scene_rays(v, n, seed)
    # shadow rays: from surface points towards points of a light above the scene
    rng = np.random.default_rng(seed + 2)
    p = v[f[rng.integers(0, len(f), n)]].mean(1)
    to = np.concatenate([rng.uniform(0.4, 0.6, (n, 2)), np.full((n, 1), 1.5)], axis=1) - p
    dist = np.linalg.norm(to, axis=1, keepdims=True)
    sd = to / dist
    return dict(e=e, n=n, org=_dev(org), d=_dev(d), out=_hits(n), so=_dev((p + 1e-3 * sd).astype(np.float32)),
                sd=_dev(sd.astype(np.float32)), st=_dev(dist[:, 0].astype(np.float32)),
                occ=torch.zeros(n, dtype=torch.uint8, device="cuda"))


def _run_rays(s):
    s["e"].trace_rays_device(s["org"], s["d"], s["n"], *s["out"])
    s["e"].occluded_device(s["so"], s["sd"], s["st"], s["n"], s["occ"])
    return s["out"] + [s["occ"]]


def _log_sizes(case, n):
    """n triangle counts and image sides, log-uniform over the case's ranges; the same for every seed."""
    rng = np.random.default_rng(n)
    logs = [np.exp(rng.uniform(math.log(case[k + "_lo"]), math.log(case[k + "_hi"]), n)) for k in ("tris", "px")]
    return [[int(round(x)) for x in a] for a in logs]


def _prepare_batch(case, seed):
    from happyray_b200.batch import Batch, SceneSpec
    specs = []
    for i, (tris, side) in enumerate(zip(*_log_sizes(case, case["scenes"]))):
        v, f = _mesh(dict(mesh=("heightfield", "clusters")[i % 2], tris=tris), seed + i)
        cam = S.camera_at_bounds(v, (side, side))
        specs.append(SceneSpec(v, f, cam["position"], cam["orientation"], cam["up"], cam["fov"], side, side,
                               ao_samples=case["spp"]))
    b = Batch(0)
    b.set_scenes(specs)
    out = torch.zeros(3 * sum(x.width * x.height for x in specs)).pin_memory().numpy()
    return dict(b=b, out=out)


def _run_batch(s):
    s["b"].run(0)
    return s["b"].download_images(s["out"])


def _prepare_served(case, seed):
    from happyray_b200.server import Server
    rng = np.random.default_rng(seed + 4)
    srv = Server(0, 16 << 30)
    kfs = []
    for i, n in enumerate(_log_sizes(case, case["scenes"])[0]):
        kf, f = _frames(dict(mesh="clusters", tris=n, keyframes=case["keyframes"]), seed + i)
        srv.add_scene(kf, f)
        kfs.append(kf)
    reqs = []
    for i, side in enumerate(_log_sizes(case, case["requests"])[1]):
        sc = i % len(kfs)
        k = len(kfs[sc])
        cam = S.camera_at_bounds(kfs[sc][0], (side, side))
        out = torch.zeros(side * side, 3).pin_memory().numpy()
        reqs.append((sc, k * int(rng.integers(0, 120)) / 120.0, (RENDER_AO, RENDER_PATH)[i // 2 % 2], (1, 4)[i % 3 % 2],
                     cam, out))
    return dict(srv=srv, reqs=reqs)


def _run_served(s):
    pend = [s["srv"].submit_render(sc, t, mode, spp, cam, SEED, out=out) for sc, t, mode, spp, cam, out in s["reqs"]]
    return [p.wait() for p in pend]


def _prepare_hier(case, seed):
    from happyray_b200.hier import Hierarchy
    v, f, counts, inst, org, d = _hier_scene(case, seed)
    h = Hierarchy(0)
    h.set_densities(1.2, 1.2)
    h.set_objects(v, f, counts)
    h.set_instances(inst)
    h.build()
    n = len(d)
    out = [torch.zeros(n, dtype=torch.int32, device="cuda")] + _hits(n)
    return dict(h=h, inst=inst, org=_dev(org), d=_dev(d), out=out)


def _run_hier(s):
    s["h"].set_instances(s["inst"])
    s["h"].build()
    s["h"].trace_rays_device(s["org"], s["d"], *s["out"])
    return s["out"]


_PREPARE = dict(query=_prepare_query, frame=_prepare_frame, rebuild=_prepare_rebuild, rays=_prepare_rays,
                batch=_prepare_batch, served=_prepare_served, hier=_prepare_hier)
_RUN = dict(query=_run_query, frame=_run_frame, rebuild=_run_rebuild, rays=_run_rays, batch=_run_batch,
            served=_run_served, hier=_run_hier)


# ---- what a pass cannot do without ------------------------------------------------------

RAY_FLOPS = 80       # a ray's set-up and one triangle test
HIT_SHARE = 0.3      # of the camera rays, in scenes of these kinds


def _build_work(tris, keyframes):
    """A grid build reads the triangles' indices and the vertices (two key frames of them
    when it interpolates) once and writes at least one reference per triangle."""
    return tris * (12 + 4) + (tris // 2) * 16 * (2 if keyframes > 1 else 1)


def work(case):
    k = case["kind"]
    if k == "query":
        return {"bytes": 40 * case["rays"], "flops": RAY_FLOPS * case["rays"]}
    if k == "frame":
        px = case["w"] * case["h"]
        per_px = {"primary": 1.0, "ao": 1.0 + HIT_SHARE * case["spp"], "path": 1.0 + 2.0 * HIT_SHARE}[case["mode"]]
        rays = px * per_px * case["frames"]
        return {"bytes": _build_work(case["tris"], case["keyframes"]) + 12 * px, "flops": RAY_FLOPS * rays}
    if k == "rebuild":
        return {"bytes": _build_work(case["tris"], case["keyframes"]) + 40 * case["rays"],
                "flops": RAY_FLOPS * case["rays"]}
    if k == "rays":
        return {"bytes": (40 + 29) * case["rays"], "flops": 2 * RAY_FLOPS * case["rays"]}
    if k == "hier":
        n = case["w"] * case["h"]
        return {"bytes": 80 * case["instances"] + 44 * n, "flops": RAY_FLOPS * n}
    px = sum(x * x for x in _log_sizes(case, case["scenes" if k == "batch" else "requests"])[1])
    tris = _log_sizes(case, case["scenes"])[0]
    if k == "batch":
        return {"bytes": _build_work(sum(tris), 1) + 12 * px, "flops": RAY_FLOPS * px * (1.0 + HIT_SHARE * case["spp"])}
    built = sum(tris[i % len(tris)] for i in range(case["requests"]))
    return {"bytes": _build_work(built, case["keyframes"]) + 12 * px,
            "flops": RAY_FLOPS * px * (1.0 + 2.0 * HIT_SHARE)}


# ---- 64-bit results ---------------------------------------------------------------------


def _closest(v, f, org, d):
    """Closest hits by brute force in binary64: hit mask, t, u, v, triangle."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    p = torch.as_tensor(np.ascontiguousarray(v[f]), device=dev).double()
    o, d = (torch.as_tensor(np.ascontiguousarray(x), device=dev).double() for x in (org, d))
    n = len(o)
    best = torch.full((n,), math.inf, dtype=torch.float64, device=dev)
    bu, bv = torch.zeros_like(best), torch.zeros_like(best)
    tri = torch.full((n,), -1, dtype=torch.int64, device=dev)
    cross = lambda a, b: (a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0])  # noqa: E731
    dot = lambda a, b: a[0] * b[0] + a[1] * b[1] + a[2] * b[2]   # noqa: E731
    step = max(1, (1 << 24) // max(1, n))
    od, dd = [o[:, None, k] for k in range(3)], [d[:, None, k] for k in range(3)]
    for a in range(0, len(p), step):
        q = p[a:a + step]
        p0, p1, p2 = ([q[None, :, j, k] for k in range(3)] for j in range(3))
        e1, e2 = [p1[k] - p0[k] for k in range(3)], [p2[k] - p0[k] for k in range(3)]
        pv = cross(dd, e2)
        inv = 1.0 / dot(e1, pv)
        sv = [od[k] - p0[k] for k in range(3)]
        u = dot(sv, pv) * inv
        qv = cross(sv, e1)
        w = dot(qv, dd) * inv
        t = dot(e2, qv) * inv
        t = torch.where((u >= 0) & (w >= 0) & (u + w <= 1) & (t > 1e-4), t, math.inf)
        tm, at = t.min(1)
        closer = tm < best
        at_ = at[:, None]
        best = torch.where(closer, tm, best)
        bu = torch.where(closer, u.gather(1, at_)[:, 0], bu)
        bv = torch.where(closer, w.gather(1, at_)[:, 0], bv)
        tri = torch.where(closer, at + a, tri)
    hit = torch.isfinite(best)
    return hit, torch.where(hit, best, FLT_MAX), bu, bv, tri


def exact(case, seed):
    """Hit distances and barycentric weights, and the shaded image of small camera frames.
    AO and path images are random estimates: they have no value of their own."""
    k = case["kind"]
    if k == "query":
        v, f = _mesh(case, seed)
        org, d = _query_rays(case["rays"], seed)
    elif k == "rebuild":
        kf, f = _frames(case, seed)
        t = _frame_time(case, seed)
        i = int(t)
        c = t - i
        v = kf[i].astype(np.float64) * (1.0 - c) + kf[(i + 1) % len(kf)].astype(np.float64) * c
        org, d = _scene_rays(kf[0], case["rays"], seed)
    elif k == "frame" and case["mode"] == "primary" and case["frames"] == 1 and case["keyframes"] == 1:
        v, f = _mesh(case, seed)
        if len(f) * case["w"] * case["h"] > 1e10:
            return None
        return _exact_image(case, v, f)
    else:
        return None
    if len(f) * len(org) > 1e10:
        return None
    _, t, u, w, _ = _closest(v, f, org, d)
    return [None, t, u, w]


def _exact_image(case, v, f):
    w, h = case["w"], case["h"]
    cam = S.camera_at_bounds(v, (w, h))
    unit = lambda a: a / np.linalg.norm(a, axis=-1, keepdims=True)   # noqa: E731
    fwd = unit(np.asarray(cam["orientation"], np.float64))
    right = unit(np.cross(fwd, cam["up"]))
    down = unit(np.cross(fwd, right))
    tn = math.tan(math.radians(cam["fov"]) / 2.0)
    row, col = right * 2.0 * tn * w / h, down * 2.0 * tn
    ys, xs = np.divmod(np.arange(w * h), w)
    d = unit(fwd - row / 2 - col / 2 + (xs[:, None] + 0.25) / w * row + (ys[:, None] + 0.25) / h * col)
    org = np.broadcast_to(np.asarray(cam["position"], np.float64), d.shape)
    hit, _, _, _, tri = _closest(v, f, org, d)
    hit, tri = hit.cpu().numpy(), tri.clamp(min=0).cpu().numpy()
    p = v[f[tri]].astype(np.float64)
    nr = np.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0])
    a = p - org[:, None, :]
    area = np.linalg.norm(nr, axis=1)
    u = np.linalg.norm(np.cross(a[:, 1], a[:, 2]), axis=1) / area
    q = np.linalg.norm(np.cross(a[:, 2], a[:, 0]), axis=1) / area
    cs = np.abs((unit(nr) * d).sum(1))
    rgb = np.stack([u, q, 1.0 - u - q], 1) * cs[:, None]
    return np.where(hit[:, None], rgb, np.array([0.15, 0.2, 0.3]))
