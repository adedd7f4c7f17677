"""Images and waves on both sides of each number of rays that a warp takes at a time.  Sizes
come from the SM count, as the rules do: a warp takes 32 rays, or 16, 8 or 4 while a launch
would not fill the resident warps often enough."""
import time

import numpy as np
import pytest

from happyray_b200 import GRID_TWO_LEVEL, GRID_UNIFORM, RENDER_AO, RENDER_PATH, RENDER_PRIMARY, Engine
from happyray_b200 import scenes as S
from happyray_b200.server import BATCHED, Server

pytestmark = pytest.mark.gpu

SEED = 41


def sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def build(engine, O, v, f, kind):
    engine.upload(v, v, f, 1.0)
    engine.set_uniform_density(5.0)
    engine.setGridDensities(0.0625, 2.0)
    engine.build(kind)
    v4, bmin, bmax = O.lerp_bounds(v, v, 1.0)
    return O.build_ug(v4, f, bmin, bmax, 5.0, True) if kind == GRID_UNIFORM else O.build_tl(v4, f, bmin, bmax, 0.0625, 2.0)


def set_camera(engine, O, v, w, h):
    cam = S.camera_at_bounds(v, (w, h))
    args = (cam["position"], cam["orientation"], cam["up"], cam["fov"], w, h)
    engine.setCamera(*args)
    return O.camera(*args)


@pytest.mark.parametrize("width", [8, 16, 32])   # the width from these sizes on; half of it below
@pytest.mark.parametrize("off", [-4, 0])
def test_uniform_camera_rays(engine, oracle, width, off):
    """Resident warps (32 per SM) filled four times over."""
    import torch
    v, f = S.clusters(2000, seed=2)
    b = build(engine, oracle, v, f, GRID_UNIFORM)
    w, h = 8 * sms(), 16 * width + off   # w * h slots: 32 warps x 4 x width per SM
    cam = set_camera(engine, oracle, v, w, h)
    n = w * h
    out = [torch.zeros(n, dtype=torch.int32, device="cuda")] + [torch.zeros(n, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    engine.trace_primary_device(*out)
    engine.sync()
    for got, want in zip(out, oracle.trace_primary(b, cam)):
        assert np.array_equal(got.cpu().numpy(), want)
    engine.set_integrator(seed=SEED)
    fb = engine.renderFrame(None, 5, RENDER_PRIMARY)
    assert np.array_equal(fb, oracle.render_primary(b, cam, 5, SEED))
    alpha = float(np.float32(0.05) * b.diag())
    engine.set_integrator(ao_samples=2, ao_radius=alpha, seed=SEED)
    assert np.array_equal(engine.renderFrame(None, 0, RENDER_AO)[:, 0], oracle.render_ao(b, cam, 2, alpha, SEED)[0])


@pytest.mark.parametrize("kind", [GRID_TWO_LEVEL, GRID_UNIFORM])
@pytest.mark.parametrize("width", [8, 16, 32])
def test_path_tracer_images(engine, oracle, kind, width):
    """Images of 9/8 of what 8 blocks of 4 warps per SM hold at `width` paths a warp, which is
    below twice what 7 hold."""
    v, f = S.clusters(2000, seed=2)
    b = build(engine, oracle, v, f, kind)
    cam = set_camera(engine, oracle, v, sms(), 36 * width + 1)
    engine.set_integrator(pt_bounces=3, albedo=0.7, seed=SEED)
    engine.setLights((0.4, 0.4, 1.0), (0.2, 0, 0), (0, 0.2, 0), 20.0)
    fb = engine.renderFrame(None, 0, RENDER_PATH)
    img, _ = oracle.render_pt(b, cam, oracle.make_light(), 3, 0.7, float(np.float32(1e-4) * b.diag()), SEED)
    assert np.array_equal(fb[:, 0], img) and img.max() > 0


@pytest.mark.parametrize("mode,fill", [(RENDER_PATH, 1.9), (RENDER_PATH, 2.1), (RENDER_PATH, 3.9), (RENDER_PATH, 4.1),
                                       (RENDER_AO, 7.8), (RENDER_AO, 8.2), (RENDER_AO, 15.8), (RENDER_AO, 16.2)])
def test_requests_of_one_wave(hrlib, mode, fill):
    """Three requests over three scenes in one wave whose 8 x 4 tiles fill the 24 warps per SM of
    the job kernel `fill` times (lines at 2 and 4 for paths, 8 and 16 for the others), each
    against the per-scene path."""
    meshes = [S.clusters(6000, seed=1), S.heightfield_tris(5000, seed=2), S.clusters(900, seed=3)]
    tiles = fill * 24 * sms()
    cols = [int((tiles * part / 2.0) ** 0.5) for part in (0.5, 0.3, 0.2)]
    spp = (1, 2, 1)

    def cam(k, rows=None):
        c = cols[k]
        w = 8 * c - 3   # c tiles across, 2 c or the rest of the total down
        h = 8 * c - 1 if rows is None else 4 * rows - 1
        return S.camera_at_bounds(meshes[k][0], (w, h))
    rest = int(round((tiles - 2 * cols[0] ** 2 - 2 * cols[1] ** 2) / cols[2]))
    cams = [cam(0), cam(1), cam(2, rest)]
    have = sum(-(-c["res_x"] // 8) * -(-c["res_y"] // 4) for c in cams)
    assert abs(have / (24.0 * sms()) - fill) < 0.05
    with Server(0, 16 << 30, BATCHED) as srv:
        for v, f in meshes:
            srv.add_scene(v, f)
        small = S.camera_at_bounds(meshes[0][0], (16, 16))
        srv.inject_stall(2, 400)   # two waves held back on the host: the requests gather behind them
        first = []
        for _ in range(2):
            first.append(srv.submit_render(0, 0.0, RENDER_PRIMARY, 1, small, SEED))
            time.sleep(0.1)
        pend = [srv.submit_render(k, 0.0, mode, spp[k], cams[k], SEED) for k in range(3)]
        got = [p.wait(60_000) for p in pend]
        assert len({p.info()["wave"] for p in pend}) == 1
        for p in first:
            p.wait(60_000)
    for k, (v, f) in enumerate(meshes):
        with Engine(0) as e:
            e.upload(v, v, f, 1.0)
            e.setGridDensities(0.0625, 2.0)
            e.build(GRID_TWO_LEVEL)
            c = cams[k]
            e.setCamera(c["position"], c["orientation"], c["up"], c["fov"], c["res_x"], c["res_y"])
            e.set_integrator(ao_samples=spp[k], ao_radius=-0.1, pt_bounces=4, albedo=0.7, seed=SEED)
            fb = None
            for im in range(spp[k] if mode == RENDER_PATH else 1):
                fb = e.renderFrame(fb, im, mode)
            assert np.array_equal(got[k], fb), f"request {k}"
