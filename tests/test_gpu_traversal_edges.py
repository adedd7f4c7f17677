"""Edges of the warp-wide traversal against the oracle, bit for bit: list lengths around the
32 pairs of a round, ray counts around a warp, axis-parallel rays, any-hit queries whose
lists end in the middle of a round, and the cell / test counters of the camera kernel."""
import numpy as np
import pytest

from happyray_b200 import GRID_TWO_LEVEL, GRID_UNIFORM
from happyray_b200 import scenes as S

pytestmark = pytest.mark.gpu


def overlapping_triangles(n, seed):
    """n triangles that each span most of the unit box: every cell near the middle lists them all."""
    rng = np.random.default_rng(seed)
    v = rng.uniform(0.0, 1.0, (n, 3, 3)).astype(np.float32)
    v[:, :, 2] = rng.uniform(0.0, 1.0, (n, 1)) + rng.normal(0, 0.05, (n, 3))
    return v.reshape(-1, 3).astype(np.float32), np.arange(3 * n, dtype=np.uint32).reshape(n, 3)


def rays(n, seed):
    rng = np.random.default_rng(seed)
    o = rng.uniform(-0.5, 1.5, (n, 3))
    d = rng.uniform(0.1, 0.9, (n, 3)) - o
    d[::5, 0] = 0.0            # axis-parallel components, both signs of zero
    d[::7, 1] = -0.0
    return o.astype(np.float32), (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)


def build(engine, O, v, f, kind):
    engine.upload(v, v, f, 1.0)
    engine.set_uniform_density(5.0)
    engine.setGridDensities(0.0625, 2.0)
    engine.build(kind)
    v4, bmin, bmax = O.lerp_bounds(v, v, 1.0)
    return O.build_ug(v4, f, bmin, bmax, 5.0, True) if kind == GRID_UNIFORM else O.build_tl(v4, f, bmin, bmax, 0.0625, 2.0)


@pytest.mark.parametrize("kind", [GRID_UNIFORM, GRID_TWO_LEVEL])
@pytest.mark.parametrize("ntri,nrays", [(1, 1), (17, 31), (31, 32), (32, 33), (33, 64), (65, 257), (300, 1000)])
def test_ray_queries_around_round_and_warp_sizes(engine, oracle, kind, ntri, nrays):
    import torch
    v, f = overlapping_triangles(ntri, ntri)
    b = build(engine, oracle, v, f, kind)
    org, d = rays(nrays, nrays)
    hid, t, u, w = engine.trace_rays(org, d)
    oid, ot, ou, ov = oracle.trace(b, org, d)
    assert np.array_equal(hid, oid) and np.array_equal(t, ot) and np.array_equal(u, ou) and np.array_equal(w, ov)
    tmax = np.random.default_rng(3).uniform(0.05, 2.0, nrays).astype(np.float32)
    do, dd, dt = (torch.from_numpy(x).cuda() for x in (org, d, tmax))
    occ = torch.full((nrays,), 7, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    engine.occluded_device(do, dd, dt, nrays, occ)
    engine.sync()
    assert np.array_equal(occ.cpu().numpy().astype(bool), np.asarray(oracle.occluded(b, org, d, tmax)).astype(bool))


def test_host_queries_around_the_staging_sizes(engine, oracle):
    """Host arrays of 40 bytes a ray around 64 and 256 KiB, growing and shrinking."""
    v, f = overlapping_triangles(300, 300)
    b = build(engine, oracle, v, f, GRID_TWO_LEVEL)
    for n in (1, 1638, 1639, 6553, 6554, 64, 6000):
        org, d = rays(n, n)
        for got, want in zip(engine.trace_rays(org, d), oracle.trace(b, org, d)):
            assert np.array_equal(got, want)


@pytest.mark.parametrize("kind", [GRID_UNIFORM, GRID_TWO_LEVEL])
@pytest.mark.parametrize("res", [(1, 1), (7, 3), (33, 17), (130, 70)])
def test_camera_rays_and_counters(engine, oracle, kind, res):
    """Camera rays of images around the 8 x 4 pixel tile, with the cells and triangle tests
    each ray reports."""
    import torch
    v, f = S.clusters(3000, seed=2)
    b = build(engine, oracle, v, f, kind)
    cam = S.camera_at_bounds(v, res)
    engine.setCamera(cam["position"], cam["orientation"], cam["up"], cam["fov"], *res)
    oc = oracle.camera(cam["position"], cam["orientation"], cam["up"], cam["fov"], *res)
    n = res[0] * res[1]
    out = [torch.zeros(n, dtype=torch.int32, device="cuda")] + [torch.zeros(n, device="cuda") for _ in range(3)]
    st = torch.zeros(2 * n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    engine.trace_primary_device(*out, st)
    engine.sync()
    oid, ot, ou, ov, ost = oracle.trace_primary(b, oc, stats=True)
    for got, want in zip(out, (oid, ot, ou, ov)):
        assert np.array_equal(got.cpu().numpy(), want)
    assert np.array_equal(st.cpu().numpy().reshape(n, 2), np.asarray(ost).reshape(n, 2).astype(np.int32))


@pytest.mark.parametrize("kind", [GRID_UNIFORM, GRID_TWO_LEVEL])
def test_ray_queries_at_every_share_per_warp(engine, oracle, kind):
    """Ray counts on both sides of each number of rays per warp, up to the refilled pool
    (more rays than the resident warps hold), whose words the next query finds cleared."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    full = sms * 32 * 32           # rays in flight at once: 32 warps per SM, 32 rays each
    v, f = S.clusters(2000, seed=3)
    b = build(engine, oracle, v, f, kind)
    org, d = rays(full + 4097, 9)
    oid, ot, ou, ov = oracle.trace(b, org, d)
    tmax = np.full(len(org), 0.7, np.float32)
    occ_o = np.asarray(oracle.occluded(b, org, d, tmax)).astype(bool)
    do, dd, dt = (torch.from_numpy(x).cuda() for x in (org, d, tmax))
    for n in (full // 32, full // 32 + 1, full // 8 + 5, full, full + 1, full + 4097, full + 4097, full // 2 + 1):
        out = [torch.zeros(n, dtype=torch.int32, device="cuda")] + [torch.zeros(n, device="cuda") for _ in range(3)]
        occ = torch.full((n,), 7, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        engine.trace_rays_device(do, dd, n, *out)
        engine.occluded_device(do, dd, dt, n, occ)
        engine.sync()
        for got, want in zip(out, (oid, ot, ou, ov)):
            assert np.array_equal(got.cpu().numpy(), want[:n])
        assert np.array_equal(occ.cpu().numpy().astype(bool), occ_o[:n])
