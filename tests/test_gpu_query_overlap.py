"""Ray queries that run side by side: captured ones replayed on other streams than the
context's, and ray counts on both sides of each way a query is shared out."""
import numpy as np
import pytest

from happyray_b200 import GRID_TWO_LEVEL, GRID_UNIFORM, Engine
from happyray_b200 import scenes as S

pytestmark = pytest.mark.gpu


def in_flight():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count * 32 * 32   # 32 warps per SM, 32 rays each


def scene_rays(v, n, seed):
    rng = np.random.default_rng(seed)
    o = rng.uniform(v.min(0), v.max(0), (n, 3))
    d = rng.normal(size=(n, 3))
    return o.astype(np.float32), (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)


def hits(n):
    import torch
    return [torch.full((n,), -7, dtype=torch.int32, device="cuda")] + [torch.zeros(n, device="cuda") for _ in range(3)]


@pytest.mark.parametrize("kind", [GRID_UNIFORM, GRID_TWO_LEVEL])
def test_captured_queries_replayed_beside_others(hrlib, kind):
    """Graphs of one context's queries, larger than its warps hold at once, replayed together on
    several streams and beside a query on the context's own: each gives what it gives alone."""
    import torch
    v, f = S.clusters(20_000, seed=3)
    st = torch.cuda.Stream()
    e = Engine(0, st.cuda_stream)
    e.upload(v, v, f, 1.0)
    e.build(kind)
    n = 3 * in_flight() + 1
    org, d = scene_rays(v, n, 5)
    do, dd, tm = torch.from_numpy(org).cuda(), torch.from_numpy(d).cuda(), torch.full((n,), 0.4, device="cuda")
    want, wocc, wfb = hits(n), torch.zeros(n, dtype=torch.uint8, device="cuda"), torch.zeros(n, 3, device="cuda")
    torch.cuda.synchronize()
    e.trace_rays_device(do, dd, n, *want)
    e.occluded_device(do, dd, tm, n, wocc)
    e.render_rays_device(do, dd, n, 0, wfb)
    e.sync()
    outs = [hits(n) for _ in range(3)]
    occ, fb = torch.full((n,), 7, dtype=torch.uint8, device="cuda"), torch.zeros(n, 3, device="cuda")
    work = [lambda k=k: e.trace_rays_device(do, dd, n, *outs[k]) for k in range(2)]
    work += [lambda: e.occluded_device(do, dd, tm, n, occ), lambda: e.render_rays_device(do, dd, n, 0, fb)]
    graphs = []
    torch.cuda.synchronize()
    for w in work:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            w()
        graphs.append((g, torch.cuda.Stream()))
    for _ in range(3):
        for x in outs:
            x[0].fill_(-7)
        occ.fill_(7)
        fb.zero_()
        torch.cuda.synchronize()
        for g, s in graphs:
            with torch.cuda.stream(s):
                g.replay()
        e.trace_rays_device(do, dd, n, *outs[2])
        torch.cuda.synchronize()
        for out in outs:
            assert all(torch.equal(a, b) for a, b in zip(out, want))
        assert torch.equal(occ, wocc) and torch.equal(fb, wfb)
    del graphs
    e.close()


@pytest.mark.parametrize("kind", [GRID_UNIFORM, GRID_TWO_LEVEL])
def test_ray_counts_around_every_share(hrlib, oracle, kind):
    """Ray counts on both sides of each number of rays per warp (all warps with 1, 2, 4, 8
    and 16 rays) and of the refilled pool, whose words the next query finds cleared."""
    import torch
    v, f = S.clusters(2000, seed=3)
    e = Engine(0)
    e.upload(v, v, f, 1.0)
    e.set_uniform_density(5.0)
    e.setGridDensities(0.0625, 2.0)
    e.build(kind)
    v4, bmin, bmax = oracle.lerp_bounds(v, v, 1.0)
    b = (oracle.build_ug(v4, f, bmin, bmax, 5.0, True) if kind == GRID_UNIFORM
         else oracle.build_tl(v4, f, bmin, bmax, 0.0625, 2.0))
    full = in_flight()
    warps = full // 32
    org, d = scene_rays(v, 2 * full + 33, 9)
    want = oracle.trace(b, org, d)
    tmax = np.full(len(org), 0.3, np.float32)
    occ_o = np.asarray(oracle.occluded(b, org, d, tmax)).astype(bool)
    do, dd, dt = (torch.from_numpy(x).cuda() for x in (org, d, tmax))
    sizes = [warps * w + k for w in (1, 2, 4, 8, 16) for k in (0, 1)]
    sizes += [full, full + 1, 2 * full + 33, 7]
    for n in sizes:
        out, occ = hits(n), torch.full((n,), 7, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        e.trace_rays_device(do, dd, n, *out)
        e.occluded_device(do, dd, dt, n, occ)
        e.sync()
        for got, x in zip(out, want):
            assert np.array_equal(got.cpu().numpy(), x[:n])
        assert np.array_equal(occ.cpu().numpy().astype(bool), occ_o[:n])
    e.close()
