"""The hierarchy's counting traversal (trace_stats_device): hits and the five work counters of
every ray against the oracle's nested loops."""
import numpy as np
import pytest

from happyray_b200 import scenes as S
from happyray_b200.hier import Hierarchy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_inst,nrays,spread", [(1, 33, False), (33, 500, True), (65, 4000, True), (300, 3000, False),
                                                 (300, 100_000, False)])
def test_hits_and_work_of_every_ray(hrlib, oracle, n_inst, nrays, spread):
    """Origins inside and outside the instance grid; instances that overlap near the centre
    (spread: cells list more than the 32 boxes of a window) or lie apart."""
    import torch
    kw = dict(world=0.2, scale_range=(0.3, 0.6)) if spread else {}
    v, f, counts, inst = S.instanced_scene(4, n_inst, seed=n_inst, tri_range=(80, 400), **kw)
    ob = oracle.hier_build(v, f, counts, inst, 1.2, 1.2)
    rng = np.random.default_rng(nrays)
    lo, hi = inst["bmin"].min(0), inst["bmax"].max(0)
    org = rng.uniform(lo - 0.5 * (hi - lo), hi + 0.5 * (hi - lo), (nrays, 3))
    d = rng.uniform(lo, hi, (nrays, 3)) - org
    d[::5, 0] = 0.0   # axis-parallel components
    d[::7, 1] = -0.0
    org, d = org.astype(np.float32), d.astype(np.float32)
    want = oracle.hier_trace(ob, org, d, stats=True)
    with Hierarchy(0) as h:
        h.set_objects(v, f, counts)
        h.set_instances(inst)
        h.build()
        o, dd = torch.from_numpy(org).cuda(), torch.from_numpy(d).cuda()
        out = ([torch.full((nrays,), -7, dtype=torch.int32, device="cuda") for _ in range(2)]
               + [torch.zeros(nrays, device="cuda") for _ in range(3)])
        work = torch.full((nrays, 5), -7, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        h.trace_stats_device(o, dd, *out, work)
        torch.cuda.synchronize()
        for got, x in zip(out, want):
            assert np.array_equal(got.cpu().numpy(), x)
        assert np.array_equal(work.cpu().numpy(), want[5].astype(np.int32))
        assert (want[5].max(0) > 0).all()
