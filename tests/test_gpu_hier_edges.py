"""Edges of the hierarchy's warp-wide traversal against the oracle, bit for bit: instance
lists around the 32 boxes of a window, ray counts around the rays a warp holds."""
import numpy as np
import pytest

from happyray_b200 import scenes as S
from happyray_b200.hier import Hierarchy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_inst,nrays", [(1, 1), (31, 31), (32, 33), (33, 500), (65, 2000), (300, 150_000)])
def test_overlapping_instances(hrlib, oracle, n_inst, nrays):
    """Instances that overlap near the centre, so that a cell lists nearly all of them."""
    v, f, counts, inst = S.instanced_scene(4, n_inst, seed=n_inst, tri_range=(80, 400), world=0.2,
                                           scale_range=(0.3, 0.6))
    ob = oracle.hier_build(v, f, counts, inst, 1.2, 1.2)
    rng = np.random.default_rng(nrays)
    org = rng.uniform(-1.0, 1.2, (nrays, 3))
    d = rng.uniform(-0.1, 0.3, (nrays, 3)) - org
    d[::5, 0] = 0.0   # axis-parallel components
    d[::7, 1] = -0.0
    org, d = org.astype(np.float32), d.astype(np.float32)
    tmax = rng.uniform(0.2, 1.5, nrays).astype(np.float32)
    with Hierarchy(0) as h:
        h.set_objects(v, f, counts)
        h.set_instances(inst)
        h.build()
        for _ in range(2):
            for got, want in zip(h.trace_rays(org, d), oracle.hier_trace(ob, org, d)):
                assert np.array_equal(got, want)
        assert np.array_equal(h.occluded(org, d, tmax), oracle.hier_trace(ob, org, d, tmax=tmax, anyhit=True)[0] >= 0)
