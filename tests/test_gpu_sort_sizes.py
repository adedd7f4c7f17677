"""Builds whose sort changes its tile size: large and small meshes in turn in one context, each
rebuilt until its captured graph is replayed, and sorts on both sides of the line."""
import numpy as np
import pytest

from happyray_b200 import GRID_TWO_LEVEL, GRID_UNIFORM, Engine
from happyray_b200 import scenes as S

pytestmark = pytest.mark.gpu


def line():
    """Keys from which tiles hold 4096 instead of 2048: four of the smaller ones per SM."""
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count * 4 * 2048


@pytest.mark.parametrize("kind", [GRID_TWO_LEVEL, GRID_UNIFORM])
def test_large_and_small_meshes_in_turn(hrlib, oracle, kind):
    grids = []
    for n in (1_000_000, 30_000, 420_000):
        v, f = S.clusters(n, seed=n)
        v4, bmin, bmax = oracle.lerp_bounds(v, v, 1.0)
        b = (oracle.build_ug(v4, f, bmin, bmax, 5.0, False) if kind == GRID_UNIFORM
             else oracle.build_tl(v4, f, bmin, bmax, 0.0625, 2.0))
        grids.append((v, f, b))
    assert max(b.npairs for _, _, b in grids) >= line() > min(b.npairs for _, _, b in grids)
    with Engine(0) as e:
        e.set_uniform_density(5.0)
        e.setGridDensities(0.0625, 2.0)
        for k in (0, 1, 2, 1, 0):
            v, f, b = grids[k]
            e.upload(v, v, f, 1.0)
            for _ in range(4):
                e.build(kind, False)
            _, cl, lv, pr = e.grid_download()
            assert np.array_equal(cl, b.cells) and np.array_equal(pr, b.prims)
            if kind == GRID_TWO_LEVEL:
                assert np.array_equal(lv, b.leaves)


@pytest.mark.parametrize("off", [-1, 0, 1])
def test_sorts_around_the_line(engine, off):
    import torch
    n = line() + off
    k = np.random.default_rng(n).integers(0, 1 << 18, n, dtype=np.uint64).astype(np.uint32)
    dk, dv = torch.from_numpy(k.view(np.int32)).cuda(), torch.arange(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    engine.radix_sort_pairs_device(dk, dv, n, 18)
    engine.sync()
    o = np.argsort(k, kind="stable")
    assert np.array_equal(dk.cpu().numpy().view(np.uint32), k[o]) and np.array_equal(dv.cpu().numpy(), o)
