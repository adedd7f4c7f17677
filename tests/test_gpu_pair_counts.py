"""Builds whose pairs come in the orders that the per-cell counts take differently: equal keys
side by side, a few crowded cells in turn or at random, keys that all differ.  Grids against
the oracle, bit for bit."""
import numpy as np
import pytest

from happyray_b200 import GRID_TWO_LEVEL, GRID_UNIFORM, Engine

pytestmark = pytest.mark.gpu


def cells_in_turn(n, cells, order, seed):
    """n tiny triangles near `cells` points, in blocks, in turn or at random."""
    rng = np.random.default_rng(seed)
    at = rng.uniform(0.05, 0.95, (cells, 3))
    i = np.arange(n)
    pick = {"blocks": i * cells // n, "turn": i % cells, "random": rng.integers(0, cells, n)}[order]
    v = at[pick][:, None, :] + rng.normal(0, 0.0005, (n, 1, 3)) + rng.normal(0, 0.0002, (n, 3, 3))
    return v.reshape(-1, 3).astype(np.float32), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)


@pytest.mark.parametrize("pipeline", [False, True])
@pytest.mark.parametrize("n,cells,order", [(31, 2, "turn"), (4000, 2, "blocks"), (4001, 2, "turn"), (4001, 3, "turn"),
                                           (4001, 12, "turn"), (4001, 13, "turn"), (4001, 2, "random"),
                                           (4001, 5, "random"), (4001, 4001, "random")])
def test_counts_by_runs_and_by_match(hrlib, oracle, monkeypatch, pipeline, n, cells, order):
    if pipeline:
        monkeypatch.setenv("HAPPYRAY_SMALL_BUILD_MAX_TRIS", "0")
    v, f = cells_in_turn(n, cells, order, n + cells)
    v4, bmin, bmax = oracle.lerp_bounds(v, v, 1.0)
    with Engine(0) as e:
        e.upload(v, v, f, 1.0)
        e.set_uniform_density(5.0)
        e.setGridDensities(0.0625, 2.0)
        for kind in (GRID_UNIFORM, GRID_TWO_LEVEL):
            b = (oracle.build_ug(v4, f, bmin, bmax, 5.0, False) if kind == GRID_UNIFORM
                 else oracle.build_tl(v4, f, bmin, bmax, 0.0625, 2.0))
            e.build(kind, False)
            gi, cl, lv, pr = e.grid_download()
            assert gi["res"] == tuple(b.grid.res) and gi["num_pairs"] == b.npairs
            assert np.array_equal(cl, b.cells) and np.array_equal(pr, b.prims)
            if kind == GRID_TWO_LEVEL:
                assert np.array_equal(lv, b.leaves)
