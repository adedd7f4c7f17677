"""Insertion of triangles over many cells against the oracle, bit for bit, through the single
launch and through the pipeline.  Exact: written by blocks instead of one thread; extents
around the serial limit, the piece size and the per-axis tables.  By bounding box: blocks
whose runs are staged in shared memory beside blocks with longer ones."""
import numpy as np
import pytest

from happyray_b200 import GRID_UNIFORM, Engine

pytestmark = pytest.mark.gpu


def scene(cells_per_side, tilt, flat, seed):
    """Small triangles that fix the grid and two large ones across it."""
    rng = np.random.default_rng(seed)
    n = max(64, cells_per_side * cells_per_side // 5)
    c = rng.uniform(0.0, 1.0, (n, 3))
    c[:, 2] *= flat
    small = c[:, None, :] + rng.normal(0, 0.01, (n, 3, 3)) * np.array([1.0, 1.0, flat])
    big = np.array([[[0.0, 0.0, 0.0], [1.0, 0.0, 0.0], [1.0, 1.0, tilt * flat]],
                    [[0.0, 0.0, 0.2 * flat], [1.0, 1.0, flat], [0.0, 1.0, 0.5 * flat]]])
    v = np.concatenate([small[: n // 2], big, small[n // 2:]]).reshape(-1, 3).astype(np.float32)
    return v, np.arange(len(v), dtype=np.uint32).reshape(-1, 3)


@pytest.mark.parametrize("exact", [True, False])
@pytest.mark.parametrize("pipeline", [False, True])
@pytest.mark.parametrize("side,tilt,flat,density", [(4, 0.0, 1.0, 1.0), (4, 1.0, 1.0, 5.0), (20, 0.0, 1.0, 5.0),
                                                    (45, 1.0, 1.0, 5.0), (130, 0.1, 0.01, 5.0), (330, 0.0, 1e-4, 130.0)])
def test_large_triangles(oracle, monkeypatch, exact, pipeline, side, tilt, flat, density):
    if pipeline:
        monkeypatch.setenv("HAPPYRAY_SMALL_BUILD_MAX_TRIS", "0")
    v, f = scene(side, tilt, flat, side)
    v4, bmin, bmax = oracle.lerp_bounds(v, v, 1.0)
    b = oracle.build_ug(v4, f, bmin, bmax, density, exact)
    with Engine(0) as e:
        e.upload(v, v, f, 1.0)
        e.set_uniform_density(density)
        for _ in range(3):   # the third replays the captured build
            e.build(GRID_UNIFORM, exact)
            gi, cells, _, prims = e.grid_download()
            assert gi["res"] == tuple(b.grid.res) and gi["num_pairs"] == b.npairs
            assert np.array_equal(cells, b.cells) and np.array_equal(prims, b.prims)
