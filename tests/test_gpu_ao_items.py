"""Ambient occlusion with about 2^32 (hit pixel, sample) items: every sample of every pixel is
traced once, so a pixel's visibility is its unoccluded samples over all of them."""
import numpy as np
import pytest

from happyray_b200 import GRID_TWO_LEVEL, GRID_UNIFORM, RENDER_AO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,w,h,spp", [
    (GRID_TWO_LEVEL, 8192, 8192, 65),     # 2^32 + 2^26 items
    (GRID_UNIFORM, 8192, 8192, 65),
    (GRID_TWO_LEVEL, 65537, 1285, 51),    # 2^32 - 1: what the warps take past the end would go beyond 2^32
    (GRID_TWO_LEVEL, 8192, 8192, 32),     # 2^31, and one sample more a pixel
    (GRID_TWO_LEVEL, 8192, 8192, 33),
])
def test_ao_samples_beyond_32_bits_of_items(engine, kind, w, h, spp):
    """A floor that fills the image; samples start 0.01 radii = 1 above it along their
    direction, clear of it, so all of them are free (a triangle below the floor makes the
    scene's box a volume)."""
    import torch
    v = np.array([[-4, -4, 0], [5, -4, 0], [5, 5, 0], [-4, 5, 0], [0.5, 0.5, -2], [0.51, 0.5, -2], [0.5, 0.51, -2]],
                 np.float32)
    f = np.array([[0, 1, 2], [0, 2, 3], [4, 5, 6]], np.uint32)
    engine.upload(v, v, f, 1.0)
    engine.build(kind)
    engine.setCamera((0.5, 0.45, 1.0), (0, 0, -1), (0, 1, 0), 1.0, w, h)
    engine.set_integrator(ao_samples=spp, ao_radius=100.0, seed=3)
    fb = torch.zeros(w * h, 3, device="cuda")
    torch.cuda.synchronize()
    engine.counters(reset=True)
    engine.render_device(fb, 0, RENDER_AO)
    assert engine.counters(reset=True)["rays2"] == w * h * spp
    assert bool((fb == 1.0).all())


@pytest.mark.parametrize("kind", [GRID_TWO_LEVEL, GRID_UNIFORM])
@pytest.mark.parametrize("side,spp", [(1, 1), (3, 31), (3, 33), (5, 3001)])
def test_ao_items_against_the_oracle(engine, oracle, kind, side, spp):
    """Items that do not divide into whole takes."""
    from happyray_b200 import scenes as S
    v, f = S.clusters(2000, seed=4)
    engine.set_uniform_density(5.0)
    engine.setGridDensities(0.0625, 2.0)
    engine.upload(v, v, f, 1.0)
    engine.build(kind)
    v4, bmin, bmax = oracle.lerp_bounds(v, v, 1.0)
    b = (oracle.build_ug(v4, f, bmin, bmax, 5.0, True) if kind == GRID_UNIFORM
         else oracle.build_tl(v4, f, bmin, bmax, 0.0625, 2.0))
    cam = S.camera_at_bounds(v, (side, side))
    args = (cam["position"], cam["orientation"], cam["up"], cam["fov"], side, side)
    engine.setCamera(*args)
    alpha = float(np.float32(0.1) * b.diag())
    engine.set_integrator(ao_samples=spp, ao_radius=alpha, seed=5)
    fb = engine.renderFrame(None, 0, RENDER_AO)
    img, _ = oracle.render_ao(b, oracle.camera(*args), spp, alpha, 5)
    assert np.array_equal(fb[:, 0], img)
