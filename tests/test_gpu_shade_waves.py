"""Shading launches small waves in CTAs of 4 warps and waves of 151,552 paths and
more in CTAs of 16 that start each path together: two samples a pixel rendered in
one large wave equal the same two rendered in two small ones, bit for bit (every
path is its own, and 0 + a + b is the same sum either way) -- at the first size
that takes the large CTAs, at ragged ones, and with the material-sorted queue."""
import numpy as np
import pytest

from vitrum_b200 import scenes
from vitrum_b200.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sort", [False, True])
@pytest.mark.parametrize("size", [(512, 148), (401, 199), (397, 330)])
@pytest.mark.parametrize("kind", ["room", "cloud"])
def test_large_and_small_waves_agree(cuda, kind, size, sort):
    w, h = size
    if kind == "room":
        sc, cam = scenes.box_room(wall_cells=8, box_cells=4)
    else:
        sc, cam = scenes.instanced_cloud(n_instances=37, seed=5, sphere_levels=(1, 2, 2, 3), torus_segments=(16, 8),
                                         cube_cells=(2, 3, 4))
    assert w * h < 2 * 148 * 512 <= 2 * w * h
    imgs = []
    for wave in (w * h, 2 * w * h):
        e = Engine(max_bounces=4, wave_paths=wave)
        e.set_tuning(wave_paths=wave, sort_by_material=sort)
        e.set_scene(sc)
        e.render_frame(cam, w, h, samples=2)
        imgs.append(e.capture_frame())
        e.dispose()
    assert np.isfinite(imgs[0]).all() and imgs[0].max() > 0
    assert np.array_equal(imgs[0], imgs[1])
