"""Small launches trace with eight lanes per ray (up to 16,384 rays), larger ones
with one: the same rays in one large batch and in small ones give the same hits
and occlusion, bit for bit -- nodes and triangles come in the same order, ties
included -- on soups, on a grid whose vertices and edges the rays meet exactly,
with finite intervals, empty and one-triangle trees, and material flags."""
import numpy as np
import pytest

from vitrum_b200 import bvh as vb
from vitrum_b200 import scenes
from vitrum_b200.engine import Engine, Material, Mesh, Scene

pytestmark = pytest.mark.gpu


def _rays(n, seed):
    r = scenes.sphere_rays(n, seed=seed, target_half=0.9)
    r[::3, 7] = 2.5        # finite intervals
    r[::5, 3] = 2.0        # starting inside
    k = n // 4             # axis-parallel through grid points
    r[:k, 4:7] = 0.0
    r[:k, 6] = -1.0
    r[:k, 0:2] = np.round(r[:k, 0:2] * 4) / 16
    r[:k, 2] = 2.0
    return r


def _meshes():
    p, t = scenes.grid_quad((-1, -1, 0), (2, 0, 0), (0, 2, 0), 32)
    pos = np.zeros((len(p), 4), np.float32)
    pos[:, :3] = p
    idx = np.zeros((len(t), 4), np.uint32)
    idx[:, :3] = t
    one = scenes.random_triangles(1, seed=1, sigma=0.5)
    soup = scenes.random_triangles(20000, seed=2)
    return {"grid": (pos, idx), "one": (one.positions, one.indices), "soup": (soup.positions, soup.indices),
            "empty": (np.zeros((0, 4), np.float32), np.zeros((0, 4), np.uint32))}


@pytest.mark.parametrize("mesh", ["grid", "one", "soup", "empty"])
def test_small_batches_equal_large(cuda, mesh):
    pos, idx = _meshes()[mesh]
    rays = _rays(40000, 5)
    with vb.build_compressed_wide_bvh(pos, idx) as g:
        hits, occ = g.intersect_first_hit(rays), g.intersect_any_hit(rays)
        at = 0
        for n in (1, 7, 16, 17, 1000, 16384, 16385):
            h, o = g.intersect_first_hit(rays[at:at + n]), g.intersect_any_hit(rays[at:at + n])
            assert np.array_equal(h.view(np.uint32), hits[at:at + n].view(np.uint32)), n
            assert np.array_equal(o, occ[at:at + n]), n
            at += n


def test_material_flags(cuda):
    p, t = scenes.grid_quad((-1, -1, 0), (2, 0, 0), (0, 2, 0), 8)
    sc = Scene(meshes=[Mesh(p, t, 0), Mesh(p + np.float32([0, 0, -0.5]), t, 1)],
               materials=[Material(double_sided=False, cast_shadow=False), Material()])
    e = Engine()
    e.set_scene(sc)
    r = _rays(20000, 8)
    r[1::2, 0:3] *= -1
    r[1::2, 4:7] *= -1
    hits, _ = e.trace_rays(r)
    for a, n in ((0, 5000), (5000, 15000)):
        h, _ = e.trace_rays(r[a:a + n])
        assert np.array_equal(h.view(np.uint32), hits[a:a + n].view(np.uint32))
    e.dispose()


@pytest.mark.parametrize("leaf", [1, 2, 4])
@pytest.mark.parametrize("n", [16385, 16400, 20001, 70003])
def test_occlusion_is_a_closest_hit(cuda, n, leaf):
    """A large occlusion batch ends with eight lanes on each of a warp's last rays:
    a segment is occluded just when the same ray has a closest hit -- long rays
    through a loose soup, in leaves of 1 to 4, with warps that hold a few rays
    only and with a trace order."""
    soup = scenes.random_triangles(30000, seed=4)
    rays = _rays(n, 11)
    rays[::7, 3] = 0.0
    rays[::7, 7] = 1e30
    with vb.build_compressed_wide_bvh(soup.positions, soup.indices, maxLeafTriangles=leaf, traversalTree="reference") as g:
        for order in (0, 3):
            g.set_trace_order(order)
            hit = g.intersect_first_hit(rays)["prim"] >= 0
            occ = g.intersect_any_hit(rays)
            assert 0 < hit.sum() < n
            assert np.array_equal(occ.astype(bool), hit), (order, int((occ.astype(bool) != hit).sum()))


@pytest.mark.parametrize("stage", [False, True])
def test_shadow_flags_in_large_waves(cuda, stage):
    """Two samples of 128 x 128 pixels in one wave of 32,768 paths or in two of
    16,384 (eight lanes on every ray): the same image, bit for bit, with geometry
    that casts no shadow."""
    sc, cam = scenes.box_room(wall_cells=8, box_cells=4)
    sc.materials[3].cast_shadow = False
    imgs = []
    for wave in (1 << 14, 1 << 15):
        e = Engine(max_bounces=4, wave_paths=wave)
        e.set_tuning(wave_paths=wave, stage_hot_nodes=stage)
        e.set_scene(sc)
        e.render_frame(cam, 128, 128, samples=2)
        imgs.append(e.capture_frame())
        e.dispose()
    assert imgs[0].max() > 0
    assert np.array_equal(imgs[0], imgs[1])
