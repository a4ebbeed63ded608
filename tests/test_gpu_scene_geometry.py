"""Scenes whose geometry is packed on the device (meshes of 512 triangles and
more on average) equal the host pipeline's word for word, with empty meshes in
any place, unused vertices, several emissive meshes and material flags, at mesh
sizes around the line; and what a host-packed scene refuses is refused with the
same message, a first fault before a later one, leaving the old scene set."""
import numpy as np
import pytest

from vitrum_b200 import _native as N
from vitrum_b200 import scenes
from vitrum_b200.engine import Camera, Engine, Material, Mesh, Scene

pytestmark = pytest.mark.gpu

MATS = [Material(), Material(double_sided=False), Material(emission=(4.0, 2.0, 1.0)), Material(cast_shadow=False)]
EMPTY = Mesh(np.zeros((0, 3), np.float32), np.zeros((0, 3), np.uint32), 1)


def _mesh(n_tri, seed, material):
    s = scenes.random_triangles(n_tri, seed=seed)
    p = np.concatenate([s.positions[:, :3], np.float32([[9, 9, 9]])])  # one vertex nobody uses
    return Mesh(p, s.indices[:, :3].copy(), material)


def _export(scene, **kw):
    e = Engine(**kw)
    e.set_scene(scene)
    out = e.export_scene()
    cam = Camera(eye=(0.0, 0.0, 4.0), target=(0.0, 0.0, 0.0))
    e.render_frame(cam, 16, 16, samples=2, bounces=3, frame_seed=3)
    img = e.capture_frame()
    st = e.stats()
    e.dispose()
    return out, img, (st["triangle_count"], st["emitter_count"])


@pytest.mark.parametrize("sizes", [(512,), (511,), (1, 2000), (300, 300), (5000, 600, 3)])
@pytest.mark.parametrize("empty_at", [None, 0, 1, -1])
def test_equals_host(cuda, sizes, empty_at):
    meshes = [_mesh(n, 10 + i, (2, 0, 3, 1)[i % 4]) for i, n in enumerate(sizes)]
    if empty_at is not None:
        meshes.insert(len(meshes) if empty_at < 0 else empty_at, EMPTY)
    sc = Scene(meshes=meshes, materials=MATS)
    (gw, gr), gi, gs = _export(sc)
    (hw, hr), hi, hs = _export(sc, scene_build="host")
    assert np.array_equal(gw, hw) and np.array_equal(gr.view(np.uint32), hr.view(np.uint32))
    assert np.array_equal(gi, hi) and gs == hs


def _fault(kind):
    m = [_mesh(1000, 3, 0), _mesh(1000, 4, 1)]
    if "position" in kind:
        m[0].positions[-1, 1] = np.nan  # the unused vertex
    if "index" in kind:
        m[1].indices[7, 2] = 3001
    if "material" in kind:
        m[1].material = 17
    return Scene(meshes=m, materials=MATS)


@pytest.mark.parametrize("kind", ["position", "index", "material", "position material", "index material"])
def test_refusals(cuda, kind):
    msgs = []
    for build in ("gpu", "host"):
        e = Engine(scene_build=build)
        e.set_scene(Scene(meshes=[_mesh(600, 5, 0)], materials=MATS))
        before = e.export_scene()[0]
        with pytest.raises(N.VtError) as err:
            e.set_scene(_fault(kind))
        msgs.append((err.value.status, str(err.value)))
        assert np.array_equal(e.export_scene()[0], before)
        e.dispose()
    assert msgs[0] == msgs[1]
