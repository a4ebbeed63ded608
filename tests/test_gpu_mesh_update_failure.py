"""A mesh update that runs out of device memory leaves the scene as it was, at
whichever allocation it fails: the scene's words (compared before anything is
traced through them), its hits and its image are those from before, and the same
update succeeds afterwards.  The failures are injected on the host."""
import dataclasses

import numpy as np
import pytest

from vitrum_b200 import _native as N
from vitrum_b200 import scenes
from vitrum_b200.engine import Engine, Mesh, debug_fail_device_allocation

from test_gpu_instance_update import rays_at, small_cloud

pytestmark = pytest.mark.gpu

VT_ERR_OUT_OF_MEMORY = 4


def _larger(sc):
    p, t = scenes.icosphere(4)
    return 1, Mesh(p * np.float32(0.8), t, sc.meshes[1].material)


def _smaller(sc):
    p, t = scenes.box_mesh((-0.5, -0.5, -0.5), (0.5, 0.5, 0.5), 1)
    return 0, Mesh(p, t, sc.meshes[0].material)


@pytest.mark.parametrize("rebuild", [False, True])
@pytest.mark.parametrize("change", [_larger, _smaller])
def test_failed_mesh_update_keeps_the_scene(cuda, change, rebuild):
    sc, cam = small_cloud()
    at, mesh = change(sc)
    rays = rays_at(1 << 14, 9)

    def state(e):
        words = [np.array(a) for a in e.export_scene()]
        h, ii = e.trace_rays(rays)
        e.reset()
        e.render_frame(cam, 32, 24, samples=4, frame_seed=5)
        return words, h.tobytes(), ii.tobytes(), e.capture_frame().tobytes()

    e = Engine(max_bounces=4)
    e.set_scene(sc)
    before = state(e)
    stages = 0
    for k in range(1, 400):
        debug_fail_device_allocation(k)
        try:
            e.update_mesh(at, mesh, rebuild=rebuild)
        except N.VtError as err:
            assert err.status == VT_ERR_OUT_OF_MEMORY and "injected" in str(err)
            stages += 1
        else:
            break
        finally:
            debug_fail_device_allocation(0)
        for a, b in zip(e.export_scene(), before[0]):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), k
        assert state(e)[1:] == before[1:], k
    assert stages >= 10, stages
    meshes = list(sc.meshes)
    meshes[at] = mesh
    f = Engine(max_bounces=4)
    f.set_scene(dataclasses.replace(sc, meshes=meshes))
    f.update_instances(sc.instances, rebuild=rebuild)
    h, _ = e.trace_rays(rays)
    hf, _ = f.trace_rays(rays)
    assert (h["prim"] == hf["prim"]).mean() > 0.9999
    e.dispose()
    f.dispose()
