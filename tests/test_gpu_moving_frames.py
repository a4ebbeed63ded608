"""Frames between instance updates: the launches captured for the first frame are
replayed after later updates where nothing they hold has changed, so every frame
equals the one an engine renders that captured nothing before its updates -- as
placements scatter and gather (the top level's encoding changes size), with
refits and rebuilds, staged nodes and every trace order."""
import dataclasses

import numpy as np
import pytest

from vitrum_b200 import _native as N
from vitrum_b200 import scenes
from vitrum_b200.engine import Engine, Instance, debug_fail_device_allocation

pytestmark = pytest.mark.gpu


def _placements(base, k):
    rng = np.random.default_rng(k)
    out = []
    for inst in base:
        M = np.asarray(inst.local_to_world, np.float32).copy()
        M[:3, 3] *= (1.0, 0.2, 2.5, 0.05)[k % 4]
        M[:3, 3] += rng.uniform(-1, 1, 3).astype(np.float32)
        out.append(Instance(mesh=int(rng.integers(0, 8)), local_to_world=M, material=inst.material))
    return out


@pytest.mark.parametrize("tuning", [dict(), dict(stage_hot_nodes=True), dict(sort_rays=2), dict(sort_rays=3)])
def test_frames_after_updates(cuda, tuning):
    sc, cam = scenes.instanced_cloud(n_instances=37, seed=5, sphere_levels=(1, 2, 2, 3), torus_segments=(16, 8),
                                     cube_cells=(2, 3, 4))
    sc = dataclasses.replace(sc)
    steps = [(_placements(sc.instances, k), k == 2) for k in range(5)]

    def engine():
        e = Engine(max_bounces=3, wave_paths=1 << 16)
        e.set_tuning(wave_paths=1 << 16, **tuning)
        e.set_scene(sc)
        return e

    def frame(e):
        e.render_frame(cam, 48, 32, samples=4, frame_seed=9)
        return e.capture_frame()

    a = engine()
    frame(a)
    for k in range(len(steps)):
        a.update_instances(*steps[k])
        got = frame(a)
        b = engine()
        for s in steps[:k + 1]:
            b.update_instances(*s)
        assert np.array_equal(got, frame(b)), k
        assert all(np.array_equal(x, y) for x, y in zip(a.export_scene(), b.export_scene())), k
        b.dispose()
    a.dispose()


def test_failed_update_keeps_the_scene(cuda):
    """An update that runs out of device memory, at any of its allocations (the
    first scattering outgrows the arrays), leaves the frame as it was."""
    sc, cam = scenes.instanced_cloud(n_instances=37, seed=5, sphere_levels=(1, 2, 2, 3), torus_segments=(16, 8),
                                     cube_cells=(2, 3, 4))

    def frame(e):
        e.reset()
        e.render_frame(cam, 48, 32, samples=4, frame_seed=9)
        return e.capture_frame()

    e = Engine(max_bounces=3, wave_paths=1 << 16, debug=True)
    e.set_scene(sc)
    want = frame(e)
    stages = 0
    for k in range(1, 200):
        debug_fail_device_allocation(k)
        try:
            e.update_instances(_placements(sc.instances, 2), True)
        except N.VtError as err:
            assert err.status == 4 and "injected" in str(err)
            stages += 1
            assert np.array_equal(frame(e), want), k
            continue
        finally:
            debug_fail_device_allocation(0)
        break
    assert stages >= 5, stages
    assert not np.array_equal(frame(e), want)
    e.dispose()
