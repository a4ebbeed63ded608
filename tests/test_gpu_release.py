"""Releasing a tree or replacing a scene while the device is in use: work in flight
is waited for, and a stream another thread is capturing (thread-local mode, as the
engine captures its own frames) is left alone."""
import threading

import numpy as np
import pytest
import torch

from vitrum_b200 import bvh as vb
from vitrum_b200 import scenes
from vitrum_b200.engine import Engine

pytestmark = pytest.mark.gpu


def _tree():
    m = scenes.random_triangles(5000, seed=3)
    return vb.build_compressed_wide_bvh(m.positions, m.indices)


def test_release_waits_for_work_in_flight(cuda):
    rays = torch.from_numpy(scenes.sphere_rays(100000, seed=4)).cuda()
    hits = torch.empty((len(rays), 4), dtype=torch.int32, device="cuda")
    g = _tree()
    want = g.intersect_first_hit(rays.cpu().numpy())
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(100_000_000)     # some 50 ms
        g.trace_closest_device(rays.data_ptr(), len(rays), hits.data_ptr(), side.cuda_stream)
    assert not side.query()
    g.close()
    assert side.query()
    assert np.array_equal(hits.cpu().numpy(), want.view(np.int32).reshape(-1, 4))


def _close_tree(kept):
    kept["tree"].close()


def _replace_scene(kept):
    kept["engine"].set_scene(kept["other"])


def _dispose(kept):
    kept["engine"].dispose()


@pytest.mark.parametrize("release", [_close_tree, _replace_scene, _dispose])
def test_release_leaves_another_threads_capture_alone(cuda, release):
    room, cam = scenes.box_room(wall_cells=8, box_cells=4)
    other, _ = scenes.box_room(wall_cells=6, box_cells=3)
    kept = {"tree": _tree(), "engine": Engine(max_bounces=2), "other": other}
    kept["engine"].set_scene(room)
    kept["engine"].render_frame(cam, 16, 16, samples=1)
    x = torch.arange(1 << 16, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    graph, errors = torch.cuda.CUDAGraph(), []

    def work():
        try:
            release(kept)
        except Exception as e:                  # noqa: BLE001 -- handed to the test
            errors.append(e)

    with torch.cuda.graph(graph, capture_error_mode="thread_local"):
        y = x * 2
        t = threading.Thread(target=work)
        t.start()
        t.join()
        y = y + 1
    graph.replay()
    torch.cuda.synchronize()
    assert not errors, errors
    assert torch.equal(y, x * 2 + 1)
    kept["tree"].close()
    if release is not _dispose:
        kept["engine"].dispose()
