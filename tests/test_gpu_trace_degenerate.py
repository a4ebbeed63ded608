"""Rays a batch carries along without meaning them to hit: directions that are
zero, NaN or infinite miss everything and cost next to nothing, and short
directions (axis-parallel segments, rays in the space of a large instance) cull
as unit ones do and hit the same triangles.  A lost cull visits every node:
hundreds of times the batch, so a factor of four tells it from noise."""
import time

import numpy as np
import pytest

from vitrum_b200 import bvh as vb
from vitrum_b200 import scenes
from vitrum_b200.engine import Engine, Instance, Material, Mesh, Scene

pytestmark = pytest.mark.gpu

BAD = np.float32([[0, 0, 0], [-0.0, 0, 0], [np.nan, 0, 1], [1, np.nan, 0], [0, 1, np.nan], [np.inf, 0, 0],
                  [1, -np.inf, 1], [np.nan, np.inf, 0]])


def _rays(n, seed):
    return scenes.sphere_rays(n, seed=seed, target_half=0.9)


def _axis_rays(n, seed):
    r = _rays(n, seed)
    rng = np.random.default_rng(seed)
    k = np.arange(n) % 3
    sign = np.where(rng.random(n) < 0.5, -1.0, 1.0)
    r[:, 0:3] = rng.uniform(-0.9, 0.9, (n, 3))
    r[np.arange(n), k] = -2.0 * sign
    r[:, 4:7] = 0.0
    r[np.arange(n), 4 + k] = sign
    return r.astype(np.float32)


def _seconds(f):
    f()
    best = np.inf
    for _ in range(3):
        t = time.perf_counter()
        f()
        best = min(best, time.perf_counter() - t)
    return best


@pytest.fixture(scope="module")
def soup():
    m = scenes.random_triangles(65536, seed=3)
    with vb.build_compressed_wide_bvh(m.positions, m.indices) as g:
        yield g


@pytest.mark.parametrize("n", [9, 16384, 200000])
def test_unusable_directions_miss_at_no_cost(cuda, soup, n):
    rays = _rays(n, 4)
    mixed = rays.copy()
    at = np.arange(0, n, 7)
    mixed[at, 4:7] = BAD[np.arange(len(at)) % len(BAD)]
    mixed[at, 7] = 3.0
    h, o = soup.intersect_first_hit(mixed), soup.intersect_any_hit(mixed)
    assert (h["prim"][at] == -1).all() and (h["t"][at] == 3.0).all() and not o[at].any()
    rest = np.setdiff1d(np.arange(n), at)
    assert np.array_equal(h[rest].view(np.uint32), soup.intersect_first_hit(rays)[rest].view(np.uint32))
    assert np.array_equal(o[rest], soup.intersect_any_hit(rays)[rest])
    for call in (soup.intersect_first_hit, soup.intersect_any_hit):
        assert _seconds(lambda: call(mixed)) < 4 * _seconds(lambda: call(rays)) + 1e-3


@pytest.mark.parametrize("n", [4096, 200000])
@pytest.mark.parametrize("length", [2.0 ** -20, 2.0 ** -40, 2.0 ** 20])
def test_short_axis_parallel_rays_cull(cuda, soup, n, length):
    unit = _axis_rays(n, 5)
    short = unit.copy()
    short[:, 4:7] *= np.float32(length)
    short[:, 3] /= np.float32(length)      # the interval is in units of the direction
    h, s = soup.intersect_first_hit(unit), soup.intersect_first_hit(short)
    assert (h["prim"] >= 0).mean() > 0.2
    assert np.array_equal(h["prim"], s["prim"])
    hit = h["prim"] >= 0
    assert np.array_equal(h["t"][hit] / np.float32(length), s["t"][hit])   # a power of two: exact
    assert np.array_equal(soup.intersect_any_hit(unit), soup.intersect_any_hit(short))
    for call in (soup.intersect_first_hit, soup.intersect_any_hit):
        assert _seconds(lambda: call(short)) < 4 * _seconds(lambda: call(unit)) + 1e-3


def test_axis_parallel_rays_cull_inside_a_large_instance(cuda):
    m = scenes.random_triangles(65536, seed=3)
    mesh = Mesh(np.ascontiguousarray(m.positions[:, :3]), np.ascontiguousarray(m.indices[:, :3]), 0)
    unit = _axis_rays(100000, 6)
    seconds, prims = [], []
    for scale in (1.0, 2.0 ** 20):
        M = np.diag([scale, scale, scale, 1.0]).astype(np.float32)
        e = Engine()
        e.set_scene(Scene(meshes=[mesh], materials=[Material()], instances=[Instance(0, M, 0)]))
        r = unit.copy()
        r[:, 0:3] *= np.float32(scale)
        h, _ = e.trace_rays(r)
        prims.append(h["prim"].copy())
        seconds.append(_seconds(lambda: e.trace_rays(r)))
        e.dispose()
    assert (prims[0] >= 0).mean() > 0.2
    assert np.array_equal(prims[0], prims[1])
    assert seconds[1] < 4 * seconds[0] + 1e-3
