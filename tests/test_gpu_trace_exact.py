"""The traversal's watertight test and slab culling where their shortcuts can go
wrong, against the CPU oracle's f32 watertight query: rays through vertices and
edges (zero edge functions), along every dominant axis and sign, with equal
dominant components, axis-parallel rays, near-grazing planes, scaled directions
and scenes far from unit size.  Decisions are f32-exact on both sides, so the
hit triangles are equal except where two hits tie in f32 t."""
import numpy as np
import pytest

import oracle
from oracle import parity
from vitrum_b200 import bvh as vb
from vitrum_b200 import scenes

pytestmark = pytest.mark.gpu


def _grid_rays(axis, sign, n, size, rng):
    """Rays onto the n x n grid of a quad normal to `axis`: through vertices, edge
    midpoints, diagonals and random points, perpendicular, oblique and diagonal."""
    u = rng.integers(0, 2 * n + 1, (600, 2)) / (2.0 * n)
    u[400:] = rng.random((200, 2))
    tgt = np.zeros((600, 3))
    tgt[:, (axis + 1) % 3], tgt[:, (axis + 2) % 3] = u[:, 0], u[:, 1]
    d = np.zeros((600, 3))
    d[:, axis] = sign
    k = np.arange(600) % 4
    off = rng.choice([-0.5, -0.25, 0.25, 0.5], (600, 2))
    d[:, (axis + 1) % 3] = np.where(k == 1, off[:, 0], np.where(k == 2, 1.0, np.where(k == 3, 1e-22, 0.0)))
    d[:, (axis + 2) % 3] = np.where(k == 1, off[:, 1], np.where(k == 2, -1.0, 0.0))
    o = tgt * size - d * (2.0 * size)
    return np.concatenate([o, np.full((600, 1), 0.0), d, np.full((600, 1), np.inf)], 1).astype(np.float32)


@pytest.mark.parametrize("size", [1.0, 2.0 ** -20, 2.0 ** 24])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -90, 2.0 ** 60])
def test_edges_and_axes(cuda, size, scale):
    rng = np.random.default_rng(7)
    n = 4
    pos, idx, rays = [], [], []
    for axis in range(3):
        eu, ev = np.zeros(3), np.zeros(3)
        eu[(axis + 1) % 3], ev[(axis + 2) % 3] = size, size
        p, t = scenes.grid_quad(np.zeros(3), eu, ev, n)
        idx.append(t + sum(len(x) for x in pos))
        pos.append(p)
        for sign in (1.0, -1.0):
            rays.append(_grid_rays(axis, sign, n, size, rng))
    p4 = np.zeros((sum(len(x) for x in pos), 4), np.float32)
    p4[:, :3] = np.concatenate(pos)
    i4 = np.zeros((sum(len(x) for x in idx), 4), np.uint32)
    i4[:, :3] = np.concatenate(idx)
    r = np.concatenate(rays)
    r[:, 4:7] *= np.float32(scale)
    with vb.build_compressed_wide_bvh(p4, i4) as g:
        hits = g.intersect_first_hit(r)
        occ = g.intersect_any_hit(r)
    w = oracle.build_compressed_wide_bvh(p4, i4)
    wp, wt, _ = oracle.first_hit_watertight(w, p4, r)
    assert np.array_equal(hits["prim"] >= 0, wp >= 0)
    assert np.array_equal(occ, wp >= 0)
    both = (hits["prim"] != wp) & (wp >= 0)
    # another triangle only at the same f32 t: the two share the vertex or edge the ray meets
    soup = scenes.TriangleSoup(p4, i4)
    ties, errors = parity.watertight_disagreements(soup.positions, soup.indices, r, hits["prim"], wp)
    assert not errors, (errors[:5], int(both.sum()))
    assert (wp >= 0).sum() > 1000


def test_grazing_side(cuda):
    """Directions within a few ulps of the plane of a triangle: the side check decides."""
    rng = np.random.default_rng(3)
    soup = scenes.random_triangles(64, seed=9, sigma=0.3)
    v = soup.positions[:, :3].reshape(-1, 3, 3).astype(np.float64)
    k = rng.integers(0, 64, 4000)
    a, b, c = v[k, 0], v[k, 1], v[k, 2]
    nrm = np.cross(b - a, c - a)
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    d = (b - a) * rng.random((4000, 1)) + (c - a) * (rng.random((4000, 1)) + 0.1)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    d += nrm * (rng.choice([-1.0, 1.0], (4000, 1)) * 10.0 ** rng.uniform(-9, -3, (4000, 1)))
    tgt = a + (b - a) * 0.3 + (c - a) * 0.3
    r = np.concatenate([tgt - 2 * d, np.full((4000, 1), 1e-4), d, np.full((4000, 1), np.inf)], 1).astype(np.float32)
    with vb.build_compressed_wide_bvh(soup.positions, soup.indices) as g:
        hits = g.intersect_first_hit(r)
    w = oracle.build_compressed_wide_bvh(soup.positions, soup.indices)
    wp, _, _ = oracle.first_hit_watertight(w, soup.positions, r)
    ties, errors = parity.watertight_disagreements(soup.positions, soup.indices, r, hits["prim"], wp)
    assert not errors, errors[:5]
