"""The traversal's triangle decisions on lattice geometry, where almost every ray
meets edges, vertices and planes exactly: small whole coordinates and directions, in
every dominant axis and sign, flat, sliver and degenerate triangles among them.  The
reference test of every triangle against every ray (bit-exact elsewhere) says which
triangles are at the smallest t; the traversal has to return one of those, from both
kernels, and to miss where none is hit.  (Rays in the plane of a triangle that the
test then counts as hit are left out: its t lies anywhere on the line, outside the
triangle's box too, where a tree need not find it.)"""
import numpy as np
import pytest
import torch

from vitrum_b200 import bvh as vb

pytestmark = pytest.mark.gpu

RESULT = np.dtype([("hit", np.int32), ("t", np.float32), ("bary", np.float32, 3), ("side", np.int32),
                   ("mask", np.int32)])


def _nearest(tri, rays):
    """Smallest watertight t of each ray, which triangles have it, the zero-edge masks, and
    whether the test hits a triangle edge-on."""
    n, m = len(rays), len(tri)
    cases = np.zeros((n, m, 16), np.float32)
    cases[:, :, 0:3] = rays[:, None, 0:3]
    cases[:, :, 3:6] = rays[:, None, 4:7]
    cases[:, :, 6:15] = tri.reshape(1, m, 9)
    cases[:, :, 15] = rays[:, None, 3]
    d = torch.from_numpy(cases.reshape(-1, 16)).cuda()
    out = torch.zeros((n * m, RESULT.itemsize // 4), dtype=torch.int32, device="cuda")
    vb.watertight_eval_device(d.data_ptr(), n * m, out.data_ptr())
    torch.cuda.synchronize()
    r = out.cpu().numpy().view(RESULT).reshape(n, m)
    t = np.where(r["hit"] != 0, r["t"], np.inf)
    t = np.where(t < rays[:, None, 7], t, np.inf)
    best = t.min(1)
    e = tri.astype(np.float64)
    normal = np.cross(e[:, 1] - e[:, 0], e[:, 2] - e[:, 0])
    d64 = rays[:, 4:7].astype(np.float64)
    d64 /= np.maximum(np.abs(d64).max(1, keepdims=True), 1e-300)
    edge_on = (np.abs(d64 @ normal.T) < 1e-5) & (r["hit"] != 0)
    return best, (t == best[:, None]) & np.isfinite(t), r["mask"], edge_on.any(1)


@pytest.mark.parametrize("seed", range(6))
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -30])
def test_lattice_hits(cuda, seed, scale):
    rng = np.random.default_rng(seed)
    tri = rng.integers(-4, 5, (150, 3, 3)).astype(np.float32)
    if seed % 2:                                     # and a lattice plane of shared edges
        tri[:50, :, seed % 3] = 0.0
    pos = np.zeros((450, 4), np.float32)
    pos[:, :3] = tri.reshape(-1, 3)
    idx = np.zeros((150, 4), np.uint32)
    idx[:, :3] = np.arange(450).reshape(150, 3)
    n = 3000
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:3] = rng.integers(-8, 9, (n, 3))
    rays[:, 4:7] = rng.integers(-3, 4, (n, 3)) * np.float32(scale)
    rays[::5, 4:7] *= rng.uniform(0.1, 3.0, (len(rays[::5]), 1)).astype(np.float32)
    rays[:, 7] = np.where(rng.random(n) < 0.2, 3.0 / scale, np.inf)
    rays[::7, 3] = 1.0 / scale
    best, at_best, mask, edge_on = _nearest(tri, rays)
    assert (mask[at_best] != 0).mean() > 0.2         # edges and vertices were met
    with vb.build_compressed_wide_bvh(pos, idx) as g:
        small, occ = g.intersect_first_hit(rays), g.intersect_any_hit(rays)
        large = g.intersect_first_hit(np.concatenate([rays] * 6))[:n]
        assert np.array_equal(small.view(np.uint32), large.view(np.uint32))
    assert edge_on.mean() < 0.01
    hit = np.isfinite(best)
    assert 0.1 < hit.mean() < 1.0
    assert np.array_equal((small["prim"] >= 0) | edge_on, hit | edge_on) and np.array_equal(occ | edge_on, hit | edge_on)
    k = np.flatnonzero(hit & ~edge_on)
    assert at_best[k, small["prim"][k]].all()
