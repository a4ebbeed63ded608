"""The GPU binary build at the sizes where its regimes meet -- subtrees built
whole in shared memory (up to 256 triangles; up to eight per direct evaluation),
larger nodes in chunks of 512 -- over bin counts around a warp's 32 lanes and
geometry that takes every decision: spread soups, clusters of coincident
centroids (sorted halves in both regimes), flat and collinear sets, zeros of
both signs.  Word for word the host build."""
import numpy as np
import pytest

from test_gpu_build import both

pytestmark = pytest.mark.gpu


def _mesh(kind, n, seed):
    rng = np.random.default_rng(seed)
    cen = rng.uniform(-1, 1, (n, 1, 3))
    off = rng.normal(0, 0.02, (n, 3, 3))
    if kind == "clusters":          # few distinct centroids, triangles of different shapes around them
        cen = rng.uniform(-1, 1, (max(1, n // 40), 1, 3))[rng.integers(0, max(1, n // 40), n)]
        off = rng.choice([-0.5, 0.0, 0.25], (n, 3, 3))
    elif kind == "flat":            # one axis without extent, zeros of both signs
        cen[:, :, 1] = 0.0
        off[:, :, 1] = rng.choice([0.0, -0.0], (n, 3))
    elif kind == "line":            # centroids along one axis, equal boxes across it
        cen[:, :, 1:] = 0.0
        off = np.broadcast_to(np.array([[0, 0, 0], [0.1, 0.1, 0], [0.0, 0.1, 0.1]]), (n, 3, 3))
    elif kind == "same":            # one triangle over and over
        cen[:] = 0.25
        off[:] = off[:1]
    v = (cen + off).reshape(-1, 3).astype(np.float32)
    pos = np.zeros((3 * n, 4), np.float32)
    pos[:, :3] = v
    idx = np.zeros((n, 4), np.uint32)
    idx[:, :3] = np.arange(3 * n, dtype=np.uint32).reshape(n, 3)
    return pos, idx


@pytest.mark.parametrize("kind", ["soup", "clusters", "flat", "line", "same"])
@pytest.mark.parametrize("n", [2, 8, 9, 33, 255, 256, 257, 512, 513, 1025, 5000])
def test_sizes(cuda, kind, n):
    pos, idx = _mesh(kind, n, n)
    (hn, hr), (dn, dr), _ = both(pos, idx)
    assert np.array_equal(hn, dn) and np.array_equal(hr, dr)


@pytest.mark.parametrize("bins", [2, 31, 32, 33, 64, 255, 256])
@pytest.mark.parametrize("leaf", [1, 4])
def test_bins(cuda, bins, leaf):
    for kind in ("soup", "clusters"):
        pos, idx = _mesh(kind, 1500, bins)
        (hn, hr), (dn, dr), _ = both(pos, idx, binCount=bins, maxLeafTriangles=leaf)
        assert np.array_equal(hn, dn) and np.array_equal(hr, dr)
