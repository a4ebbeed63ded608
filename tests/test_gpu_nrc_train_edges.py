"""Training gradients where the four-threads-per-sample division can go wrong:
partial tiles, one more tile than SMs, level counts that leave a thread's four
levels empty or cut them, and every level of the full grid; against the numpy
oracle in fp16 storage, with the bound of the gradient test beside it (3e-2
relative: fp16 activations and deltas of six layers at 2^-11 each, summed)."""
import numpy as np
import pytest

from oracle import nrc as O
from test_gpu_nrc import randomise, training_samples
from vitrum_b200.nrc import NrcConfig, RadianceCache

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,levels", [(1, 16), (127, 5), (129, 1), (129, 13), (1000, 16), (148 * 128 + 1, 4)])
def test_gradients(cuda, n, levels):
    cfg = NrcConfig(levels=levels, log2_table_size=10, base_resolution=4, growth=1.4)
    c = RadianceCache(cfg)
    W, T = randomise(c, 3, w_scale=0.2, t_scale=0.3)
    s = training_samples(n, 5)
    gw, gt, loss = c.gradients(s)
    res = O.level_resolutions(cfg.base_resolution, cfg.growth, cfg.levels)
    dW, dT, oloss = O.gradients(W, O.f16(T), s, res, cfg.aabb_min, cfg.aabb_max)
    for l in range(6):
        assert np.linalg.norm(gw[l] - dW[l]) < 3e-2 * np.linalg.norm(dW[l]) + 1e-30, l
    for l in range(levels):
        assert np.linalg.norm(gt[l] - dT[l]) < 3e-2 * np.linalg.norm(dT[l]) + 1e-30, l
    assert abs(loss - oloss) <= 1e-2 * abs(oloss)
    c.close()
