"""The minimum-contrast summary at the edges of its tiles: rows that are shorter than a step of 4 voxels or than the 25
voxels of the longest offset, lengths around the 32 bits of a mask word, images of one row or one plane, rows without data, NaN, and
values below zero.  Counts and distances equal the oracle's; the sums are the same FP64 products in another order: within
1e-12 of the sum of their magnitudes."""
import numpy as np
import pytest

from dualres_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 1, 3), (2, 3, 4), (1, 30, 5), (27, 1, 31), (3, 5, 32), (4, 3, 33),
                                   (5, 7, 63), (9, 6, 97)])
def test_edges(oracle, shape):
    rng = np.random.default_rng(sum(shape))
    img = rng.standard_normal(shape).astype(np.float32)
    img[rng.random(shape) < 0.3] = 0
    img[rng.random(shape) < 0.1] = np.nan
    if shape[1] > 2:
        img[:, 1] = 0
    Q = np.diag([1.0, 1.5, 2.0, 1.0]).astype(np.float32)
    g, o = api.mce_summary(img, Q, with_sums=True), oracle.mce_summary(img, Q)
    assert np.array_equal(g["npairs"], o["npairs"]) and np.array_equal(g["distance"], o["distance"])
    v = np.abs(np.nan_to_num(img)).astype(np.float64)
    assert np.max(np.abs(g["sums"] - o["sums"])) <= 1e-12 * max(1.0, v.sum(), (v * v).sum())
