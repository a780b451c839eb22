"""The minimum-contrast summary of images with infinite voxels: an infinite voxel takes part in the sums of the offsets that pair
it with a voxel of the mask, and in no others (0 * inf, with a masked voxel or the padding, would be NaN at every offset).

Counts equal the oracle's; each sum and covariance that is finite there is finite here, within 1e-12 of the sum of the
magnitudes of the finite values, and the others are the same infinity or NaN."""
import numpy as np
import pytest

from dualres_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 3), (4, 3, 33), (27, 1, 31), (9, 6, 97)])
@pytest.mark.parametrize("values", [(np.inf,), (-np.inf,), (np.inf, -np.inf), (np.inf, np.inf, np.nan, -np.inf, np.inf)])
def test_infinite_voxels(oracle, shape, values):
    rng = np.random.default_rng(sum(shape))
    img = rng.standard_normal(shape).astype(np.float32)
    img[rng.random(shape) < 0.4] = 0
    img.ravel()[rng.choice(img.size, min(len(values), img.size), replace=False)] = values[:img.size]
    Q = np.diag([1.0, 1.5, 2.0, 1.0]).astype(np.float32)
    g, o = api.mce_summary(img, Q, with_sums=True), oracle.mce_summary(img, Q)
    assert np.array_equal(g["npairs"], o["npairs"])
    v = np.abs(np.where(np.isfinite(img), img, 0)).astype(np.float64)
    for a, b in ((g["sums"], o["sums"]), (g["covariance"], o["covariance"])):
        fine = np.isfinite(b)
        assert np.array_equal(fine, np.isfinite(a)) and np.array_equal(a[~fine], b[~fine], equal_nan=True)
    fine = np.isfinite(o["sums"])
    assert fine.sum() > fine.size // 2
    assert np.max(np.abs(g["sums"][fine] - o["sums"][fine])) <= 1e-12 * max(1.0, v.sum(), (v * v).sum())
