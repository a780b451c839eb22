"""Kriging weights solved on the device against the host builder at system sizes around the solver's blocks: panels
of 32 columns in groups of 8, product tiles of 64, and neighbourhoods from 7 to 257 voxels, complete (K^-1 alone) and
cut by a mask that leaves rows with any number of absent voxels.  Both sides solve in FP64 and round each weight to
float, so two weights differ by at most one rounding of a float: 2^-23 of its size."""
import numpy as np
import pytest

import dualres_b200 as d
from dualres_b200 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius", [1.2, 1.8, 2.1, 2.6, 3.1, 3.5, 4.01])
@pytest.mark.parametrize("fill", [1.0, 0.6])
def test_weights_match_host_builder(radius, fill):
    vol = synth.make_volume((13, 11, 12), 1.0, (0.9, 0.4, 1.0), 0.5, 0.3, radius, "ellipsoid", 0.8, 3)
    if fill < 1.0:
        keep = np.random.default_rng(5).random(vol.highres.shape) < fill
        vol.highres = np.where(keep, vol.highres, 0.0).astype(np.float32)
    hr = np.where(vol.hmask == 0, 0, vol.highres) if vol.hmask is not None else vol.highres
    hrp, hcol, hval = api.kriging_matrix(hr, vol.qform_hr, vol.stdres, vol.qform_sr, vol.theta, vol.radius)
    dv = d.MultiResData.from_volume(vol)
    rp, col, val = dv.W()
    dv.close()
    assert np.array_equal(rp, hrp) and np.array_equal(col, hcol)
    sizes = np.diff(rp)
    assert sizes.max() > 0
    assert np.all(np.abs(val.astype(np.float64) - hval) <= 2.0 ** -23 * np.abs(hval) + 1e-12)
