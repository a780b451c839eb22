"""|S| counts the modes that are masked: those whose eigenvalue, taken as the mean of lambda(k) and lambda(-k) (one number, which
the transform leaves a rounding apart), is not positive.  The covariances 1 - b d^e with b near the unit roundoff of 64 bits put
most eigenvalues within rounding of zero."""
import numpy as np
import pytest

import dualres_b200 as d
from dualres_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(8, 8, 8), (17, 9, 12)])
@pytest.mark.parametrize("theta", [(1.0, 1e-15, 1.0), (1.0, 1e-14, 0.7), (0.8, 0.3, 1.0)])
def test_count_of_masked_modes(dims, theta):
    vol = synth.make_volume(dims, 1.0, (0.75, 0.25, 1.0), 0.5, 0.3, 2.3, "full", 1.0, 1, dual=False)
    vol.theta = theta
    data = d.MultiResData.from_volume(vol)
    lam = data.lambda_re()
    mirrored = lam[np.ix_(*[(-np.arange(n)) % n for n in lam.shape])]
    assert data.info.n_nonpositive == np.count_nonzero(0.5 * (lam + mirrored) <= 0)
    data.close()
