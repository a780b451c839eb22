"""The row-group products with counts of chains that are no multiple of 4: lanes then take their 4 chains in rounds of one or two.
Every width of an entry's group of lanes, first and last count of each; few groups and more than 8 per SM.  The oracle and the
tolerance are test_gpu_row_products.py's."""
import numpy as np
import pytest

import dualres_b200 as d
from dualres_b200 import synth
from test_gpu_row_products import _dense, _products

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def row_groups(monkeypatch):
    monkeypatch.setenv("DRB_AUTOTUNE", "0")
    monkeypatch.setenv("DRB_TC_PRODUCTS", "0")


@pytest.mark.parametrize("chains", [7, 9, 10, 14, 15, 17, 18, 31, 34, 62, 63, 65, 126, 127, 129, 254])
def test_rounds(chains):
    data = d.MultiResData.from_volume(synth.small_volume(seed=82, dims=(11, 10, 9), radius=3.6))
    W = _dense(data)
    ch = d.MultiResParameters(data, d.HMCParameters(burnin=2, nsave=1, thin=1, leapfrog=2, seed=1), chains)
    rng = np.random.default_rng(chains)
    for c in {0, 1, 4, chains // 2, chains - 1}:
        mu = (4 * rng.standard_normal(data.shape)).astype(np.complex64)
        sq, wt, sq_x, wt_x = _products(data, ch, c, mu, W)
        assert abs(sq / sq_x - 1) < 1e-5
        assert np.linalg.norm(wt - wt_x) < 1e-5 * np.linalg.norm(wt_x)
    ch.run()
    assert all(x["done"] for x in ch.stats())
    ch.close(), data.close()


@pytest.mark.parametrize("chains", [3, 5, 6, 9, 10, 33])
def test_rounds_with_many_groups(chains):
    data = d.MultiResData.from_volume(synth.make_volume((44, 41, 40), 1.0, (0.75, 0.25, 1.0), 0.5, 0.3, 2.3, "full", 1.0, 4))
    assert data.n_stdres > 4 * 8 * 148
    rp, col, val = data.W()
    ys, flat = data.data()[1], data.indices()[0]
    ch = d.MultiResParameters(data, d.HMCParameters(burnin=2, nsave=1, thin=1, leapfrog=2, seed=1), chains)
    mu = (4 * np.random.default_rng(5).standard_normal(data.shape)).astype(np.complex64)
    m = mu.ravel()[flat].real.astype(np.float64)
    wm = np.add.reduceat(np.append(val.astype(np.float64) * m[col], 0.0), rp[:-1])
    wm[rp[1:] == rp[:-1]] = 0.0
    rs = ys.astype(np.float64) - wm
    for c in (0, chains - 1):
        ch.set_state(c, mu, (0.0, 1.0))
        assert abs(ch.log_prior_likelihood(c, mu)[1] / (-0.5 * rs @ rs) - 1) < 1e-5
    ch.close(), data.close()
