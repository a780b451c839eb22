"""The plane kernels with 256 threads, which chain sets of more planes than SMs run: k_xyplane at every pair of sides 16 to 128
(the other tests of these sizes have few planes and run its 512 threads) and k_plane_square at 4 to 64.  Gradient, one
trajectory and its energies of the first and the last chain against the FP64 oracle at the repository's bars (1e-5, 1e-4);
embedding, covariance and boxes are test_gpu_plane_sizes.py's."""
import numpy as np
import pytest

import dualres_b200 as d
from dualres_b200 import synth
from test_gpu_plane_sizes import INSIDE, WIDE, rel

pytestmark = pytest.mark.gpu
CHAINS = 60  # x 3 planes (E2 = 4): more than the 148 SMs


def _check(oracle, dims, E):
    vol = synth.make_volume(dims, 1.0, (0.75, 1.0, 1.0), 0.5, 0.3, 2.6, "full", 1.0, 5, dual=False)
    data = d.MultiResData.from_volume(vol)
    assert data.E == E and (E[2] // 2 + 1) * CHAINS > 148
    ch = d.MultiResParameters(data, d.HMCParameters(burnin=4, nsave=2, thin=1, leapfrog=3, seed=7), CHAINS)
    assert ch.config()["path"] != "lines"
    prep = oracle.prepare(vol.highres)
    m = oracle.Model(prep["D"], prep["Yh"], vol.qform_hr, vol.theta, None, None, prep["O"])
    m.set_sigma(1.5, 1.0)
    rng = np.random.default_rng(1)
    for c in (0, CHAINS - 1):
        mu, p = ((rng.standard_normal(m.shape) + 1j * rng.standard_normal(m.shape)).astype(np.complex64) for _ in range(2))
        ch.set_state(c, mu, (1.5, 1.0))
        assert rel(ch.gradient(c, mu), m.gradient(mu)) < 1e-5
        mu1, p1, en = ch.leapfrog(c, mu, p, 0.05, 3)
        mu_o, p_o = m.leapfrog(mu, p, 0.05, 3)
        assert rel(mu1, mu_o) < 1e-4 and rel(p1, p_o) < 1e-4
        want = [m.log_prior(mu), m.log_likelihood(mu), m.kinetic(p), m.log_prior(mu_o), m.log_likelihood(mu_o),
                m.kinetic(p_o)]
        assert np.allclose(en, want, rtol=1e-4)
    ch.run()
    assert all(x["done"] for x in ch.stats())
    ch.close(), data.close()


@pytest.mark.parametrize("e0", [16, 32, 64, 128])
@pytest.mark.parametrize("e1", [16, 32, 64, 128])
@pytest.mark.parametrize("sizes", [WIDE, INSIDE])
def test_rows_in_registers(oracle, monkeypatch, e0, e1, sizes):
    monkeypatch.setenv("DRB_PLANE_PREFETCH", "1")
    _check(oracle, (sizes[e0], sizes[e1], 3), (e0, e1, 4))


@pytest.mark.parametrize("e,n", [(4, 3), (8, 5), (8, 4), (16, 9), (16, 6), (32, 17), (32, 11), (64, 33), (64, 20)])
def test_square_planes(oracle, monkeypatch, e, n):
    monkeypatch.setenv("DRB_AUTOTUNE", "0")
    monkeypatch.delenv("DRB_PLANE_PREFETCH", raising=False)
    _check(oracle, (n, n, 3), (e, e, 4))
