"""The plane kernel with rows in registers (k_xyplane) at every plane size it is built for, 16 to 128 along each axis, with
boxes as wide as the embedding allows (half of it and its middle) and boxes that end inside a tile: gradient, one trajectory and
its energies against the FP64 oracle at the repository's bars (1e-5, 1e-4), through the kernel's forcing switch.

A short-range covariance keeps 1/lambda within two decades, so that the bars are not about conditioning."""
import numpy as np
import pytest

import dualres_b200 as d
from dualres_b200 import synth

pytestmark = pytest.mark.gpu
WIDE = {16: 9, 32: 17, 64: 33, 128: 65}
INSIDE = {16: 6, 32: 11, 64: 20, 128: 41}


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a) - b) / np.linalg.norm(b))


@pytest.mark.parametrize("e0", [16, 32, 64, 128])
@pytest.mark.parametrize("e1", [16, 32, 64, 128])
@pytest.mark.parametrize("sizes", [WIDE, INSIDE])
def test_plane(oracle, monkeypatch, e0, e1, sizes):
    monkeypatch.setenv("DRB_PLANE_PREFETCH", "1")
    vol = synth.make_volume((sizes[e0], sizes[e1], 3), 1.0, (0.75, 1.0, 1.0), 0.5, 0.3, 2.6, "full", 1.0, 5, dual=False)
    data = d.MultiResData.from_volume(vol)
    assert data.E == (e0, e1, 4)
    ch = d.MultiResParameters(data, d.HMCParameters(burnin=4, nsave=2, thin=1, leapfrog=3, seed=7), 2)
    assert ch.config()["path"] != "lines"
    prep = oracle.prepare(vol.highres)
    m = oracle.Model(prep["D"], prep["Yh"], vol.qform_hr, vol.theta, None, None, prep["O"])
    rng = np.random.default_rng(1)
    mu, p = ((rng.standard_normal(m.shape) + 1j * rng.standard_normal(m.shape)).astype(np.complex64) for _ in range(2))
    ch.set_state(1, mu, (1.5, 1.0))
    m.set_sigma(1.5, 1.0)
    assert rel(ch.gradient(1, mu), m.gradient(mu)) < 1e-5
    mu1, p1, en = ch.leapfrog(1, mu, p, 0.05, 3)
    mu_o, p_o = m.leapfrog(mu, p, 0.05, 3)
    assert rel(mu1, mu_o) < 1e-4 and rel(p1, p_o) < 1e-4
    want = [m.log_prior(mu), m.log_likelihood(mu), m.kinetic(p), m.log_prior(mu_o), m.log_likelihood(mu_o),
            m.kinetic(p_o)]
    assert np.allclose(en, want, rtol=1e-4)
    ch.run()
    assert all(x["done"] for x in ch.stats())
    ch.close(), data.close()
