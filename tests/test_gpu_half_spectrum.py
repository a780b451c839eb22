"""The half-spectrum state (planes kz = 0 .. E2/2 of the spectra of Re mu and Im mu) on embeddings where its
self-conjugate planes, pair lines and tiles are at their edges: axes of length 2, one plane between the
self-conjugate ones, pair lines that do not fill a tile, chain groups of 8 that are not full.

Position and momentum are complex white fields, so both spectra and every plane carry weight.  The covariance
parameters are exact in 32 bits, as the library holds them.  Tolerances are the repository's bars against the FP64 oracle: gradient 1e-5, energies 1e-5, leapfrog 1e-4 (norm-wise relative)."""
import numpy as np
import pytest

import dualres_b200 as d
from dualres_b200 import synth

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a) - b) / np.linalg.norm(b))


@pytest.mark.parametrize("dims,dual", [((2, 2, 2), False), ((3, 2, 9), False), ((9, 5, 3), True), ((5, 17, 2), False),
                                       ((7, 6, 33), True), ((34, 3, 5), True), ((13, 33, 9), True)])
@pytest.mark.parametrize("chains,ztile", [(1, 8), (9, 8), (9, 1)])
@pytest.mark.parametrize("lines", [False, True])
def test_gradient_and_leapfrog(oracle, monkeypatch, dims, dual, chains, ztile, lines):
    monkeypatch.setenv("DRB_AUTOTUNE", "0")
    monkeypatch.setenv("DRB_ZTILE", str(ztile))
    if lines:
        monkeypatch.setenv("DRB_NO_PLANE", "1")
    vol = synth.make_volume(dims, 1.0, (0.75, 0.25, 1.0), 0.5, 0.3, 2.6, "full", 1.0, 5, dual=dual)
    data = d.MultiResData.from_volume(vol)
    ch = d.MultiResParameters(data, d.HMCParameters(burnin=4, nsave=2, thin=1, leapfrog=3, seed=7), chains)
    prep = oracle.prepare(vol.highres)
    ys = W = None
    if dual:
        rp, col, val = data.W()
        ys, W = data.data()[1], (rp, col, val.astype(np.float64))
    m = oracle.Model(prep["D"], prep["Yh"], vol.qform_hr, vol.theta, ys, W, prep["O"])
    rng = np.random.default_rng(1)
    mu, p = ((rng.standard_normal(m.shape) + 1j * rng.standard_normal(m.shape)).astype(np.complex64) for _ in range(2))
    c = chains - 1
    ch.set_state(c, mu, (1.5, 3.0))
    m.set_sigma(1.5, 3.0)
    back, s = ch.get_state(c)
    assert rel(back, mu) < 1e-6 and tuple(s) == (1.5, 3.0)
    lp, ll = ch.log_prior_likelihood(c, mu)
    assert abs(lp / m.log_prior(mu) - 1) < 1e-5 and abs(ll / m.log_likelihood(mu) - 1) < 1e-5
    assert rel(ch.gradient(c, mu), m.gradient(mu)) < 1e-5
    mu1, p1, en = ch.leapfrog(c, mu, p, 0.05, 3)
    mu_o, p_o = m.leapfrog(mu, p, 0.05, 3)
    assert rel(mu1, mu_o) < 1e-4 and rel(p1, p_o) < 1e-4
    want = [m.log_prior(mu), m.log_likelihood(mu), m.kinetic(p), m.log_prior(mu_o), m.log_likelihood(mu_o),
            m.kinetic(p_o)]
    assert np.allclose(en, want, rtol=1e-4)
    ch.run()
    assert all(x["done"] for x in ch.stats()) and np.isfinite(ch.summary(-1)["mean"]).all()
    ch.close(), data.close()


def test_checkpoint_of_the_full_spectrum_is_still_read():
    """A version-1 checkpoint holds each chain's spectrum u = N IFFT(mu) on all N modes, and the accepted mu at the
    data and output voxels in either half (here in both); restoring it gives the state it was written from, to the
    rounding of one split, and the fit goes on as the other one does."""
    vol = synth.small_volume(seed=9, dims=(9, 8, 6))
    data = d.MultiResData.from_volume(vol)
    hmc = d.HMCParameters(burnin=4, nsave=4, thin=1, leapfrog=3, seed=2)
    a = d.MultiResParameters(data, hmc, 2)
    a.update(3)
    ck = a.checkpoint()
    head = np.frombuffer(ck[:64], np.int64).copy()
    nh = data.N // data.shape[0] * (data.shape[0] // 2 + 1)
    assert head[1] == 3 and head[3] == data.N
    head[1] = 1
    u = [(np.fft.ifftn(a.get_state(c)[0].astype(np.complex128)) * data.N).astype(np.complex64) for c in range(2)]
    at = 64 + 2 * 2 * nh * 8
    halves = []
    for n in (data.n_highres, data.n_output):
        mu = ck[at:at + n * 2 * 4]
        halves.append(mu + mu)
        at += 2 * len(mu)
    b = d.MultiResParameters(data, hmc, 2)
    b.restore(head.tobytes() + b"".join(x.tobytes() for x in u) + b"".join(halves) + ck[at:])
    for steps in (0, 2):
        a.update(steps), b.update(steps)
        for c in range(2):
            (mu, s), (want, t) = b.get_state(c), a.get_state(c)
            assert rel(mu, want) < (1e-4 if steps else 1e-6) and np.allclose(s, t, rtol=1e-4)
    head[1] = 4
    with pytest.raises(d.api.DrError):
        b.restore(head.tobytes() + ck[64:])
    a.close(), b.close(), data.close()
