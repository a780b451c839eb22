"""The row-group kriging products (chain sets off the tensor cores): every lane layout (vectors of 4, 2 and 1 chains,
one to 32 lanes, several rounds), groups that are not full, W's groups shared by 4 and by 8 warps, batches of columns that span
more than 16 bits, and columns that only some rows of a group have meeting a value that is not finite.

The products are FP32 sums of FP32 weights: against the same sums in 64 bits they are within 1e-5, the repository's
bar for gradients (a sum of n <= 1400 terms is within n 2^-24 = 8e-5 at worst and sqrt(n) 2^-24 = 2e-6 typically)."""
import numpy as np
import pytest

import dualres_b200 as d
from dualres_b200 import synth

pytestmark = pytest.mark.gpu


def _products(data, ch, c, mu, W):
    """(||rs||^2, W^T rs) of chain c at mu, from the likelihood and from two gradients that differ by s_sr W^T rs."""
    n = data.n_highres
    yh, ys = data.data()
    flat, _ = data.indices()
    out = {}
    for s_sr in (0.0, 1024.0):
        ch.set_state(c, mu, (0.0, s_sr))
        out[s_sr] = ch.gradient(c, mu).ravel()[flat].real.astype(np.float64)
    ll = ch.log_prior_likelihood(c, mu)[1]
    rs = ys.astype(np.float64) - W @ mu.ravel()[flat].real.astype(np.float64)
    assert n == len(yh)
    return -2 * ll / 1024.0, (out[1024.0] - out[0.0]) / 1024.0, rs @ rs, W.T @ rs


def _dense(data):
    rp, col, val = data.W()
    W = np.zeros((data.n_stdres, data.n_highres))
    for r in range(data.n_stdres):
        np.add.at(W[r], col[rp[r]:rp[r + 1]], val[rp[r]:rp[r + 1]].astype(np.float64))
    return W


@pytest.mark.parametrize("chains", [1, 2, 3, 4, 5, 6, 8, 12, 30, 33, 66, 72, 100, 130, 200, 255])
def test_lane_layouts(monkeypatch, chains):
    monkeypatch.setenv("DRB_AUTOTUNE", "0")
    monkeypatch.setenv("DRB_TC_PRODUCTS", "0")
    data = d.MultiResData.from_volume(synth.small_volume(seed=81, dims=(13, 11, 9), radius=3.6))
    assert data.n_stdres % 4 or data.n_highres % 4
    W = _dense(data)
    ch = d.MultiResParameters(data, d.HMCParameters(burnin=2, nsave=1, thin=1, leapfrog=2, seed=1), chains)
    rng = np.random.default_rng(3)
    for c in {0, chains // 2, chains - 1}:
        mu = (4 * rng.standard_normal(data.shape)).astype(np.complex64)
        sq, wt, sq_x, wt_x = _products(data, ch, c, mu, W)
        assert abs(sq / sq_x - 1) < 1e-5
        assert np.linalg.norm(wt - wt_x) < 1e-5 * np.linalg.norm(wt_x)
    ch.run()
    assert all(x["done"] for x in ch.stats())
    ch.close(), data.close()


@pytest.mark.parametrize("chains", [2, 16])
def test_many_groups(monkeypatch, chains):
    """More than 8 groups of W per SM: the groups of 16 chains are shared by 4 warps."""
    monkeypatch.setenv("DRB_AUTOTUNE", "0")
    monkeypatch.setenv("DRB_TC_PRODUCTS", "0")
    vol = synth.make_volume((44, 41, 40), 1.0, (0.75, 0.25, 1.0), 0.5, 0.3, 2.3, "full", 1.0, 4)
    data = d.MultiResData.from_volume(vol)
    assert data.n_stdres > 4 * 8 * 148
    rp, col, val = data.W()
    yh, ys = data.data()
    flat, _ = data.indices()
    ch = d.MultiResParameters(data, d.HMCParameters(burnin=2, nsave=1, thin=1, leapfrog=2, seed=1), chains)
    mu = (4 * np.random.default_rng(5).standard_normal(data.shape)).astype(np.complex64)
    ch.set_state(chains - 1, mu, (0.0, 1.0))
    m = mu.ravel()[flat].real.astype(np.float64)
    wm = np.add.reduceat(np.append(val.astype(np.float64) * m[col], 0.0), rp[:-1])
    wm[rp[1:] == rp[:-1]] = 0.0
    rs = ys.astype(np.float64) - wm
    assert abs(ch.log_prior_likelihood(chains - 1, mu)[1] / (-0.5 * rs @ rs) - 1) < 1e-5
    ch.close(), data.close()


def test_columns_far_apart(monkeypatch):
    """Std-res voxels in a cavity whose neighbours lie only in its floor and its roof: consecutive columns of their
    rows are more than 65535 data voxels apart."""
    monkeypatch.setenv("DRB_AUTOTUNE", "0")
    g, b = (116, 116, 14), 8
    hr = np.zeros((g[2] + 2 * b, g[1] + 2 * b, g[0] + 2 * b), np.float32)
    rng = np.random.default_rng(8)
    box = rng.uniform(0.5, 1.5, (g[2], g[1], g[0])).astype(np.float32)
    y, x = np.mgrid[:g[1], :g[0]]
    box[2:12, (x - 58.5) ** 2 + (y - 58.5) ** 2 < 10.5 ** 2] = 0
    hr[b:-b, b:-b, b:-b] = box
    Qh = np.diag([1, 1, 1, 1]).astype(np.float32)
    sr = np.zeros(tuple(n // 2 for n in hr.shape), np.float32)
    sr[(b + 6) // 2, (b + 58) // 2:(b + 58) // 2 + 2, (b + 57) // 2:(b + 57) // 2 + 3] = 1.25
    Qs = np.array([[2, 0, 0, .5], [0, 2, 0, .5], [0, 0, 2, .5], [0, 0, 0, 1]], np.float32)
    data = d.MultiResData(hr, Qh, sr, Qs, (0.75, 0.25, 1.0), 6.9)
    rp, col, _ = data.W()
    assert data.n_stdres == 6 and any(np.diff(col[a:e]).max() > 65535 for a, e in zip(rp[:-1], rp[1:]))
    W = _dense(data)
    for chains in (1, 12):
        ch = d.MultiResParameters(data, d.HMCParameters(burnin=2, nsave=1, thin=1, leapfrog=2, seed=1), chains)
        mu = (4 * rng.standard_normal(data.shape)).astype(np.complex64)
        sq, wt, sq_x, wt_x = _products(data, ch, chains - 1, mu, W)
        assert abs(sq / sq_x - 1) < 1e-5
        assert np.linalg.norm(wt - wt_x) < 1e-5 * np.linalg.norm(wt_x)
        ch.close()
    data.close()


@pytest.mark.parametrize("chains", [1, 12])
def test_a_value_that_is_not_finite_stays_in_its_rows(monkeypatch, chains):
    """An infinite mu at one voxel makes the residuals of the rows that have it infinite and no others NaN: the
    likelihood is -inf."""
    monkeypatch.setenv("DRB_AUTOTUNE", "0")
    monkeypatch.setenv("DRB_TC_PRODUCTS", "0")
    data = d.MultiResData.from_volume(synth.small_volume(seed=81, dims=(13, 11, 9), radius=3.6))
    ch = d.MultiResParameters(data, d.HMCParameters(burnin=2, nsave=1, thin=1, leapfrog=2, seed=1), chains)
    mu = np.zeros(data.shape, np.complex64)
    flat, _ = data.indices()
    mu.ravel()[flat[len(flat) // 2]] = np.inf
    ch.set_state(0, np.zeros(data.shape, np.complex64), (1.0, 1.0))
    st = ch.log_prior_likelihood(0, mu)
    assert st[1] == -np.inf
    ch.close(), data.close()
