"""Whole transitions of the sampler (MultiResParameters.h:674-727) against 64 bits: from the state that each iteration starts in, with
the momentum, step-size and accept draws that the library makes from its counter-based generator, numpy runs the same
trajectory in 64 bits with four transforms a step; compared are the logarithm of the Metropolis ratio, the decision, the position
and the Gibbs draws of both sigmas.

Bars.  The Hamiltonian at either end is a sum of 32-bit quantities: its difference is within four roundings (2^-22) of the sum of the two
energies' magnitudes.  A decision is compared unless the uniform is within that of the ratio.  Position: the bar of fixed
leapfrogs, 1e-4; sigma: 1e-5, the bar of likelihoods (at most 2 sqrt(n) standard deviations of a draw whose rate is a residual norm)."""
import math

import numpy as np
import pytest

import dualres_b200 as d
from dualres_b200 import synth

pytestmark = pytest.mark.gpu
MOMENTUM, SCALAR = 1, 3  # generator streams


def philox(x, y, z, w, key):
    """Philox4x32-10 (Salmon et al., SC'11) of arrays of counters."""
    m = np.uint64(0xFFFFFFFF)
    c = [np.broadcast_to(np.asarray(a, np.uint64), np.shape(x)).copy() for a in (x, y, z, w)]
    k0, k1 = key & 0xFFFFFFFF, key >> 32
    for _ in range(10):
        p, q = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(q >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), q & m, (p >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p & m]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def normals(n, iteration, chain, seed):
    """n complex normals by Box-Muller of 24-bit uniforms, two to a counter."""
    r = philox(np.arange(n // 2, dtype=np.uint64), iteration, chain, MOMENTUM, seed)
    u = [((v >> np.uint64(8)).astype(np.float64) + 0.5) / 2 ** 24 for v in r]
    out = np.empty(n, np.complex128)
    for k in (0, 1):
        out[k::2] = np.sqrt(-2 * np.log(u[2 * k])) * np.exp(2j * np.pi * u[2 * k + 1])
    return out


def scalars(x, iteration, chain, seed):
    """The two 53-bit uniforms of a counter."""
    r = [int(v[0]) for v in philox(np.array([x], np.uint64), iteration, chain, SCALAR, seed)]
    return [(((a >> 5) << 26 | (b >> 6)) + 0.5) / 2 ** 53 for a, b in (r[:2], r[2:])]


def gamma(shape, scale, base, iteration, chain, seed):
    """Marsaglia & Tsang (2000) as the library draws it, shape > 1."""
    a = shape - 1 / 3
    c = 1 / math.sqrt(9 * a)
    for k in range(64):
        n, u = scalars(base + 2 * k, iteration, chain, seed), scalars(base + 2 * k + 1, iteration, chain, seed)[0]
        x = math.sqrt(-2 * math.log(n[0])) * math.cos(2 * math.pi * n[1])
        v = (1 + c * x) ** 3
        if v > 0 and math.log(u) < 0.5 * x * x + a - a * v + a * math.log(v):
            return a * v * scale
    raise AssertionError


@pytest.mark.parametrize("dims,dual,chains", [((12, 10, 8), True, 2), ((9, 18, 5), True, 3), ((11, 6, 17), False, 2),
                                              ((12, 10, 8), True, 32), ((9, 9, 8), True, 9)])
@pytest.mark.parametrize("eps", [0.1, 0.45, 1.2])
def test_transition(monkeypatch, dims, dual, chains, eps):
    monkeypatch.setenv("DRB_AUTOTUNE", "0")
    L, seed, c = 10, 11, chains - 1
    half = min(synth.embedding_dims(dims)) / 2
    vol = synth.make_volume(dims, 1.0, (0.806, round(min(0.132, 4.2 / half), 4), 1.0), 0.5, 0.3, 3.2, "ellipsoid", 0.6, 4, dual=dual)
    data = d.MultiResData.from_volume(vol)
    lam = data.lambda_re()
    live = lam > 0
    inv = np.where(live, 1 / np.where(live, lam, 1), 0)
    flat, n = data.indices()[0], data.N
    yh, ys = (np.asarray(v, np.float64) for v in data.data())
    W = np.zeros((data.n_stdres if dual else 0, data.n_highres))
    if dual:
        rp, col, val = data.W()
        W[np.repeat(np.arange(len(rp) - 1), np.diff(rp)), col] = val
    ch = d.MultiResParameters(data, d.HMCParameters(burnin=0, nsave=99, thin=1, leapfrog=L, starting_eps=eps, seed=seed), chains)
    assert ch.config()["tensor_products"] == (chains >= 32)

    def residuals(u):
        m = np.fft.fftn(u).ravel()[flat].real / n
        return yh - m, (ys - W @ m if dual else np.zeros(0))

    for it in range(4):
        mu, s = ch.get_state(c)
        sh, ss = map(float, s)
        before = ch.stats()[c]["accepted"]
        ch.update(1)
        after = ch.stats()[c]
        u = np.fft.ifftn(mu.astype(np.complex128)) * n
        jitter, accept = scalars(0, it, c, seed)
        # without a burn-in the step size is the given one once and the average's initial 1 from then on (HMCParameters.h:259-263)
        e = float(np.float32((np.float64(np.float32(eps)) if it == 0 else 1.0) * (0.9 + 0.2 * jitter)))
        assert after["last_eps"] == e
        lm = inv + sh
        w = normals(n, it, c, seed).reshape(lam.shape)
        q = np.where(live, np.sqrt(n * lm), 0) * w

        def kick(u, q, step):
            rh, rs = residuals(u)
            g = np.zeros(n, np.complex128)
            g[flat] = sh * rh + (ss * (W.T @ rs) if dual else 0)
            return q + step * (np.fft.ifftn(g.reshape(lam.shape)) * n - u * inv)

        def energy(u):
            rh, rs = residuals(u)
            return 0.5 * (np.abs(u) ** 2 * inv).sum() / n + 0.5 * (sh * (rh @ rh) + ss * (rs @ rs)), rh @ rh, rs @ rs

        e0, *r0 = energy(u)
        e0 += 0.5 * (np.abs(w) ** 2).sum()
        v, q = u, kick(u, q, e / 2)
        for t in range(1, L + 1):
            v = v + np.where(live, e / lm, 0) * q
            q = kick(v, q, e / 2 if t == L else e)
        ep, *rl = energy(v)
        ep += 0.5 * np.where(live, np.abs(q) ** 2 / lm, 0).sum() / n
        bar = 2.0 ** -22 * (e0 + ep)
        assert abs(after["last_log_ratio"] - (e0 - ep)) < bar
        moved = math.log(accept) < e0 - ep
        if abs(math.log(accept) - (e0 - ep)) < bar:
            moved = after["accepted"] > before
        assert moved == (after["accepted"] > before)
        mu1, s1 = ch.get_state(c)
        want = np.fft.fftn(v if moved else u) / n
        assert np.linalg.norm(mu1 - want) < 1e-4 * np.linalg.norm(want)
        kept = rl if moved else r0
        for k, (count, r, base) in enumerate(((len(yh), kept[0], 16), (len(ys), kept[1], 4096))):
            if dual or k == 0:
                assert abs(s1[k] / gamma(0.5 * count + 1, 2 / r, base, it, c, seed) - 1) < 1e-5
    ch.close(), data.close()
