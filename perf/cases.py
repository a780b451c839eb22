"""The work that a user has this library do, as measurable cases.

Most use is sampling: `MultiResParameters.update` on one volume with one chain (what `dualgpmf` runs), with a few,
and with a batch of chains.  Volumes run from a small region of interest to a whole brain at 1 mm, their sizes come
from scanners and are seldom powers of two, and some fits have no standard-resolution image.  Beside it stand single
evaluations of the model (the gradient, the log posterior, one leapfrog trajectory), the covariance estimate that
precedes a fit, a whole fit with its set-up, and a stream of small fits through the server.

`listed()` names one case for each; `draw(rng)` gives more of the same ranges; `prepare(case, seed)` makes what a
program has in hand before the call; `run(state)` is one pass; `work(case)` is what a pass cannot do without; and
`exact(case, seed)` is the same result in 64 bits, from numpy alone.
"""
import math

import numpy as np

import dualres_b200 as d
from dualres_b200 import synth

# A fit that goes on for as long as it is asked to: it is past its burn-in, in which the step size settles, and has
# more draws to save than any pass reaches.
BURNIN = 20
ENDLESS = 1_000_000
SIGMA = (1.7, 4.3)  # sigma^-2 of the two images in the evaluation cases


def _case(name, kind, nx, ny, nz, chains=1, steps=25, iterations=1, dual=True, voxel=1.0, radius=6.9,
          mask="ellipsoid", jobs=1):
    # a covariance whose range reaches across the volume, as the benchmark's (0.132 / mm at 32 mm); the embedding
    # then has non-positive modes, and acceptance does not hang on the last digits of an energy
    half = min(synth.embedding_dims((nx, ny, nz))) / 2 * voxel
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, chains=chains, steps=steps, iterations=iterations, dual=dual,
             voxel=voxel, bandwidth=round(min(0.132, 4.2 / half), 4), radius=radius, mask=mask, jobs=jobs)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # a small region of interest, one chain: every kernel is tiny, launches and latency count
        _case("update_roi", "update", 12, 10, 8, steps=10, iterations=20, radius=3.2),
        # one chain on a 32^3 volume: the command line's default use
        _case("update_32_1", "update", 32, 32, 32, iterations=8),
        # a batch of 64 chains on the same volume: the benchmark's workload
        _case("update_32_64", "update", 32, 32, 32, chains=64, iterations=6),
        # 16 chains on a larger volume at 1.5 mm with a ragged mask
        _case("update_64_16", "update", 64, 64, 48, chains=16, iterations=4, voxel=1.5, mask="smooth"),
        # the largest volumes, a couple of chains
        _case("update_80_2", "update", 80, 80, 64, chains=2, iterations=6),
        # odd sizes whose embedding is longer along x than along y (128 x 64 x 64), a dozen chains
        _case("update_ragged_12", "update", 43, 23, 17, chains=12, iterations=6),
        # no standard-resolution image: no kriging, transforms only
        _case("update_single_4", "update", 49, 37, 33, chains=4, iterations=6, dual=False),
        # one trajectory from given position and momentum (host arrays in and out): a custom sampler's inner call
        _case("leapfrog_20", "leapfrog", 20, 18, 15, radius=3.6),
        # gradient and log posterior at a given field (host arrays in and out): an optimiser's or a checker's call
        _case("evaluate_32", "evaluate", 32, 32, 32, radius=3.6),
        # the covariance estimate of a fit that is given no covariance parameters
        _case("estimate_64", "estimate", 64, 64, 48, voxel=1.5, mask="smooth"),
        # a whole fit: set-up, sampling, posterior summary
        _case("fit_30", "fit", 30, 28, 26, iterations=30),
        # a handful of one-chain fits through the server
        _case("serve_16", "serve", 18, 16, 15, iterations=20, jobs=6, radius=4.2),
    ]


def _cost(c):
    """Gradient evaluations x embedding points, the measure by which a drawn case stays below the largest."""
    n = np.prod(synth.embedding_dims((c["nx"], c["ny"], c["nz"])))
    if c["kind"] == "estimate":
        return 0
    iterations = c["iterations"] + (BURNIN if c["kind"] in ("fit", "serve") else 0)
    return float(n) * c["chains"] * c["jobs"] * iterations * (c["steps"] + 1)


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["update"] * 7 + ["leapfrog", "evaluate", "estimate", "fit", "serve"])
        top = {"update": 80, "leapfrog": 24, "evaluate": 32, "estimate": 64, "fit": 28, "serve": 20}[kind]
        # sizes over their logarithm, each axis on its own: odd ones and unequal axes as they come
        nx, ny, nz = (int(round(math.exp(rng.uniform(math.log(8), math.log(top))))) for _ in range(3))
        chains = 1
        if kind == "update":
            chains = int(round(math.exp(rng.uniform(0, math.log(96)))))
        steps = rng.choice([10, 25, 25]) if kind == "update" else 25
        iterations = {"update": rng.choice([2, 4, 6]), "fit": 15, "serve": 8}.get(kind, 1)
        radius = rng.choice([3.6, 5.1, 6.9]) if kind in ("update", "fit") else 3.6
        c = _case(None, kind, nx, ny, nz, chains=chains, steps=steps, iterations=iterations,
                  dual=rng.random() < 0.8, radius=radius, mask=rng.choice(["ellipsoid", "smooth"]),
                  jobs=4 if kind == "serve" else 1)
        if _cost(c) <= 0.8 * most:
            return c


def _volume(c, seed, dual=None):
    return synth.make_volume((c["nx"], c["ny"], c["nz"]), c["voxel"], (0.806, c["bandwidth"], 1.0), 0.5, 0.3,
                             c["radius"], c["mask"], 0.60, seed, dual=c["dual"] if dual is None else dual)


def _field(c, seed):
    """A position that is typical of the prior and a momentum that is typical of the mass matrix, as a sampler meets
    them, on the embedding."""
    E = synth.embedding_dims((c["nx"], c["ny"], c["nz"]))
    lam = synth.circulant_spectrum(E, [c["voxel"]] * 3, (0.806, c["bandwidth"], 1.0))
    live = lam > 0
    rng = np.random.default_rng(seed)
    w, v = (rng.standard_normal(lam.shape) + 1j * rng.standard_normal(lam.shape) for _ in range(2))
    mass = np.where(live, 1 / np.where(live, lam, 1.0) + SIGMA[0], 0.0)
    mu = np.fft.fftn(np.sqrt(np.where(live, lam, 0.0) / lam.size) * w)
    p = np.fft.fftn(np.sqrt(mass / lam.size) * v)
    return mu.astype(np.complex64), p.astype(np.complex64)


def _image(vol, values):
    """Values of the output voxels (the non-zero voxels, in the image's order) as an image."""
    out = np.zeros(vol.highres.shape, np.float32)
    out[vol.highres != 0] = values
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "estimate":
        vol = _volume(case, seed, dual=False)
        return dict(kind=kind, img=vol.highres, qform=vol.qform_hr)
    if kind == "fit":
        hmc = d.HMCParameters(burnin=BURNIN, nsave=case["iterations"], thin=1, leapfrog=case["steps"], seed=seed)
        return dict(kind=kind, vol=_volume(case, seed), hmc=hmc, chains=case["chains"])
    if kind == "serve":
        vols = [_volume(case, seed + 7919 * j) for j in range(case["jobs"])]
        hmc = [d.HMCParameters(burnin=BURNIN, nsave=case["iterations"], thin=1, leapfrog=case["steps"], seed=seed + j)
               for j in range(case["jobs"])]
        return dict(kind=kind, vols=vols, hmc=hmc, server=d.Server())
    data = d.MultiResData.from_volume(_volume(case, seed))
    hmc = d.HMCParameters(burnin=BURNIN, nsave=ENDLESS, thin=3, leapfrog=case["steps"], seed=seed)
    chains = d.MultiResParameters(data, hmc, case["chains"])
    st = dict(kind=kind, data=data, chains=chains, iterations=case["iterations"])
    if kind == "update":
        chains.update(BURNIN + 1)
    else:
        st["mu"], st["p"] = _field(case, seed)
        st["steps"] = case["steps"]
        chains.set_state(0, st["mu"], SIGMA)
    return st


def run(state):
    kind = state["kind"]
    if kind == "update":
        ch = state["chains"]
        ch.update(state["iterations"])
        mu, s = ch.get_state(ch.n_chains - 1)
        st = ch.stats()
        return dict(mu=mu, sigma_sq_inv=s, sigma_hr=np.array([x["sigma_hr"] for x in st], np.float32),
                    sigma_sr=np.array([x["sigma_sr"] for x in st], np.float32))
    if kind == "leapfrog":
        # the energies of a 32-bit state: as 32-bit numbers
        mu, p, en = state["chains"].leapfrog(0, state["mu"], state["p"], 1.0 / state["steps"], state["steps"])
        return dict(mu=mu, p=p, energies=en.astype(np.float32))
    if kind == "evaluate":
        g = state["chains"].gradient(0, state["mu"])
        e = state["chains"].log_prior_likelihood(0, state["mu"])
        return dict(gradient=g, energies=np.array(e, np.float32))
    if kind == "estimate":
        return d.api.mce_summary(state["img"], state["qform"])
    if kind == "fit":
        data = d.MultiResData.from_volume(state["vol"])
        fit = d.fit_model(data, state["hmc"], state["chains"])
        out = {k: _image(state["vol"], fit[k]) for k in ("mean", "var", "activation")}
        fit["chains"].close()
        data.close()
        return out
    sv = state["server"]
    ids = [sv.submit_volume(v, h) for v, h in zip(state["vols"], state["hmc"])]
    sv.drain()
    res = [sv.result(j, forget=True) for j in ids]
    return [dict(mean=_image(v, r.mean), var=_image(v, r.var), activation=_image(v, r.activation))
            for v, r in zip(state["vols"], res)]


def work(case):
    g = (case["nx"], case["ny"], case["nz"])
    n = float(np.prod(synth.embedding_dims(g)))
    vox = float(np.prod(g))
    if case["kind"] == "estimate":
        # each voxel pair of the lattice offsets: one product and two sums in 64 bits, for the pairs inside the mask
        return {"bytes": 4.0 * vox + 12.0 * len(_offsets()), "flops": 4.0 * len(_offsets()) * vox * 0.36}
    n_h = 0.6 * vox
    n_s = n_h / 8 if case["dual"] else 0.0
    per_row = 4.19 * (case["radius"] / case["voxel"]) ** 3 * 0.8
    nnz = n_s * per_row
    c = float(case["chains"])
    # One gradient evaluation of a chain: position and momentum of the real field (n floats each) read and written,
    # the data vectors, and once for all chains W in both directions; a forward and an inverse real transform, the
    # products with W and its transpose, the update.
    grad_bytes = c * (16.0 * n + 8.0 * n_h + 4.0 * n_s) + 16.0 * nnz
    grad_flops = c * (5.0 * n * math.log2(n) + 4.0 * nnz + 8.0 * n)
    fit = (BURNIN + case["iterations"]) * (case["steps"] + 1)
    evals = {"update": case["iterations"] * (case["steps"] + 1), "fit": fit, "serve": case["jobs"] * fit, "leapfrog": case["steps"] + 1,
             "evaluate": 2}[case["kind"]]
    host = {"update": 8.0 * n, "leapfrog": 32.0 * n, "evaluate": 24.0 * n}.get(case["kind"], 8.0 * n_h)
    return {"bytes": evals * grad_bytes + host, "flops": evals * grad_flops}


# ---------------------------------------------------------------- the same results in 64 bits
def _offsets():
    """The lattice offsets of the minimum-contrast summary in their order (perturbation_matrix.h:19-109)."""
    unit = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, 0, 1), (-1, 1, 0), (1, 0, -1), (0, 1, 1),
            (0, 1, -1), (1, 1, 1), (1, 1, -1), (-1, 1, 1), (-1, 1, -1)]
    seen = {}
    for k in range(1, 19):
        for j in range(1, 19):
            for i in range(1, 19):
                for u in unit:
                    seen.setdefault((u[0] * i, u[1] * j, u[2] * k))
    for e in range(19, 26):
        for a in range(3):
            seen.setdefault(tuple(e if b == a else 0 for b in range(3)))
    return np.array(list(seen), np.int64)


def _exact_estimate(case, seed):
    """Pair sums as correlations by zero-padded transforms (estimate_kernel_parameters.h:50-101)."""
    vol = _volume(case, seed, dual=False)
    img = vol.highres.astype(np.float64)
    m = (img != 0).astype(np.float64)
    shape = [n + 26 for n in img.shape]
    F = np.fft.rfftn(img, shape)
    M = np.fft.rfftn(m, shape)
    P = _offsets()
    at = tuple(P[:, 2 - a] % shape[a] for a in range(3))

    def pairs(a, b):  # sum_x a(x) b(x + p)
        return np.fft.irfftn(np.conj(a) * b, shape)[at]

    sxy, sx, sy, n = pairs(F, F), pairs(F, M), pairs(M, F), np.rint(pairs(M, M))
    cov = np.where(n > 1, (sxy - sx * sy / np.maximum(n, 1)) / np.maximum(n - 1, 1), 0.0)
    dist = np.sqrt(((P @ vol.qform_hr[:3, :3].astype(np.float64).T) ** 2).sum(1))
    return dict(distance=dist, covariance=cov, npairs=n.astype(np.int32))


def _cov(dist, theta):
    return theta[0] * np.exp(-theta[1] * np.abs(dist) ** theta[2])


def _kriging(vol, theta):
    """The kriging weights of every standard-resolution voxel over its high-resolution neighbourhood, dense
    (kriging_matrix.h:148-343; the images of these cases keep the neighbourhoods inside the grid)."""
    h = float(vol.qform_hr[0, 0])
    r = int(vol.radius / h)
    ax = np.arange(-r, r + 1)
    P = np.array([(i, j, k) for k in ax for j in ax for i in ax if (i * i + j * j + k * k) * h * h <= vol.radius ** 2])
    K = _cov(h * np.sqrt(((P[:, None] - P[None]) ** 2).sum(-1)), theta)
    np.fill_diagonal(K, 1.0)
    hr = vol.highres
    order = np.full(hr.shape, -1)
    order[hr != 0] = np.arange(np.count_nonzero(hr))
    z, y, x = np.nonzero(vol.stdres)
    W = np.zeros((len(x), np.count_nonzero(hr)))
    kp_all = _cov(h * np.sqrt(((P - 0.5) ** 2).sum(1)) + 1e-5, theta)
    for row, (i, j, k) in enumerate(zip(x, y, z)):
        q = np.array([2 * i, 2 * j, 2 * k]) + P
        c = order[q[:, 2], q[:, 1], q[:, 0]]
        on = np.nonzero(c >= 0)[0]
        if len(on):
            w = np.linalg.solve(K[np.ix_(on, on)], kp_all[on])
            W[row, c[on]] = w / w.sum()
    return W


def _spectrum(E, h, theta):
    """Eigenvalues of the wrapped covariance, in 64 bits, of distances in 32 (circulant_base.inl:83-84)."""
    o = [np.where(np.arange(n) <= n // 2, np.arange(n), n - np.arange(n)).astype(np.float32) * np.float32(h) for n in E]
    q = [a * a for a in o]
    dist = np.sqrt((q[0][None, None, :] + q[1][None, :, None]) + q[2][:, None, None])
    return np.fft.fftn(_cov(dist.astype(np.float64), theta)).real


class _Model:
    """The log posterior of a field on the embedding (MultiResParameters.h:337-514, 674-700) with transforms of numpy."""

    def __init__(self, vol):
        theta = [float(np.float32(t)) for t in vol.theta]
        z, y, x = np.nonzero(vol.highres)
        lo = [x.min(), y.min(), z.min()]
        g = [int(a.max() - b + 1) for a, b in zip((x, y, z), lo)]
        E = synth.embedding_dims(g)
        self.shape, self.N = (E[2], E[1], E[0]), float(np.prod(E))
        self.lam = _spectrum(E, vol.qform_hr[0, 0], theta)
        self.live = self.lam > 0
        self.inv = np.where(self.live, 1 / np.where(self.live, self.lam, 1.0), 0.0)
        self.at = (z - lo[2], y - lo[1], x - lo[0])
        self.Yh = vol.highres[z, y, x].astype(np.float64)
        self.Ys = self.W = None
        if vol.stdres is not None:
            self.Ys = vol.stdres[np.nonzero(vol.stdres)].astype(np.float64)
            self.W = _kriging(vol, theta)
        self.s = [float(np.float32(v)) for v in SIGMA]

    def residuals(self, mu):
        m = mu.real[self.at]
        return self.Yh - m, None if self.W is None else self.Ys - self.W @ m

    def prior(self, mu):
        return -0.5 * self.N * float((np.abs(np.fft.ifftn(mu)) ** 2 * self.inv).sum())

    def likelihood(self, mu):
        rh, rs = self.residuals(mu)
        return -0.5 * (self.s[0] * float(rh @ rh) + (0.0 if rs is None else self.s[1] * float(rs @ rs)))

    def gradient(self, mu):
        g = -np.fft.fftn(np.fft.ifftn(mu) * self.inv)
        rh, rs = self.residuals(mu)
        g[self.at] += self.s[0] * rh + (0.0 if rs is None else self.s[1] * (self.W.T @ rs))
        return g

    def mass_inv(self):
        return np.where(self.live, 1.0 / (self.inv + self.s[0]), 0.0)

    def kinetic(self, p):
        return -0.5 * self.N * float((np.abs(np.fft.ifftn(p)) ** 2 * self.mass_inv()).sum())

    def leapfrog(self, mu, p, eps, steps):
        mi = self.mass_inv()
        p = p + 0.5 * eps * self.gradient(mu)
        for s in range(steps):
            mu = mu + eps * np.fft.fftn(np.fft.ifftn(p) * mi)
            p = p + (0.5 if s == steps - 1 else 1.0) * eps * self.gradient(mu)
        return mu, p


def exact(case, seed):
    kind = case["kind"]
    if kind == "estimate":
        return _exact_estimate(case, seed)
    if kind not in ("leapfrog", "evaluate"):
        return None  # the sampler's random draws, or a volume whose kriging takes minutes
    m = _Model(_volume(case, seed))
    mu, p = (a.astype(np.complex128) for a in _field(case, seed))
    if kind == "evaluate":
        return dict(gradient=m.gradient(mu), energies=np.array([m.prior(mu), m.likelihood(mu)]))
    eps = float(np.float32(1.0 / case["steps"]))
    mu1, p1 = m.leapfrog(mu, p, eps, case["steps"])
    en = [m.prior(mu), m.likelihood(mu), m.kinetic(p), m.prior(mu1), m.likelihood(mu1), m.kinetic(p1)]
    return dict(mu=mu1, p=p1, energies=np.array(en))
