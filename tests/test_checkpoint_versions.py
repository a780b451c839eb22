"""Checkpoints of the two earlier layouts, in which mu_D and mu_O of a chain's accepted state lie in the half that its state says
(ChainState.acc) and the other half is the last proposal's: with that other half NaN, chains of either half go on as the chain
set they were taken from.  Version 2 holds the same half spectra as the present version, so its continuation is bit-identical;
version 1 holds the full spectrum, whose split rounds once (the bar of fixed leapfrogs, 1e-4, after three iterations)."""
import numpy as np
import pytest

import dualres_b200 as d
from dualres_b200 import synth

pytestmark = pytest.mark.gpu
CHAINS, HEADER, STATE, ACC = 6, 64, 240, 132  # bytes of the header and of a ChainState, offset of its acc


@pytest.mark.parametrize("version", [1, 2])
def test_accepted_half(version):
    data = d.MultiResData.from_volume(synth.small_volume(seed=9, dims=(9, 8, 6)))
    hmc = d.HMCParameters(burnin=6, nsave=30, thin=1, leapfrog=3, seed=2, store_samples=True)
    a, b = (d.MultiResParameters(data, hmc, CHAINS) for _ in range(2))
    nh = data.N // data.shape[0] * (data.shape[0] // 2 + 1)
    for _ in range(20):
        a.update(1)
        ck = np.frombuffer(a.checkpoint(), np.uint8)
        at_mu = HEADER + CHAINS * 2 * nh * 8
        at_st = at_mu + 2 * (data.n_highres + data.n_output) * CHAINS * 4
        st = ck[at_st:at_st + CHAINS * STATE].reshape(CHAINS, STATE)
        acc = st[:, ACC:ACC + 4].copy().view(np.int32).ravel()
        it = a.stats()[0]["saved"]
        if it > 2 and set(acc) == {0, 1}:
            break
    assert set(acc) == {0, 1}
    halves, at = [], at_mu
    for n in (data.n_highres, data.n_output):
        new = ck[at:at + n * CHAINS * 4].copy().view(np.float32).reshape(n, CHAINS)
        both = np.full((2, n, CHAINS), np.nan, np.float32)
        for c in range(CHAINS):
            both[acc[c], :, c] = new[:, c]
        halves.append(both.tobytes())
        at += 2 * n * CHAINS * 4
    head = ck[:HEADER].copy().view(np.int64)
    assert head[1] == 3
    head[1] = version
    spectra = ck[HEADER:at_mu].tobytes()
    if version == 1:
        spectra = b"".join((np.fft.ifftn(a.get_state(c)[0].astype(np.complex128)) * data.N).astype(np.complex64).tobytes()
                           for c in range(CHAINS))
    b.restore(head.tobytes() + spectra + b"".join(halves) + ck[at_st:].tobytes())
    for ch in (a, b):
        ch.update(3)
    for c in range(CHAINS):
        (mu, s), (want, t) = b.get_state(c), a.get_state(c)
        if version == 2:
            assert np.array_equal(mu, want) and np.array_equal(s, t)
            assert np.array_equal(b.samples(c), a.samples(c))
        else:
            assert np.linalg.norm(mu - want) < 1e-4 * np.linalg.norm(want) and np.allclose(s, t, rtol=1e-4)
            assert np.linalg.norm(b.samples(c) - a.samples(c)) < 1e-4 * np.linalg.norm(a.samples(c))
    if version == 2:
        assert a.stats() == b.stats()
    a.close(), b.close(), data.close()
