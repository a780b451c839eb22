"""The tuner's choice is kept per shape of work: volumes of equal embedding and voxel counts whose kriging radii differ are tuned on
their own (the number of nonzeros of W decides between the products), and a choice made while the tensor-core products were
turned off is not taken over once they are on again."""
import pytest

import dualres_b200 as d
from dualres_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture
def config(monkeypatch):
    for k in ("DRB_AUTOTUNE", "DRB_NO_PLANE", "DRB_PLANE_PREFETCH", "DRB_FFT_PLAN", "DRB_ZTILE", "DRB_TC_PRODUCTS"):
        monkeypatch.delenv(k, raising=False)

    def make(vol, chains):
        data = d.MultiResData.from_volume(vol)
        ch = d.MultiResParameters(data, d.HMCParameters(burnin=4, nsave=3, thin=1, leapfrog=13, seed=2), chains)
        c = ch.config()
        ch.close(), data.close()
        return c
    return make


def _volume(radius, dims=(24, 24, 20)):
    return synth.make_volume(dims, 1.0, (0.75, 0.25, 1.0), 0.5, 0.3, radius, "full", 1.0, 5)


def test_radius(config):
    near, far, again = (config(_volume(r), 12) for r in (2.3, 6.9, 2.3))
    assert again == near and near["tuned_ms"] > 0
    assert far["tuned_ms"] != near["tuned_ms"]


def test_products_turned_off_and_on(config, monkeypatch):
    vol = _volume(6.9, (32, 32, 32))
    monkeypatch.setenv("DRB_TC_PRODUCTS", "0")
    assert not config(vol, 64)["tensor_products"]
    monkeypatch.delenv("DRB_TC_PRODUCTS")
    assert config(vol, 64)["tensor_products"]
