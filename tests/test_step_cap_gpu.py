"""The step cap of a photon: 0 means none, in the forward pass and in the gradient's replay."""
import numpy as np
import pytest

from conftest import have_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA GPU")]

from ppc_b200 import workloads as W  # noqa: E402
from ppc_b200.api import PPC  # noqa: E402


@pytest.mark.parametrize("opts", [{"photon_streams": True}, {"deterministic": True}], ids=["photon_streams", "static"])
def test_gradient_without_a_step_cap(ice_full, opts):
    """No photon comes near the default cap of 1e6 steps, so without one the gradient is the
    same (its sums are made in another order: 1e-9)."""
    out = []
    for cap in (1_000_000, 0):
        c = PPC()
        c.initialize(1.0, ice_full)
        c.set_seed(11)
        c.set_options(max_steps=cap, **opts)
        c.choose(0)
        c.ini()
        k = 20 * 60 + 29
        b = W.flasher(k, c.tables()["oms"]["r"][k], 1_000_000, q=0)
        out.append(c.gradient(b, weights=np.ones(c.info()["gsize"], np.float32)))
        c.close()
    a, b = out
    assert a["info"]["hits"] > 1000 and np.array_equal(a["counts"], b["counts"])
    assert b["info"]["replayed"] == a["info"]["replayed"] and b["info"]["unmatched"] == a["info"]["unmatched"]
    assert np.abs(a["g_ba"]).max() > 0 and np.abs(a["g_be"]).max() > 0
    for g in ("g_ba", "g_be"):
        np.testing.assert_allclose(b[g], a[g], rtol=1e-9, atol=1e-9 * np.abs(a[g]).max())
