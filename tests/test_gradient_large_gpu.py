"""The gradient's charges and counts through kept buffers and, for very many events, without."""
import numpy as np
import pytest

from conftest import have_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA GPU")]

from ppc_b200 import workloads as W  # noqa: E402
from ppc_b200.api import PPC  # noqa: E402


@pytest.mark.parametrize("given", ["observed", "weights"])
def test_many_events(ice_full, given):
    """Events that no photon belongs to change nothing: 900 events (4.6e6 bins) give what 2 give.
    (The sums are made in another order: 1e-9.)"""
    c = PPC()
    c.initialize(1.0, ice_full)
    c.set_seed(11)
    c.set_options(photon_streams=True)
    c.choose(0)
    c.ini()
    oms, gsize = c.tables()["oms"], c.info()["gsize"]
    b = np.concatenate([W.flasher(k, oms["r"][k], 300_000, q=i) for i, k in enumerate((20 * 60 + 29, 44 * 60 + 35))])
    rng, out = np.random.default_rng(1), []
    q = rng.poisson(3.0, 2 * gsize).astype(np.float32)
    for events in (2, 900):
        bins = np.zeros(events * gsize, np.float32)
        bins[:len(q)] = q
        out.append(c.gradient(b, events=events, **{given: bins}))
    few, many = out
    n, m = few["counts"].reshape(-1), many["counts"].reshape(-1)
    assert few["info"]["hits"] > 100 and np.array_equal(m[:len(n)], n) and not m[len(n):].any()
    for g in ("g_ba", "g_be"):
        np.testing.assert_allclose(many[g], few[g], rtol=1e-9, atol=1e-9 * np.abs(few[g]).max())
    c.close()
