"""The likelihood's counters in each of their places, and evaluations inside a CUDA graph that is
replayed after other calls on the same object."""
import numpy as np
import pytest

from conftest import have_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA GPU")]

import oracle_util as O  # noqa: E402
from ppc_b200 import types as T  # noqa: E402
from ppc_b200.api import PPC, Likelihood  # noqa: E402


def _hits(n, doms, seed):
    rng = np.random.default_rng(seed)
    h = np.zeros(n, T.HIT_DTYPE)
    h["i"], h["z"] = rng.integers(0, doms, n), rng.integers(0, T.WNUM, n)
    h["t"] = rng.uniform(0, 1200.0, n)
    h["pth"], h["dth"] = np.arccos(rng.uniform(-1, 1, n)), np.arccos(rng.uniform(-1, 1, n))
    h["pph"], h["dph"] = rng.uniform(-np.pi, np.pi, n), rng.uniform(-np.pi, np.pi, n)
    return h


@pytest.mark.parametrize("doms,ndt", [(12, 5), (60, 64), (400, 64)], ids=["shared", "parts", "global"])
def test_likelihood_replayed_after_a_larger_call(ice_full2d, doms, ndt):
    """The counters' three places (ids).  The replay sees the hits that its buffer holds then, and
    gives what a plain call gives."""
    import torch
    c = PPC()
    c.initialize(1.0, ice_full2d)
    c.set_seed(3)
    c.choose(0)
    c.ini()
    dom, per = np.repeat(np.arange(doms), 20), np.tile(np.arange(20), doms)
    d = np.zeros(20 * doms, T.LLH_HIT_DTYPE)
    d["str"], d["om"], d["t"], d["q"] = dom // 60 + 1, dom % 60 + 1, 100.0 + 50.0 * per, 20.0
    L = Likelihood(c, d, lbin=25.0)
    dts, n = np.linspace(-100.0, 100.0, ndt), 4001
    first, second = _hits(n, doms, 1), _hits(n, doms, 2)
    buf = torch.from_numpy(first.view(np.uint8).copy()).cuda()
    out = torch.zeros(ndt, dtype=torch.float64, device="cuda")
    plain = [L.eval(h, dts, nsim=3.0, seed=6) for h in (first, second)]
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s, capture_error_mode="thread_local"):
        L.eval_device(buf.data_ptr(), n, dts, 3.0, out.data_ptr(), seed=6, stream=s.cuda_stream)
    L.eval(_hits(50 * n, doms, 3), dts, nsim=3.0, seed=6)
    for h, ref in ((first, plain[0]), (second, plain[1])):
        buf.copy_(torch.from_numpy(h.view(np.uint8).copy()))
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), ref)
    L.close()
    c.close()


@pytest.mark.parametrize("norm", [0, 1])
@pytest.mark.parametrize("doms,ndt", [(38, 64), (39, 64), (60, 33), (100, 64), (145, 64), (155, 64), (700, 17)])
def test_likelihood_counters_against_oracle(ice_full2d, doms, ndt, norm):
    """Counters of all shifts in one CTA (up to 768 at 64 shifts), in parts (up to 3072) and in
    global memory, with the DOMs' own counters (norm) among them.  Tolerance as for the sums of
    test_stage_kernels_gpu.py: the same FP64 terms in another order."""
    c = PPC()
    c.initialize(1.0, ice_full2d)
    c.set_seed(3)
    c.choose(0)
    c.ini()
    dom, per = np.repeat(np.arange(doms), 20), np.tile(np.arange(20), doms)
    d = np.zeros(20 * doms, T.LLH_HIT_DTYPE)
    d["str"], d["om"], d["t"], d["q"] = dom // 60 + 1, dom % 60 + 1, 100.0 + 50.0 * per, 20.0
    L = Likelihood(c, d, lbin=25.0, norm=norm, unh=1)
    h, dts = _hits(4001, doms + 20, 4), np.linspace(-300.0, 100.0, ndt)
    h["t"][::3] = 100.0 + 12.5 + 25.0 * (np.arange(len(h["t"][::3])) % 48)  # between two bins
    out = L.eval(h, dts, nsim=3.0, seed=6)
    ref, err = O.llh_fllh(d, c.accept(h, seed=6), dts, 3.0, opts={"lbin": 25.0, "norm": norm, "unh": 1})
    assert err == 0
    np.testing.assert_allclose(out, ref, rtol=1e-10, atol=1e-13)
    L.close()
    c.close()
