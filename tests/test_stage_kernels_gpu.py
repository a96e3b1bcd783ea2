"""The back end's and the likelihood's kernels at the sizes where they change their way: tiles
of hits and the scan over tiles, unaligned hit buffers, and the counters of a likelihood
evaluation in one pass, in several passes over the shifts, and in global memory."""
import numpy as np
import pytest

from conftest import have_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA GPU")]

import oracle_util as O  # noqa: E402
from ppc_b200 import types as T  # noqa: E402
from ppc_b200.api import PPC, Likelihood  # noqa: E402


def _ctx(ice):
    c = PPC()
    c.initialize(1.0, ice)
    c.set_seed(3)
    c.choose(0)
    c.ini()
    return c


def _hits(n, doms, seed, tmax=4000.0):
    rng = np.random.default_rng(seed)
    h = np.zeros(n, T.HIT_DTYPE)
    h["i"] = rng.choice(doms, n)
    h["n"], h["z"] = 1, rng.integers(0, T.WNUM, n)
    h["t"] = rng.uniform(0, tmax, n)
    h["pth"], h["dth"] = np.arccos(rng.uniform(-1, 1, n)), np.arccos(rng.uniform(-1, 1, n))
    h["pph"], h["dph"] = rng.uniform(-np.pi, np.pi, n), rng.uniform(-np.pi, np.pi, n)
    return h


SIZES = [1, 31, 32, 33, 255, 256, 257, 511, 512, 513, 1025, 512 * 4096, 512 * 4096 + 1]


@pytest.mark.parametrize("kind", ["full2d", "full_ng"])
def test_back_end_sizes(kind, request):
    """Hit k is decided by its record and (seed, k) alone: the accepted hits of the first n
    are the first accepted hits of a longer list.  A record's impact point and direction
    follow from the hit's angles (single precision: 1e-6 and the modules' 0.5 m size)."""
    c = _ctx(request.getfixturevalue("ice_" + kind))
    h = _hits(SIZES[-1] + 4321, np.arange(c.info()["gsize"]), 1)
    whole = c.accept(h, seed=9)
    assert 0.2 * len(h) < len(whole) < 0.9 * len(h)
    assert np.all(np.diff(whole["hit"].astype(np.int64)) > 0)
    for n in SIZES:
        part = c.accept(h[:n], seed=9)
        assert part.tobytes() == whole[:np.searchsorted(whole["hit"], n)].tobytes(), n
    s = h[whole["hit"]].astype([(k, "f8") for k in h.dtype.names])
    d = np.stack([np.sin(s["pth"]) * np.cos(s["pph"]), np.sin(s["pth"]) * np.sin(s["pph"]), np.cos(s["pth"])], 1)
    np.testing.assert_allclose(whole["d"], d, atol=3e-6)
    if kind == "full2d":  # spherical modules
        r = -T.OMR * np.stack([np.sin(s["dth"]) * np.cos(s["dph"]), np.sin(s["dth"]) * np.sin(s["dph"]),
                               np.cos(s["dth"])], 1)
        np.testing.assert_allclose(whole["r"], r, atol=1e-6)
        assert np.array_equal(whole["t"], h["t"][whole["hit"]])
    c.close()


@pytest.mark.parametrize("shift", [4, 8, 16])
def test_back_end_takes_unaligned_hits(ice_full2d, shift):
    """Hit buffers on a 4-byte boundary, as the C record allows, give the same hits."""
    import torch
    c = _ctx(ice_full2d)
    n = 1000
    h = _hits(n, np.arange(c.info()["gsize"]), 2)
    whole = c.accept(h, seed=4)
    buf = torch.zeros(32 * n + 32, dtype=torch.uint8, device="cuda")
    buf[shift:shift + 32 * n] = torch.from_numpy(h.view(np.uint8).copy()).cuda()
    out = torch.zeros(56 * n + 4, dtype=torch.uint8, device="cuda")
    cnt = torch.zeros(1, dtype=torch.int64, device="cuda")
    c.accept_device(buf.data_ptr() + shift, n, 4, out.data_ptr() + 4, cnt.data_ptr())
    torch.cuda.synchronize()
    got = out[4:4 + 56 * int(cnt)].cpu().numpy().tobytes()
    assert got == whole.tobytes()
    c.close()


def _pulses(doms, per_dom):
    """Pulses of 20 charges in every other bin of 25 ns: every bin is a block of its own."""
    d = np.zeros(len(doms) * per_dom, T.LLH_HIT_DTYPE)
    dom, k = np.repeat(doms, per_dom), np.tile(np.arange(per_dom), len(doms))
    d["str"], d["om"], d["t"], d["q"] = dom // 60 + 1, dom % 60 + 1, 100.0 + 50.0 * k, 20.0
    return d


# observed DOMs, the counters' place that they are chosen for (bytes per shift of the blocks)
PLACES = {"one_pass": (12, 0, 3 << 10), "parts": (400, 3 << 10, 192 << 10), "global": (5160, 192 << 10, 1 << 30)}


@pytest.mark.parametrize("place", list(PLACES))
@pytest.mark.parametrize("ndt,n", [(1, 33), (2, 4001), (4, 31), (5, 4001), (9, 257), (17, 4001), (33, 32), (64, 4001)])
def test_likelihood_counters(ice_full2d, place, ndt, n):
    """Against the oracle, with hit times on the middle between two bins, far outside the bins
    and not finite."""
    c = _ctx(ice_full2d)
    doms, lo, hi = PLACES[place]
    dom = np.arange(doms)
    data = _pulses(dom, 20)
    L = Likelihood(c, data, lbin=25.0)
    assert lo < 4 * L.info()["blocks"] <= hi, L.info()
    h = _hits(n, dom, ndt, tmax=1200.0)
    h["t"][::3] = 100.0 + 12.5 + 25.0 * (np.arange(len(h["t"][::3])) % 48)  # between two bins
    h["t"][5::50], h["t"][6::50], h["t"][7::50] = 3e5, -2e7, np.inf
    h["t"][8::50] = np.nan
    dts = np.array([0.0]) if ndt == 1 else np.linspace(-100.0, 100.0, ndt)
    if ndt > 4:
        dts[1], dts[2] = 25.0, -3e5  # a bin's width; a shift that brings the far hits back
    out = L.eval(h, dts, nsim=3.0, seed=6)
    ref, err = O.llh_fllh(data, c.accept(h, seed=6), dts, 3.0, opts={"lbin": 25.0})
    assert err == 0
    np.testing.assert_allclose(out, ref, rtol=1e-10, atol=1e-13)
    L.close()
    c.close()
