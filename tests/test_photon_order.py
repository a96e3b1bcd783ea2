"""The order in which a launch takes its photons: dealt out at the start (few photons), from
the queue, or screened by absorption depth first (three photons per lane and more), on some
or all of the warps.  Whatever the order, every photon is propagated exactly once, with its own random
numbers."""
import numpy as np
import pytest

from conftest import have_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA GPU")]

from ppc_b200 import types as T  # noqa: E402
from ppc_b200.api import PPC  # noqa: E402


def _ctx(ice, **opts):
    c = PPC()
    c.initialize(1.0, ice)
    c.set_seed(17)
    c.set_options(**opts)
    c.choose(0)
    c.ini()
    return c


def _iso(num, q=1):
    # two metres off the central string: some per cent of the photons are seen, at any size
    return T.bunch_led([2, 0, 10, 0], [0, 0, 1], q, num, 1, ka=-1, up=0, fldr=-1)


def _sizes(threads):
    return [1, 31, 32, 33, 749, 750, 751, 23_968, 23_969, threads - 1, threads, threads + 1, 3 * threads - 1, 3 * threads,
            3 * threads + 1, 17 * threads + 5, 144_000, 6 * threads - 1, 6 * threads + 1]


def _sorted(h):
    return np.sort(np.ascontiguousarray(h).view("V32").ravel())


@pytest.mark.parametrize("k", range(19))
def test_every_photon_once(ice_small, k):
    """The hits of a launch of n photons are the hits of the first n photons of a larger launch
    (another order: photon i draws from its own stream wherever it runs)."""
    c = _ctx(ice_small, photon_streams=True)
    n = _sizes(c.info()["threads"])[k]
    small, info = c.propagate(_iso(n))
    assert info["photons"] == n and info["steps"] >= n
    large, _ = c.propagate(np.concatenate([_iso(n), _iso(20 * c.info()["threads"] + 77, q=2)]))
    part = large[large["n"] == 1]
    assert len(small) == len(part) and (n < 500 or len(small) > 0)
    assert np.array_equal(_sorted(small), _sorted(part))
    c.close()


@pytest.mark.parametrize("k", range(6))
def test_every_photon_once_in_hole_ice(ice_small_hole, k):
    """The same where hole ice has more warps at work for a given number of photons."""
    c = _ctx(ice_small_hole, photon_streams=True)
    threads = c.info()["threads"]
    n = [47_935, 47_937, 120_000, 2 * threads - 1, 2 * threads + 1, 6 * threads + 1][k]
    small, info = c.propagate(_iso(n))
    large, _ = c.propagate(np.concatenate([_iso(n), _iso(7 * threads + 77, q=2)]))
    part = large[large["n"] == 1]
    assert info["photons"] == n and len(small) == len(part) > 0
    assert np.array_equal(_sorted(small), _sorted(part))
    c.close()


@pytest.mark.parametrize("mult", [0.5, 2, 3, 17.3])
def test_thread_streams_keep_the_absorption_law(ice_small, mult):
    """Thread streams draw the absorption depth when a photon is screened: the mean number of
    steps per photon and the fraction seen agree with per-photon streams.  Steps per photon
    spread by at most twice their mean, so the bound is five standard errors of that; the
    fraction seen has a binomial error."""
    c = _ctx(ice_small)
    n = int(mult * c.info()["threads"])
    h1, i1 = c.propagate(_iso(n))
    d = _ctx(ice_small, photon_streams=True)
    h2, i2 = d.propagate(_iso(n))
    assert i1["photons"] == i2["photons"] == n
    mean = i2["steps"] / n
    assert abs(i1["steps"] - i2["steps"]) < 5 * 2 * mean * np.sqrt(2 * n), (i1["steps"] / n, mean)
    seen1, seen2 = len(h1), len(h2)
    # a photon may be seen several times (DOMs are transparent at this size): clusters of two
    assert abs(seen1 - seen2) < 5 * np.sqrt(2 * (seen1 + seen2)), (seen1, seen2)
    c.close()
    d.close()
