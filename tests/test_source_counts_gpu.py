"""Photon counts of the device front end, source for source, against the double-precision
sampler of the reference (gpu/f2k.cxx:387-433) restated in numpy on the same random streams,
and the kernels' block edges and record splitting."""
import numpy as np
import pytest

from conftest import have_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA GPU")]

from ppc_b200 import types as T  # noqa: E402
from ppc_b200.api import PPC, PPCError  # noqa: E402


@pytest.fixture(scope="module")
def ctx(ice_small):
    c = PPC()
    c.initialize(1.0, ice_small)
    c.choose(0)
    c.ini()
    yield c
    c.close()


class Streams:
    """One multiply-with-carry stream per source: a SplitMix64 hash of (seed, k), a multiplier."""

    def __init__(self, seed, n, rm):
        u64 = np.uint64
        k = np.arange(n, dtype=u64)
        with np.errstate(over="ignore"):
            z = u64(seed << 32 | 0x3C6EF372) + (k + u64(1)) * u64(0x9E3779B97F4A7C15)
            z = (z ^ (z >> u64(30))) * u64(0xBF58476D1CE4E5B9)
            z = (z ^ (z >> u64(27))) * u64(0x94D049BB133111EB)
        z ^= z >> u64(31)
        self.a = rm[k % u64(1024)].astype(u64)
        self.x, self.y = z & u64(0xFFFFFFFF), ((z >> u64(32)) * self.a) >> u64(32)

    def u(self, at):
        s = self.a[at] * self.x[at] + self.y[at]
        self.x[at], self.y[at] = s & np.uint64(0xFFFFFFFF), s >> np.uint64(32)
        return 1.0 - (self.x[at] >> np.uint64(9)).astype(np.float64) / 2 ** 23


def lgamma(xx):
    cof = (76.18009172947146, -86.50532032941677, 24.01409824083091, -1.231739572450155, 0.1208650973866179e-2,
           -0.5395239384953e-5)
    tmp = xx + 4.5 - (xx - 0.5) * np.log(xx + 4.5)
    return -tmp + np.log(2.5066282746310005 * (1 + sum(q / (xx + j) for j, q in enumerate(cof))))


def poisson(mean, s):
    num = np.zeros(len(mean), np.int64)
    at = np.flatnonzero(mean < 12)
    g, t = np.exp(-mean[at]), s.u(at)
    while len(at):
        more = t > g
        at, g, t = at[more], g[more], t[more]
        num[at] += 1
        t = t * s.u(at)
    at = np.flatnonzero(mean >= 12)
    y, em = np.zeros(len(mean)), np.zeros(len(mean))
    while len(at):
        draw = at
        while len(draw):
            y[draw] = np.tan((np.float32(np.pi) * s.u(draw).astype(np.float32)).astype(np.float64))
            em[draw] = np.sqrt(2 * mean[draw]) * y[draw] + mean[draw]
            draw = draw[em[draw] < 0]
        m, um, lm = mean[at], np.floor(em[at]), np.log(mean[at])
        with np.errstate(over="ignore"):
            t = 0.9 * (1 + y[at] ** 2) * np.exp(um * lm - lgamma(um + 1) - (m * lm - lgamma(m + 1)))
        num[at] = um.astype(np.int64)
        at = at[s.u(at) > t]
    return num


@pytest.mark.parametrize("mean", [3.0, 11.9, 12.1, 14.0, 25.0, 100.0, 1e3, 1e4, 1e6, 3e7, 9e8, 2e9])
def test_counts_equal_the_double_precision_sampler(ctx, mean):
    """Every count equal: the two differ only where CUDA's and numpy's double-precision
    functions (a few ulps apart) straddle a comparison, about once in 1e12 proposals below
    means of 1e6; from there the terms of the Poisson ratio (mean x log mean) round by up to
    1e-15 of themselves, which moves the acceptance by that much: at 2e9 by 5e-5, so a few
    of 2e4 samples."""
    n = 20_000
    info, src = ctx.info(), np.zeros(n, T.SOURCE_DTYPE)
    src["kind"], src["n"], src["beta"], src["q"] = T.SRC_MOPO, [0, 0, 1], 1, np.arange(n)
    light = np.float32(mean * info["ovr"] / info["eff"]) * (1 + 0.01 * (np.arange(n) % 7)).astype(np.float32)
    src["amount"] = light
    bunches, bstart, photons = ctx.sources(src, seed=5)
    got = np.zeros(n, np.int64)
    np.add.at(got, bunches["q"], bunches["num"].astype(np.int64))
    assert photons == got.sum() == bstart[-1]
    m = (light * np.float32(info["eff"]) / np.float32(info["ovr"])).astype(np.float64)
    ref = poisson(m, Streams(5, n, ctx.tables()["rm"]))
    differ = int((got != ref).sum())
    assert differ <= (0 if mean <= 1e6 else 20), (differ, mean)


@pytest.mark.parametrize("n", [1, 31, 32, 127, 128, 129, 255, 257, 4096 * 128 - 1, 4096 * 128 + 1])
def test_block_edges_and_splits(ctx, n):
    """Exact counts: one record per source, none for a count of zero, ceil(count / 2^31) for a
    large one, in source order, whether a block writes its records as one run or one by one."""
    src = np.zeros(n, T.SOURCE_DTYPE)
    src["kind"], src["q"] = T.SRC_POINT, np.arange(n)
    src["r"][:, 0] = np.arange(n)
    src["amount"] = 1 + np.arange(n) % 5
    src["amount"][::7] = 0
    src["amount"][n // 2] = 5_000_000_000  # three records
    bunches, bstart, photons = ctx.sources(src, seed=1)
    num = src["amount"].astype(np.int64)
    recs = -(-num // 2 ** 31)
    q = np.repeat(np.arange(n), recs)
    assert np.array_equal(bunches["q"], q) and np.array_equal(bunches["r"][:, 0], q.astype(np.float32))
    assert photons == num.sum() and np.array_equal(np.diff(bstart.astype(np.int64)), bunches["num"])
    assert np.array_equal(np.bincount(q, bunches["num"], minlength=n).astype(np.int64), num)


@pytest.mark.parametrize("cap", [0, 1, 100, 300])
def test_small_buffer_and_unaligned_output(ctx, cap):
    """A buffer for fewer records than there are receives the first of them; record buffers
    on a 4-byte boundary receive the same records."""
    import torch
    n = 300
    src = np.zeros(n, T.SOURCE_DTYPE)
    src["kind"], src["q"], src["amount"] = T.SRC_POINT, np.arange(n), 7
    whole, _, _ = ctx.sources(src, seed=1)
    d = torch.from_numpy(src.view(np.uint8).copy()).cuda()
    for off in (0, 4, 8):
        out = torch.zeros(64 * n + 64, dtype=torch.uint8, device="cuda")
        bs = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        cnt = torch.zeros(2, dtype=torch.int64, device="cuda")
        ctx.sources_device(d.data_ptr(), n, 1, out.data_ptr() + off, bs.data_ptr(), cap, cnt.data_ptr())
        torch.cuda.synchronize()
        assert cnt.tolist() == [n, 7 * n]
        got = out.cpu().numpy()
        assert got[off:off + 64 * cap].tobytes() == whole[:cap].tobytes()
        assert not got[:off].any() and not got[off + 64 * cap:].any()


@pytest.mark.parametrize("n", [3, 200_000])
def test_failed_source_is_reported_once(ctx, n):
    """A source that cannot be sampled fails its call (staged or not), not the next one."""
    src = np.zeros(n, T.SOURCE_DTYPE)
    src["kind"], src["amount"], src["q"] = T.SRC_POINT, 5, np.arange(n)
    bad = src.copy()
    bad["kind"][1], bad["type"][1] = T.SRC_PARTICLE, -1
    with pytest.raises(PPCError):
        ctx.sources(bad, seed=2)
    bunches, _, photons = ctx.sources(src, seed=2)
    assert len(bunches) == n and photons == 5 * n


def test_counts_do_not_depend_on_the_neighbours(ctx):
    """Warps with 0 to 31 sources above the mean from which a warp leaves the screening out, just
    below and above it: the counts of the double-precision sampler (tolerance as above)."""
    n = 32 * 600
    info, src = ctx.info(), np.zeros(n, T.SOURCE_DTYPE)
    k = np.arange(n)
    large = k % 32 < np.array([0, 1, 2, 3, 4, 31])[k // 32 % 6]
    mean = np.where(large, np.where(k % 2, 1.01e8, 6e8), np.array([0.5, 20.0, 1e3, 9.9e7])[k // 192 % 4])
    src["kind"], src["n"], src["beta"], src["q"] = T.SRC_MOPO, [0, 0, 1], 1, k
    src["amount"] = light = (mean * info["ovr"] / info["eff"]).astype(np.float32)
    bunches, bstart, photons = ctx.sources(src, seed=8)
    got = np.zeros(n, np.int64)
    np.add.at(got, bunches["q"], bunches["num"].astype(np.int64))
    m = (light * np.float32(info["eff"]) / np.float32(info["ovr"])).astype(np.float64)
    ref = poisson(m, Streams(8, n, ctx.tables()["rm"]))
    assert photons == got.sum() and int((got != ref)[m < 1e6].sum()) == 0 and int((got != ref).sum()) <= 20
