"""The kernels compiled for an ice model (tilt kind, plain ice) against the general one and the
oracle: the tilt shift and every index bit for bit, at the radii of the 1-d maps and at the
edges of the 2-d map, for maps that the interval cells and reciprocal quotients allow and for
maps that they do not."""
import os
import shutil

import numpy as np
import pytest

from conftest import have_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA GPU")]

import oracle_util as O  # noqa: E402
from ppc_b200 import types as T  # noqa: E402
from ppc_b200 import workloads as W  # noqa: E402
from ppc_b200.api import PPC  # noqa: E402


def _tilted(ice_full, path, radii):
    """The full detector with 1-d tilt maps at the given distances."""
    shutil.copytree(ice_full, path)
    depths = 1200.0 + 10.0 * np.arange(125)
    with open(os.path.join(path, "tilt.par"), "w") as f:
        for k, r in enumerate(radii):
            f.write(f"{k + 1} {r}\n")
    with open(os.path.join(path, "tilt.dat"), "w") as f:
        for d in depths:
            f.write(f"{d:.2f} " + " ".join("%.4f" % (20.0 * np.sin(d / 80.0 + r / 400.0)) for r in radii) + "\n")
    return str(path)


def _ctx(ice, **opts):
    c = PPC()
    c.initialize(1.0, ice)
    c.set_seed(7)
    c.set_options(**opts)
    c.choose(0)
    c.ini()
    return c


def _points(c, n, rng):
    pos = np.zeros((n, 8), np.float32)
    pos[:, :2] = rng.uniform(-900, 900, (n, 2))
    pos[:, 2] = rng.uniform(-700, 700, n)
    d = rng.normal(size=(n, 3))
    pos[:, 4:7] = d / np.linalg.norm(d, axis=1)[:, None]
    pos[:, 7] = rng.uniform(0, 200, n)
    return pos


def _same(c, pos):
    import torch
    oi = torch.zeros((len(pos), 8), dtype=torch.int32, device="cuda")
    of = torch.zeros((len(pos), 2), dtype=torch.float32, device="cuda")
    d = torch.from_numpy(pos).cuda()
    c.index_probe_device(d.data_ptr(), len(pos), oi.data_ptr(), of.data_ptr())
    torch.cuda.synchronize()
    ri, rf = O.index_probe(O.tables_from_product(c), pos)
    gf = of.cpu().numpy()
    same = (gf.view(np.uint32) == rf.view(np.uint32)) | (np.isnan(gf) & np.isnan(rf)) | ((gf == 0) & (rf == 0))
    assert same.all(), pos[~same.all(axis=1)][:3]
    # indices, but for exact .5 ties of the layer and of the cell range's ends (rounded half to
    # even here, half away from zero there)
    gi = oi.cpu().numpy()
    rows = np.flatnonzero((gi != ri).any(axis=1))
    for k in rows:
        t = _rounded(c.params(), pos[k], rf[k, 0])
        cols = np.flatnonzero(gi[k] != ri[k])
        assert set(cols) <= {0, 1, 2, 3, 4} and all(abs(t[j]) % 1 == 0.5 for j in cols), (pos[k], gi[k], ri[k], t)
    assert len(rows) <= 1e-4 * len(pos)


def _rounded(p, q, zs):
    """What is rounded to the layer and to the cell range's ends (x low, x high, y low, y high)."""
    f = np.float32
    cb, cl, cr = [f(x) for x in p.cb], [f(x) for x in p.cl], [f(x) for x in p.crst]
    x1, y1 = q[0] + q[7] * q[4], q[1] + q[7] * q[5]
    u = [cb[0] * q[0] + cb[2] * q[1], cb[0] * x1 + cb[2] * y1]
    v = [cb[1] * q[0] + cb[3] * q[1], cb[1] * x1 + cb[3] * y1]
    ends = [(min(u) - f(p.rx) - cl[0]) * cr[0], (max(u) + f(p.rx) - cl[0]) * cr[0],
            (min(v) - f(p.rx) - cl[1]) * cr[1], (max(v) + f(p.rx) - cl[1]) * cr[1]]
    return [((q[2] - zs) - f(p.hmin)) * f(p.rdh)] + ends


RADII = {
    "six": [-500.0, -250.0, 0.0, 250.0, 500.0, 750.0],
    "three": [-100.0, 3.25, 90.0],
    "two": [-200.0, 300.0],
    "forty": [25.0 * k - 490.0 for k in range(40)],
    "eighty": [12.5 * k - 490.0 for k in range(80)],          # two radii per cell: no cells
    "close": [-531.2, -164.0, -163.1, 0.0, 302.0, 368.0],     # likewise
    "equal": [-500.0, -250.0, 0.0, 0.0, 250.0, 500.0],        # an interval of no width
}


@pytest.mark.parametrize("vthk", [0, 1])
@pytest.mark.parametrize("name", list(RADII))
def test_1d_tilt_at_the_radii(ice_full, tmp_path, name, vthk, monkeypatch):
    monkeypatch.setenv("VTHK", str(vthk))  # variable layer thickness: the general kernel
    c = _ctx(_tilted(ice_full, tmp_path / "ice", RADII[name]))
    p, rng = c.params(), np.random.default_rng(5)
    assert p.tmod == 1 and p.lnum == len(RADII[name])
    pos = _points(c, 60_000, rng)
    # half of the points on a radius, within a few ulps of the distance, or within a cell of it
    near = slice(0, 30_000)
    lr = np.asarray(RADII[name])[rng.integers(0, p.lnum, 30_000)]
    off = rng.choice([0.0, 3e-5, -3e-5, 1e-3, -1e-3, 0.1, -0.1, 7.0, -7.0], 30_000)
    pos[near, 0] = (lr + off + p.r0 - p.lny * pos[near, 1].astype(np.float64)) / p.lnx
    _same(c, pos)
    c.close()


@pytest.mark.parametrize("vthk", [0, 1])
def test_2d_tilt_at_the_edges(ice_full2d, vthk, monkeypatch):
    monkeypatch.setenv("VTHK", str(vthk))
    c = _ctx(ice_full2d)
    p, rng = c.params(), np.random.default_rng(6)
    assert p.tmod == 2
    pos = _points(c, 60_000, rng)
    pos[:20_000, :2] *= 3  # far outside the map
    # on grid lines and corners: positions from grid coordinates near integers
    q = np.round(rng.uniform(-1.4, 11.4, (20_000, 2))) + rng.choice([0.0, 1e-6, -1e-6, 1e-3, -1e-3], (20_000, 2))
    a = np.array([[p.cb[0], p.cb[2]], [p.cb[1], p.cb[3]]], np.float64)  # grid = a . (x, y)
    g = q * np.array([p.mstp[0], p.mstp[1]]) + np.array([p.mmin[0], p.mmin[1]])
    pos[20_000:40_000, :2] = np.linalg.solve(a, g.T).T
    _same(c, pos)
    c.close()


def test_models_propagate_alike(ice_full, tmp_path):
    """A second map at the radius and with the shifts of another leaves the ice as it is but
    needs the general kernel: every photon's path, and so every hit, is the same."""
    a = _ctx(_tilted(ice_full, tmp_path / "fast", RADII["six"]), photon_streams=True)
    b = _ctx(_tilted(ice_full, tmp_path / "general", sorted(RADII["six"] + [250.0])), photon_streams=True)
    k = 39 * 60 + 29
    bunch = np.concatenate([W.flasher(k, a.tables()["oms"]["r"][k], 3_000_000, q=1),
                            W.cascade([30, -20, 100], [0.3, 0.4, 0.8660254], 3_000_000, q=2)])
    (h1, i1), (h2, i2) = a.propagate(bunch), b.propagate(bunch)
    assert len(h1) > 1000 and i1["steps"] == i2["steps"]
    assert np.array_equal(np.sort(h1.view("V32").ravel()), np.sort(h2.view("V32").ravel()))
    # the same through the gradient's recording and replay kernels
    w = np.ones(a.info()["gsize"], np.float32)
    r1, r2 = a.gradient(bunch, weights=w), b.gradient(bunch, weights=w)
    assert np.array_equal(r1["counts"], r2["counts"])
    np.testing.assert_allclose(r1["g_ba"], r2["g_ba"], rtol=1e-9)
    np.testing.assert_allclose(r1["g_be"], r2["g_be"], rtol=1e-6, atol=1e-9 * np.abs(r1["g_be"]).max())
    a.close()
    b.close()


@pytest.mark.parametrize("name", ["six", "two", "forty"])
def test_1d_tilt_at_points_that_are_not_finite(ice_full, tmp_path, name, monkeypatch):
    """NaN, infinite and huge positions give the general kernel's tilt shift."""
    import torch
    ice, rng, got = _tilted(ice_full, tmp_path / "ice", RADII[name]), np.random.default_rng(9), []
    xy = rng.choice([np.nan, np.inf, -np.inf, 3e38, -3e38, 1.0], (4096, 2))
    for vthk in (0, 1):
        monkeypatch.setenv("VTHK", str(vthk))
        c = _ctx(ice)
        pos = _points(c, 4096, np.random.default_rng(9))
        pos[:, :2] = xy
        oi = torch.zeros((4096, 8), dtype=torch.int32, device="cuda")
        of = torch.zeros((4096, 2), dtype=torch.float32, device="cuda")
        d = torch.from_numpy(pos).cuda()
        c.index_probe_device(d.data_ptr(), 4096, oi.data_ptr(), of.data_ptr())
        torch.cuda.synchronize()
        got.append(of.cpu().numpy()[:, 0])
        c.close()
    np.testing.assert_array_equal(got[0], got[1])  # NaN where it is NaN
    assert np.isfinite(got[1]).any() and np.isnan(got[1]).any()
