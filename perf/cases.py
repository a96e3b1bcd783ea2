"""Performance cases of the propagator and of the stages around it, through the Python API.

Every case runs with per-photon random streams (photon i draws from the stream of (seed, i)),
so that a call on the same inputs registers the same hits; the order in which hits are
appended changes from run to run, and a reader of hits sorts them by event, DOM and time.
Outputs are whole buffers: what lies beyond the records of a pass is zero.  Detector
configurations are the synthetic ones of ppc_b200/synth.py; one context per configuration is
kept for the whole program, as a user's program keeps its detector.

  kind      entry point                         what a program does there
  call      PPC.propagate                       host bunches in, host hits out
  device    PPC.propagate_device                bunches and hits stay on the GPU
  batch     Batch.run, counts, hits             many events in one launch
  gradient  PPC.gradient                        one likelihood and ice-gradient evaluation
  fit       PPC.gradient_graph, GradGraph.run   one iteration of an ice fit
  accept    PPC.accept_device / PPC.accept      the hit back end
  llh       Likelihood.eval_device              DirectFit's likelihood over time shifts
  sources   PPC.sources_device                  the source front end
"""
import math
import os

import numpy as np
import torch

from ppc_b200 import synth
from ppc_b200 import types as T
from ppc_b200 import workloads as W
from ppc_b200.api import PPC, Batch, Likelihood

os.environ.setdefault("PPCB_QUIET", "1")
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HIT_SEED, SRC_SEED, LLH_SEED = 7, 11, 5

# photon steps per photon and hits per photon of the configurations (round figures, for work())
STEPS = {"small": 36, "small_tilt": 36, "small_hole": 60, "small_xr1": 36, "full": 26, "full2d": 26, "full_ng": 26}
HITS = {"small": 7e-3, "small_tilt": 7e-3, "small_hole": 2e-3, "small_xr1": 3e-4, "full": 7e-3, "full2d": 7e-3,
        "full_ng": 7e-3}
STEP_FLOPS = 383  # single-precision and special-function operations of one propagation step
TABLE_BYTES = 1.1e6  # ice, tilt, detector and birefringence tables


def listed():
    return [
        # the smallest call: one low-energy secondary, a launch and its latency
        {"name": "call_cascade_1e3", "kind": "call", "ice": "full", "source": "cascade", "photons": 1000},
        # an ordinary call: one cascade of about a GeV, host buffers on both sides
        {"name": "call_cascade_1e6", "kind": "call", "ice": "full", "source": "cascade", "photons": 1_000_003},
        # the benchmark's workload: one bright cascade of 1e8 photons
        {"name": "device_cascade_1e8", "kind": "device", "ice": "full", "source": "cascade",
         "photons": 100_000_000},
        # a calibration flasher on the detector with the two-dimensional tilt map
        {"name": "device_flasher_1e7_2d", "kind": "device", "ice": "full2d", "source": "flasher",
         "photons": 10_000_000},
        # hole ice: a point source beside a string, short steps in and out of the column
        {"name": "device_point_1e6_hole", "kind": "device", "ice": "small_hole", "source": "point",
         "photons": 1_000_000},
        # a simulation file's events, half flashers and half cascades, very uneven sizes
        {"name": "batch_512", "kind": "batch", "ice": "full", "events": 512, "lo": 1e3, "hi": 1e6},
        # one evaluation of the charge likelihood and its ice gradient from host buffers
        {"name": "gradient_64x1e5", "kind": "gradient", "ice": "full", "events": 64, "photons": 100_000},
        # one iteration of the ice fit, captured once and replayed with new coefficients
        {"name": "fit_64x1e6", "kind": "fit", "ice": "full", "events": 64, "photons": 1_000_000},
        # back end over the hits of a bright cascade, on the GPU
        {"name": "accept_1.4e6_2d", "kind": "accept", "ice": "full2d", "hits": 1_379_861, "host": False},
        # back end over an ordinary event's hits on the multi-PMT detector, host buffers
        {"name": "accept_2e4_ng_host", "kind": "accept", "ice": "full_ng", "hits": 20_011, "host": True},
        # the time scan of a reconstruction: one event, 64 time shifts per evaluation
        {"name": "llh_1.4e6x64", "kind": "llh", "ice": "full2d", "hits": 1_379_861, "shifts": 64},
        # a muon bundle's secondaries turned into photon bunches
        {"name": "sources_1e6", "kind": "sources", "ice": "full", "sources": 1_000_000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "call", "device", "device", "batch", "gradient", "fit", "accept", "accept", "llh",
                       "llh", "sources", "sources"])
    if kind in ("call", "device"):
        ice = rng.choice(["full", "full", "full2d", "full_ng", "small", "small_tilt", "small_hole", "small_xr1"])
        hi = 3e6 if kind == "call" else 5e7
        return {"kind": kind, "ice": ice, "source": rng.choice(["cascade", "flasher", "point", "muon"]),
                "photons": _log(rng, 1e3, hi if ice.startswith("full") else hi / 5)}
    if kind == "batch":
        return {"kind": kind, "ice": "full", "events": _log(rng, 8, 512), "lo": 1e3,
                "hi": float(_log(rng, 1e4, 1e6))}
    if kind in ("gradient", "fit"):
        return {"kind": kind, "ice": "full", "events": _log(rng, 2, 64), "photons": _log(rng, 1e4, 1e6)}
    if kind == "accept":
        host = rng.random() < 0.5
        return {"kind": kind, "ice": rng.choice(["full", "full2d", "full_ng"]),
                "hits": _log(rng, 1e2, 2e5 if host else 2e6), "host": host}
    if kind == "llh":
        return {"kind": kind, "ice": rng.choice(["full", "full2d"]), "hits": _log(rng, 1e3, 2e6),
                "shifts": rng.choice([1, 1, 5, 16, 33, 64])}
    return {"kind": kind, "ice": "full", "sources": _log(rng, 1e2, 2e6)}


# ---------------------------------------------------------------- what a program has at hand
_contexts = {}


def _ice_dir(ice):
    path = os.path.join(ROOT, "ppc_b200", "data", "ice", ice)
    if not os.path.exists(os.path.join(path, "cfg.txt")):
        synth.write(ice, path)
    return path


def _context(ice, role="", gpu=True):
    """The program's context for a configuration (the fit has its own: it changes the ice)."""
    key = (ice, role, gpu)
    if key not in _contexts:
        c = PPC()
        c.initialize(1.0, _ice_dir(ice))
        c.set_seed(20)
        c.set_options(photon_streams=True)
        if gpu:
            c.choose(0)
            c.ini()
        _contexts[key] = c
    return _contexts[key]


def _direction(rng):
    ct, ph = rng.uniform(-1, 1), rng.uniform(0, 2 * math.pi)
    st = math.sqrt(1 - ct * ct)
    return [st * math.cos(ph), st * math.sin(ph), ct]


def _bunch(case, c, rng):
    num, source, full = case["photons"], case["source"], case["ice"].startswith("full")
    reach = 400.0 if full else 120.0
    v = rng.uniform(-reach, reach, 3)
    if source == "cascade":
        return W.cascade(v, _direction(rng), num, q=1)
    if source == "flasher":
        oms = c.tables()["oms"]
        k = int(rng.integers(0, len(oms)))
        return W.flasher(k, oms["r"][k], num, q=1)
    if source == "muon":  # a bare muon's track segment
        return T.bunch_particle([*v, 0.0], _direction(rng), 1, num, 0, f=0.84, length=float(rng.uniform(5, 50)))
    # an isotropic point source; among the 7 strings it sits within the column of the central one
    x, y = (rng.uniform(-0.5, 0.5, 2) if not full else v[:2])
    return T.bunch_led([x, y, rng.uniform(-200, 200), 0.0], [0, 0, 1], 1, num, 1, ka=-1, up=0, fldr=-1)


def _on_gpu(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1).copy()).cuda()


def _flashers(case, c, rng):
    oms = c.tables()["oms"]
    k = rng.integers(0, len(oms), case["events"])
    b = np.concatenate([W.flasher(int(j), oms["r"][j], case["photons"], q=e) for e, j in enumerate(k)])
    # observed charges: falling with the distance from the flasher, Poisson
    d = np.linalg.norm(oms["r"][k][:, None, :] - oms["r"][None], axis=2)
    mean = case["photons"] * 4e-4 * np.exp(-d / 25.0) / (1 + d / 17.0)
    return b, rng.poisson(mean).astype(np.float32)


def _hits(case, c, n, gen):
    """Kernel-level hits of one cascade as the back end meets them: n records on the GPU."""
    oms = torch.from_numpy(np.ascontiguousarray(c.tables()["oms"]["r"])).cuda()
    u = lambda *s: torch.rand(*s, generator=gen, device="cuda")
    v = (u(3) - 0.5) * 800
    d = (oms - v).norm(dim=1)
    i = torch.multinomial(torch.exp(-d / 30) / (5 + d), n, replacement=True, generator=gen)
    di = d[i]
    h = torch.empty((n, 8), dtype=torch.float32, device="cuda")
    w = h.view(torch.int32)
    w[:, 0] = i.int()
    w[:, 1] = 1
    w[:, 2] = (u(n) * 512).int().clamp_(max=511)
    h[:, 3] = di / 0.22 - torch.log1p(-u(n)) * (20 + 1.5 * di)
    h[:, 4] = torch.arccos(2 * u(n) - 1)
    h[:, 5] = (u(n) - 0.5) * (2 * math.pi)
    h[:, 6] = torch.arccos(2 * u(n) - 1)
    h[:, 7] = (u(n) - 0.5) * (2 * math.pi)
    return h


def _pulses(h, gen):
    """Observed pulses of the same cascade: about half of the hits, on (string, DOM)."""
    keep = h[torch.rand(len(h), generator=gen, device="cuda") < 0.5].cpu().numpy()
    data = np.zeros(len(keep), T.LLH_HIT_DTYPE)
    i = keep[:, 0].view(np.int32)
    data["str"], data["om"], data["t"], data["q"] = i // 60 + 1, i % 60 + 1, keep[:, 3], 1.0
    return data


def _source_list(case, seed):
    n = case["sources"]
    rng = np.random.default_rng(seed)
    s = np.zeros(n, T.SOURCE_DTYPE)
    s["kind"] = T.SRC_PARTICLE
    s["r"][:, :3] = rng.uniform(-400, 400, (n, 3))
    s["r"][:, 3] = rng.uniform(0, 5000, n)
    s["n"] = [0.3, 0.4, 0.8660254]
    s["amount"] = 10 ** rng.uniform(-1, 1, n)
    s["type"] = rng.choice(np.array([0, 11, 12, 13, 14, 101, 102, 105]), n)
    s["dr"] = np.where(s["type"] == 0, rng.uniform(1, 20, n), 0)
    s["scale"] = 1
    s["q"] = np.arange(n)
    return s


def _hit_capacity(photons):
    return max(1 << 16, photons // 16)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _event(case, c, seed):
    """Simulated hits (GPU), observed pulses (host) and time shifts of an llh case."""
    gen = _generator(seed)
    h = _hits(case, c, case["hits"], gen)
    obs = _pulses(h[: max(64, case["hits"] // 10)], gen)
    dts = np.linspace(-200.0, 200.0, case["shifts"]) if case["shifts"] > 1 else np.array([12.5])
    return h, obs, dts


def prepare(case, seed):
    kind, rng = case["kind"], np.random.default_rng(seed)
    c = _context(case["ice"], "fit" if kind == "fit" else "")
    s = {"case": case, "ctx": c}
    if kind == "call":
        s["bunches"] = _bunch(case, c, rng)
        cap = _hit_capacity(case["photons"])
        s["out"] = np.empty(cap, T.HIT_DTYPE)
        s["ordered"] = np.zeros((cap, 8), np.int32)
    elif kind == "device":
        cap = _hit_capacity(case["photons"])
        s["bunches"] = _on_gpu(_bunch(case, c, rng))
        s["bstart"] = torch.tensor([0, case["photons"]], dtype=torch.int64, device="cuda")
        s["hits"] = torch.empty((cap, 8), dtype=torch.int32, device="cuda")
        s["ordered"] = torch.zeros((cap, 8), dtype=torch.int32, device="cuda")
        s["ctrl"] = torch.zeros(7, dtype=torch.int64, device="cuda")
    elif kind == "batch":
        s["bunches"] = W.batched_events(c.tables()["oms"], case["events"], case["lo"], case["hi"], seed)
        cap = case["events"] * int(case["hi"] * 0.05 + 66)
        s["batch"] = Batch(c, case["events"], case["events"], cap)
        s["ordered"] = torch.zeros((case["events"] * 20_000, 8), dtype=torch.int32, device="cuda")
    elif kind == "gradient":
        s["bunches"], s["observed"] = _flashers(case, c, rng)
    elif kind == "fit":
        b, obs = _flashers(case, c, rng)
        if "be0" not in _contexts:
            _contexts["be0"] = c.get_ice()
        be, ba = _contexts["be0"]
        s["be"] = (be * np.exp(0.1 * rng.normal(size=len(be)))).astype(np.float32)
        s["ba"] = (ba * np.exp(0.1 * rng.normal(size=len(ba)))).astype(np.float32)
        s["graph"] = c.gradient_graph(b, obs, events=case["events"], scale=1.0)
    elif kind == "accept":
        h = _hits(case, c, case["hits"], _generator(seed))
        if case["host"]:
            s["hits"] = h.cpu().numpy().view(T.HIT_DTYPE).reshape(-1)
            s["out"] = np.zeros((case["hits"], 14), np.int32)
        else:
            s["hits"] = h
            s["out"] = torch.zeros((case["hits"], 14), dtype=torch.int32, device="cuda")
            s["count"] = torch.zeros(1, dtype=torch.int64, device="cuda")
    elif kind == "llh":
        s["hits"], obs, s["dts"] = _event(case, c, seed)
        s["llh"] = Likelihood(c, obs)
        s["out"] = torch.empty(case["shifts"], dtype=torch.float64, device="cuda")
    else:
        n = case["sources"]
        s["sources"] = _on_gpu(_source_list(case, seed))
        s["bunches"] = torch.zeros((n + 1024, 16), dtype=torch.int32, device="cuda")
        s["bstart"] = torch.zeros(n + 1025, dtype=torch.int64, device="cuda")
        s["counts"] = torch.zeros(2, dtype=torch.int64, device="cuda")
    return s


# ---------------------------------------------------------------- one pass
def _columns(h, names, ints):
    """Records (rows of 4-byte words, numpy or torch int32) as named columns."""
    f = h.view(torch.float32 if isinstance(h, torch.Tensor) else np.float32)
    return {n: (h if n in ints else f)[:, k] for k, n in enumerate(names)}


def _in_order(w, to):
    """Hit records (int32 words) by event, DOM and time, at the head of the buffer `to`."""
    x = w.long() if isinstance(w, torch.Tensor) else w.astype(np.int64)
    key = (((x[:, 1] << 13) | x[:, 0]) << 41) | (x[:, 3] << 10) | (x[:, 5] & 1023)
    to[: len(w)] = w[key.argsort()]
    return _columns(to, ("i", "n", "z", "t", "pth", "pph", "dth", "dph"), ("i", "n", "z"))


def _words(rec):
    return rec.view(np.int32).reshape(len(rec), rec.itemsize // 4)


def run(s):
    kind, c = s["case"]["kind"], s["ctx"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "call":
        hits, info = c.propagate(s["bunches"], out=s["out"])
        return {"hits": _in_order(_words(hits), s["ordered"]), "steps": info["steps"], "photons": info["photons"]}
    if kind == "device":
        s["ctrl"].zero_()
        c.propagate_device(s["bunches"].data_ptr(), s["bstart"].data_ptr(), 1, s["case"]["photons"],
                           s["hits"].data_ptr(), len(s["hits"]), s["ctrl"].data_ptr(), stream)
        n = min(int(s["ctrl"][1].item()), len(s["hits"]))
        return {"hits": _in_order(s["hits"][:n], s["ordered"]), "steps": s["ctrl"][3]}
    if kind == "batch":
        info = s["batch"].run(s["bunches"], s["case"]["events"], hits_per_photon=0.05)
        produced, offsets = s["batch"].counts()
        hits = torch.from_numpy(_words(s["batch"].hits())).cuda()
        return {"hits": _in_order(hits, s["ordered"]), "produced": produced.astype(np.int64),
                "offsets": offsets.astype(np.int64), "steps": info["steps"]}
    if kind == "gradient":
        r = c.gradient(s["bunches"], observed=s["observed"], events=s["case"]["events"])
        return {"ll": r["ll"], "counts": r["counts"].astype(np.int64), "g_be": r["g_be"], "g_ba": r["g_ba"]}
    if kind == "fit":
        r = s["graph"].run(s["be"], s["ba"])
        return {"ll": r["ll"], "counts": r["counts"].astype(np.int64), "g_be": r["g_be"], "g_ba": r["g_ba"]}
    if kind == "accept":
        if s["case"]["host"]:
            acc = c.accept(s["hits"], seed=HIT_SEED)
            s["out"][: len(acc)] = _words(acc)
            count = len(acc)
        else:
            c.accept_device(s["hits"].data_ptr(), len(s["hits"]), HIT_SEED, s["out"].data_ptr(),
                            s["count"].data_ptr(), stream)
            count = s["count"]
        names = ("i", "n", "hit", "str", "om", "pmt", "t", "wv", "rx", "ry", "rz", "dx", "dy", "dz")
        return {"hits": _columns(s["out"], names, names[:6]), "count": count}
    if kind == "llh":
        s["llh"].eval_device(s["hits"].data_ptr(), len(s["hits"]), s["dts"], 10.0, s["out"].data_ptr(),
                             seed=LLH_SEED, stream=stream)
        return s["out"]
    n = s["case"]["sources"]
    c.sources_device(s["sources"].data_ptr(), n, SRC_SEED, s["bunches"].data_ptr(), s["bstart"].data_ptr(), n + 1024,
                     s["counts"].data_ptr(), stream)
    b, f = s["bunches"], s["bunches"].view(torch.float32)
    return {"r": f[:, 0:4], "n": f[:, 4:8], "q": b[:, 8], "num": b[:, 9], "type": b[:, 10], "f": f[:, 11],
            "u": f[:, 12:16], "bstart": s["bstart"], "counts": s["counts"]}


def work(case):
    """Bytes in and out once, and the arithmetic of the path (propagation: its steps)."""
    kind = case["kind"]
    if kind in ("call", "device"):
        n, h = case["photons"], case["photons"] * HITS[case["ice"]]
        return {"bytes": 64 + TABLE_BYTES + 32 * h, "flops": STEP_FLOPS * STEPS[case["ice"]] * n}
    if kind == "batch":
        n = case["events"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        return {"bytes": 64 * case["events"] + TABLE_BYTES + 32 * 7e-3 * n, "flops": STEP_FLOPS * 26 * n}
    if kind in ("gradient", "fit"):
        n, bins = case["events"] * case["photons"], case["events"] * 5160
        return {"bytes": TABLE_BYTES + 96 * 1e-3 * n + 8 * bins, "flops": STEP_FLOPS * 30 * n}
    if kind == "accept":
        return {"bytes": 32 * case["hits"] + 56 * 0.4 * case["hits"], "flops": 120 * case["hits"]}
    if kind == "llh":
        return {"bytes": 32 * case["hits"], "flops": 120 * case["hits"] + 6 * 0.4 * case["hits"] * case["shifts"]}
    return {"bytes": (72 + 64 + 8) * case["sources"], "flops": 600 * case["sources"]}


# ---------------------------------------------------------------- the same in 64 bits
class _Stream:
    """The multiply-with-carry stream of record k: a SplitMix64 hash of (seed, k) and a multiplier."""

    def __init__(self, seed, word, k, rm):
        k = k.astype(np.uint64)
        with np.errstate(over="ignore"):
            z = np.uint64(seed << 32 | word) + (k + np.uint64(1)) * np.uint64(0x9E3779B97F4A7C15)
            z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
            z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z ^= z >> np.uint64(31)
        self.a = rm[k % np.uint64(1024)].astype(np.uint64)
        self.x = z & np.uint64(0xFFFFFFFF)
        self.y = ((z >> np.uint64(32)) * self.a) >> np.uint64(32)

    def u(self, at=slice(None)):
        s = self.a[at] * self.x[at] + self.y[at]
        self.x[at], self.y[at] = s & np.uint64(0xFFFFFFFF), s >> np.uint64(32)
        return 1.0 - (self.x[at] >> np.uint64(9)).astype(np.float64) / 2 ** 23


def _wavelength_acceptance(ice):
    """Acceptance of the standard sensor in each of the 512 bins of its own emission spectrum."""
    frac, wv = np.loadtxt(os.path.join(_ice_dir(ice), "wv.dat")).T
    step = np.diff(wv)
    qw, qf = wv[1:] - step / 2, np.diff(frac) / step
    qw = np.concatenate([[qw[0] - step[0]], qw, [qw[-1] + step[-1]]])
    dat = np.interp(250.5 + np.arange(450), qw, np.concatenate([[0], qf, [0]]), left=0, right=0)
    cum = np.cumsum(dat) / dat.sum()

    def position(p):  # where the cumulative spectrum reaches p, in bins of a nanometre
        first = int(np.argmax(cum > 0)) - 1
        j = max(min(int(np.searchsorted(cum, p)), 449), first + 1)
        d = cum[j] - cum[j - 1]
        return j - 1 + ((p - cum[j - 1]) / d if d > 0 else 0)

    rat = np.zeros(512)
    for n in range(512):
        a, b = position(n / 512), position(min((n + 1) / 512, cum[-1]))
        x = np.arange(450)
        rat[n] = 512 / dat.sum() * (dat * np.clip(np.minimum(b, x + 1) - np.maximum(a, x), 0, 1)).sum()
    return rat


def _accepted(case, c, h, seed):
    """Which hits a standard sensor registers: acceptance, angular sensitivity, cable shadow."""
    h = h.cpu().numpy()
    i = h[:, 0].view(np.int32)
    a = h[:, 3:].astype(np.float64)
    s = _Stream(seed, 0x6A09E667, np.arange(len(h)), c.tables()["rm"])
    ok = s.u() < _wavelength_acceptance(case["ice"])[h[:, 2].view(np.int32)]
    u = s.u()
    axis = np.tile([0.0, 0.0, 1.0], (5160, 1))
    cable = np.full(5160, np.nan)
    if case["ice"] == "full2d":
        for name, to in (("cx.dat", axis), ("dx.dat", cable)):
            rows = np.loadtxt(os.path.join(_ice_dir(case["ice"]), name))
            at = ((rows[:, 0] - 1) * 60 + rows[:, 1] - 1).astype(int)
            to[at] = rows[:, 2:5] if name == "cx.dat" else rows[:, 2]
    n = np.stack([np.sin(a[:, 1]) * np.cos(a[:, 2]), np.sin(a[:, 1]) * np.sin(a[:, 2]), np.cos(a[:, 1])], 1)
    x = (n * axis[i]).sum(1)
    ok &= u < 0.35 + 0.5 * x + 0.15 * x * x
    R, rc, p = T.OMR, 0.023, np.radians(cable[i])
    qx = -R * np.sin(a[:, 3]) * np.cos(a[:, 4]) - (R + rc) * np.cos(p)
    qy = -R * np.sin(a[:, 3]) * np.sin(a[:, 4]) - (R + rc) * np.sin(p)
    aa, b = n[:, 0] ** 2 + n[:, 1] ** 2, n[:, 0] * qx + n[:, 1] * qy
    with np.errstate(invalid="ignore"):
        D = b * b - aa * (qx * qx + qy * qy - rc * rc)
        ok &= ~((D >= 0) & (b + np.sqrt(np.maximum(D, 0)) > 0))
    return ok, i, a[:, 0]


def _llf(s, d, nsim, sig=0.10):
    """DirectFit's saturated likelihood of s simulated (nsim times) against d observed (once)."""
    if s == 0 and d == 0:
        return 0.0
    sd, s2 = s + d, sig * sig
    ls = ld = sd / (1 + nsim)
    while True:
        f = nsim * ls - s - math.log(ld / ls) / s2
        step = -f / (nsim * (1 + (1 / ld + 1 / (nsim * ls)) / s2))
        ls += step
        ld = sd - nsim * ls
        if abs(step) <= 1e-8 * ls:
            break
    r = math.log(ld / ls) ** 2 / (2 * s2)
    r += s * math.log(s / nsim / ls) if s > 0 else 0.0
    return r + (d * math.log(d / ld) if d > 0 else 0.0)


def _exact_llh(case, seed):
    c = _context(case["ice"])
    h, obs, dts = _event(case, c, seed)
    like = Likelihood(c, obs)
    info, blocks = like.info(), like.blocks()
    ok, dom, t = _accepted(case, c, h, LLH_SEED)
    dom, t = dom[ok], t[ok]
    table = np.full((5160, 201), -1)
    for k, b in enumerate(blocks):
        at = (b["str"] - 1) * 60 + b["om"] - 1
        table[at, min(b["first"], b["last"]):max(b["first"], b["last"]) + 1] = k
    out = np.zeros(len(dts))
    for j, dt in enumerate(dts):
        q = (t + dt - info["t0"]) / info["lbin"]
        q = np.copysign(np.floor(np.abs(q) + 0.5), q)  # halves away from zero
        inside = (q >= 0) & (q < 200)
        k = table[dom[inside], q[inside].astype(int)]
        n = np.bincount(k[k >= 0], minlength=len(blocks))
        out[j] = sum(_llf(float(x), float(y), 10.0) for x, y in zip(n, blocks["dat"])) / info["ndof"]
    return out


def _lgamma(xx):
    """log Gamma by the Lanczos series of the sampler."""
    cof = (76.18009172947146, -86.50532032941677, 24.01409824083091, -1.231739572450155, 0.1208650973866179e-2,
           -0.5395239384953e-5)
    tmp = xx + 4.5 - (xx - 0.5) * np.log(xx + 4.5)
    return -tmp + np.log(2.5066282746310005 * (1 + sum(q / (xx + j) for j, q in enumerate(cof))))


def _poisson(mean, s):
    """The sampler's counts: products of uniforms below 12, rejection from a Lorentzian above."""
    num = np.zeros(len(mean), np.int64)
    at = np.flatnonzero(mean < 12)
    g, t = np.exp(-mean[at]), s.u(at)
    while True:
        more = t > g
        at, g, t = at[more], g[more], t[more]
        if not len(at):
            break
        num[at] += 1
        t = t * s.u(at)
    at = np.flatnonzero(mean >= 12)
    y, em = np.zeros(len(mean)), np.zeros(len(mean))
    pi32 = np.float32(3.141592653589793)
    while len(at):
        draw = at
        while len(draw):
            y[draw] = np.tan((pi32 * s.u(draw).astype(np.float32)).astype(np.float64))
            em[draw] = np.sqrt(2 * mean[draw]) * y[draw] + mean[draw]
            draw = draw[em[draw] < 0]
        m, um, lm = mean[at], np.floor(em[at]), np.log(mean[at])
        with np.errstate(over="ignore"):
            t = 0.9 * (1 + y[at] ** 2) * np.exp(um * lm - _lgamma(um + 1) - (m * lm - _lgamma(m + 1)))
        num[at] = um.astype(np.int64)
        at = at[s.u(at) > t]
    return num


def _exact_sources(case, seed):
    c = _context(case["ice"])
    src = _source_list(case, seed)
    s = _Stream(SRC_SEED, 0x3C6EF372, np.arange(len(src)), c.tables()["rm"])
    E, typ = src["amount"].astype(np.float32).astype(np.float64), src["type"]
    logE = np.log(np.maximum(0.105658389, E))
    rho = 0.910 / 0.9216
    extr = 1 + np.maximum(0.0, 0.1880 + 0.0206 * logE) * rho
    muon = typ == 0
    nph = np.where(muon, src["dr"] * extr, 5.321 * rho * E)
    f = np.where(muon, 1 / extr, 0.0)
    a, b = np.zeros(len(src)), np.zeros(len(src))
    L = 0.39652 * rho
    for kinds, a0, a1, bb in (((11, 12), 2.01849, 0.63176, 0.63207), ((13,), 2.00035, 0.63190, 0.63008),
                              ((14,), 2.83923, 0.58209, 0.64526), ((101, 102), 1.58357292, 0.41886807, 0.33833116),
                              ((105,), 1.47495778, 0.40450398, 0.35226706)):
        at = np.isin(typ, kinds)
        a[at], b[at] = a0 + a1 * logE[at], L / bb
    for kinds, E0, m, f0, rms0, gamma in (((101, 102), 0.18791678, 0.16267529, 0.30974123, 0.95899551, 1.35589541),
                                          ((105,), 0.29579368, 0.19373018, 0.02455403, 1.01619344, 1.45477346)):
        at = np.flatnonzero(np.isin(typ, kinds))
        e = np.maximum(2.71828183, E[at])
        F = 1 - (e / E0) ** -m * (1 - f0)
        w, todo = np.zeros(len(at)), np.arange(len(at))
        while len(todo):  # the hadronic fluctuation, truncated to [0, 1.1]
            k = at[todo]
            r = np.sqrt(-2 * np.log(s.u(k)))
            w[todo] = F[todo] * (1 + rms0 * np.log(e[todo]) ** -gamma * r * np.sin(2 * np.pi * s.u(k)))
            todo = todo[(w[todo] < 0) | (w[todo] > 1.1)]
        nph[at] *= w
    info = c.info()
    num = _poisson(info["eff"] * nph / info["ovr"], s)
    k = np.flatnonzero(num > 0)
    r, n, u = (np.zeros((len(src) + 1024, 4)) for _ in range(3))
    m = len(k)
    r[:m], n[:m, :3], n[:m, 3] = src["r"][k], src["n"][k], src["dr"][k]
    u[:m, 0], u[:m, 1], u[:m, 2] = a[k], b[k], 1.0
    fr = np.zeros(len(src) + 1024)
    fr[:m] = f[k]
    return {"r": r, "n": n, "q": None, "num": None, "type": None, "f": fr, "u": u, "bstart": None, "counts": None}


def exact(case, seed):
    """Outputs in 64 bits: the likelihoods and the bunch templates.  The hits of a random walk and
    which hits a random draw accepts have no such value, nor has a gradient along those walks."""
    if case["kind"] == "llh":
        return _exact_llh(case, seed)
    if case["kind"] == "sources":
        return _exact_sources(case, seed)
    return None
