"""What the library asks of the CUDA runtime, on a runtime without a GPU (fake_cudart.cpp):
kernels and attributes inside stream captures, memory held between calls."""
import json
import os
import subprocess
import sys

import pytest

from ppc_b200 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HEAD = """
import ctypes as C, json, sys
sys.path.insert(0, {root!r})
import numpy as np
import ppc_b200._lib as native
native.LIBPATH = {lib!r}
from ppc_b200 import types as T, workloads as W
from ppc_b200.api import PPC, Batch, Likelihood
rt = C.CDLL({lib!r})
rt.fake_log.restype = C.c_char_p
rt.fake_pinned.restype = rt.fake_device.restype = C.c_size_t

def log():
    return rt.fake_log().decode().splitlines()

def ctx(**opts):
    c = PPC()
    c.initialize(1.0, {ice!r})
    c.set_seed(1)
    c.set_options(**opts)
    c.choose(0)
    c.ini()
    return c
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    build.build()
    d = tmp_path_factory.mktemp("fake")
    names = build.CU + [f"{f}.{k}" for f, k in build.PARTS] + build.CPP
    objs = [os.path.join(build.OBJ, n + ".o") for n in names]
    rt, lib = str(d / "fake_cudart.o"), str(d / "libppcb_fake.so")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "fake_cudart.cpp")
    subprocess.run([build.CXX, "-std=c++17", "-O1", "-fPIC", "-I" + os.path.join(build.CUDA_HOME, "include"), "-c", src,
                    "-o", rt], check=True)
    subprocess.run([build.CXX, "-shared", "-Wl,-Bsymbolic", "-o", lib, rt] + objs, check=True)
    return lib


def _run(lib, ice, body):
    """What `body` leaves in `result`, in a process of its own."""
    code = HEAD.format(root=ROOT, lib=lib, ice=ice) + body + "\nprint('RESULT', json.dumps(result))\n"
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return json.loads(r.stdout.split("RESULT", 1)[1])


CAPTURES = {
    "propagate": """
buf, bs = np.zeros(1 << 20, np.uint8), np.array([0, 1000], np.uint64)
st, graph = C.addressof(C.create_string_buffer(8)), C.c_void_p()
rt.cudaStreamBeginCapture(C.c_void_p(st), 0)
c.propagate_device(buf.ctypes.data, bs.ctypes.data, 1, 1000, buf.ctypes.data, 10, buf.ctypes.data, stream=st)
rt.cudaStreamEndCapture(C.c_void_p(st), C.byref(graph))
""",
    "batch": """
b = W.cascade([0, 0, -100], [0, 0, 1], 1000, q=0)
Batch(c, 1, 1, 10000).run(b, 1)
""",
    "fit": """
b = W.cascade([0, 0, -100], [0, 0, 1], 1000, q=0)
c.gradient_graph(b, np.ones(c.info()["gsize"], np.float32), hit_cap=1000)
""",
    "likelihood": """
d = np.zeros(1, T.LLH_HIT_DTYPE)
d["str"], d["om"], d["t"], d["q"] = 1, 1, 100.0, 20.0
L = Likelihood(c, d)
h, out = np.zeros(100, T.HIT_DTYPE), np.zeros(1)
st, graph = C.addressof(C.create_string_buffer(8)), C.c_void_p()
rt.cudaStreamBeginCapture(C.c_void_p(st), 0)
L.eval_device(h.ctypes.data, 100, [0.0], 1.0, out.ctypes.data, stream=st)
rt.cudaStreamEndCapture(C.c_void_p(st), C.byref(graph))
""",
}


@pytest.mark.parametrize("opts", [{}, {"deterministic": True}, {"photon_streams": True}],
                         ids=["threads", "static", "photon_streams"])
@pytest.mark.parametrize("what", list(CAPTURES))
@pytest.mark.parametrize("kind", ["small_tilt", "full2d"])
def test_attributes_are_set_before_a_capture(fake, what, kind, opts, request):
    """A process's first call is a captured one: the kernels that it launches have their
    shared-memory limits, and are loaded, before the capture begins."""
    log = _run(fake, request.getfixturevalue("ice_" + kind), f"c = ctx(**{opts!r})" + CAPTURES[what]
               + "result = log()")
    assert any(x.startswith("captured ") for x in log)
    assert not [x for x in log if x.startswith("attribute-in-capture")]


@pytest.mark.parametrize("doms", [60, 400])
def test_likelihood_scratch_does_not_follow_the_hits(fake, ice_full2d, doms):
    """An evaluation's device memory does not depend on the number of hits or shifts: a later call
    of more gives nothing back that a captured call would still write to."""
    sizes = _run(fake, ice_full2d, """
c = ctx()
dom, per = np.repeat(np.arange(%d), 20), np.tile(np.arange(20), %d)
d = np.zeros(len(dom), T.LLH_HIT_DTYPE)
d["str"], d["om"], d["t"], d["q"] = dom // 60 + 1, dom %% 60 + 1, 100.0 + 50.0 * per, 20.0
L = Likelihood(c, d, lbin=25.0)
assert L.info()["blocks"] > 768  # 64 shifts' counters are more than one CTA's shared memory
dts, h, out = np.linspace(-100, 100, 64), np.zeros(5000, T.HIT_DTYPE), np.zeros(64)
L.eval_device(h.ctypes.data, 10, dts[:5], 1.0, out.ctypes.data)  # and the back end's tables
result = []
for n, ndt in ((1000, 5), (1000, 64), (5000, 64)):
    L.eval_device(h.ctypes.data, n, dts[:ndt], 1.0, out.ctypes.data)
    result.append(rt.fake_device())
""" % (doms, doms))
    assert sizes[0] == sizes[1] == sizes[2]


@pytest.mark.parametrize("given", ["observed", "weights"])
def test_gradient_keeps_little_pinned_memory(fake, ice_small, given):
    """Charges and counts of very many events do not stay behind in pinned memory."""
    few, many, counts = _run(fake, ice_small, """
c = ctx()
gsize = c.info()["gsize"]
b = W.cascade([0, 0, -100], [0, 0, 1], 1000, q=0)
result = []
for events in (64, 40 * (16 << 20) // (10 * gsize)):
    n = events * gsize
    r = c.gradient(b, events=events, %s=np.ones(n, np.float32), hit_cap=1000)
    result.append(rt.fake_pinned())
result.append(int(r["counts"].sum()))
""" % given)
    assert many - few <= 32 << 20 and counts == 0
