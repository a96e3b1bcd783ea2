"""A process whose first GPU work is a captured one."""
import os
import subprocess
import sys

import pytest

from conftest import have_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA GPU")]

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CODE = """
import sys
sys.path.insert(0, {root!r})
import numpy as np
from ppc_b200 import workloads as W
from ppc_b200.api import PPC, Batch
c = PPC()
c.initialize(1.0, {ice!r})
c.set_seed(11)
c.set_options(photon_streams=True)
c.choose(0)
c.ini()
k = int(c.info()["gsize"]) // 2
b = W.flasher(k, c.tables()["oms"]["r"][k], 200_000, q=0)
if {what!r} == "fit":
    q = np.ones(c.info()["gsize"], np.float32)
    first = c.gradient_graph(b, q, events=1).run()
    then = c.gradient(b, events=1, observed=q)
    assert then["info"]["hits"] > 10 and first["info"]["hits"] == then["info"]["hits"]
    assert np.array_equal(first["counts"].reshape(-1), then["counts"].reshape(-1))
    for g in ("g_ba", "g_be"):
        np.testing.assert_allclose(first[g], then[g], rtol=1e-9, atol=1e-9 * np.abs(then[g]).max())
else:
    B = Batch(c, 1, len(b), 200_000)
    first = B.run(b, 1, 0.5)
    B.set_graph(False)
    then = B.run(b, 1, 0.5)
    assert then["hits"] > 10 and (first["hits"], first["steps"]) == (then["hits"], then["steps"])
print("same")
"""


@pytest.mark.parametrize("what", ["fit", "batch"])
@pytest.mark.parametrize("kind", ["small", "full", "full2d", "small_hole"])
def test_graph_first(what, kind, request):
    """The graph's results are those of the plain calls after it (sums in another order: 1e-9)."""
    code = CODE.format(root=ROOT, ice=request.getfixturevalue("ice_" + kind), what=what)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr
