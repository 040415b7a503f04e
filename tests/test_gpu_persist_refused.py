"""The fallback of the persistent solve.  WL_PERSIST=3 makes the library refuse every cooperative launch on the host,
before anything is launched (a child process, since the switch is read once).  The solve must then be the ordinary one
from the first iteration on: the same kernels in the same order as an engine stepped from the host, so bitwise the same
solutions and iteration counts, driven by the loop graph and from the host."""

import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("CUDA device required", allow_module_level=True)

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import json, sys
import numpy as np, torch
sys.path.insert(0, ROOT)
from jaxqft_b200.lib import SLOT_CONVERGED, Engine, WilsonContext
from oracle import wilson as W

shape, n = (4, 4, 4, 8), 3
rng = np.random.default_rng(5)
U = W.hot_links(rng, shape, 1, 0.25)
ctx = WilsonContext(shape, bc=(1, 1, 1, -1))
gauge = ctx.gauge(torch.from_numpy(U[0]))
masses = np.array([-0.2, 0.05, -0.1])
rep = []
for inner in ("double", "single", "half"):
    for op in ("eo_normal", "normal"):
        b = W.gaussian_spinor(rng, shape, n)
        b = torch.from_numpy(W.project(b, 0) if op == "eo_normal" else b).cuda()
        eng = Engine(ctx, gauge, n, op=op, inner=inner, tol=1e-10, maxiter=2000)
        eng.admit(np.arange(n), b, masses)
        while eng.poll()[1]:
            eng.step(8)
        ref = [eng.retire(r) for r in range(n)]
        eng.close()
        for use_graph in (True, False):
            for again in range(2):
                x, st = ctx.solve(gauge, b, masses, op=op, tol=1e-10, maxiter=2000, inner=inner, use_graph=use_graph)
                rep.append({"case": [inner, op, use_graph, again],
                            "converged": all(s["status"] == SLOT_CONVERGED and s["true_res"] <= 1e-10 for s in st),
                            "same": all(torch.equal(x[r], ref[r][0]) and s["iters"] == ref[r][1]["iters"]
                                        for r, s in enumerate(st))})
print(json.dumps(rep))
"""


def test_a_refused_launch_leaves_the_solve_to_the_ordinary_iterations():
    res = subprocess.run([sys.executable, "-c", CHILD.replace("ROOT", repr(ROOT), 1)], cwd=ROOT, capture_output=True,
                         text=True, timeout=900, env=dict(os.environ, WL_PERSIST="3"))
    assert res.returncode == 0, res.stdout[-2000:] + res.stderr[-4000:]
    rep = json.loads(res.stdout.strip().splitlines()[-1])
    assert len(rep) == 24
    for case in rep:
        assert case["converged"] and case["same"], case
