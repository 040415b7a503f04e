"""The bounded waits of the persistent solve.  WL_PERSIST_POLLS=0 (read once: a child process) makes every barrier wait
that is not over at its first poll run out, which on a grid of many blocks happens in the first barriers.  The kernel
then gives up, the loop ends, and the solve starts again with the ordinary launches from the caller's data: bitwise the
result of an engine stepped from the host.  The next solve of the same engine and a solve of another context run as
usual, and nothing is left on the device that waits."""

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

shape = (8, 8, 8, 8)
rng = np.random.default_rng(8)
U = W.hot_links(rng, shape, 1, 0.25)
masses = np.array([-0.1, 0.05, 0.2, 0.0])
rep = []
for inner, n in (("double", 1), ("single", 3), ("half", 4)):
    ctx = WilsonContext(shape, bc=(1, 1, 1, -1))
    gauge = ctx.gauge(torch.from_numpy(U[0]))
    b = torch.from_numpy(W.project(W.gaussian_spinor(rng, shape, n), 0)).cuda()
    x0 = torch.from_numpy(W.project(W.gaussian_spinor(rng, shape, n), 0)).cuda()
    eng = Engine(ctx, gauge, n, inner=inner, tol=1e-10, maxiter=2000)
    eng.admit(np.arange(n), b, masses[:n])
    while eng.poll()[1]:
        eng.step(8)
    ref = [eng.retire(r) for r in range(n)]
    eng.close()
    for use_graph in (True, False):
        for again in range(2):
            x, st = ctx.solve(gauge, b, masses[:n], tol=1e-10, maxiter=2000, inner=inner, use_graph=use_graph)
            rep.append({"case": [inner, use_graph, again],
                        "converged": all(s["status"] == SLOT_CONVERGED and s["true_res"] <= 1e-10 for s in st),
                        "same": all(torch.equal(x[r], ref[r][0]) and s["iters"] == ref[r][1]["iters"]
                                    for r, s in enumerate(st))})
        x, st = ctx.solve(gauge, b, masses[:n], tol=1e-10, maxiter=2000, inner=inner, use_graph=use_graph, x0=x0)
        rep.append({"case": [inner, use_graph, "x0"],
                    "converged": all(s["status"] == SLOT_CONVERGED and s["true_res"] <= 1e-10 for s in st),
                    "same": True})
    ctx.close()
print(json.dumps(rep))
"""


@pytest.mark.parametrize("polls", ["0", "2"])
def test_a_wait_that_runs_out_restarts_the_solve_with_the_ordinary_launches(polls):
    res = subprocess.run([sys.executable, "-c", CHILD.replace("ROOT", repr(ROOT), 1)], cwd=ROOT, capture_output=True,
                         text=True, timeout=900, env=dict(os.environ, WL_PERSIST="2", WL_PERSIST_POLLS=polls))
    assert res.returncode == 0, res.stdout[-2000:] + res.stderr[-4000:]
    rep = json.loads(res.stdout.strip().splitlines()[-1])
    assert len(rep) == 3 * 2 * 3
    for case in rep:
        assert case["converged"] and case["same"], case
