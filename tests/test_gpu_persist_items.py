"""The persistent iteration kernel where a warp has more than one item: sweeps over several groups of sites per warp,
several slots on one block, several lane tiles per warp with the links staged anew, blocks whose share crosses the
parities of the full operator, ragged last items.  WL_PERSIST_BLOCKS=3 spreads a small lattice over three blocks (a
child process, since the switch is read once); without it the lattice takes the default dispatch.

The kernel must really have run: a solve then makes fewer than four launches an iteration (one per reliable update and
what belongs to that), the ordinary one seven or nine.  Reference: an engine stepped from the host and the numpy oracle.
Both run the same CG in the same precision with sums grouped differently, so they take the same number of iterations up
to one reliable update's worth of rounding (two iterations), and the FP64 residual is at most tol."""

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
from jaxqft_b200.lib import SLOT_CONVERGED, Engine, WilsonContext, kernel_launches
from oracle import wilson as W

shape, bc, tol = (6, 6, 10, 14), (1, 1, 1j, -1), 1e-10
rng = np.random.default_rng(31)
U = W.hot_links(rng, shape, 1, 0.25)
ctx = WilsonContext(shape, bc=bc)
gauge = ctx.gauge(torch.from_numpy(U[0]))
field = W.gaussian_spinor(rng, shape, 16)
rep = []
for op in ("eo_normal", "normal"):
    b = W.project(field, 0) if op == "eo_normal" else field
    bt = torch.from_numpy(b).cuda()
    for inner, counts in (("double", (1, 3)), ("single", (1, 3, 5, 8, 16)), ("half", (1, 3, 4, 12, 16))):
        for n in counts:
            masses = np.linspace(0.3, 0.0, n)
            solve = lambda: ctx.solve(gauge, bt[:n], masses, op=op, tol=tol, maxiter=2000, inner=inner)
            solve()
            before = kernel_launches()
            x, st = solve()
            launches = kernel_launches() - before
            eng = Engine(ctx, gauge, n, op=op, inner=inner, tol=tol, maxiter=2000)
            eng.admit(np.arange(n), bt[:n], masses)
            while eng.poll()[1]:
                eng.step(8)
            ref = [eng.retire(r)[1] for r in range(n)]
            eng.close()
            r = n - 1  # the slot that takes the most iterations, against the oracle
            xr = x[r].cpu().numpy()[None]
            if op == "eo_normal":
                s = W.schur_even(U, xr, masses[r], bc, normalized=True)
                ax = W.schur_even(U, s, masses[r], bc, normalized=True, dag=True)[0]
            else:
                ax = W.apply_normal(U, xr, masses[r], bc)[0]
            rep.append({"case": [op, inner, n], "launches": launches, "iters": [s["iters"] for s in st],
                        "ref_iters": [s["iters"] for s in ref],
                        "converged": all(s["status"] == SLOT_CONVERGED and s["true_res"] <= tol for s in st),
                        "residual": float(np.linalg.norm(b[r] - ax) / np.linalg.norm(b[r]))})
print(json.dumps(rep))
"""


@pytest.mark.parametrize("blocks", ["3", None])
def test_several_items_per_warp(blocks):
    env = dict(os.environ, WL_PERSIST="2", WL_PERSIST_BLOCKS=blocks) if blocks else dict(os.environ)
    res = subprocess.run([sys.executable, "-c", CHILD.replace("ROOT", repr(ROOT), 1)], cwd=ROOT, capture_output=True,
                         text=True, timeout=900, env=env)
    assert res.returncode == 0, res.stdout[-2000:] + res.stderr[-4000:]
    rep = json.loads(res.stdout.strip().splitlines()[-1])
    assert len(rep) == 2 * (2 + 5 + 5)
    for case in rep:
        assert case["converged"] and case["residual"] <= 1e-10, case
        assert all(abs(i - j) <= 2 for i, j in zip(case["iters"], case["ref_iters"])), case
        assert case["launches"] < 4 * max(case["iters"]), case
