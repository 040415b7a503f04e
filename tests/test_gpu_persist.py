"""The persistent iteration kernel of wl_solve (wl_persist.cuh) at the sizes where its work split can go wrong: fewer
sites than one warp, ragged last blocks and warps, groups of right-hand sides that do not fill their lanes, the largest
slot count it takes and one more, slots that finish at different iterations, and a solve stopped at maxiter.

Reference: the ordinary kernels (an Engine stepped from the host) and the numpy oracle.  Both run the same CG in the
same precision with sums grouped differently, so they take the same number of iterations up to one reliable update's
worth of rounding (two iterations), and either solution has an FP64 residual of at most tol, checked by the oracle."""

import numpy as np
import pytest

from oracle import wilson as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("CUDA device required", allow_module_level=True)

from jaxqft_b200.lib import SLOT_CONVERGED, SLOT_MAXITER, Engine, WilsonContext  # noqa: E402

BC = (1, 1, 1j, -1)
TOL = 1e-10


def _residual(U, x, b, mass, op):
    if op == "eo_normal":
        s = W.schur_even(U, x[None], mass, BC, normalized=True)
        ax = W.schur_even(U, s, mass, BC, normalized=True, dag=True)[0]
    else:
        ax = W.apply_normal(U, x[None], mass, BC)[0]
    return np.linalg.norm(b - ax) / np.linalg.norm(b)


@pytest.mark.parametrize("shape", [(2, 2, 2, 2), (2, 4, 6, 10)])
@pytest.mark.parametrize("inner,n", [("double", 1), ("double", 3), ("single", 1), ("single", 2), ("single", 5),
                                     ("single", 16), ("half", 1), ("half", 3), ("half", 4), ("half", 9),
                                     ("half", 16), ("half", 17)])
@pytest.mark.parametrize("op", ["eo_normal", "normal"])
def test_matches_the_ordinary_kernels(shape, inner, n, op):
    rng = np.random.default_rng(n)
    U = W.hot_links(rng, shape, 1, 0.3)
    b = W.gaussian_spinor(rng, shape, n)
    if op == "eo_normal":
        b = W.project(b, 0)
    masses = np.linspace(0.4, 0.05, n)
    ctx = WilsonContext(shape, bc=BC)
    gauge = ctx.gauge(torch.from_numpy(U[0]))
    x, st = ctx.solve(gauge, torch.from_numpy(b), masses, op=op, tol=TOL, maxiter=2000, inner=inner)
    eng = Engine(ctx, gauge, n, op=op, inner=inner, tol=TOL, maxiter=2000)
    eng.admit(np.arange(n), torch.from_numpy(b), masses)
    active = n
    while active:
        eng.step(8)
        _, active = eng.poll()
    for r in range(n):
        _, ref = eng.retire(r)
        assert st[r]["status"] == ref["status"] == SLOT_CONVERGED, (r, st[r], ref)
        assert abs(st[r]["iters"] - ref["iters"]) <= 2, (r, st[r], ref)
        assert _residual(U, x[r].cpu().numpy(), b[r], masses[r], op) <= TOL
    eng.close()


@pytest.mark.parametrize("inner,n", [("double", 2), ("single", 1), ("half", 8)])
def test_stops_at_maxiter_and_solves_again(inner, n):
    shape = (2, 4, 2, 6)
    rng = np.random.default_rng(9)
    U = W.hot_links(rng, shape, 1, 0.3)
    b = W.project(W.gaussian_spinor(rng, shape, n), 0)
    ctx = WilsonContext(shape, bc=BC)
    gauge = ctx.gauge(torch.from_numpy(U[0]))
    for maxiter in (1, 5):
        _, st = ctx.solve(gauge, torch.from_numpy(b), 0.0, tol=1e-13, maxiter=maxiter, inner=inner)
        assert all(s["status"] == SLOT_MAXITER and s["iters"] == maxiter for s in st), st
    zero = np.zeros_like(b)
    zero[0] = b[0]  # the other slots have nothing to solve
    x, st = ctx.solve(gauge, torch.from_numpy(zero), 0.0, tol=TOL, maxiter=2000, inner=inner)
    assert all(s["status"] == SLOT_CONVERGED for s in st)
    assert _residual(U, x[0].cpu().numpy(), b[0], 0.0, "eo_normal") <= TOL
    assert not torch.any(x[1:] != 0)
