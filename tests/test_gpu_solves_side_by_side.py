"""Solves of several threads on one device.  A solve that starts while another is in flight must take the ordinary
launches (two persistent ones could wait for each other's blocks, and taking turns would undo the overlap): its result
is then bitwise that of an engine stepped from the host, which runs the same kernels in the same order.  Threads that
solve all the time must all get converged solutions, whichever form each solve took."""

import threading

import numpy as np
import pytest

from oracle import wilson as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("CUDA device required", allow_module_level=True)

from jaxqft_b200.lib import SLOT_CONVERGED, Engine, WilsonContext  # noqa: E402

SHAPE, BC, MASS = (4, 4, 6, 8), (1, 1, 1, -1), 0.0


def _system(seed, n, shape=SHAPE):
    rng = np.random.default_rng(seed)
    ctx = WilsonContext(shape, bc=BC)
    gauge = ctx.gauge(torch.from_numpy(W.hot_links(rng, shape, 1, 0.3)[0]))
    b = torch.from_numpy(W.project(W.gaussian_spinor(rng, shape, n), 0)).cuda()
    torch.cuda.synchronize()
    return ctx, gauge, b


@pytest.mark.parametrize("inner", ["double", "single", "half"])
@pytest.mark.parametrize("use_graph", [True, False])
def test_a_solve_beside_another_takes_the_ordinary_launches(inner, use_graph):
    ctx, gauge, b = _system(1, 2)
    eng = Engine(ctx, gauge, 2, inner=inner, tol=1e-10, maxiter=2000)
    eng.admit(np.arange(2), b, MASS)
    while eng.poll()[1]:
        eng.step(8)
    ref = [eng.retire(r) for r in range(2)]
    eng.close()
    solve = lambda: ctx.solve(gauge, b, MASS, tol=1e-10, maxiter=2000, inner=inner, use_graph=use_graph)  # noqa: E731
    solve()
    # 17 slots never take the persistent form; an unreachable tolerance keeps this solve going for some tenths of a second
    other, other_gauge, other_b = _system(2, 17, (8, 8, 8, 8))
    other.solve(other_gauge, other_b, MASS, tol=1e-10, maxiter=10, inner="double")
    started = threading.Event()

    def long_solve():
        started.set()
        other.solve(other_gauge, other_b, MASS, tol=1e-30, maxiter=8000, inner="double")

    thread = threading.Thread(target=long_solve)
    thread.start()
    started.wait()
    threading.Event().wait(0.05)
    x, st = solve()
    beside = thread.is_alive()
    thread.join()
    assert beside, "the other solve ended too early to say anything"
    for r in range(2):
        assert st[r]["status"] == SLOT_CONVERGED and st[r]["iters"] == ref[r][1]["iters"], (st[r], ref[r][1])
        assert torch.equal(x[r], ref[r][0])


@pytest.mark.parametrize("inner,n", [("double", 1), ("single", 2), ("half", 12)])
def test_threads_that_solve_all_the_time(inner, n):
    nthreads, solves, found, go = 4, 25, {}, threading.Barrier(4)

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            ctx, gauge, b = _system(10 + k, n)
            go.wait()
            got = [ctx.solve(gauge, b, MASS, tol=1e-10, maxiter=2000, inner=inner)[1] for _ in range(solves)]
            found[k] = [s for st in got for s in st]
            ctx.close()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(nthreads)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert sorted(found) == list(range(nthreads))
    for k, stats in found.items():
        assert len(stats) == n * solves
        assert all(s["status"] == SLOT_CONVERGED and s["true_res"] <= 1e-10 for s in stats), k
        per_slot = [{s["iters"] for s in stats[r::n]} for r in range(n)]
        assert all(max(i) - min(i) <= 2 for i in per_slot), per_slot  # both forms: sums grouped differently
