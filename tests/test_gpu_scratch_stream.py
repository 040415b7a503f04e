"""A context whose stream is not torch's current one: the scratch of the gauge force and of the even-odd force must not
be handed to the current stream's next tensors while the context's kernels still have to use it.  The context's stream
is held up first, so that a tensor made right after the call would get the scratch's block and be overwritten later."""

import numpy as np
import pytest

from oracle import wilson as W
from tests.conftest import rel

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("CUDA device required", allow_module_level=True)

from jaxqft_b200.lib import WilsonContext  # noqa: E402

SHAPE, BC, MASS = (8, 8, 8, 8), (1, 1, 1, -1), 0.1


@pytest.mark.parametrize("what", ["gauge", "even-odd"])
@pytest.mark.parametrize("swap", [False, True])
def test_scratch_belongs_to_the_stream_of_the_context(what, swap):
    rng = np.random.default_rng(12)
    nconf = 8 if what == "gauge" else 1
    U = W.hot_links(rng, SHAPE, nconf, 0.4)
    X, Y = (W.project(W.gaussian_spinor(rng, SHAPE, 1), 0) for _ in range(2))
    side, main = torch.cuda.Stream(), torch.cuda.default_stream()
    own, current = (main, side) if swap else (side, main)
    with torch.cuda.stream(current):
        u, x, y = (torch.from_numpy(a).cuda() for a in (U, X[0], Y[0]))
        ctx = WilsonContext(SHAPE, bc=BC)
        ctx.set_stream(own)
        torch.cuda.synchronize()
        gauge = ctx.gauge(u[0])
        F = torch.empty((nconf, 4, *SHAPE, 3, 3), dtype=torch.complex128, device="cuda")
        size = u.shape if what == "gauge" else (2, *SHAPE, 4, 3)
        torch.cuda.synchronize()
        with torch.cuda.stream(own):
            torch.cuda._sleep(200_000_000)  # about 0.1 s
        if what == "gauge":
            ctx.gauge_force(u, 5.6, out=F)
        else:
            ctx._force_into(gauge, x, y, F[0], eo_coef=-1.0 / (MASS + 4.0) ** 2)
        others = [torch.full(size, 7.0, dtype=torch.complex128, device="cuda") for _ in range(3)]
        torch.cuda.synchronize()
    assert all(bool((t == 7.0).all()) for t in others)
    ref = W.gauge_force(U, 5.6) if what == "gauge" else W.eop_force_from_solution(U, X, Y, MASS, BC)
    assert rel(F.cpu().numpy(), ref) < 1e-13
    ctx.close()
