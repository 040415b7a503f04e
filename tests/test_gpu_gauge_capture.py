"""The gauge force allocates nothing and is one launch: the first call of a context can be captured into a graph, which
then follows the links in place; and a caller's scratch pointer changes nothing.  Oracle: the numpy restatement, with
the tolerance of the other gauge-force tests (fewer than 200 products of numbers of order one in FP64)."""

import numpy as np
import pytest

from oracle import wilson as W
from tests.conftest import rel

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("CUDA device required", allow_module_level=True)

from jaxqft_b200.lib import WilsonContext, kernel_launches  # noqa: E402


@pytest.mark.parametrize("shape,nconf", [((2, 2, 2, 2), 1), ((4, 2, 6, 10), 3)])
def test_first_call_of_a_context_under_capture(shape, nconf):
    rng = np.random.default_rng(21)
    U0, U1 = (W.hot_links(rng, shape, nconf, 0.5) for _ in range(2))
    stream = torch.cuda.Stream()
    u = torch.from_numpy(U0).cuda()
    F = torch.empty_like(u)
    torch.cuda.synchronize()
    ctx = WilsonContext(shape)
    ctx.set_stream(stream)
    graph = torch.cuda.CUDAGraph()
    before = kernel_launches()
    with torch.cuda.graph(graph, stream=stream):
        ctx.gauge_force(u, 5.6, out=F)
    assert kernel_launches() - before == 1
    for U in (U0, U1):
        u.copy_(torch.from_numpy(U))
        graph.replay()
        torch.cuda.synchronize()
        assert rel(F.cpu().numpy(), W.gauge_force(U, 5.6)) < 1e-13


def test_a_scratch_pointer_changes_nothing():
    shape = (4, 4, 2, 6)
    u = torch.from_numpy(W.hot_links(np.random.default_rng(22), shape, 2, 0.5)).cuda()
    ctx = WilsonContext(shape)
    F = ctx.gauge_force(u, 5.6)
    for scratch in (None, torch.empty_like(u)):
        G = torch.empty_like(u)
        ctx._check(ctx.lib.wl_gauge_force_ws(ctx.handle, u.data_ptr(), 2, 5.6,
                                             None if scratch is None else scratch.data_ptr(), G.data_ptr()))
        assert torch.equal(F, G)
