"""Which form a solve takes near the line of the FP16 site form: even-odd solves of two and three slots with 899 sites a
multiprocessor were slower in the persistent kernel and take the ordinary launches (nine an iteration); one slot, and
the full operator, take the persistent kernel (a few per reliable update)."""

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("CUDA device required", allow_module_level=True)

from jaxqft_b200.lib import WilsonContext, kernel_launches  # noqa: E402


@pytest.mark.skipif(torch.cuda.get_device_properties(0).multi_processor_count != 148,
                    reason="the lattices are chosen for 148 multiprocessors")
@pytest.mark.parametrize("shape,op,n,persistent", [((16, 16, 20, 52), "eo_normal", 1, True),
                                                   ((16, 16, 20, 52), "eo_normal", 2, False),
                                                   ((16, 16, 20, 52), "eo_normal", 3, False),
                                                   ((16, 16, 14, 52), "eo_normal", 2, True),
                                                   ((16, 16, 16, 32), "normal", 2, True)])
def test_form_of_fp16_site_solves(shape, op, n, persistent):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)
    h = torch.randn((4, *shape, 3, 3), generator=gen, device="cuda", dtype=torch.complex128)
    h = 0.1 * (h - h.conj().transpose(-1, -2))
    h = h - torch.diagonal(h, dim1=-2, dim2=-1).sum(-1)[..., None, None] / 3 * torch.eye(3, device="cuda")
    ctx = WilsonContext(shape, bc=(1, 1, 1, -1))
    gauge = ctx.gauge(torch.linalg.matrix_exp(h))
    psi = torch.randn((n, *shape, 4, 3), generator=gen, device="cuda", dtype=torch.complex128)
    b = ctx.apply("SCHUR_E_DAG", gauge, -0.2, psi, normalized=True) if op == "eo_normal" else psi
    for _ in range(2):
        before = kernel_launches()
        _, st = ctx.solve(gauge, b, -0.2, op=op, tol=1e-12, maxiter=40, inner="half")
        launches = kernel_launches() - before
    assert all(s["iters"] == 40 for s in st)
    assert (launches < 4 * 40) == persistent, launches
