"""Force and gauge-sector kernels at the sizes where their tiling can go wrong: lattices smaller than, filling and ragged
against the 32-site blocks of the gauge force and the 64-site blocks of the pseudofermion force, extents of two (both
neighbours the same site), fields that are not 32-byte aligned, accumulation, in-place drift.

Oracle: the numpy restatement.  Tolerances: every force entry is a sum of fewer than 200 products of numbers of
order one in FP64, so a relative 2-norm error of 1e-13 leaves a factor of more than two over the worst case
200 eps; the drift squares s ~ log2 ||dt P|| times, each doubling the relative error of a few eps."""

import numpy as np
import pytest

from oracle import wilson as W
from tests.conftest import rel

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("CUDA device required", allow_module_level=True)

from jaxqft_b200.lib import WilsonContext  # noqa: E402
from jaxqft_b200.su3_wilson_nf2 import SU3WilsonNf2  # noqa: E402

SHAPES = [(2, 2, 2, 2), (2, 4, 6, 16), (4, 2, 2, 18), (2, 2, 4, 34), (6, 2, 4, 10), (2, 6, 2, 10)]
BC = (1, 1j, 1, -1)


def _unaligned(a):
    """A device copy of `a` whose first element is 16 but not 32 bytes aligned."""
    flat = torch.empty(a.size + 1, dtype=torch.complex128, device="cuda")
    out = flat[1:].view(a.shape)
    out.copy_(torch.from_numpy(np.ascontiguousarray(a)))
    assert out.data_ptr() % 32 == 16
    return out


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("aligned", [True, False])
def test_pseudofermion_force(shape, aligned):
    rng = np.random.default_rng(3)
    U, X, Y = W.hot_links(rng, shape, 1, 0.4), W.gaussian_spinor(rng, shape, 1), W.gaussian_spinor(rng, shape, 1)
    ctx = WilsonContext(shape, bc=BC)
    g = ctx.gauge(torch.from_numpy(U[0]))
    put = (lambda a: torch.from_numpy(a).cuda()) if aligned else _unaligned
    ref = W.force_from_solution(U, X, Y, BC)[0]
    F = ctx.pf_force(g, put(X[0]), put(Y[0]))
    assert rel(F.cpu().numpy(), ref) < 1e-13
    F = ctx.pf_force(g, put(X[0]), put(Y[0]), coef=-0.25, F=F)
    assert rel(F.cpu().numpy(), 0.75 * ref) < 1e-13


@pytest.mark.parametrize("shape", SHAPES)
def test_even_odd_force_ignores_odd_input_sites(shape):
    rng = np.random.default_rng(4)
    mass = W.kappa_to_mass(0.13)
    U = W.hot_links(rng, shape, 2, 0.4)
    X, Y = W.gaussian_spinor(rng, shape, 2), W.gaussian_spinor(rng, shape, 2)
    th = SU3WilsonNf2(lattice_shape=shape, beta=5.6, batch_size=2, mass=mass, fermion_bc=BC,
                      fermion_monomial_kind="eo_preconditioned")
    ref = W.eop_force_from_solution(U, W.project(X, 0), W.project(Y, 0), mass, BC)
    F = th.eop_pseudofermion_force_from_solution(torch.from_numpy(U).cuda(), torch.from_numpy(X).cuda(),
                                                 torch.from_numpy(Y).cuda())
    assert rel(F.cpu().numpy(), ref) < 1e-13


@pytest.mark.parametrize("shape", SHAPES)
def test_gauge_force(shape):
    U = W.hot_links(np.random.default_rng(5), shape, 2, 0.6)
    F = WilsonContext(shape).gauge_force(torch.from_numpy(U), 5.6).cpu().numpy()
    assert rel(F, W.gauge_force(U, 5.6)) < 1e-13


@pytest.mark.parametrize("dt", [0.0, 1e-9, 0.2, 0.9, 12.0])
def test_drift_in_place_and_general_generators(dt):
    """Momenta that are neither traceless nor anti-Hermitian exercise every coefficient of the characteristic
    polynomial; the output may be the links or the momenta."""
    shape = (2, 2, 4, 6)  # 384 links: three full blocks of 128 threads
    rng = np.random.default_rng(6)
    U = W.hot_links(rng, shape, 1, 0.4)
    P = W.algebra_field(rng, shape, 1)
    if dt < 1.0:
        P = P + 0.3 * (rng.standard_normal(P.shape) + 1j * rng.standard_normal(P.shape))
    A = torch.from_numpy(dt * P)
    ref = (torch.linalg.matrix_exp(A) @ torch.from_numpy(U)).numpy()
    norm = float(A.abs().sum(-1).max())
    ctx = WilsonContext(shape)
    tol = 40 * np.finfo(float).eps * (1.0 + norm)
    for alias in (None, "U", "P"):
        u, p = torch.from_numpy(U).cuda(), torch.from_numpy(P).cuda()
        out = ctx.gauge_evolve(dt, p, u, out={None: None, "U": u, "P": p}[alias])
        assert rel(out.cpu().numpy(), ref) < tol, alias
