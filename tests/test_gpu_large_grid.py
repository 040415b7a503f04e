"""The drop-in hop on a lattice whose site blocks do not fit one grid dimension (65536 blocks of 32 sites at 32^3x64):
with unit links and periodic boundaries a constant spinor is an eigenvector, D psi = mass psi, at every site.  Each of
the eight contributions is exact up to one rounding, so 16 eps of the largest term (m0 |psi|) bounds the error."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("CUDA device required", allow_module_level=True)

from jaxqft_b200.lib import WilsonContext  # noqa: E402


def test_constant_field_on_a_lattice_of_two_grid_layers():
    shape, mass = (32, 32, 32, 64), 0.3
    U = torch.eye(3, dtype=torch.complex128, device="cuda").expand(4, *shape, 3, 3).contiguous()
    ctx = WilsonContext(shape)
    gauge = ctx.gauge(U)
    site = torch.complex(torch.arange(1.0, 13.0, dtype=torch.float64), -torch.arange(12.0, dtype=torch.float64))
    psi = site.reshape(4, 3).cuda().expand(*shape, 4, 3).contiguous()
    out = ctx.apply("D", gauge, mass, psi)
    bound = 16 * np.finfo(float).eps * (mass + 4.0) * float(site.abs().max())
    assert float((out - mass * psi).abs().max()) <= bound
