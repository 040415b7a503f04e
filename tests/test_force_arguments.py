"""The forces read whole-lattice fields through raw pointers, so a field of another size (a compact half-lattice field,
two fields in one tensor) must be refused before anything is launched, and a strided one copied.  No GPU: the library
is a stand-in that records its calls."""

import types

import numpy as np
import pytest
import torch

from jaxqft_b200.lib import WilsonContext
from jaxqft_b200.su3_wilson_nf2 import SU3WilsonNf2

SHAPE = (2, 4, 2, 6)
VOLUME = int(np.prod(SHAPE))


class _Library:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda *args: self.calls.append((name, args)) or 0


def _context():
    ctx = WilsonContext.__new__(WilsonContext)
    ctx.lib, ctx.device, ctx.lattice_shape, ctx.volume = _Library(), torch.device("cpu"), SHAPE, VOLUME
    ctx._torch, ctx._index, ctx._field = torch, -1, 12 * VOLUME
    ctx.handle = None
    return ctx


def _theory(ctx):
    th = SU3WilsonNf2.__new__(SU3WilsonNf2)
    th.ctx, th.device, th.lattice_shape, th.layout, th.dtype = ctx, ctx.device, SHAPE, "BMXYIJ", torch.complex128
    th.mass, th._m0 = 0.1, 4.1
    th._gauges_for = lambda U: [types.SimpleNamespace(handle=None)] * 2
    return th


def _field(n, *shape):
    return torch.zeros((n, *shape), dtype=torch.complex128)


WHOLE = (*SHAPE, 4, 3)
WRONG = [(VOLUME // 2, 4, 3), (2, *WHOLE), (VOLUME, 4, 2)]


@pytest.mark.parametrize("bad", WRONG)
@pytest.mark.parametrize("which", [0, 1])
def test_a_field_of_the_wrong_size_is_refused_before_any_launch(bad, which):
    ctx = _context()
    th = _theory(ctx)
    args = [_field(2, *WHOLE), _field(2, *WHOLE)]
    args[which] = _field(2, *bad)
    for force in (th.pseudofermion_force_from_solution, th.eop_pseudofermion_force_from_solution):
        with pytest.raises(ValueError, match="is not one field on lattice"):
            force(None, *args)
    with pytest.raises(ValueError, match="is not one field on lattice"):
        ctx.pf_force(types.SimpleNamespace(handle=None), args[0][0], args[1][0])
    assert ctx.lib.calls == []


def test_a_strided_field_reaches_the_library_as_a_contiguous_copy():
    ctx = _context()
    x = _field(1, *WHOLE)[0].transpose(0, 1).contiguous().transpose(0, 1)  # the right shape, other strides
    assert not x.is_contiguous()
    y = _field(1, *WHOLE)[0]
    F = torch.empty((4, *SHAPE, 3, 3), dtype=torch.complex128)
    ctx._force_into(types.SimpleNamespace(handle=None), x, y, F)
    (name, args), = ctx.lib.calls
    assert name == "wl_pf_force"
    assert args[2] != x.data_ptr() and args[3] == y.data_ptr() and args[6] == F.data_ptr()
