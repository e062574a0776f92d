"""Bounds in host memory that starts anywhere: the kernels' loads and stores need
8-byte alignment, so other arrays are copied. Results are the bits of the aligned
call, and a failed call leaves its inputs in the outputs."""
import ctypes as C

import numpy as np
import pytest

import gdp
import gdpgen

pytestmark = pytest.mark.gpu

DOUBLES = C.POINTER(C.c_double)


def _shifted(a, by):
    """A copy of `a` that starts `by` bytes past an 8-byte boundary."""
    raw = np.zeros(8 * len(a) + 16, np.uint8)
    at = (-raw.ctypes.data) % 8 + by
    out = raw[at:at + 8 * len(a)].view(np.float64)
    out[:] = a
    assert out.ctypes.data % 8 == by
    return out


@pytest.mark.parametrize("m", [2, 400, 20_000])
@pytest.mark.parametrize("shift", [(4, 0), (0, 1), (7, 4)])
@pytest.mark.parametrize("sync", [gdp.CPU_LOOP, gdp.MEGAKERNEL])
def test_unaligned_inputs(m, shift, sync):
    mip = gdpgen.random_mip(0, seed=31, m=m, n=max(3 * m // 4, 3))
    with gdp.Context(mip, sync_type=sync) as ctx:
        lb, ub, st = ctx.propagate()
        for _ in range(2):  # the second call finds the device copies in place
            ulb, uub, ust = ctx.propagate(_shifted(mip.lb, shift[0]), _shifted(mip.ub, shift[1]))
            assert ust["rounds"] == st["rounds"] and ust["infeasible"] == st["infeasible"]
            assert ulb.tobytes() == lb.tobytes() and uub.tobytes() == ub.tobytes()
        alb, aub, _ = ctx.propagate()
        assert alb.tobytes() == lb.tobytes() and aub.tobytes() == ub.tobytes()


def test_unaligned_outputs_and_in_place():
    mip = gdpgen.random_mip(0, seed=32)
    at = lambda a: C.cast(a.ctypes.data, DOUBLES)
    with gdp.Context(mip) as ctx:
        lb, ub, _ = ctx.propagate()
        ilb, iub = mip.lb.copy(), mip.ub.copy()
        olb, oub = _shifted(np.zeros(mip.n), 4), _shifted(np.zeros(mip.n), 2)
        assert ctx._lib.gdp_propagate_into(ctx._h, at(ilb), at(iub), at(olb), at(oub), None) == gdp.GDP_OKAY
        assert olb.tobytes() == lb.tobytes() and oub.tobytes() == ub.tobytes()
        olb[:], oub[:] = mip.lb, mip.ub
        assert ctx._lib.gdp_propagate(ctx._h, at(olb), at(oub), None) == gdp.GDP_OKAY
        assert olb.tobytes() == lb.tobytes() and oub.tobytes() == ub.tobytes()
