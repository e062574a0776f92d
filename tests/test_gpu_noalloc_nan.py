"""Bounds and sides that are NaN in the allocation-free call: a NaN is no infinity, as
in the oracle's compares, in rows read by lanes, by a warp and by a CTA."""
import numpy as np
import pytest

import gdp
import gdpgen
import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _check(mip):
    d = [torch.tensor(a, device="cuda") for a in (mip.col, mip.row_ptr, mip.val, mip.lhs, mip.rhs, mip.lb, mip.ub,
                                                  mip.vartype)]
    torch.cuda.synchronize()
    st = gdp.propagate_noalloc(mip.m, mip.n, mip.nnz, *(t.data_ptr() for t in d))
    ref = oracle.propagate(mip, oracle.JACOBI)
    assert st["rounds"] == ref.rounds and bool(st["infeasible"]) == ref.infeasible
    for got, want in ((d[5], ref.lb), (d[6], ref.ub)):
        assert np.array_equal(got.cpu().numpy(), want, equal_nan=True)


@pytest.mark.parametrize("seed", range(8))
@pytest.mark.parametrize("where", ["lb", "ub", "lhs"])
def test_random_problems(seed, where):
    mip = gdpgen.random_mip(0, seed=seed, m=300, n=220)
    rng = np.random.default_rng(seed)
    a = {"lb": mip.lb, "ub": mip.ub, "lhs": mip.lhs}[where].copy()
    a[rng.random(len(a)) < 0.02] = np.nan
    _check(gdp.MIP(mip.row_ptr, mip.col, mip.val, a if where == "lhs" else mip.lhs, mip.rhs,
                   a if where == "lb" else mip.lb, a if where == "ub" else mip.ub, mip.vartype))


@pytest.mark.parametrize("length", [2, 32, 33, 1024, 1025, 3000])
@pytest.mark.parametrize("nan_lb", [False, True])
def test_one_nan_beside_a_candidate(length, nan_lb):
    """3 x + 1e-300 y + (variables fixed at 0) <= 6 with y's upper (lower) bound NaN: the
    minimum activity is a number (a NaN)."""
    n = length
    val = np.ones(n)
    val[0], val[1] = 3.0, 1e-300
    lb, ub = np.zeros(n), np.zeros(n)
    lb[0], ub[0], lb[1], ub[1] = -9.0, 20.0, -9.0, 5.0
    (lb if nan_lb else ub)[1] = np.nan
    _check(gdp.MIP(np.array([0, n], np.int32), np.arange(n, dtype=np.int32), val, np.array([-50.0]), np.array([6.0]),
                   lb, ub, np.full(n, 3, np.int32)))
