"""gdp_propagate_noalloc at the row lengths where its kernel changes its way of
reading a row (one flat list up to 32 non-zeros, one warp up to 1,024, one CTA
above; windows of 128 staged elements) and at values that the FP32 screen
cannot bound, against the oracle's left-to-right Jacobi rounds, bit for bit."""
import numpy as np
import pytest

import gdp
import gdpgen
import oracle
from gdp_testutil import assert_bitexact
from test_zz_no_alloc import _noalloc

pytestmark = pytest.mark.gpu


def _check(torch, mip, what, same=None):
    """same: the MIP the oracle propagates (the problem without its empty rows)."""
    lb, ub, st = _noalloc(torch, mip)
    ref = oracle.propagate(same or mip, oracle.JACOBI, nthreads=8)
    assert st["rounds"] == ref.rounds and bool(st["infeasible"]) == ref.infeasible, what
    assert_bitexact(lb, ub, ref.lb, ref.ub, what=what)


@pytest.mark.parametrize("m", [1, 33, 700])
@pytest.mark.parametrize("lens", [(1, 1), (2, 40), (31, 33), (126, 130), (1022, 1027), (2040, 2060)])
def test_row_lengths(lens, m):
    torch = pytest.importorskip("torch")
    for slack in (5.0, 0.05):
        mip = gdpgen.random_mip(0, seed=410 + m, m=m, n=max(3000, m), len_min=lens[0], len_max=lens[1], slack_max=slack)
        _check(torch, mip, f"rows of {lens}, m={m}, slack {slack}")


@pytest.mark.parametrize("seed", [1, 2])
def test_values_outside_the_screen(seed):
    torch = pytest.importorskip("torch")
    mip = gdpgen.random_mip(0, seed=420 + seed, len_max=60)
    rng = np.random.default_rng(seed)
    pick = lambda a, share: rng.random(len(a)) < share
    mip.val[pick(mip.val, 0.02)] *= 1e-12   # coefficients below the EPS
    mip.val[pick(mip.val, 0.01)] *= 1e-22   # below 2^-60
    mip.val[pick(mip.val, 0.01)] *= 1e14    # above 2^40
    tiny = pick(mip.lb, 0.02) & (mip.lb == 0.0) & (mip.vartype == 3)
    mip.lb[tiny] = 1e-300                   # below 2^-126
    far = pick(mip.ub, 0.02) & (mip.ub >= 1e20)
    mip.ub[far] = np.inf
    _check(torch, mip, "values outside the screen")


def test_power_law_with_empty_rows():
    torch = pytest.importorskip("torch")
    mip = gdpgen.random_mip(1, seed=431, m=20_011, n=15_000, n_dense_rows=3, dense_len=9_001)
    keep = np.diff(mip.row_ptr) != 3  # every row of three non-zeros becomes empty
    counts = np.where(keep, np.diff(mip.row_ptr), 0)
    inside = np.repeat(keep, np.diff(mip.row_ptr))
    mip.col, mip.val = mip.col[inside].copy(), mip.val[inside].copy()
    mip.row_ptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    # an empty row is no constraint to the library, whatever its sides; the oracle checks its sides
    filled = gdp.MIP(np.concatenate([[0], np.cumsum(counts[keep])]).astype(np.int32), mip.col, mip.val, mip.lhs[keep],
                     mip.rhs[keep], mip.lb, mip.ub, mip.vartype)
    _check(torch, mip, "power-law rows, some empty", same=filled)
