"""Which calls the grid-barrier limit ends: gdp_options.barrier_wait_kcycles covers
the persistent loops, while the rounds that the host drives may take any time."""
import pytest

import gdp
import gdpgen
import oracle
from gdp_testutil import assert_bitexact

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sync", [gdp.CPU_LOOP, gdp.GPU_LOOP])
@pytest.mark.parametrize("m", [2_000, 30_000])
def test_driven_rounds_have_no_limit(sync, m):
    mip = gdpgen.random_mip(1, seed=61, m=m, n=3 * m // 4, n_dense_rows=2, dense_len=m // 4)
    with gdp.Context(mip, sync_type=sync, barrier_wait_kcycles=1) as ctx:
        lb, ub, st = ctx.propagate()
    ref = oracle.propagate(mip, oracle.JACOBI, split_len=32, split_tile=1024, nthreads=8)
    assert st["rounds"] == ref.rounds and bool(st["infeasible"]) == ref.infeasible
    assert_bitexact(lb, ub, ref.lb, ref.ub)
