"""Which calls the grid-barrier limit ends: gdp_options.barrier_wait_kcycles covers
the persistent loops, while the rounds that the host drives may take any time."""
import numpy as np
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


def test_allocation_free_call_with_a_phase_of_seconds():
    """One row of 64M elements: its sums, one element after the other, take 4.5e9
    cycles (over 2 s), for which the rest of the grid waits."""
    torch = pytest.importorskip("torch")
    n, nnz = 64, 64_000_000
    dev = dict(device="cuda")
    col = torch.arange(nnz, dtype=torch.int32, **dev) % (n - 1)
    col[-1] = n - 1
    val = torch.ones(nnz, dtype=torch.float64, **dev)
    row_ptr = torch.tensor([0, nnz], dtype=torch.int32, **dev)
    lhs, rhs = (torch.tensor([v], dtype=torch.float64, **dev) for v in (-1e20, 5.0))
    lb, ub = torch.zeros(n, dtype=torch.float64, **dev), torch.zeros(n, dtype=torch.float64, **dev)
    ub[-1] = 10.0  # every other variable is fixed at 0
    vartype = torch.full((n,), 3, dtype=torch.int32, **dev)
    torch.cuda.synchronize()
    st = gdp.propagate_noalloc(1, n, nnz, *(t.data_ptr() for t in (col, row_ptr, val, lhs, rhs, lb, ub, vartype)))
    assert st["rounds"] == 2 and st["converged"] and not st["infeasible"]
    assert not lb.any() and np.array_equal(ub.cpu().numpy(), [0.0] * (n - 1) + [5.0])
