"""Round loops whose grid is a single CTA and whose barrier is __syncthreads: what the
CTA changes by atomics (the bitmap, the drift bounds of split rows, round state) is
what it reads in the next round. Several rounds each, bit for bit against the
oracle."""
import numpy as np
import pytest

import gdp
import gdpgen
import oracle
from gdp_testutil import assert_bitexact

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("seed", range(12))
@pytest.mark.parametrize("m,n", [(100, 75), (60, 1000), (180, 40)])
def test_allocation_free_call(seed, m, n):
    # at most 256 rows, 1,024 variables and 1,024 non-zeros: one CTA
    mip = gdpgen.random_mip(0, seed=seed, m=m, n=n, len_max=8 if m == 180 else 16)
    assert mip.m <= 256 and mip.n <= 1024 and mip.nnz <= 1024
    d = [torch.tensor(a, device="cuda") for a in (mip.col, mip.row_ptr, mip.val, mip.lhs, mip.rhs, mip.lb, mip.ub,
                                                  mip.vartype)]
    torch.cuda.synchronize()
    st = gdp.propagate_noalloc(mip.m, mip.n, mip.nnz, *(t.data_ptr() for t in d))
    ref = oracle.propagate(mip, oracle.JACOBI)
    assert st["rounds"] == ref.rounds and bool(st["infeasible"]) == ref.infeasible
    assert_bitexact(d[5].cpu().numpy(), d[6].cpu().numpy(), ref.lb, ref.ub)


def _with_split_row(seed):
    """x_{i+1} <= x_i + c_i over 60 variables, and one row of 14 elements, in two
    tiles of 8, whose slack shrinks round by round until it binds."""
    rng = np.random.default_rng(seed)
    n = 60
    cols, vals, rhs = [], [], []
    for i in rng.permutation(n - 1):
        cols.append([i, i + 1])
        vals.append([-1.0, 1.0])
        rhs.append(-rng.uniform(0.01, 0.2))
    for _ in range(3):
        c = np.sort(rng.choice(n, 4, replace=False))
        cols.append(list(c))
        vals.append(list(rng.uniform(0.5, 2.0, 4)))
        rhs.append(rng.uniform(5, 20))
    c = np.sort(rng.choice(n, 14, replace=False))
    cols.append(list(c))
    vals.append(list(rng.uniform(-2.0, -0.5, 14)))  # -sum a x <= -r: the falling upper bounds eat its slack
    rhs.append(-rng.uniform(2, 40))
    row_ptr = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    ub = np.full(n, 10.0)
    ub[0] = 8.0
    return gdp.MIP(row_ptr, np.concatenate(cols).astype(np.int32), np.concatenate(vals), np.full(len(cols), -1e20),
                   np.array(rhs), np.full(n, -5.0), ub, np.full(n, 3, np.int32))


@pytest.mark.parametrize("sync", [gdp.CPU_LOOP, gdp.MEGAKERNEL])
@pytest.mark.parametrize("cta_threads", [256, 512])
def test_context_with_a_split_row(sync, cta_threads):
    drift = 0
    for seed in range(12):
        mip = _with_split_row(seed)
        with gdp.Context(mip, sync_type=sync, cta_threads=cta_threads, thread_row_max=4, split_tile=8,
                         use_marking=2) as ctx:
            lay = ctx.layout()
            assert lay["mega_grid"] == 1 and lay["split_rows"] == 1 and lay["split_tiles"] == 2
            lb, ub, st = ctx.propagate()
        ref = oracle.propagate(mip, oracle.JACOBI, split_len=4, split_tile=8)
        assert st["rounds"] == ref.rounds > 2 and bool(st["infeasible"]) == ref.infeasible, seed
        assert_bitexact(lb, ub, ref.lb, ref.ub, what=f"seed {seed}")
        drift += st["rows_drift"]
    assert drift > 0
