"""The sizes at which the round loops change instantiation, bit for bit against a
loop that does not: batches on both sides of the work that takes the loop with
more warps and fewer registers (4 items per warp of 24 warps per SM), and problems
of one-lane rows on both sides of the exact pass in place (48 slices per SM)."""
import numpy as np
import pytest

import gdp
import gdpgen
from gdp_testutil import assert_bitexact

pytestmark = pytest.mark.gpu

SMS = 152


def _single(mip, sync):
    ctx = gdp.Context(mip, sync_type=sync)
    out = ctx.propagate()
    ctx.close()
    return out


@pytest.mark.parametrize("members", [2, 9])
def test_batch_loops(members):
    # 9 x 60,000 short rows: 16,875 slices, above 4 x 24 x 152 = 14,592
    mips = [gdpgen.random_mip(0, seed=90 + k, m=60_000, n=45_000) for k in range(members)]
    b = gdp.Batch.instances(mips)
    lb, ub, st, _ = b.propagate([p.lb for p in mips], [p.ub for p in mips])
    b.close()
    for k in (0, members - 1):
        slb, sub, sst = _single(mips[k], gdp.MEGAKERNEL)
        assert st[k]["rounds"] == sst["rounds"] and st[k]["infeasible"] == sst["infeasible"]
        assert_bitexact(lb[k], ub[k], slb, sub, what=f"member {k}")


@pytest.mark.parametrize("slices", [24 * SMS, 48 * SMS - 1, 48 * SMS, 48 * SMS + 1])
def test_exact_pass_in_place(slices):
    m = 32 * slices - 5
    mip = gdpgen.random_mip(0, seed=70, m=m, n=3 * m // 4)
    ref = _single(mip, gdp.GPU_LOOP)  # always queues the exact rows
    for sync in (gdp.MEGAKERNEL, gdp.CPU_LOOP):
        lb, ub, st = _single(mip, sync)
        for key in ("rounds", "infeasible", "rows_processed", "nnz_processed", "nnz_exact", "changed_vars"):
            assert st[key] == ref[2][key], key
        assert_bitexact(lb, ub, ref[0], ref[1], what=f"{sync}")
