"""The exact pass and the round loops at the sizes where they change their way of
working, against the oracle's GPU mode, bit for bit: one CTA up to 16 slices of
one-lane rows, the exact pass in place with a warp for each slice, and items of
fewer rows with more lanes per chain when a round has few rows (rows of 1 to 32
lanes). Batch members run the exact pass in place for every row length."""
import numpy as np
import pytest

import gdp
import gdpgen
from gdp_testutil import assert_bitexact
from test_gpu_parity import check_vs_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 31, 33, 512, 513, 1100])
def test_one_lane_problems(m):
    mip = gdpgen.random_mip(0, seed=510 + m, m=m, n=max(40, 3 * m // 4))
    for sync in (gdp.CPU_LOOP, gdp.GPU_LOOP, gdp.MEGAKERNEL):
        check_vs_oracle(mip, sync)
    check_vs_oracle(mip, gdp.MEGAKERNEL, marking=2)


@pytest.mark.parametrize("m", [1, 5, 150, 6000])
@pytest.mark.parametrize("lens", [(30, 34), (60, 70), (120, 260), (500, 530), (1000, 1030)])
def test_lanes_per_chain(lens, m):
    if m * lens[1] > 800_000:
        m = 800_000 // lens[1]
    mip = gdpgen.random_mip(0, seed=530 + m, m=m, n=2500, len_min=lens[0], len_max=lens[1], slack_max=0.5)
    check_vs_oracle(mip, gdp.MEGAKERNEL)
    check_vs_oracle(mip, gdp.CPU_LOOP, marking=2)
    lb, ub, st = gdp.propagate(mip, sync_type=gdp.MEGAKERNEL)
    b = gdp.Batch.instances([mip, mip])
    blb, bub, bst, _ = b.propagate([mip.lb, mip.lb], [mip.ub, mip.ub])
    for k in range(2):
        assert bst[k]["rounds"] == st["rounds"] and bst[k]["infeasible"] == st["infeasible"]
        assert_bitexact(blb[k], bub[k], lb, ub, what=f"batch member {k}")
    b.close()


def test_more_candidates_than_the_list_holds():
    """Rows whose every element is a candidate overflow the collected list: they are read again."""
    rng = np.random.default_rng(3)
    m, n = 40, 64
    rows = [np.sort(rng.choice(n, 24, replace=False)) for _ in range(m)]
    val = rng.choice([-1.0, 1.0], 24 * m) * rng.uniform(1, 2, 24 * m)
    mip = gdp.MIP((24 * np.arange(m + 1)).astype(np.int32), np.concatenate(rows).astype(np.int32), val,
                  np.full(m, -1e20), rng.uniform(-60, -50, m), np.full(n, -100.0), np.full(n, 100.0),
                  rng.choice([1, 3], n).astype(np.int32))
    act = np.add.reduceat(np.where(val > 0, -100.0 * val, 100.0 * val), mip.row_ptr[:-1])
    mip.rhs = act + rng.uniform(10, 40, m)  # far below every |a| (ub - lb)
    for sync in (gdp.CPU_LOOP, gdp.GPU_LOOP, gdp.MEGAKERNEL):
        check_vs_oracle(mip, sync)
