"""The schedule of small problems, one CTA of 512 threads by default (unless they have
many variables, whose change bitmap that CTA reads every round): it survives a
change of options, and the tuner hands back the schedule that it timed."""
import numpy as np
import pytest

import gdp
import gdpgen
import oracle
from gdp_testutil import assert_bitexact

pytestmark = pytest.mark.gpu


def _exact(mip, ctx, split_len=32):
    lb, ub, st = ctx.propagate()
    ref = oracle.propagate(mip, oracle.JACOBI, split_len=split_len)
    assert st["rounds"] == ref.rounds and bool(st["infeasible"]) == ref.infeasible
    assert_bitexact(lb, ub, ref.lb, ref.ub)


@pytest.mark.parametrize("m", [30, 400, 512])
def test_options_keep_the_default_schedule(m):
    mip = gdpgen.random_mip(0, seed=5, m=m, n=3 * m // 4)
    with gdp.Context(mip) as ctx:
        assert ctx.layout()["mega_grid"] == 1
        for sync in (gdp.MEGAKERNEL, gdp.GPU_LOOP, gdp.CPU_LOOP):
            ctx.set_options(sync_type=sync)
            assert ctx.layout()["mega_grid"] == 1
            _exact(mip, ctx)


def test_explicit_sizes_are_kept():
    mip = gdpgen.random_mip(0, seed=5, m=400, n=300)
    grids = []
    for threads in (128, 256, 512):
        with gdp.Context(mip, cta_threads=threads) as ctx:
            grids.append(ctx.layout()["mega_grid"])
            ctx.set_options(sync_type=gdp.MEGAKERNEL)
            assert ctx.layout()["mega_grid"] == grids[-1] > 1
            _exact(mip, ctx)
    assert grids == sorted(grids, reverse=True)


def test_tuned_schedule_is_the_timed_one():
    gdp.autotune_clear_cache()
    mip = gdpgen.random_mip(0, seed=5, m=400, n=300)
    opts, ms, trials = gdp.autotune(mip, repeats=2)
    # short rows in every layout: stage 1 times the one CTA, stage 2 all of its schedules
    assert [t["cta_threads"] for t in trials[:9]] == [0] * 9
    assert [(t["ctas_per_sm"], t["cta_threads"]) for t in trials[9:]] == [(0, 128), (4, 128), (0, 256), (2, 256),
                                                                         (0, 512), (0, 256)]
    best = min(trials, key=lambda t: t["ms"])
    assert ms == best["ms"] and opts["cta_threads"] == best["cta_threads"]
    with gdp.Context(mip, **{k: opts[k] for k in ("sync_type", "thread_row_max", "split_tile", "ctas_per_sm",
                                                  "cta_threads")}) as ctx:
        assert (ctx.layout()["mega_grid"] == 1) == (opts["cta_threads"] == 0)
        _exact(mip, ctx, split_len=opts["thread_row_max"])


def _spread(mip, n):
    """The rows of `mip` over n variables, most of them in no row."""
    at = np.sort(np.random.default_rng(0).choice(n, mip.n, replace=False)).astype(np.int32)
    lb, ub, vartype = np.zeros(n), np.full(n, 10.0), np.full(n, 3, np.int32)
    lb[at], ub[at], vartype[at] = mip.lb, mip.ub, mip.vartype
    return gdp.MIP(mip.row_ptr, at[mip.col], mip.val, mip.lhs, mip.rhs, lb, ub, vartype)


@pytest.mark.parametrize("m,n,one", [(30, 6144, True), (30, 6145, False), (100, 1536, True), (100, 1537, False),
                                     (512, 384, True), (512, 385, False), (400, 1_000_000, False)])
def test_many_variables_take_the_grid(m, n, one):
    mip = _spread(gdpgen.random_mip(0, seed=5, m=m, n=min(n, 3 * m // 4)), n)
    with gdp.Context(mip) as ctx:
        assert (ctx.layout()["mega_grid"] == 1) == one
        for sync in (gdp.CPU_LOOP, gdp.MEGAKERNEL):
            ctx.set_options(sync_type=sync)
            _exact(mip, ctx)
