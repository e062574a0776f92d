"""Candidates of value zero keep the sign that lhs - maxact or rhs - minact and the
division give: a row side of -0.0 with activities of 0 yields bounds whose zeros
have the oracle's signs, in every exact pass (lanes, lane groups, tiles, batches, the
allocation-free call)."""
import numpy as np
import pytest

import gdp
import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _rows(length):
    """One row a x_i (+ variables fixed at 0) >= / <= a zero per sign of a, of the zero
    and of the side; every x_i is free and its bound becomes a zero."""
    cols, vals, lhs, rhs = [], [], [], []
    n = 8 + length
    k = 0
    for a in (-2.0, 3.0):
        for zero in (0.0, -0.0):
            for side in (0, 1):
                cols.append([k] + list(range(8, 8 + length - 1)))
                vals.append([a] + [1.0] * (length - 1))
                lhs.append(zero if side == 0 else -1e20)
                rhs.append(zero if side == 1 else 1e20)
                k += 1
    lb, ub = np.zeros(n), np.zeros(n)
    lb[:8], ub[:8] = -np.inf, np.inf
    row_ptr = (np.arange(9) * length).astype(np.int32)
    return gdp.MIP(row_ptr, np.concatenate(cols).astype(np.int32), np.concatenate(vals), np.array(lhs), np.array(rhs),
                   lb, ub, np.full(n, 3, np.int32))


def _same_bits(lb, ub, ref):
    assert np.array_equal(np.asarray(lb).view(np.int64), ref.lb.view(np.int64))
    assert np.array_equal(np.asarray(ub).view(np.int64), ref.ub.view(np.int64))


@pytest.mark.parametrize("length", [1, 2, 32, 33, 200, 1025, 3000])
def test_zero_signs(length):
    mip = _rows(length)
    ref = oracle.propagate(mip, oracle.JACOBI, split_len=32, split_tile=1024)
    zeros = np.concatenate([ref.lb[:8], ref.ub[:8]])
    zeros = zeros[zeros == 0.0]
    assert len(zeros) == 8 and 0 < np.signbit(zeros).sum() < 8
    for sync in (gdp.CPU_LOOP, gdp.GPU_LOOP, gdp.MEGAKERNEL):
        with gdp.Context(mip, sync_type=sync) as ctx:
            lb, ub, st = ctx.propagate()
        assert st["rounds"] == ref.rounds
        _same_bits(lb, ub, ref)
    batch = gdp.Batch.instances([mip, mip])
    lbs, ubs, _, _ = batch.propagate([mip.lb] * 2, [mip.ub] * 2)
    batch.close()
    _same_bits(lbs[1], ubs[1], ref)
    d = [torch.tensor(a, device="cuda") for a in (mip.col, mip.row_ptr, mip.val, mip.lhs, mip.rhs, mip.lb, mip.ub,
                                                  mip.vartype)]
    torch.cuda.synchronize()
    gdp.propagate_noalloc(mip.m, mip.n, mip.nnz, *(t.data_ptr() for t in d))
    _same_bits(d[5].cpu().numpy(), d[6].cpu().numpy(), ref)
