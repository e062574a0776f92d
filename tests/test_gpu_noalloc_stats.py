"""The allocation-free call counts the rows that it sweeps: all of them in a dense
round, those with a variable changed in the round before in a sparse one, whether
they are read by lanes, by a warp (more than 32 elements) or by a CTA (more than
1,024)."""
import numpy as np
import pytest

import gdp

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _chain(k, extra, touched):
    """x_{i+1} <= x_i, x_0 <= 1, the others <= 10: round r changes x_r alone, and
    round k + 1 nothing. Then one loose row per length in `extra` over variables of
    its own, with x_1 in place of one of them if `touched`."""
    rows = [(np.array([i, i + 1]), np.array([-1.0, 1.0]), 0.0) for i in range(k)]
    n = k + 1
    for length in extra:
        cols = np.arange(n, n + length)
        n += length
        if touched:
            cols[length // 2] = 1
        rows.append((cols, np.ones(length), 1e6))
    ub = np.full(n, 10.0)
    ub[0] = 1.0
    row_ptr = np.concatenate([[0], np.cumsum([len(c) for c, _, _ in rows])])
    return dict(row_ptr=row_ptr.astype(np.int32), col=np.concatenate([c for c, _, _ in rows]).astype(np.int32),
                val=np.concatenate([v for _, v, _ in rows]), lhs=np.full(len(rows), -1e20),
                rhs=np.array([r for _, _, r in rows]), lb=np.zeros(n), ub=ub, vartype=np.full(n, 3, np.int32))


@pytest.mark.parametrize("extra", [(), (32,), (33,), (1024,), (1025,), (7, 40, 3000)])
@pytest.mark.parametrize("touched", [False, True])
def test_rows_counted_as_swept(extra, touched):
    k = 64
    p = _chain(k, extra, touched)
    m, n, nnz = len(p["lhs"]), len(p["lb"]), len(p["col"])
    d = {key: torch.tensor(a, device="cuda") for key, a in p.items()}
    torch.cuda.synchronize()
    st = gdp.propagate_noalloc(m, n, nnz, *(d[key].data_ptr() for key in (
        "col", "row_ptr", "val", "lhs", "rhs", "lb", "ub", "vartype")))
    assert st["rounds"] == k + 1 and st["changed_vars"] == k
    rows = m + 2 * (k - 1) + 1  # the changed variable's two rows, in the end the last one's
    swept = nnz + 2 * (2 * (k - 1) + 1)
    if touched:  # round 2 follows the change of x_1
        rows += len(extra)
        swept += sum(extra)
    assert (st["rows_processed"], st["nnz_processed"]) == (rows, swept)
    assert st["bytes_algorithmic"] == 12.0 * swept + 20.0 * rows + 36.0 * n * st["rounds"]
    assert np.all(d["ub"].cpu().numpy()[:k + 1] == 1.0)
