"""changed_vars counts every committed variable: a context with a model, whose commit
loop leaves a warp's lanes at different times, counts what the batch loop counts for
the same rounds."""
import numpy as np
import pytest

import gdp
import gdpgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,seed", [(3_000, 3), (20_000, 4), (60_000, 5)])
def test_learned_context_counts_like_the_batch(m, seed):
    mip = gdpgen.random_mip(0, seed=seed, m=m, n=3 * m // 4)
    model = gdp.Mlp(seed=5)
    batch = gdp.Batch.instances([mip])
    batch.set_model(model, 0.0, 1)
    lbs, ubs, sts, _ = batch.propagate([mip.lb], [mip.ub])
    batch.close()
    with gdp.Context(mip, sync_type=gdp.MEGAKERNEL) as ctx:
        ctx.set_model(model, 0.0, 1)
        lb, ub, st = ctx.propagate()
    assert lb.tobytes() == lbs[0].tobytes() and ub.tobytes() == ubs[0].tobytes()
    assert st["rounds"] == sts[0]["rounds"] and st["changed_vars"] == sts[0]["changed_vars"]
    moved = int(np.sum((lb != mip.lb) | (ub != mip.ub)))
    assert st["changed_vars"] >= moved > 0
