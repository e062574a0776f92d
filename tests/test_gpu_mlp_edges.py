"""The MLP kernels at the sizes where their tiles and grids change: a last tile
that is partly empty, one tile per warp against several, features that are not
16-byte aligned. Tolerances are those of the FP32 summation order and of the
rare BF16 tie that it rounds the other way; sums run in a fixed order, so equal
calls give equal bits."""
import numpy as np
import pytest

import gdp
from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu


def _data(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(0, 1, (n, mo.IN)).astype(np.float32)
    y = (x[:, 0] - 0.5 * x[:, 1] > 0.1).astype(np.float32)
    w = rng.uniform(0.5, 2.0, n).astype(np.float32)
    return x, y, w


@pytest.mark.parametrize("n", [17, 31, 4095, 200_003])
def test_forward_unaligned_features(n):
    m = gdp.Mlp(seed=3)
    x, _, _ = _data(n, 5)
    raw = np.empty(x.size + 5, np.float32)
    off = next(k for k in range(1, 5) if (raw.ctypes.data + 4 * k) % 16)
    xu = raw[off:off + x.size].reshape(x.shape)
    xu[:] = x
    z = m.forward(x)
    assert np.array_equal(z, m.forward(xu))
    z_ref, _ = mo.forward(m.params, x)
    scale = np.abs(z_ref).mean() + 1e-3
    err = np.abs(z - z_ref)
    assert np.median(err) <= 1e-3 * scale + 1e-5
    assert err.max() <= 0.05 * scale + 1e-3


# 9,728 = 16 x 4 x 152: one tile per warp of four-warp CTAs; 17,024 = 16 x 7 x 152
@pytest.mark.parametrize("n", [17, 31, 65, 9727, 9728, 9729, 17_023, 17_025, 70_001])
def test_gradient_edges(n):
    m = gdp.Mlp(seed=2)
    x, y, w = _data(n, 11)
    loss, g = m.gradient(x, y, w)
    loss2, g2 = m.gradient(x, y, w)
    assert loss == loss2 and np.array_equal(g, g2)
    loss_ref, g_ref = mo.loss_and_grad(m.params, x, y, w)
    assert abs(loss - loss_ref) <= 1e-3 * abs(loss_ref) + 1e-5
    for a, b in ((mo.OFF_W1, mo.OFF_B1), (mo.OFF_B1, mo.OFF_W2), (mo.OFF_W2, mo.OFF_B2), (mo.OFF_B2, mo.OFF_W3),
                 (mo.OFF_W3, mo.OFF_B3), (mo.OFF_B3, mo.N_PARAMS)):
        assert np.linalg.norm(g[a:b] - g_ref[a:b]) < 2e-2 * np.linalg.norm(g_ref[a:b]) + 1e-12


@pytest.mark.parametrize("n,batch", [(1, 1), (33, 16), (1000, 4096), (20_011, 9729)])
def test_training_equal_bits(n, batch):
    x, y, w = _data(n, 17)
    runs = []
    for _ in range(2):
        m = gdp.Mlp(seed=6)
        loss = m.train(x, y, w, epochs=3, batch=batch, lr=1e-3, seed=9)
        runs.append((loss, m.params))
    assert runs[0][0] == runs[1][0] and np.isfinite(runs[0][0])
    assert np.array_equal(runs[0][1], runs[1][1])
