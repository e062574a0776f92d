"""The host arrays a caller may give the MLP's forward pass: logits that share
memory with the features, features and logits that start on any byte. Results are
the bits of the plain call."""
import ctypes as C
import mmap

import numpy as np
import pytest

import gdp

pytestmark = pytest.mark.gpu

FLOATS = C.POINTER(C.c_float)


def _forward_at(model, n, x_addr, z_addr):
    """gdp_mlp_forward on raw addresses."""
    rc = model._lib.gdp_mlp_forward(model._h, n, C.cast(x_addr, FLOATS), C.cast(z_addr, FLOATS))
    assert rc == gdp.GDP_OKAY, gdp.last_error()


def _features(n, seed=5):
    return np.random.default_rng(seed).normal(0, 1, (n, gdp.MLP_FEATURES)).astype(np.float32)


# 262,144 rows are the last whose logits (1 MB) are written by one launch
@pytest.mark.parametrize("n", [1, 17, 5000, 262_144, 262_145])
@pytest.mark.parametrize("where", ["front", "middle", "last row"])
def test_logits_over_the_features(n, where):
    m = gdp.Mlp(seed=3)
    x = _features(n)
    z = m.forward(x)
    buf = np.concatenate([x.ravel(), np.zeros(n, np.float32)])
    at = {"front": 0, "middle": 16 * (n // 2), "last row": 16 * n - 16}[where]
    _forward_at(m, n, buf.ctypes.data, buf.ctypes.data + 4 * at)
    assert np.array_equal(buf[at:at + n], z)


@pytest.mark.parametrize("n", [1, 17, 5000, 262_145])
@pytest.mark.parametrize("x_by,z_by", [(0, 1), (0, 2), (4, 3), (2, 0), (3, 3)])
def test_arrays_off_their_alignment(n, x_by, z_by):
    m = gdp.Mlp(seed=3)
    x = _features(n)
    z = m.forward(x)
    xraw, zraw = np.zeros(x.nbytes + 32, np.uint8), np.zeros(z.nbytes + 32, np.uint8)
    x0 = (-xraw.ctypes.data) % 16 + x_by
    z0 = (-zraw.ctypes.data) % 16 + z_by
    xraw[x0:x0 + x.nbytes] = x.view(np.uint8).ravel()
    _forward_at(m, n, xraw.ctypes.data + x0, zraw.ctypes.data + z0)
    assert zraw[z0:z0 + z.nbytes].tobytes() == z.tobytes()
    assert not zraw[:z0].any() and not zraw[z0 + z.nbytes:].any()


# above 262,144 rows the first quarter's logits go by way of device memory
@pytest.mark.parametrize("n", [262_143, 262_144, 262_145, 262_207, 1_000_003])
@pytest.mark.parametrize("z_by", [0, 4, 2052])
def test_split_logits_equal_chunks(n, z_by):
    m = gdp.Mlp(seed=7)
    x = _features(n, seed=9)
    z = np.concatenate([m.forward(x[k:k + 100_000]) for k in range(0, n, 100_000)])
    pages = mmap.mmap(-1, 4 * n + (1 << 17))  # pages that nothing has touched
    raw = np.frombuffer(pages, np.uint8)
    page = mmap.PAGESIZE
    at = (-raw.ctypes.data) % page + z_by
    _forward_at(m, n, x.ctypes.data, raw.ctypes.data + at)
    assert raw[at:at + 4 * n].tobytes() == z.tobytes()
    assert not raw[:at].any() and not raw[at + 4 * n:].any()
