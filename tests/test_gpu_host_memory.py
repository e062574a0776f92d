"""A host allocation that fails inside a call is the call's error, not the end of the
process."""
import subprocess
import sys
from pathlib import Path

import pytest

import gdp

pytestmark = pytest.mark.gpu

PKG = Path(gdp.__file__).resolve().parent
CHILD = """
import resource, sys
sys.path.insert(0, sys.argv[1])
import numpy as np, gdp
n = 8_000_000
x = np.zeros((n, 16), np.float32)
y, w = np.zeros(n, np.float32), np.ones(n, np.float32)
m = gdp.Mlp(seed=1)
m.train(x[:1000], y[:1000], w[:1000], epochs=1)
now = int(next(s for s in open("/proc/self/status") if s.startswith("VmSize")).split()[1]) * 1024
resource.setrlimit(resource.RLIMIT_AS, (now + (16 << 20), resource.RLIM_INFINITY))
try:  # 96 MB for the order of the samples and their weights
    m.train(x, y, w, epochs=1)
    print("trained")
except gdp.GDPError as e:
    print("error:", e)
resource.setrlimit(resource.RLIMIT_AS, (resource.RLIM_INFINITY, resource.RLIM_INFINITY))
print("loss", m.train(x[:1000], y[:1000], w[:1000], epochs=1) >= 0)
"""


def test_training_without_host_memory():
    out = subprocess.run([sys.executable, "-c", CHILD, str(PKG)], capture_output=True, text=True)
    assert out.returncode == 0, out.stderr[-500:]
    assert "host allocation failed" in out.stdout and "loss True" in out.stdout
