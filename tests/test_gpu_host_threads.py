"""A context built by fewer host threads than it asks for (OMP_THREAD_LIMIT, a call
from inside a caller's parallel region) has every row: its results are those of
this process."""
import hashlib
import os
import subprocess
import sys
from pathlib import Path

import pytest

import gdp
import gdpgen

pytestmark = pytest.mark.gpu

PKG = Path(gdp.__file__).resolve().parent
CHILD = """
import sys, hashlib
sys.path.insert(0, sys.argv[1])
import gdp, gdpgen
mip = gdpgen.random_mip(1, seed=71, m=400_000, n=300_000, n_dense_rows=4, dense_len=9_000)
with gdp.Context(mip) as ctx:
    lb, ub, st = ctx.propagate()
    print(ctx.layout()["thread_rows"], ctx.layout()["split_rows"], st["rounds"],
          hashlib.sha256(lb.tobytes() + ub.tobytes()).hexdigest())
"""


@pytest.mark.parametrize("env", [{"OMP_THREAD_LIMIT": "1"}, {"OMP_THREAD_LIMIT": "3"}, {"OMP_NUM_THREADS": "2"}])
def test_small_teams(env):
    mip = gdpgen.random_mip(1, seed=71, m=400_000, n=300_000, n_dense_rows=4, dense_len=9_000)
    with gdp.Context(mip) as ctx:
        lb, ub, st = ctx.propagate()
        lay = ctx.layout()
    out = subprocess.run([sys.executable, "-c", CHILD, str(PKG)], env={**os.environ, **env}, check=True,
                         capture_output=True, text=True).stdout.split()
    assert out == [str(lay["thread_rows"]), str(lay["split_rows"]), str(st["rounds"]),
                   hashlib.sha256(lb.tobytes() + ub.tobytes()).hexdigest()]
