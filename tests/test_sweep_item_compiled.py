"""sweep_item (csrc/gdp_sweep.h), the function that the batch loop runs, compiled as
plain C++: every item of every unit exactly once, each unit's items in their order,
and an equal part of every unit's list at a time."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "gpu-domain-propagator_gb300" / "csrc"
PARTS = 8

PROGRAM = r"""
#include "gdp_sweep.h"
#include <cstdio>
#include <cstdlib>
#include <vector>
static_assert(gdp::kSweepParts == 8, "the test's share of a list");
int main(int argc, char **argv) {
    std::vector<int> prefix(1, 0);
    for (int k = 1; k < argc; k++) prefix.push_back(prefix.back() + atoi(argv[k]));
    for (int i = 0; i < prefix.back(); i++) {
        const gdp::SweepItem at = gdp::sweep_item(prefix.data(), argc - 1, prefix.back(), i);
        printf("%d %d\n", at.unit, at.item);
    }
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("sweep")
    (d / "t.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", f"-I{CSRC}", str(d / "t.cpp"), "-o", str(d / "t")], check=True)
    return str(d / "t")


@pytest.mark.parametrize("sizes", [[1], [7], [8], [9], [1, 1, 1], [3, 0, 5], [0, 0, 1], [1, 0, 0], [17, 4, 100, 1, 33],
                                   [1000, 2, 2, 2], list(range(40)), [5000, 4999, 0, 8, 7]])
def test_every_item_once(program, sizes):
    out = subprocess.run([program, *map(str, sizes)], check=True, capture_output=True, text=True).stdout
    got = [tuple(map(int, line.split())) for line in out.splitlines()]
    total = sum(sizes)
    assert sorted(got) == [(k, a) for k, n in enumerate(sizes) for a in range(n)]
    done = [0] * len(sizes)
    for c, (k, a) in enumerate(got, 1):
        assert a == done[k]  # each unit's items in their order
        done[k] = a + 1
        # each unit is at its share of the claims, up to a part and a few items
        assert abs(done[k] - sizes[k] * c / total) <= sizes[k] / PARTS + 3
    assert done == sizes
