"""touch_pages (csrc/gdp_pages.h), compiled by itself: the bytes of the array and
around it keep their values, and every page of a new mapping is resident after
it."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "gpu-domain-propagator_gb300" / "csrc"

PROGRAM = r"""
#include "gdp_pages.h"
#include <cstdio>
#include <cstdlib>
#include <sys/mman.h>
#include <unistd.h>
#include <vector>

int main(int argc, char **argv) {
    const size_t off = atoll(argv[1]), bytes = atoll(argv[2]);
    const int threads = atoi(argv[3]);
    std::vector<unsigned char> a(off + bytes + 64), b;
    for (size_t i = 0; i < a.size(); i++) a[i] = (unsigned char)(1 + i % 251);
    b = a;
    gdp::touch_pages(a.data() + off, bytes, threads);
    if (a != b) return printf("contents changed\n"), 1;
    const size_t page = sysconf(_SC_PAGESIZE), len = (off + bytes + page - 1) / page * page;
    char *m = (char *)mmap(nullptr, len, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (m == MAP_FAILED) return 2;
    madvise(m, len, MADV_NOHUGEPAGE);
    gdp::touch_pages(m + off % page, bytes, threads);
    std::vector<unsigned char> in(len / page);
    if (mincore(m, len, in.data())) return 3;
    for (size_t i = 0; i < (off % page + bytes + page - 1) / page; i++)
        if (!(in[i] & 1)) return printf("page %zu untouched\n", i), 1;
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("pages")
    (d / "t.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O2", "-fopenmp", f"-I{CSRC}", str(d / "t.cpp"), "-o", str(d / "t")], check=True)
    return str(d / "t")


@pytest.mark.parametrize("off", [0, 4, 4092, 4095])
@pytest.mark.parametrize("size", [1, 4, 4096, 4097, 8192, 1_048_580])
@pytest.mark.parametrize("threads", [1, 3])
def test_contents_kept_and_pages_resident(program, off, size, threads):
    out = subprocess.run([program, str(off), str(size), str(threads)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
