"""csrc/parallel_rows.h: every row once, also where threads or memory for them
run out part of the way."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "ollinaxis-bib_gb300", "csrc")

DRIVER = r"""
#include "parallel_rows.h"
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>
// the n-th allocation from now on fails, and all after it
static std::atomic<long> left{1l << 60};
void* operator new(std::size_t n) {
    if (--left < 0) throw std::bad_alloc();
    void* p = std::malloc(n);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
int main(int argc, char** argv) {
    const int lo = -2, hi = std::atoi(argv[1]);
    const long points = std::atol(argv[2]), fail = std::atol(argv[3]);
    std::vector<std::atomic<int>> done(hi - lo);
    for (auto& d : done) d = 0;
    if (fail >= 0) left = fail;
    ollin::parallel_rows(lo, hi, (std::size_t)points, [&](int j) { ++done[j - lo]; });
    left = 1l << 60;
    for (auto& d : done)
        if (d != 1) return 3;
    std::puts("every row once");
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("rows")
    (d / "driver.cpp").write_text(DRIVER)
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", CSRC, "-o", str(d / "driver"), str(d / "driver.cpp")], check=True)
    return str(d / "driver")


@pytest.mark.parametrize("rows, points", [(1, 10), (5, 32768 * 16), (300, 32768 * 3), (1027, 1 << 20)])
@pytest.mark.parametrize("fail", [-1, 0, 1, 2, 5])
def test_every_row_once(program, rows, points, fail):
    r = subprocess.run([program, str(rows), str(points), str(fail)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "every row once\n", (r.returncode, r.stderr)
