"""Host threads of a solve (csrc/host_pool.h, compiled here): every piece runs
once, also when memory runs out while the threads are started."""
import shutil
import subprocess

import pytest

from ultrasound_solver_b200 import build

SOURCE = r"""
#include "host_pool.h"
#include <atomic>
#include <cstdlib>
#include <new>
static std::atomic<long> left{-1};  // allocations until one fails; below zero: none does
void* operator new(std::size_t n) {
    if (left.load() >= 0 && left.fetch_sub(1) == 0) throw std::bad_alloc();
    if (void* p = std::malloc(n)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
int main(int, char** argv) {
    left = std::atol(argv[1]);
    usv::HostPool pool(std::atoi(argv[2]));
    left = -1;
    for (int count : {0, 1, 2, 3, 64, 1000}) {
        static std::atomic<int> hits[1000];
        for (auto& h : hits) h = 0;
        pool.run(count, [&](int i) { ++hits[i]; });
        for (int i = 0; i < 1000; ++i)
            if (hits[i] != (i < count)) return 1;
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("pool")
    (d / "pool.cpp").write_text(SOURCE)
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-I", str(build.CSRC), str(d / "pool.cpp"),
                    "-o", str(d / "pool")], check=True)
    return str(d / "pool")


@pytest.mark.parametrize("helpers", [0, 1, 7])
@pytest.mark.parametrize("fail", [-1, 0, 1, 2, 3, 5, 8])
def test_every_piece_runs_once(program, helpers, fail):
    assert subprocess.run([program, str(fail), str(helpers)], timeout=60).returncode == 0
