"""rtb::parallel_for (csrc/rt_parallel.h) when host memory runs out while it
starts its threads: the ranges whose thread could not be started run on the
caller, and every element is visited once.  A C++ program whose operator new
fails at a chosen allocation of the calling thread."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r'''
#include "rt_parallel.h"
#include <atomic>
#include <cstdio>
#include <cstdlib>

static thread_local int fail_at = 0;         /* fails the fail_at-th allocation of this thread; 0: none */
void* operator new(std::size_t n) {
    if (fail_at > 0 && --fail_at == 0) throw std::bad_alloc();
    void* p = std::malloc(n ? n : 1);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

int main(int, char** argv) {
    const int at = std::atoi(argv[1]);
    const int n = 100003;
    std::vector<std::atomic<int>> seen(n);
    rtb::parallel_for(1, 1, [](int64_t, int64_t) {});
    bool thrown = false;
    fail_at = at;
    try {
        rtb::parallel_for(n, 1, [&](int64_t a, int64_t b) { for (int64_t i = a; i < b; i++) seen[i]++; });
    } catch (const std::bad_alloc&) {
        thrown = true;                       /* before any thread was started: nothing has run */
    }
    fail_at = 0;
    for (int i = 0; i < n; i++)
        if (seen[i] != (thrown ? 0 : 1)) { std::printf("element %d visited %d times\n", i, (int)seen[i]); return 1; }
    std::printf("parallel ok\n");
    return 0;
}
'''


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("parallel")
    (d / "p.cpp").write_text(SRC)
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", os.path.join(ROOT, "radiantium_gb300", "csrc"),
                        str(d / "p.cpp"), "-o", str(d / "p")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return str(d / "p")


@pytest.mark.parametrize("fail_at", [0, 1, 2, 3, 4])
def test_out_of_memory_while_threads_start(program, fail_at):
    r = subprocess.run([program, str(fail_at)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
    assert "parallel ok" in r.stdout
