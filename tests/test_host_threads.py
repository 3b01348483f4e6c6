"""CPU test of the host threads behind the uploads: a thread that cannot be started is done without, and nothing is thrown."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_UNIT = r"""
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>
#include "host_threads.h"
static std::atomic<int> allowed{1 << 30};
void *operator new(std::size_t n) {
    if (allowed.fetch_sub(1) <= 0) throw std::bad_alloc();
    return std::malloc(n);
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, std::size_t) noexcept { std::free(p); }
int main(int, char **argv) {
    std::atomic<int> next{0}, done{0}, workers{0};
    auto work = [&](int) { workers++; while (next.fetch_add(1) < 1000) done++; };
    allowed = std::atoi(argv[1]);          // every thread's state is one allocation
    q36::run_on_threads<8>(8, work);
    allowed = 1 << 30;
    std::printf("%d %d\n", done.load(), workers.load());
    return 0;
}
"""


@pytest.mark.parametrize("allowed", [0, 1, 3, 100])
def test_missing_threads_are_done_without(tmp_path, allowed):
    src, exe = tmp_path / "unit.cpp", tmp_path / "unit"
    src.write_text(_UNIT)
    r = subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-pthread", "-I", os.path.join(ROOT, "q36_b200", "csrc"), str(src),
                        "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe), str(allowed)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, (r.returncode, r.stderr)
    done, workers = map(int, r.stdout.split())
    assert done == 1000 and workers == 1 + min(allowed, 7)


def test_the_uploads_start_threads_nowhere_else():
    for f in os.listdir(os.path.join(ROOT, "q36_b200", "csrc")):
        if f != "host_threads.h":
            assert "std::thread(" not in open(os.path.join(ROOT, "q36_b200", "csrc", f)).read(), f
