"""The threads that carry large results: every share is carried, by the caller where a
thread or the memory for one cannot be had, and nothing ends the process."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ferrolearn_gb300", "csrc")

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>
#include "fk_workers.h"

static std::atomic<int> left{-1};  // allocations until they fail (negative: none do)
void *operator new(std::size_t n) {
    if (left >= 0 && left-- == 0) {
        left = 0;
        throw std::bad_alloc();
    }
    void *p = std::malloc(n);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, std::size_t) noexcept { std::free(p); }

int main(int, char **argv) {
    const int n = std::atoi(argv[1]);
    std::atomic<int> ran[8] = {};
    left = std::atoi(argv[2]);
    fk::run_workers<8>(n, [&](int w) { ran[w]++; });
    left = -1;
    for (int w = 0; w < 8; w++) std::printf("%d", (int)ran[w]);
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("workers")
    (d / "p.cpp").write_text(PROGRAM)
    exe = str(d / "p")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-o", exe, str(d / "p.cpp")], check=True)
    return exe


@pytest.mark.parametrize("n", [0, 1, 2, 7, 8])
@pytest.mark.parametrize("fail_at", [-1, 0, 1, 3])
def test_every_share_is_carried_once(program, n, fail_at):
    r = subprocess.run([program, str(n), str(fail_at)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    assert r.stdout == "1" * n + "0" * (8 - n)
