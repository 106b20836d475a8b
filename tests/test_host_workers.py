"""The threads of a staged copy (csrc/host_workers.h) where not all can be started:
the work is done by those that were, whatever kept the others from starting."""
from __future__ import annotations

import ctypes as C
import os
import subprocess

import pytest

from conftest import PKG

HARNESS = r"""
#include "host_workers.h"
#include <atomic>
#include <cstdlib>
#include <new>
static thread_local int left = -1;  // allocations of this thread until one fails
void* operator new(std::size_t n) {
    if (left >= 0 && left-- == 0) { left = -1; throw std::bad_alloc(); }
    if (void* p = std::malloc(n)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
int main(int argc, char** argv) {
    const int started = std::atoi(argv[1]), chunks = 1000;
    std::atomic<int> next{0}, done{0};
    left = started;
    gcu::run_workers(8, [&](unsigned) {
        while (next.fetch_add(1) < chunks) done.fetch_add(1);
    });
    return done.load() == chunks ? 0 : 1;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("host_workers")
    src, exe = d / "t.cpp", d / "t"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", os.path.join(PKG, "csrc"), str(src), "-o", str(exe)],
                   check=True)
    return str(exe)


@pytest.mark.parametrize("started", [0, 1, 3, 7, 100])
def test_work_is_done_by_the_threads_that_started(program, started):
    assert subprocess.run([program, str(started)], timeout=60).returncode == 0
