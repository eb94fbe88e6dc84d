"""Host-only parts of the engine, compiled with the C++ compiler and run without a GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "braketsimulator.jl_gb300", "csrc")


def run_cpp(tmp_path, source, *extra):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(source)
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(src), *extra, "-o", str(exe)], check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


def test_a_result_whose_ticket_never_comes_is_an_error(tmp_path):
    """The wait for a result in mapped memory: a ticket that is there, that comes while polling and that comes with the
    stream's end is a result; a failed stream and one that ends without the ticket (an earlier ticket in the word) are
    errors, not the stale memory."""
    run_cpp(tmp_path, r"""
#include "bs_ticket.h"
#include <cstdio>
#include <thread>
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
int main() {
    volatile int64_t word = 7;
    int synced = 0;
    auto ok = [&] { synced++; return BS_OK; };
    CHECK(bs_poll_ticket(&word, 7, 0.01, ok) == BS_OK && synced == 0);
    std::thread late([&] { std::this_thread::sleep_for(std::chrono::milliseconds(20)); word = 8; });
    CHECK(bs_poll_ticket(&word, 8, 10.0, ok) == BS_OK && synced == 0);
    late.join();
    CHECK(bs_poll_ticket(&word, 9, 0.01, [&] { synced++; word = 9; return BS_OK; }) == BS_OK && synced == 1);
    CHECK(bs_poll_ticket(&word, 10, 0.01, [&] { return BS_ERR_CUDA; }) == BS_ERR_CUDA);
    CHECK(bs_poll_ticket(&word, 10, 0.01, ok) == BS_ERR_TIMEOUT);
    return 0;
}
""")
