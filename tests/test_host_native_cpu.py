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


def test_blocks_kept_between_calls_are_given_back(tmp_path):
    """The pool of kept device blocks on a fake of the allocator with room for 100 bytes: at most its cap is kept, the
    oldest block goes first, a block goes with its owner, and an allocation that does not fit frees the pool and is
    tried again, also from another thread."""
    run_cpp(tmp_path, r"""
#include "bs_keep.h"
#include <cstdio>
#include <map>
#include <thread>
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
struct Fake {
    static std::mutex m;
    static std::map<void*, size_t> live;
    static size_t used() { size_t n = 0; for (auto& k : live) n += k.second; return n; }
    static void* get(size_t n) {
        std::lock_guard<std::mutex> lock(m);
        if (used() + n > 100) return nullptr;
        void* p = new char[n];
        live[p] = n;
        return p;
    }
    static void put(void* p) {
        std::lock_guard<std::mutex> lock(m);
        if (!live.erase(p)) std::abort();   // freed twice
        delete[] (char*)p;
    }
};
std::mutex Fake::m;
std::map<void*, size_t> Fake::live;
int main() {
    KeepPool<Fake> pool(60);
    int a, b, c;
    size_t got = 0;
    CHECK(!pool.take(&a, 10, &got));
    void* p = pool.get(40);
    pool.keep(&a, p, 40);
    CHECK(!pool.take(&b, 10, &got));                        // another handle's
    CHECK(pool.take(&a, 30, &got) == p && got == 40 && pool.idle_bytes() == 0);
    pool.keep(&a, p, 40);
    CHECK(!pool.take(&a, 50, &got) && Fake::used() == 0);   // too small: freed
    pool.keep(&a, pool.get(30), 30);
    pool.keep(&b, pool.get(30), 30);
    pool.keep(&c, pool.get(20), 20);                        // above the cap: the oldest goes
    CHECK(pool.idle_bytes() == 50 && !pool.take(&a, 1, &got));
    pool.drop(&b);
    CHECK(Fake::used() == 20);
    pool.keep(&b, pool.get(40), 40);
    void* big = pool.get(90);                               // does not fit beside the kept blocks
    CHECK(big && pool.idle_bytes() == 0 && Fake::used() == 90);
    CHECK(!pool.get(20));
    Fake::put(big);
    auto work = [&](void* me) {
        for (int i = 0; i < 2000; i++) {
            size_t n = 0;
            void* q = pool.take(me, 10, &n);
            if (!q) { n = 10 + i % 7; q = pool.get(n); }
            if (q) pool.keep(me, q, n);
        }
        pool.drop(me);
    };
    std::thread t1(work, &a), t2(work, &b), t3(work, &c);
    t1.join(); t2.join(); t3.join();
    CHECK(pool.idle_bytes() == 0 && Fake::used() == 0);
    return 0;
}
""")


PLAN = r"""
#include <cstdio>
#include <cstdlib>
#include "bs_internal.h"
int bs_fail(bs_sim*, int code, const std::string&) { return code; }
int bs_vec_bits(const bs_sim* s) { return s->n; }
double bs_fuse_tc(const std::vector<const HostGate*>&, const int*, int, double, std::vector<HostGate>*) { return 0; }
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
"""


def run_plan(tmp_path, main):
    cuda = next((p for p in (os.environ.get("CUDA_HOME"), "/usr/local/cuda") if p and os.path.exists(os.path.join(p, "include"))), None)
    if not cuda:
        pytest.skip("no CUDA headers")
    run_cpp(tmp_path, PLAN + main, "-I", os.path.join(cuda, "include"), os.path.join(CSRC, "bs_plan.cpp"))


def test_threads_of_a_sweep_follow_what_is_set(tmp_path):
    """512 threads for sweeps of up to 152 tiles is the choice where nothing is set: BS_TILE_THREADS and a handle's tuning
    hold for every size."""
    run_plan(tmp_path, r"""
int main() {
    bs_sim s;
    unsetenv("BS_TILE_THREADS");
    CHECK(bs_sweep_threads(&s, 152) == 512 && bs_sweep_threads(&s, 153) == 256);
    setenv("BS_TILE_THREADS", "256", 1);
    CHECK(bs_sweep_threads(&s, 1) == 256 && bs_sweep_threads(&s, 4096) == 256);
    setenv("BS_TILE_THREADS", "512", 1);
    CHECK(bs_sweep_threads(&s, 4096) == 512);
    s.tune.tile_threads = 256;
    CHECK(bs_sweep_threads(&s, 1) == 256);
    unsetenv("BS_TILE_THREADS");
    CHECK(bs_sweep_threads(&s, 1) == 256);
    return 0;
}
""")


def test_eight_handles_of_a_batch_hold_at_most_8_gib(tmp_path):
    """Eight handles for lists of 8192 instructions and more, unless their states take more than 8 GiB together; four
    otherwise; never more than circuits; BS_BATCH_STREAMS as set."""
    run_plan(tmp_path, r"""
int main() {
    const double gib = 1 << 30;
    unsetenv("BS_BATCH_STREAMS");
    CHECK(bs_batch_handles(48, 8191, gib) == 4 && bs_batch_handles(48, 8192, gib) == 8);
    CHECK(bs_batch_handles(48, 100000, 8 * gib) == 8 && bs_batch_handles(48, 100000, 8.5 * gib) == 4);
    CHECK(bs_batch_handles(3, 100000, gib) == 3 && bs_batch_handles(0, 0, 0) == 0);
    setenv("BS_BATCH_STREAMS", "6", 1);
    CHECK(bs_batch_handles(48, 100000, 128 * gib) == 6 && bs_batch_handles(48, 1, gib) == 6);
    return 0;
}
""")
