"""Words of the geometry's bitmap pool: none is given twice.

gpk_pool.h is compiled for the host and its requests are made from several
threads at once, of very different sizes and past the end of the pool.  The
given ranges lie in the pool and do not overlap, and a request is refused only
where it does not fit behind what was given.
"""
import os
import subprocess

import pytest

ROOT = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..")

SOURCE = r"""
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <thread>
#include <utility>
#include <vector>
#include "gpk_pool.h"

static std::atomic<unsigned> g_taken;
static std::atomic<int> g_go;

struct Counter {
    unsigned load() { return g_taken.load(); }
    unsigned exchange(unsigned old, unsigned next) {
        g_taken.compare_exchange_strong(old, next);
        return old;
    }
};

int main(int argc, char** argv) {
    const unsigned pool = std::atoi(argv[1]);
    const int rounds = std::atoi(argv[2]), T = 8, per = 40;
    for (int r = 0; r < rounds; ++r) {
        g_taken = 0;
        g_go = 0;
        std::vector<std::vector<std::pair<unsigned, unsigned>>> got(T);
        std::vector<std::vector<unsigned>> refused(T);
        std::vector<std::thread> th;
        for (int t = 0; t < T; ++t)
            th.emplace_back([&, t]() {
                std::mt19937 rng(r * T + t);
                g_go++;
                while (g_go < T) {}
                Counter c;
                for (int k = 0; k < per; ++k) {
                    const unsigned need = 1u << (rng() % 8);
                    unsigned at = 0;
                    if (pool_take(c, need, pool, at)) got[t].push_back({at, need});
                    else refused[t].push_back(need);
                }
            });
        for (auto& x : th) x.join();
        std::vector<std::pair<unsigned, unsigned>> all;
        for (auto& g : got) all.insert(all.end(), g.begin(), g.end());
        std::sort(all.begin(), all.end());
        unsigned end = 0;
        for (auto& a : all) {
            if (a.first < end) { std::printf("round %d: words from %u given twice\n", r, a.first); return 1; }
            end = a.first + a.second;
        }
        if (end > pool) { std::printf("round %d: past the end\n", r); return 1; }
        for (auto& q : refused)
            for (unsigned n : q)
                if (pool - end >= n) { std::printf("round %d: %u refused with %u left\n", r, n, pool - end); return 1; }
    }
    std::printf("ok\n");
    return 0;
}
"""


@pytest.mark.parametrize("pool", [1, 1000, 3000, 100000])
def test_no_word_is_given_twice(tmp_path, pool):
    src, exe = tmp_path / "pool.cpp", tmp_path / "pool"
    src.write_text(SOURCE)
    inc = os.path.join(ROOT, "gpk_b200", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", inc, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe), str(pool), "300"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
