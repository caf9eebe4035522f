"""Words of the geometry's bitmap pool: none is given twice.

gpk_pool.h is compiled for the host and its requests are made from several
threads at once, of very different sizes and past the end of the pool.  The
given ranges lie in the pool and do not overlap, and a request is refused only
where it does not fit behind what was asked for (with one thread: behind what
was given).
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

static std::atomic<unsigned long long> g_taken;
static std::atomic<int> g_go;

struct Counter {
    unsigned long long load() { return g_taken.load(); }
    unsigned long long add(unsigned v) { return g_taken.fetch_add(v); }
};

int main(int argc, char** argv) {
    const unsigned pool = std::atoi(argv[1]);
    const int rounds = std::atoi(argv[2]), T = std::atoi(argv[3]), per = 320 / T;
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
        const unsigned long long behind = T == 1 ? end : g_taken.load();
        for (auto& q : refused)
            for (unsigned n : q)
                if (behind + n <= pool) { std::printf("round %d: %u refused with %u left\n", r, n, pool - end); return 1; }
    }
    std::printf("ok\n");
    return 0;
}
"""


@pytest.mark.parametrize("pool,threads", [(1, 8), (1000, 8), (3000, 8), (100000, 8), (1000, 1), (3000, 1)])
def test_no_word_is_given_twice(tmp_path, pool, threads):
    src, exe = tmp_path / "pool.cpp", tmp_path / "pool"
    src.write_text(SOURCE)
    inc = os.path.join(ROOT, "gpk_b200", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", inc, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe), str(pool), "300", str(threads)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
