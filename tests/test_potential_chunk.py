"""The chunk rule of the orbit potentials (csrc/potential_chunk.h), compiled for the host: it finds the minimum of its
cost over every chunk count, in a small part of the time that looking at every count takes."""

import os
import subprocess

from conftest import ROOT

SOURCE = r"""
#include <stdio.h>
#include <stdlib.h>
#include <chrono>
#include "potential_chunk.h"
static int64_t every(int64_t n, int64_t p, int64_t slots) {
    int64_t cmax = std::min<int64_t>((n + 7) / 8, 65535);
    cmax = std::max<int64_t>(1, std::min<int64_t>(cmax, 8 * ((slots + p - 1) / p)));
    int64_t chunk = n, best = 0;
    for (int64_t c = 1; c <= cmax; ++c) {
        const int64_t e = (n + c - 1) / c, t = (p * c + slots) * ((e + 3) / 4 + 2);
        if (c == 1 || t < best) best = t, chunk = e;
    }
    return chunk;
}
template <class F> static double seconds(F f) {
    double best = 1e9;
    for (int r = 0; r < 5; ++r) {
        const auto a = std::chrono::steady_clock::now();
        int64_t sum = 0;
        for (int64_t i = 0; i < 200; ++i) sum += f(131072 + i);
        if (sum == 0) abort();
        best = std::min(best, std::chrono::duration<double>(std::chrono::steady_clock::now() - a).count());
    }
    return best;
}
int main() {
    int bad = 0;
    srand(7);
    for (int i = 0; i < 6000; ++i) {
        const int64_t n = 1 + (int64_t)exp(log(3e5) * rand() / RAND_MAX), p = 1 + (int64_t)exp(log(5e4) * rand() / RAND_MAX);
        const int64_t slots = 148 * (1 + rand() % 10);
        if (every(n, p, slots) != bc::potential_chunk(n, p, slots)) {
            printf("%ld %ld %ld\n", (long)n, (long)p, (long)slots);
            ++bad;
        }
    }
    const double slow = seconds([](int64_t n) { return every(n, 1, 740); });
    const double fast = seconds([](int64_t n) { return bc::potential_chunk(n, 1, 740); });
    if (fast > 0.25 * slow) printf("%g s against %g s\n", fast, slow), ++bad;
    return bad != 0;
}
"""


def test_finds_the_minimum_quickly(tmp_path):
    (tmp_path / "probe.cpp").write_text(SOURCE)
    exe = str(tmp_path / "probe")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "bempp-cl_b200", "csrc"), "-o", exe,
                    str(tmp_path / "probe.cpp")], check=True)
    done = subprocess.run([exe], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout
