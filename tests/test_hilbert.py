"""The Hilbert key of the spatial sort (csrc/tdp_hilbert.h), compiled for the host: the key of the
transform as it is stated, a curve whose neighbours are neighbours, and at a fraction of the time."""
import os
import subprocess

import pytest

from tholedipoleplugin_b200 import build as B

SOURCE = r"""
#include "tdp_hilbert.h"
#include <algorithm>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

// Skilling's transform and the interleaved Gray code, bit by bit.
static uint64_t stated(uint32_t x, uint32_t y, uint32_t z) {
    uint32_t v[3] = {x, y, z}, g = 0;
    for (uint32_t q = 1u << 20; q > 1; q >>= 1)
        for (int k = 0; k < 3; k++) {
            const uint32_t low = q - 1, d = (v[0] ^ v[k]) & low;
            if (v[k] & q) { v[0] ^= low; }
            else { v[0] ^= d; v[k] ^= d; }
        }
    v[1] ^= v[0];
    v[2] ^= v[1];
    for (uint32_t q = 1u << 20; q > 1; q >>= 1)
        if (v[2] & q) g ^= q - 1;
    uint64_t key = 0;
    for (int b = 20; b >= 0; b--)
        for (int k = 0; k < 3; k++) key = key << 1 | (((v[k] ^ g) >> b) & 1u);
    return key;
}

template <class F>
static double seconds(const std::vector<uint32_t>& p, uint64_t& sum, F f) {
    double best = 1e9;
    for (int rep = 0; rep < 5; rep++) {
        const auto t0 = std::chrono::steady_clock::now();
        for (size_t i = 0; i < p.size(); i += 3) sum += f(p[i], p[i + 1], p[i + 2]);
        best = std::min(best, std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count());
    }
    return best;
}

int main() {
    std::mt19937 rng(7);
    std::vector<uint32_t> p(3 * 32768);
    for (auto& v : p) v = rng() & 0x1fffff;
    for (int c = 0; c < 8; c++)   // the cube's corners
        for (int k = 0; k < 3; k++) p[3 * c + k] = c >> k & 1 ? 0x1fffff : 0;
    for (size_t i = 0; i < p.size(); i += 3)
        if (tdp::kHilbert.key(p[i], p[i + 1], p[i + 2]) != stated(p[i], p[i + 1], p[i + 2])) {
            printf("key %zu differs\n", i / 3);
            return 1;
        }
    // The 16^3 cells of the top four bits: every position once, each step to an adjacent cell.
    std::vector<int> cell(4096, -1);
    for (int c = 0; c < 4096; c++)
        cell[tdp::kHilbert.key((c & 15) << 17, (c >> 4 & 15) << 17, (c >> 8) << 17) >> 51] = c;
    for (int k = 0; k < 4096; k++) {
        if (cell[k] < 0) { printf("no cell at %d\n", k); return 1; }
        if (k == 0) continue;
        int d = 0;
        for (int s = 0; s < 12; s += 4) d += std::abs((cell[k] >> s & 15) - (cell[k - 1] >> s & 15));
        if (d != 1) { printf("step %d jumps\n", k); return 1; }
    }
    uint64_t sum = 0;
    const double slow = seconds(p, sum, stated),
                 fast = seconds(p, sum, [](uint32_t x, uint32_t y, uint32_t z) { return tdp::kHilbert.key(x, y, z); });
    printf("stated %.3f ms, table %.3f ms (%llu)\n", 1e3 * slow, 1e3 * fast, (unsigned long long)sum);
    return fast < 0.4 * slow ? 0 : 2;
}
"""


def test_key(tmp_path):
    src, exe = tmp_path / "hilbert.cpp", tmp_path / "hilbert"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", B.CSRC, "-o", str(exe), str(src)], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
