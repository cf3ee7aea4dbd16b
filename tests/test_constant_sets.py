"""The sets of constant values of a batch (host code,
superspinsim_gb300/csrc/sss_constant.h), compiled with g++: random programs with
ascending, repeated, out-of-order and infinite segment ends, one to four live
channels, channels the programs lack.  Every set found is held by the programs
(each channel's segment looked up at a time as the kernels look it up), every
stretch of at least dt between two segment ends whose values are constant is
found, and the time grows with the segments, not with their square.  No GPU."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r'''
#include "sss_constant.h"
#include <chrono>
#include <cstdio>
#include <random>
using namespace sss;

static bool lookup(const double* prog, int nch, int nseg, int ch, double t, double* x) {
    *x = 0.0;
    for (int s = 0; s < nseg && ch < nch; s++) {
        const double* g = prog + ((size_t)ch * nseg + s) * 5;
        if (!(t < g[0])) continue;
        *x = g[1];
        return g[2] == 0.0;
    }
    return true;
}

int main() {
    std::mt19937_64 rng(9);
    auto pick = [&](int n) { return (int)(rng() % n); };
    int fails = 0, found = 0;
    for (int run = 0; run < 4000; run++) {
        const int nch = 1 + pick(4), nseg = 1 + pick(7);
        std::vector<int> live;
        for (int c = 0; c < 4; c++)
            if (pick(2) || (c == 3 && live.empty())) live.push_back(c);
        std::vector<double> p((size_t)nch * nseg * 5, 0.0), cut;
        for (int c = 0; c < nch; c++)
            for (int s = 0; s < nseg; s++) {
                double* g = &p[((size_t)c * nseg + s) * 5];
                const int kind = pick(8);
                g[0] = kind == 0 ? INFINITY : kind == 1 ? -INFINITY : kind == 2 ? 3.0 : kind == 3 ? -1.0 : 0.25 * pick(40);
                g[1] = pick(3);
                g[2] = pick(3) ? 0.0 : 1.0;
                if (std::isfinite(g[0])) cut.push_back(g[0]);
            }
        const double dt = 0.5;
        const std::vector<ConstSet> sets = constant_sets(p.data(), 1, nch, nseg, live, dt);
        std::sort(cut.begin(), cut.end());
        std::vector<double> times{cut.empty() ? 0.0 : cut.front() - 1.0, cut.empty() ? 0.0 : cut.back() + 1.0};
        for (size_t i = 1; i < cut.size(); i++) times.push_back(0.5 * (cut[i - 1] + cut[i]));
        auto values = [&](double t, std::vector<double>* v) {
            bool constant = true;
            v->clear();
            for (int c : live) {
                double x;
                constant = lookup(p.data(), nch, nseg, c, t, &x) && constant;
                v->push_back(x);
            }
            return constant;
        };
        std::vector<double> v;
        for (const ConstSet& s : sets) {
            bool held = false;
            for (double t : times) held = held || (values(t, &v) && v == s.value);
            found++;
            if (!held) fails++;
        }
        for (size_t i = 0; i < times.size(); i++) {
            if (i >= 2 && cut[i - 1] - cut[i - 2] < dt) continue;
            if (!values(times[i], &v)) continue;
            bool has = sets.size() == (size_t)kConstMax;
            for (const ConstSet& s : sets) has = has || s.value == v;
            if (!has) fails++;
        }
    }
    // 16 times the segments, 16 times the time (within a factor of 8 for the
    // machine's noise; 256 times were it quadratic)
    double best[2] = {1e9, 1e9};
    for (int k = 0; k < 2; k++) {
        const int nseg = k ? 4096 : 256;
        std::vector<double> p((size_t)4 * nseg * 5, 0.0);
        for (int c = 0; c < 4; c++)
            for (int s = 0; s < nseg; s++) {
                p[((size_t)c * nseg + s) * 5] = s + 0.1 * c;
                p[((size_t)c * nseg + s) * 5 + 1] = s % 3;
            }
        for (int rep = 0; rep < 9; rep++) {
            const auto a = std::chrono::steady_clock::now();
            found += (int)constant_sets(p.data(), 1, 4, nseg, {0, 1, 2, 3}, 0.05).size();
            best[k] = std::min(best[k], std::chrono::duration<double>(std::chrono::steady_clock::now() - a).count());
        }
    }
    if (best[1] > 128.0 * best[0]) {
        std::printf("FAIL: %g s for 256 segments, %g s for 4096\n", best[0], best[1]);
        fails++;
    }
    std::printf("%d sets, %d failures\n", found, fails);
    return fails || found < 1000;
}
'''


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_sets_of_constant_values(tmp_path):
    src = tmp_path/"sets.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path/"sets"
    inc = os.path.join(ROOT, "superspinsim_gb300", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-I", inc, str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
