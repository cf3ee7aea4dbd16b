"""Maps of output samples over which nothing varies (host code,
superspinsim_gb300/csrc/sss_constant.h), compiled with g++: the map of F steps
of K exponentials, as hi + lo, against stepping every unit vector in long
double, and the sets of values found in hand-made programs.  Tolerance: the
long double steps round F K times, each M products of 2^-64 (x86; less on
Arm).  No GPU."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r'''
#include "sss_constant.h"
#include <cstdio>
#include <random>
using namespace sss;
using pow_detail::dd;

static int fails = 0;
#define CHECK(c) do { if (!(c)) { std::printf("FAIL line %d: %s\n", __LINE__, #c); fails++; } } while (0)

int main() {
    std::mt19937_64 rng(3);
    std::uniform_real_distribution<double> u(-1.0, 1.0);
    for (int M : {1, 2, 5, 19, 32})
        for (int F : {1, 7, 16, 100})
            for (int K : {1, 2, 5}) {
                std::vector<int> rp(1, 0), col;
                for (int r = 0; r < M; r++) {
                    for (int c = 0; c < M; c++)
                        if (c == r || u(rng) > 0.6) col.push_back(c);
                    rp.push_back((int)col.size());
                }
                std::vector<std::vector<dd>> ex(K);
                for (auto& e : ex)
                    for (size_t q = 0; q < col.size(); q++) e.push_back({0.04 / M * u(rng), 1e-19 * u(rng)});
                std::vector<double> hi, lo;
                CHECK(constant_sample(M, F, rp, col, ex, &hi, &lo));
                for (int c = 0; c < M; c++) {
                    std::vector<long double> x(M, 0.0L);
                    x[c] = 1.0L;
                    for (int n = 0; n < F; n++)
                        for (int e = K - 1; e >= 0; e--) {
                            std::vector<long double> T(x), d(M, 0.0L);
                            for (int j = 1; j < 30; j++) {
                                std::vector<long double> y(M, 0.0L);
                                for (int r = 0; r < M; r++)
                                    for (int q = rp[r]; q < rp[r + 1]; q++)
                                        y[r] += ((long double)ex[e][q].hi + ex[e][q].lo) * T[col[q]] / j;
                                for (int r = 0; r < M; r++) d[r] += y[r];
                                T = y;
                            }
                            for (int r = 0; r < M; r++) x[r] += d[r];
                        }
                    for (int r = 0; r < M; r++) {
                        const long double m = (long double)hi[r * M + c] + lo[r * M + c] + (r == c ? 1.0L : 0.0L);
                        CHECK(std::fabs((double)(m - x[r])) <= std::ldexp(2.0 * F * K * (M + 30), -64));
                    }
                }
            }
    std::vector<double> hi, lo;
    CHECK(!constant_sample(1, 4, {0, 1}, {0}, {{dd{1.5, 0.0}}}, &hi, &lo));
    CHECK(!constant_sample(1, 4, {0, 1}, {0}, {{dd{NAN, 0.0}}}, &hi, &lo));
    // two channels, three segments: drive off / on / off, laser on until 4
    const double inf = INFINITY;
    const double p[2][3][5] = {{{1.0, 0, 0, 0, 0}, {3.0, 0, 2.0, 5.0, 0}, {inf, 0, 0, 0, 0}},
                               {{4.0, 0.5, 0, 0, 0}, {inf, 0, 0, 0, 0}, {-inf, 9.0, 0, 0, 0}}};
    const double* prog = &p[0][0][0];
    auto has = [](const std::vector<ConstSet>& s, std::vector<double> v) {
        for (const ConstSet& c : s)
            if (c.value == v) return true;
        return false;
    };
    std::vector<ConstSet> s = constant_sets(prog, 1, 2, 3, {0, 1}, 0.5);
    CHECK(s.size() == 2 && has(s, {0.0, 0.5}) && has(s, {0.0, 0.0}));
    s = constant_sets(prog, 1, 2, 3, {1}, 0.5);
    CHECK(s.size() == 2 && has(s, {0.5}) && has(s, {0.0}));
    s = constant_sets(prog, 1, 1, 3, {0, 1}, 0.5);   // a channel the programs lack is zero
    CHECK(s.size() == 1 && has(s, {0.0, 0.0}));
    // too short to hold a sample
    const double q[1][3][5] = {{{1.0, 0, 1.0, 1.0, 0}, {1.25, 3.0, 0, 0, 0}, {inf, 0, 1.0, 1.0, 0}}};
    CHECK(constant_sets(&q[0][0][0], 1, 1, 3, {0}, 0.5).empty());
    CHECK(constant_sets(&q[0][0][0], 1, 1, 3, {0}, 0.25).size() == 1);
    std::printf("%d failures\n", fails);
    return fails ? 1 : 0;
}
'''


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_constant_samples(tmp_path):
    src = tmp_path/"constant.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path/"constant"
    inc = os.path.join(ROOT, "superspinsim_gb300", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", inc, str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
