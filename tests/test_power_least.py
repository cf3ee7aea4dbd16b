"""The bound that decides about a large system's power series before it is made
(host code, superspinsim_gb300/csrc/sss_power.h), compiled with g++: on random
chains, bands and sparse matrices of 65 to 300 rows, with and without a varying
coefficient, at weak and strong exponents and vanishing drives, the series never
has fewer entries than power_least_entries says, and for all but the weakest the
bound is worth having (a tenth of the entries).  No GPU."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r'''
#include "sss_power.h"
#include <cstdio>
#include <random>
using namespace sss;

int main() {
    std::mt19937_64 rng(5);
    std::uniform_real_distribution<double> u(0.3, 1.0);
    int fails = 0, runs = 0;
    for (int M : {65, 128, 171, 300})
        for (int kind : {0, 1, 2})
            for (int live : {0, 1})
                for (double x : {1e-6, 1e-3, 0.05, 0.4})
                    for (double b : {1e-12, 1e-5, 1e-3}) {
                        if (!live && b != 1e-3) continue;
                        std::vector<int> rp(1, 0), col;
                        for (int r = 0; r < M; r++) {
                            for (int c = 0; c < M; c++) {
                                const bool in = kind == 0   ? c == r || c + 1 == r
                                                : kind == 1 ? std::abs(c - r) <= 3
                                                            : c == r || u(rng) > 0.99;
                                if (in) col.push_back(c);
                            }
                            rp.push_back((int)col.size());
                        }
                        const size_t nnz = col.size();
                        // positive entries: no term cancels another
                        std::vector<std::vector<double>> A(1), Al(1, std::vector<double>(nnz, 0.0)), G(live);
                        std::vector<double> rho(live, 0.75), sa(M, 0.0), sg(M, 0.0);
                        for (size_t q = 0; q < nnz; q++) {
                            A[0].push_back(q % 3 ? u(rng) : 0.0);
                            sa[col[q]] += A[0][q];
                            if (live) G[0].push_back(q % 2 ? u(rng) : 0.0);
                            if (live) sg[col[q]] += G[0][q];
                        }
                        const double na = *std::max_element(sa.begin(), sa.end()), ng = *std::max_element(sg.begin(), sg.end());
                        for (double& v : A[0]) v *= x / na;
                        if (live)
                            for (double& v : G[0]) v *= b / (0.75 * ng);
                        PowSeries ps;
                        if (!power_series(M, rp, col, A, Al, G, rho, &ps)) {
                            std::printf("FAIL refused\n");
                            fails++;
                            continue;
                        }
                        const long least = power_least_entries(M, rp, col, A[0], live ? &G[0] : nullptr, x, live ? b : 0.0);
                        runs++;
                        if (least > (long)ps.ent.size()) {
                            std::printf("FAIL M %d kind %d live %d x %g b %g: %ld of %zu\n", M, kind, live, x, b, least,
                                        ps.ent.size());
                            fails++;
                        }
                    }
    std::printf("%d series, %d failures\n", runs, fails);
    return fails ? 1 : 0;
}
'''


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_series_has_at_least_these_entries(tmp_path):
    src = tmp_path/"least.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path/"least"
    inc = os.path.join(ROOT, "superspinsim_gb300", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-I", inc, str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
