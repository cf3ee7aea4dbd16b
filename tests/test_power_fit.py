"""Shared memory of the large systems' power-series layouts (host code,
superspinsim_gb300/csrc/sss_power.h), compiled with g++: over series from a few
hundred entries up, in steps of one slot's worth, every layout that
power_pack_big returns for 1 to 8 CTAs, for every quadrature's exponentials and
nodes, is within the kernel's limit with all that k_power_big keeps there (its
own sum, written out here), and a series that outgrows c CTAs fits 2 c.  No GPU."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r'''
#include "sss_power.h"
#include <cstdio>
using namespace sss;

static int fails = 0;
#define CHECK(c) do { if (!(c)) { std::printf("FAIL line %d: %s\n", __LINE__, #c); fails++; } } while (0)

int main() {
    int packed = 0, refused = 0;
    const int M = 171;
    for (int nm : {1, 5, 7})
        for (int KQ : {11, 22, 32, 53, 63}) {
            const int K = KQ / 10, Q = KQ % 10;
            for (int ctas : {1, 2, 4, 8}) {
                const int T = power_big_threads(ctas);
                for (int ne = 400; ne < 200000; ne += ctas * T) {
                    PowSeries ps;
                    ps.M = M;
                    ps.n_live = nm > 1;
                    ps.n_tables = 1;
                    for (int m = 0; m < nm; m++) ps.mono.push_back(std::vector<int>(ps.n_live, m));
                    for (int i = 0; i < ne; i++) ps.ent.push_back({i % M, i / M % M, i % nm});
                    PowLayout p;
                    if (!power_pack_big(ps, ctas, T, &p, K, Q, ps.n_live)) {
                        refused++;
                        PowLayout q;
                        CHECK(ctas == 8 || ne > 30 * ctas * T || power_pack_big(ps, 2 * ctas, power_big_threads(2 * ctas), &q, K, Q, ps.n_live));
                        break;
                    }
                    packed++;
                    const size_t n_x = (size_t)nm * M + 1, R = ctas == 1 ? 16 : 64;
                    const size_t bytes = 8 * (2 * n_x + R * Q * ps.n_live + (R * K + 1) * nm) + 10 * (size_t)p.E * T;
                    CHECK(p.E * T * ctas >= ne);
                    CHECK(bytes == power_smem(p, M, K, Q, ps.n_live, 1));
                    CHECK(bytes + 1024 <= 227 * 1024);   // the kernel's static arrays
                }
            }
        }
    CHECK(packed > 500 && refused > 20);
    std::printf("%d layouts, %d failures\n", packed, fails);
    return fails ? 1 : 0;
}
'''


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_large_layouts_fit_shared_memory(tmp_path):
    src = tmp_path/"fit.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path/"fit"
    inc = os.path.join(ROOT, "superspinsim_gb300", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", inc, str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
