"""The launches of a drop-in run by propagator columns (host code,
superspinsim_gb300/csrc/sss_columns.h), compiled with g++: over trajectories,
samples, rows, SMs and bounds of memory, a launch's propagators stay below the
bound, a run of several launches has whole blocks of the chain in each, and every
launch has the columns that fill the GPU where its samples allow it.  No GPU."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include "sss_columns.h"
#include <cstdio>
using namespace sss;

static int fails = 0;
#define CHECK(c) do { if (!(c)) { std::printf("FAIL line %d: %s (ntraj %d T %d M %d sms %d)\n", __LINE__, #c, ntraj, T, M, sms); fails++; } } while (0)

int main() {
    int cut = 0, runs = 0;
    for (size_t bytes : {(size_t)1 << 22, (size_t)1 << 26, kColBytes})
        for (int sms : {16, 152})
            for (int M : {1, 4, 9, 19, 49, 52})
                for (int T : {1, 15, 16, 17, 500, 6000, 111848, 111849, 120000, 5000000, 50000000})
                    for (int ntraj : {1, 3, 1000, 70000}) {
                        const ColumnsCut c = columns_cut(ntraj, T, M, sms, bytes);
                        const int Tc = std::min(T, c.samples);
                        const long n = (long)Tc * c.traj, want = 16L * 4 * sms;
                        runs++;
                        CHECK(c.len >= 1 && c.traj >= 1 && c.traj <= std::min(ntraj, 65535) && Tc >= 1);
                        CHECK(8 * (size_t)M * M * n <= bytes);
                        // several launches per trajectory: one trajectory, whole blocks
                        if (Tc < T) {
                            cut++;
                            CHECK(c.traj == 1 && Tc % (16 * c.len) == 0);
                            CHECK(2 * (size_t)Tc * 8 * M * M > bytes);       // and more than half the bound
                        }
                        CHECK(c.runs == (long)c.traj * ((Tc + c.len - 1) / c.len));
                        // a launch with enough samples has at least half of the wanted columns
                        CHECK(n * M < want || 2 * c.runs * M >= want);
                    }
    if (cut < 50) {
        std::printf("FAIL: %d runs of several launches\n", cut);
        fails++;
    }
    std::printf("%d cuts, %d failures\n", runs, fails);
    return fails ? 1 : 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_launches_of_column_runs(tmp_path):
    src = tmp_path/"cut.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path/"cut"
    inc = os.path.join(ROOT, "superspinsim_gb300", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", inc, str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
