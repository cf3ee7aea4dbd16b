"""The share of constant samples in a batch's programs (host code,
superspinsim_gb300/csrc/sss_constant.h), compiled with g++: hand-made programs.
No GPU."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r'''
#include "sss_constant.h"
#include <cstdio>
using namespace sss;

static int fails = 0;
static void check(const double* prog, int ntraj, int nch, int nseg, const std::vector<int>& live, double want) {
    double share = -1.0;
    constant_sets(prog, ntraj, nch, nseg, live, 0.5, &share);
    if (!(std::fabs(share - want) <= 1e-15)) {
        std::printf("FAIL: %g, expected %g\n", share, want);
        fails++;
    }
}

int main() {
    const double inf = INFINITY;
    // drive off to 2, on to 3, off to 5 (then off for ever): 1.5 and 1.5 of 5
    const double a[1][4][5] = {{{2, 0, 0, 0, 0}, {3, 0, 1, 1, 0}, {5, 0, 0, 0, 0}, {inf, 0, 0, 0, 0}}};
    check(&a[0][0][0], 1, 1, 4, {0}, 0.6);
    // from before time 0; a stretch shorter than dt does not count
    const double b[1][4][5] = {{{-3, 0, 0, 0, 0}, {4, 0, 0, 0, 0}, {4.25, 1, 0, 0, 0}, {5, 0, 1, 0, 0}}};
    check(&b[0][0][0], 1, 1, 4, {0}, 0.7);
    // two channels: constant only while both are
    const double c[2][2][5] = {{{4, 0, 0, 0, 0}, {8, 0, 1, 1, 0}}, {{2, 0, 1, 1, 0}, {8, 3, 0, 0, 0}}};
    check(&c[0][0][0], 1, 2, 2, {0, 1}, 1.5 / 8.0);
    check(&c[0][0][0], 1, 2, 2, {1}, 5.5 / 8.0);
    check(&c[0][0][0], 2, 1, 2, {0}, 9.0 / 16.0);   // the same as two trajectories
    // no end at all
    const double d[1][1][5] = {{{inf, 0, 1, 1, 0}}};
    check(&d[0][0][0], 1, 1, 1, {0}, 0.0);
    std::printf("%d failures\n", fails);
    return fails ? 1 : 0;
}
'''


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_share_of_constant_stretches(tmp_path):
    src = tmp_path/"share.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path/"share"
    inc = os.path.join(ROOT, "superspinsim_gb300", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", inc, str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
