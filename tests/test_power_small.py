"""The total degree of the power series of small exponents (host code,
superspinsim_gb300/csrc/sss_power.h), compiled with g++: over constant parts of
norm 1e-4 to 0.1 and drives of 1e-7 to 1e-2, the first degree left out is below
what may be dropped at these norms, min(2^-62, 2^-56 n^(3/2)) of the state, and
the last one kept is not.  In one dimension the terms are known: e^x b^k / k!.
No GPU."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r'''
#include "sss_power.h"
#include <cstdio>
using namespace sss;

int main() {
    int fails = 0, runs = 0;
    for (double x : {1e-4, 1e-3, 1e-2, 0.1})
        for (double b = 1e-7; b < 1e-2; b *= 1.15) {
            PowSeries ps;
            if (!power_series(1, {0, 1}, {0}, {{-x}}, {{0.0}}, {{b}}, {1.0}, &ps)) {
                std::printf("FAIL refused: x %g b %g\n", x, b);
                fails++;
                continue;
            }
            const double drop = std::min(0x1p-62, 0x1p-56 * std::pow(x + b, 1.5));
            int degree = 0;
            for (const auto& m : ps.mono) degree = std::max(degree, m[0]);
            double term = std::exp(x);
            for (int k = 1; k <= degree; k++) term *= b / k;
            runs++;
            if (term <= drop || !(term * b / (degree + 1) <= drop)) {
                std::printf("FAIL x %g b %g degree %d: term %g, next %g, drop %g\n", x, b, degree, term,
                            term * b / (degree + 1), drop);
                fails++;
            }
        }
    std::printf("%d series, %d failures\n", runs, fails);
    return fails ? 1 : 0;
}
'''


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_degree_of_small_exponents(tmp_path):
    src = tmp_path/"small.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path/"small"
    inc = os.path.join(ROOT, "superspinsim_gb300", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", inc, str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
