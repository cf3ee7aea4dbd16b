"""The power series of an exponential and its lane programs (host code,
superspinsim_gb300/csrc/sss_power.h), compiled with g++ into a small test
program: on random sparse exponents the packed program of every lane count,
run slot by slot as the kernels run it, gives e^{A + sum a G} x - x.  The
reference is the Taylor action in long double.  Tolerance per row: the n
products and sums of a row in binary64, n 2^-53 sum |c x| (doubled for the
monomials' roundings), and the dropped entries, at most 2^-62 of every column.  No
GPU."""
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

static int fails = 0;
#define CHECK(c) do { if (!(c)) { std::printf("FAIL line %d: %s\n", __LINE__, #c); fails++; } } while (0)

static std::vector<double> monomials(const PowLayout& p, const std::vector<double>& a) {
    std::vector<double> v(p.mono.size(), 1.0);
    for (size_t i = 1; i < v.size(); i++) v[i] = v[p.p1[i]] * a[p.p2[i]];
    return v;
}

// d[row], row by row, as k_batch_power / k_batch_power_rows compute it
static std::vector<double> run(const PowSeries& ps, const PowLayout& p, int tab, const std::vector<double>& a,
                               const std::vector<double>& x) {
    const int M = ps.M, L = p.L;
    const std::vector<double> mv = monomials(p, a);
    const double* val = &ps.val[tab * ps.ent.size()];
    std::vector<double> d(M, 0.0);
    auto coef = [&](int q, int l) {
        const int e = p.entry[(size_t)q * L + l];
        return e < 0 ? 0.0 : val[e];
    };
    if (p.rows) {
        const int nm = (int)mv.size();
        std::vector<double> X(nm * M + 1, 0.0), s(L);
        for (int m = 0; m < nm; m++)
            for (int r = 0; r < M; r++) X[m * M + r] = mv[m] * x[r];
        for (int l = 0; l < L; l++) {
            s[l] = 0.0;
            for (int q = 0; q < p.E; q++) s[l] += coef(q, l) * X[p.xoff[(size_t)q * L + l]];
        }
        for (int o = 1; o < p.W; o *= 2) {
            std::vector<double> t(s);
            for (int l = 0; l < L; l++)
                if (o < (int)((p.mask[l] >> 16) & 0xff)) s[l] = t[l] + t[l ^ o];
        }
        for (int l = 0; l < L; l++) {
            const int row = p.mask[l] & 0xffff;
            if (row < M && (p.mask[l] >> 24) == 0) d[row] = s[l];
            CHECK(row < M || ((p.mask[l] >> 16) & 0xff) == 1);
        }
        return d;
    }
    std::vector<double> X(x), part(p.n_part + 1, 0.0);
    X.push_back(0.0);
    for (int l = 0; l < L; l++)
        for (int s = 0; s < p.NS; s++) {
            int pb = p.pbase[(size_t)s * L + l];
            double sum = 0.0;
            for (int q = 0; q * p.NS + s < p.E; q++) {
                if ((p.mask[(size_t)(2 * s) * L + l] >> q) & 1u) sum = 0.0;
                sum += coef(q * p.NS + s, l) * X[p.xoff[(size_t)(q * p.NS + s) * L + l]];
                if ((p.mask[(size_t)(2 * s + 1) * L + l] >> q) & 1u) part[pb++] = sum;
            }
        }
    CHECK(part[p.n_part] == 0.0);
    const int slots = p.W > 1 ? M * p.W : L;
    std::vector<double> m(slots, 0.0);
    for (int k = 0; k < slots; k++)
        for (int j = 0; j < p.RM; j++) {
            const unsigned w = p.merge[(size_t)j * slots + k];
            m[k] += mv[w >> 16] * part[w & 0xffff];
        }
    for (int r = 0; r < M; r++) {
        if (p.W > 1) {
            for (int k = 0; k < p.W; k++) d[r] += m[r * p.W + k];
        } else {
            d[r] = m[r] + (p.helper[r] >= 0 ? m[p.helper[r]] : 0.0);
        }
    }
    return d;
}

// the same for a cluster's CTAs (k_power_big): rows in the layout's order,
// the segmented sum over a row's lanes, each row on one CTA and inside a warp
static std::vector<double> run_big(const PowSeries& ps, const PowLayout& p, int tab,
                                   const std::vector<double>& a, const std::vector<double>& x) {
    const int M = ps.M, T = p.L, nm = (int)p.mono.size();
    const std::vector<double> mv = monomials(p, a);
    const double* val = &ps.val[tab * ps.ent.size()];
    std::vector<double> X(nm * M + 1, 0.0), d(M, 0.0);
    std::vector<int> seen(M, 0);
    for (int m = 0; m < nm; m++)
        for (int k = 0; k < M; k++) X[m * M + k] = mv[m] * x[p.order[k]];
    CHECK((int)p.first_row.size() == p.ctas + 1 && p.first_row.back() == M);
    for (int c = 0; c < p.ctas; c++) {
        std::vector<double> s(T);
        for (int l = 0; l < T; l++)
            for (int q = 0; q < p.E; q++) {
                const size_t at = ((size_t)c * p.E + q) * T + l;
                s[l] += (p.entry[at] < 0 ? 0.0 : val[p.entry[at]]) * X[p.xoff[at]];
            }
        auto word = [&](int l) { return p.mask[(size_t)c * T + l]; };
        for (int o = 1; o < p.W; o <<= 1) {
            const std::vector<double> t(s);
            for (int l = 0; l < T; l++) {
                const int W = (word(l) >> 16) & 0xff, sub = word(l) >> 24;
                if ((sub & (2 * o - 1)) == 0 && sub + o < W) s[l] = t[l] + t[l + o];
            }
        }
        for (int l = 0; l < T; l++) {
            const int row = word(l) & 0xffff, W = (word(l) >> 16) & 0xff, sub = word(l) >> 24;
            if (row == M) continue;
            CHECK(row >= p.first_row[c] && row < p.first_row[c + 1] && l % 32 - sub + W <= 32);
            if (sub) continue;
            d[p.order[row]] = s[l];
            seen[row]++;
        }
    }
    for (int n : seen) CHECK(n == 1);
    return d;
}

int main() {
    std::mt19937_64 rng(7);
    std::uniform_real_distribution<double> u(-1.0, 1.0);
    int packed = 0, clusters = 0;
    for (int M : {1, 2, 3, 8, 9, 16, 17, 19, 32, 33, 64, 65, 130})
        for (int n_live : {0, 1, 2})
            for (int n_tab : {1, 3}) {
                if (M > 64 && (n_live > 1 || n_tab > 1)) continue;
                std::vector<int> rp(1, 0), col;
                for (int r = 0; r < M; r++) {
                    for (int c = 0; c < M; c++)
                        if (c == r || u(rng) > (M > 64 ? 0.98 : M > 8 ? 0.8 : 0.0)) col.push_back(c);
                    rp.push_back((int)col.size());
                }
                const size_t nnz = col.size();
                std::vector<std::vector<double>> Ah(n_tab, std::vector<double>(nnz)), Al(Ah), G(n_live);
                for (int t = 0; t < n_tab; t++)
                    for (size_t q = 0; q < nnz; q++) {
                        Ah[t][q] = 0.05 * u(rng) / (1 + t);
                        Al[t][q] = Ah[t][q] * 1e-17 * u(rng);
                    }
                std::vector<double> rho(n_live), a(n_live);
                for (int g = 0; g < n_live; g++) {
                    rho[g] = 0.75;
                    a[g] = 0.75 * u(rng);
                    for (size_t q = 0; q < nnz; q++) G[g].push_back(u(rng) > 0.5 ? 1e-4 * u(rng) : 0.0);
                }
                PowSeries ps;
                CHECK(power_series(M, rp, col, Ah, Al, G, rho, &ps));
                std::vector<double> x(M);
                double xs = 0.0;
                for (double& v : x) {
                    v = u(rng);
                    xs += std::fabs(v);
                }
                for (int tab = 0; tab < n_tab; tab++) {
                    std::vector<long double> T(x.begin(), x.end()), ref(M, 0.0L);
                    for (int j = 1; j < 60; j++) {
                        std::vector<long double> n(M, 0.0L);
                        for (int r = 0; r < M; r++)
                            for (int q = rp[r]; q < rp[r + 1]; q++) {
                                long double o = (long double)Ah[tab][q] + Al[tab][q];
                                for (int g = 0; g < n_live; g++) o += (long double)a[g] * G[g][q];
                                n[r] += o * T[col[q]] / j;
                            }
                        for (int r = 0; r < M; r++) ref[r] += n[r];
                        T = n;
                    }
                    std::vector<double> mag(M, 0.0);
                    std::vector<int> n_ent(M, 0);
                    for (size_t k = 0; k < ps.ent.size(); k++) {
                        double m = 1.0;
                        for (int g = 0; g < n_live; g++) m *= std::pow(std::fabs(a[g]), ps.mono[ps.ent[k].mono][g]);
                        mag[ps.ent[k].row] += std::fabs(ps.val[tab * ps.ent.size() + k]) * m * std::fabs(x[ps.ent[k].col]);
                        n_ent[ps.ent[k].row]++;
                    }
                    // lane counts, and clusters of 1 to 8 CTAs for the large systems
                    for (int L : {16, 32, 64, 128, -1, -2, -4, -8}) {
                        PowLayout p;
                        if (L < 0) {
                            if (M <= 64) continue;
                            if (!power_pack_big(ps, -L, power_big_threads(-L), &p)) continue;
                            clusters |= -L;
                        } else if (!power_pack(ps, L, &p)) {
                            continue;
                        }
                        packed++;
                        CHECK(L < 0 || (p.L <= L && (L <= 32 ? p.L == L : p.L % 32 == 0 && p.L >= 64)));
                        const std::vector<double> d = L < 0 ? run_big(ps, p, tab, a, x) : run(ps, p, tab, a, x);
                        for (int r = 0; r < M; r++) {
                            const double tol = 2.0 * (n_ent[r] + 8) * std::ldexp(mag[r], -53) + std::ldexp(xs, -61);
                            if (!(std::fabs((double)(d[r] - ref[r])) <= tol)) {
                                std::printf("FAIL M %d live %d L %d row %d: %g against %g\n", M, n_live, L, r,
                                            std::fabs((double)(d[r] - ref[r])), tol);
                                fails++;
                            }
                        }
                    }
                }
            }
    CHECK(packed > 100 && clusters == 15);
    // too large an exponent is refused
    PowSeries ps;
    CHECK(!power_series(1, {0, 1}, {0}, {{1.5}}, {{0.0}}, {}, {}, &ps));
    CHECK(!power_series(1, {0, 1}, {0}, {{0.1}}, {{0.0}}, {{0.5}}, {1.0}, &ps));
    CHECK(!power_series(1, {0, 1}, {0}, {{NAN}}, {{0.0}}, {}, {}, &ps));
    std::printf("%d layouts, %d failures\n", packed, fails);
    return fails ? 1 : 0;
}
'''


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_power_series_programs(tmp_path):
    src = tmp_path/"power.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path/"power"
    inc = os.path.join(ROOT, "superspinsim_gb300", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", inc, str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
