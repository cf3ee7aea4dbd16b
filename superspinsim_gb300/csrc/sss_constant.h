// Propagators of whole output samples over which nothing varies (host code,
// used by sss_batch.cu; no reference counterpart).
//
// In a pulse protocol most samples are free evolution or plain laser: every
// coefficient is constant from the sample's first node to its last, and the
// F fine steps of K exponentials are the same linear map.  That map depends
// only on the constant values, so a batch needs one matrix per set of values
// -- laser on and laser off, for a Ramsey batch -- and a sample of it costs
// one dense product in place of F K exponentials.  The matrices are formed in
// double-double from the same rounded exponents as the kernels' and kept as
// two doubles, minus the identity.
#pragma once
#include <algorithm>
#include <cmath>
#include <vector>

#include "sss_power.h"

namespace sss {

constexpr int kConstMax = 8;       // sets of values of a batch
constexpr int kConstMaxRows = 32;  // reachable rows (the products cost M^3 on the host)
constexpr int kConstMinExps = 16;  // exponentials per sample a dense product is worth
// Groups that share a warp stop refilling their coefficient rings together once
// one of them skips a sample, and each refill looks every node up in the
// program.  Programs of more segments than this take maps on such groups only
// where constant samples make up this share of them: 4,096 programs of 128
// segments and almost none constant, groups of 8 lanes, 320 ms with maps and 269
// without; 1,024 of 1,000 segments at 16 lanes 443 and 358; at 32 lanes (a warp
// to itself, 200 segments) 65.1 and 66.0; 7 segments, half of them constant, 16
// lanes 23.6 and 23.4.
constexpr int kConstLong = 32;
constexpr double kConstShare = 0.3;

namespace pow_detail {

using Matrix = std::vector<dd>;  // M x M row-major, a map minus the identity

// (I + A)(I + B) - I
inline Matrix compose(const Matrix& A, const Matrix& B, int M) {
    Matrix C((size_t)M * M);
    for (int r = 0; r < M; r++)
        for (int c = 0; c < M; c++) {
            dd s = dd_add(A[(size_t)r * M + c], B[(size_t)r * M + c]);
            for (int k = 0; k < M; k++) {
                const dd a = A[(size_t)r * M + k];
                if (a.hi != 0.0) s = dd_add(s, dd_mul(a, B[(size_t)k * M + c]));
            }
            C[(size_t)r * M + c] = s;
        }
    return C;
}

// e^A - I by the Taylor series on the sparse pattern
inline Matrix exponential(int M, const std::vector<int>& row_ptr, const std::vector<int>& col,
                          const std::vector<dd>& A) {
    Matrix T((size_t)M * M, dd{0.0, 0.0}), N(T), S(T);
    for (int i = 0; i < M; i++) T[(size_t)i * M + i] = {1.0, 0.0};
    for (int j = 1; j <= 60; j++) {
        double big = 0.0;
        for (int r = 0; r < M; r++) {
            dd* n = &N[(size_t)r * M];
            for (int c = 0; c < M; c++) n[c] = {0.0, 0.0};
            for (int q = row_ptr[r]; q < row_ptr[r + 1]; q++) {
                if (A[q].hi == 0.0) continue;
                const dd* t = &T[(size_t)col[q] * M];
                for (int c = 0; c < M; c++)
                    if (t[c].hi != 0.0) n[c] = dd_add(n[c], dd_mul(A[q], t[c]));
            }
            for (int c = 0; c < M; c++) {
                n[c] = dd_div(n[c], j);
                S[(size_t)r * M + c] = dd_add(S[(size_t)r * M + c], n[c]);
                big = std::max(big, std::fabs(n[c].hi));
            }
        }
        T.swap(N);
        if (big < 1e-36) break;
    }
    return S;
}

}  // namespace pow_detail

// The map of F steps, each of the exponentials of `exponents` (the last acts
// first), minus the identity: hi and lo parts, M x M row-major.  False when an
// exponent's 1-norm exceeds 1 or is not finite.
inline bool constant_sample(int M, int F, const std::vector<int>& row_ptr, const std::vector<int>& col,
                            const std::vector<std::vector<pow_detail::dd>>& exponents,
                            std::vector<double>* hi, std::vector<double>* lo) {
    using namespace pow_detail;
    const size_t MM = (size_t)M * M;
    Matrix step(MM, dd{0.0, 0.0});
    for (size_t e = 0; e < exponents.size(); e++) {
        std::vector<double> s(M, 0.0);
        for (size_t q = 0; q < col.size(); q++) s[col[q]] += std::fabs(exponents[e][q].hi);
        for (double v : s)
            if (!(v <= 1.0)) return false;
        step = compose(step, exponential(M, row_ptr, col, exponents[e]), M);
    }
    Matrix out(MM, dd{0.0, 0.0});
    bool any = false;
    for (int n = F; n; n >>= 1) {
        if (n & 1) {
            out = any ? compose(out, step, M) : step;
            any = true;
        }
        if (n > 1) step = compose(step, step, M);
    }
    hi->resize(MM);
    lo->resize(MM);
    for (size_t i = 0; i < MM; i++) {
        (*hi)[i] = out[i].hi;
        (*lo)[i] = out[i].lo;
    }
    return true;
}

// One set of values found constant together, and the time it lasts in all.
struct ConstSet {
    std::vector<double> value;   // per live channel
    double total = 0.0;
};

// The sets of values that the live channels of a batch's programs
// [b][channel][segment][5] hold together for at least dt, longest total first,
// at most kConstMax.  A run's start and end are not known here: before the
// first segment end and after the last one counts as long.  One walk over the
// channels' segments: a channel's segment lasts from the largest end before it
// to its own, if that is larger.  share: the part of the programs, from time 0
// to their last end, that whole samples inside constant stretches make up (a
// stretch holds its length less one sample of them, wherever it starts).
inline std::vector<ConstSet> constant_sets(const double* prog, int ntraj, int nch, int nseg,
                                           const std::vector<int>& live, double dt, double* share = nullptr) {
    std::vector<ConstSet> sets;
    double held = 0.0, span = 0.0;
    struct Channel {
        const double* seg;      // its segments
        int s;                  // the current one (nseg: past the last)
        double end;
    };
    std::vector<Channel> at(live.size());
    std::vector<double> v(live.size());
    auto next = [nseg](Channel& c) {
        const double from = c.end;
        do c.s++;
        while (c.s < nseg && !(c.seg[c.s * 5] > from));
        c.end = c.s < nseg ? c.seg[c.s * 5] : INFINITY;
    };
    for (int b = 0; b < ntraj; b++) {
        for (size_t i = 0; i < live.size(); i++) {
            at[i] = {prog + ((size_t)b * nch + live[i]) * nseg * 5, -1, -INFINITY};
            if (live[i] < nch)
                next(at[i]);
            else
                at[i] = {nullptr, nseg, INFINITY};
        }
        double from = -INFINITY;
        while (true) {
            double to = INFINITY;
            for (const Channel& c : at) to = std::min(to, c.end);
            const double length = std::isfinite(from) && std::isfinite(to) ? to - from : 1e3 * dt;
            bool constant = length >= dt;
            for (size_t i = 0; i < at.size() && constant; i++) {
                const double* sg = at[i].s < nseg ? at[i].seg + (size_t)at[i].s * 5 : nullptr;
                constant = !sg || (sg[2] == 0.0 && std::isfinite(sg[1]));
                v[i] = sg ? sg[1] : 0.0;
            }
            if (constant) {
                size_t k = 0;
                while (k < sets.size() && sets[k].value != v) k++;
                if (k == sets.size() && k < 64) sets.push_back({v, 0.0});
                if (k < sets.size()) sets[k].total += length;
                if (to < INFINITY) held += std::max(0.0, to - std::max(0.0, from) - dt);
            }
            if (!(to < INFINITY)) break;
            span += std::max(0.0, to - std::max(0.0, from));
            for (Channel& c : at)
                if (c.end == to) next(c);
            from = to;
        }
    }
    if (share) *share = span > 0.0 ? held / span : 0.0;
    std::stable_sort(sets.begin(), sets.end(), [](const ConstSet& a, const ConstSet& b) { return a.total > b.total; });
    if (sets.size() > (size_t)kConstMax) sets.resize(kConstMax);
    return sets;
}

}  // namespace sss
