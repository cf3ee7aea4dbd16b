// Power-series form of the exponentials of a batch (host code, used by
// sss_batch.cu; no reference counterpart).
//
// With the generators whose coefficients are constant over the batch summed
// in A and the varying ones written a_g G_g, an exponential is
//     e^{A + sum_g a_g G_g} = sum_alpha a^alpha C_alpha,
// a power series in the few varying coefficients whose matrices C_alpha are
// the same for every trajectory and every step.  The drives are weak per
// step (|a| ||G|| is 1e-4 to 1e-3 for the NV workloads), so the total degree
// that reaches the unit roundoff is 3 to 6 and the matrices hold a few
// hundred entries: one multiplication by a constant sparse matrix on
// a^alpha-scaled copies of the state takes the place of the d dependent
// Horner terms of the Taylor action (7-level NV at 5 ps: 530 multiply-adds
// against 8 x 106, and one exchange between lanes against 16).
//
// power_series() computes C_alpha - [alpha = 0] I from the Taylor series on
// the sparse pattern.  The alpha = 0 part -- the only one above 1e-3 -- is
// summed in double-double and its entries keep their low parts as further
// entries, because an entry's rounding is the same at every step: 2^-58 at
// an entry of 0.05 would be a drift of 3e-12 over 800,000 exponentials.
// Entries are dropped, smallest first, while the dropped sum of every
// column stays below a bound (kPowDrop), and degrees are left out once all of
// the next one is below it.
//
// power_pack() deals the entries to the lanes of a group.
#pragma once
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <functional>
#include <numeric>
#include <system_error>
#include <thread>
#include <utility>
#include <vector>

namespace sss {

constexpr int kPowMaxLive = 2;     // varying coefficients in the series
constexpr int kPowMaxDegree = 9;   // total degree
constexpr int kPowMaxMono = 28;    // monomial values per exponential (kernel ring; degree 6 of two)
// Entries and low parts below 2^-62 of the state are dropped: the 16,000
// exponentials of the 1024-frequency sweep keep the Taylor action's error of
// 3e-15 (2^-58 drops 10 % more and drifts to 1.2e-13).  A propagator column is
// kept minus its unit vector, so an exponent of norm x rounds it by 2^-53 x
// only; over the 1/x exponentials that change it by its own size those
// roundings add up to 2^-53 x^(1/2), a drop d to d/x: below x^(3/2) 2^-56 the
// drop stays the smaller one.
constexpr double kPowDrop = 0x1p-62, kPowDropSmall = 0x1p-56;
constexpr int kPowMaxTables = 8;   // coefficient tables of a batch
constexpr int kPowMaxRows = 64;    // reachable rows (the series fills in towards M^2)
// FMA slots per lane and merge slots per row with a compiled kernel: groups of
// 16 and of 32 lanes, and FMA slots of the row-aligned kernel (64 to 128)
constexpr int kPowSlots[2][16] = {{8, 10, 12, 14, 16, 20, 24},
                                   {2, 3, 4, 6, 8, 10, 12, 14, 16, 17, 18, 19, 20, 22, 24, 28}};
constexpr int kPowMerges[2][6] = {{3, 4, 5, 6, 8}, {3, 4, 5, 6, 7, 8}};
constexpr int kPowRowSlots[] = {1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 12, 14, 16, 20};
template <int N>
inline int pow_pick(const int (&table)[N], int want) {
    for (int s : table)
        if (s >= want) return s;
    return 0;
}
// Fine steps of coefficients per ring refill of the row-aligned kernel: enough
// to give all 128 lanes a node to sample, so that the cosine's latency, which
// the whole group waits for, is paid every 64 steps (28.4 against 27.1 ms on
// the spin-1 sweep of 64 with 16 steps).
constexpr int kPowRowsRing = 64;
constexpr int kPowRing = 16;       // and of the other kernels (kRing)
constexpr int kPowRowLanes = 16;   // lanes of a row, at most

struct PowEntry {
    int row, col, mono;   // output row, state column, monomial index
};

struct PowSeries {
    int M = 0, n_live = 0, n_tables = 0;
    std::vector<std::vector<int>> mono;   // exponents of the varying coefficients; [0] = all zero
    std::vector<PowEntry> ent;
    std::vector<double> val;              // [table * ent.size() + i]
};

namespace pow_detail {
struct dd {
    double hi, lo;
};
inline dd two_sum(double a, double b) {
    const double s = a + b, z = s - a;
    return {s, (a - (s - z)) + (b - z)};
}
inline dd dd_mul(dd a, dd b) {
    const double p = a.hi * b.hi;
    const double e = std::fma(a.hi, b.hi, -p) + (a.hi * b.lo + a.lo * b.hi);
    const double s = p + e;
    return {s, e - (s - p)};
}
inline dd dd_add(dd a, dd b) {
    const dd s = two_sum(a.hi, b.hi);
    const double e = s.lo + (a.lo + b.lo);
    const double h = s.hi + e;
    return {h, e - (h - s.hi)};
}
inline dd dd_div(dd a, double j) {
    const double q = a.hi / j;
    const double r = std::fma(-q, j, a.hi) + a.lo;
    return two_sum(q, r / j);
}

// The matrices of a power series, column by column: [column][table][monomial][row].
struct Columns {
    int M = 0, n_live = 0, nm = 0, n_tab = 0;
    double drop = 0.0;
    const std::vector<std::vector<int>>* lower = nullptr;   // monomial less one factor, or -1
    std::vector<double> size;                               // largest value of each monomial
    // a matrix by columns, without its zeros
    struct Sparse {
        std::vector<int> ptr, row;
        std::vector<dd> val;
        Sparse(int M, const std::vector<int>& row_ptr, const std::vector<int>& col, const std::vector<double>& hi,
               const std::vector<double>* lo)
            : ptr(M + 1, 0) {
            for (size_t q = 0; q < col.size(); q++) ptr[col[q] + 1] += hi[q] != 0.0;
            std::partial_sum(ptr.begin(), ptr.end(), ptr.begin());
            row.resize(ptr.back());
            val.resize(ptr.back());
            std::vector<int> at(ptr.begin(), ptr.end() - 1);
            for (int r = 0; r < M; r++)
                for (int q = row_ptr[r]; q < row_ptr[r + 1]; q++)
                    if (hi[q] != 0.0) {
                        row[at[col[q]]] = r;
                        val[at[col[q]]++] = {hi[q], lo ? (*lo)[q] : 0.0};
                    }
        }
        void add(const double* x, double* y) const {
            for (int k = 0; k + 1 < (int)ptr.size(); k++)
                if (x[k] != 0.0)
                    for (int q = ptr[k]; q < ptr[k + 1]; q++) y[row[q]] += val[q].hi * x[k];
        }
    };
    std::vector<Sparse> A, G;                               // constant part of each table, varying generators
    std::vector<double> C, lo;
    std::vector<char> keep;

    // what one thread needs, allocated before it starts
    struct Scratch {
        std::vector<dd> D, Dn, Cd;
        std::vector<double> T, N;                           // [monomial][row]
        std::vector<char> alive, next;                      // monomials with terms left
        std::vector<std::pair<double, int>> sorted;
        Scratch(int M, int nm)
            : D(M), Dn(M), Cd(M), T((size_t)nm * M), N((size_t)nm * M), alive(nm), next(nm), sorted((size_t)nm * M) {}
    };

    // Taylor terms T_j of column c, all monomials at once.  The constant part
    // is in double-double until a term's rounding no longer shows in the low
    // parts (2^-53 of it below 2^-7 of what is dropped).
    void run(int c, Scratch& s) {
        for (int tab = 0; tab < n_tab; tab++) {
            double* Cc = &C[((size_t)c * n_tab + tab) * nm * M];
            const Sparse& a = A[tab];
            std::fill(s.D.begin(), s.D.end(), dd{0.0, 0.0});
            std::fill(s.Cd.begin(), s.Cd.end(), dd{0.0, 0.0});
            std::fill(s.T.begin(), s.T.end(), 0.0);
            s.D[c] = {1.0, 0.0};
            s.T[c] = 1.0;
            std::fill(s.alive.begin(), s.alive.end(), 0);
            s.alive[0] = s.next[0] = 1;
            bool exact = true;
            for (int j = 1; j <= 60; j++) {
                double big = 0.0;
                std::fill(s.N.begin(), s.N.end(), 0.0);
                if (exact) {
                    std::fill(s.Dn.begin(), s.Dn.end(), dd{0.0, 0.0});
                    for (int k = 0; k < M; k++) {
                        if (s.D[k].hi == 0.0) continue;
                        for (int q = a.ptr[k]; q < a.ptr[k + 1]; q++)
                            s.Dn[a.row[q]] = dd_add(s.Dn[a.row[q]], dd_mul(a.val[q], s.D[k]));
                    }
                    for (int r = 0; r < M; r++) {
                        if (s.Dn[r].hi == 0.0) continue;
                        s.Dn[r] = dd_div(s.Dn[r], j);
                        s.Cd[r] = dd_add(s.Cd[r], s.Dn[r]);
                        s.N[r] = s.Dn[r].hi;
                        big = std::max(big, std::fabs(s.Dn[r].hi));
                    }
                    s.D.swap(s.Dn);
                    exact = std::ldexp(big, -53) > std::ldexp(drop, -7);
                } else {
                    a.add(s.T.data(), s.N.data());
                    for (int r = 0; r < M; r++) {
                        s.N[r] /= j;
                        s.Cd[r] = dd_add(s.Cd[r], {s.N[r], 0.0});
                        big = std::max(big, std::fabs(s.N[r]));
                    }
                }
                for (int m = 1; m < nm; m++) {
                    double* n = &s.N[(size_t)m * M];
                    double most = 0.0;
                    if (s.alive[m]) a.add(&s.T[(size_t)m * M], n);
                    bool fed = s.alive[m];
                    for (int g = 0; g < n_live; g++)
                        if ((*lower)[m][g] >= 0 && s.alive[(*lower)[m][g]]) {
                            G[g].add(&s.T[(size_t)(*lower)[m][g] * M], n);
                            fed = true;
                        }
                    s.next[m] = 0;
                    if (!fed) continue;
                    double* cm = Cc + (size_t)m * M;
                    for (int r = 0; r < M; r++) {
                        n[r] /= j;
                        cm[r] += n[r];
                        most = std::max(most, std::fabs(n[r]));
                    }
                    // a monomial whose terms no longer show, at its largest value,
                    // feeds nothing any more
                    most *= size[m];
                    s.next[m] = most >= std::ldexp(drop, -10);
                    big = std::max(big, most);
                }
                s.T.swap(s.N);
                s.alive.swap(s.next);
                if (big < std::ldexp(drop, -10)) break;
            }
            for (int r = 0; r < M; r++) {
                Cc[r] = s.Cd[r].hi;
                lo[((size_t)c * n_tab + tab) * M + r] = s.Cd[r].lo;
            }
        }
        // all but the smallest entries (by their largest value over the tables)
        // whose sum stays below the bound
        int n = 0;
        for (int m = 0; m < nm; m++)
            for (int r = 0; r < M; r++) {
                double v = 0.0;
                for (int tab = 0; tab < n_tab; tab++)
                    v = std::max(v, std::fabs(C[(((size_t)c * n_tab + tab) * nm + m) * M + r]));
                v *= size[m];
                if (v > 0.0) s.sorted[n++] = {v, m * M + r};
            }
        std::sort(s.sorted.begin(), s.sorted.begin() + n);
        double sum = 0.0;
        for (int i = 0; i < n; i++) {
            sum += s.sorted[i].first;
            if (sum > drop) keep[(size_t)c * nm * M + s.sorted[i].second] = 1;
        }
    }
};

// All columns, on as many threads as `work` (multiply-adds of a Taylor term) is
// worth; a thread that cannot be started leaves its share to the others.
inline void run_columns(Columns& w, double work) {
    int want = (int)std::min({16.0, work / 1e5, (double)w.M});
    if (want > 1) want = std::min(want, (int)std::thread::hardware_concurrency());   // (a system call)
    std::vector<Columns::Scratch> scratch(std::max(1, want), Columns::Scratch(w.M, w.nm));
    std::atomic<int> next{0};
    auto body = [&](Columns::Scratch& s) {
        for (int c = next++; c < w.M; c = next++) w.run(c, s);
    };
    std::vector<std::thread> helpers;
    helpers.reserve(scratch.size());
    try {
        for (size_t i = 1; i < scratch.size(); i++) helpers.emplace_back(body, std::ref(scratch[i]));
    } catch (const std::system_error&) {
    }
    body(scratch[0]);
    for (std::thread& t : helpers) t.join();
}
}  // namespace pow_detail

// The power series on a square pattern of M rows (CSR row_ptr/col).
//   A: n_tables double-double matrices on the pattern (hi then lo, each nnz
//      values) -- the constant part of the exponent of each table;
//   G: the varying generators' values on the pattern (n_live x nnz), scaled
//      by a power of two so that |a_g| <= rho[g] <= 1.
// False when the exponent is too large for the series to pay (1-norm of A
// above 1, or a total degree above kPowMaxDegree).
inline bool power_series(int M, const std::vector<int>& row_ptr, const std::vector<int>& col,
                         const std::vector<std::vector<double>>& A_hi,
                         const std::vector<std::vector<double>>& A_lo,
                         const std::vector<std::vector<double>>& G, const std::vector<double>& rho,
                         PowSeries* out) {
    using namespace pow_detail;
    const int nnz = (int)col.size(), n_live = (int)G.size(), n_tab = (int)A_hi.size();
    if (n_live > kPowMaxLive || n_tab > kPowMaxTables || n_tab < 1) return false;
    auto norm1 = [&](const std::vector<double>& v) {
        std::vector<double> s(M, 0.0);
        double m = 0.0;
        for (int q = 0; q < nnz; q++) {
            s[col[q]] += std::fabs(v[q]);
            if (!(s[col[q]] <= m)) m = s[col[q]];   // a NaN sticks
            if (m != m) break;
        }
        return m;
    };
    double x = 0.0, b = 0.0;
    for (const auto& a : A_hi) {
        const double n = norm1(a);
        if (!(n <= 1.0)) return false;
        x = std::max(x, n);
    }
    for (int g = 0; g < n_live; g++) b += rho[g] * norm1(G[g]);
    if (!(b <= 0.25)) return false;
    // the terms left out are below what may be dropped, as the entries are: they
    // are missing at every exponential too
    const double drop = std::min(kPowDrop, kPowDropSmall * std::pow(x + b, 1.5));
    int deg = 0;
    for (double t = b * std::exp(x); n_live && t > drop; deg++) t *= b / (deg + 2);
    if (deg > kPowMaxDegree) return false;
    // monomials by total degree
    PowSeries& ps = *out;
    ps.M = M;
    ps.n_live = n_live;
    ps.n_tables = n_tab;
    ps.mono.clear();
    for (int t = 0; t <= deg; t++) {
        if (n_live == 2)
            for (int i = t; i >= 0; i--) ps.mono.push_back({i, t - i});
        else if (n_live == 1)
            ps.mono.push_back({t});
        else
            ps.mono.push_back({});
    }
    const int nm = (int)ps.mono.size();
    std::vector<std::vector<int>> lower(nm, std::vector<int>(n_live, -1));
    for (int m = 0; m < nm; m++)
        for (int g = 0; g < n_live; g++) {
            if (!ps.mono[m][g]) continue;
            std::vector<int> al = ps.mono[m];
            al[g]--;
            lower[m][g] = (int)(std::find(ps.mono.begin(), ps.mono.end(), al) - ps.mono.begin());
        }
    // the columns of all matrices are independent: dealt to a few threads where
    // there is work for them
    pow_detail::Columns w;
    w.M = M;
    w.n_live = n_live;
    w.nm = nm;
    w.n_tab = n_tab;
    w.drop = drop;
    w.lower = &lower;
    for (int tab = 0; tab < n_tab; tab++) w.A.emplace_back(M, row_ptr, col, A_hi[tab], &A_lo[tab]);
    for (int g = 0; g < n_live; g++) w.G.emplace_back(M, row_ptr, col, G[g], nullptr);
    w.size.assign(nm, 1.0);
    for (int m = 0; m < nm; m++)
        for (int g = 0; g < n_live; g++) w.size[m] *= std::pow(rho[g], ps.mono[m][g]);
    w.C.assign((size_t)M * n_tab * nm * M, 0.0);
    w.lo.assign((size_t)M * n_tab * M, 0.0);
    w.keep.assign((size_t)M * nm * M, 0);
    pow_detail::run_columns(w, (double)M * nnz * nm * n_tab);
    // entries by row, then monomial, then column; a low part before its entry
    std::vector<size_t> at((size_t)M * nm + 1, 0);
    auto keeps_low = [&](int c, int r) {
        double v = 0.0;
        for (int tab = 0; tab < n_tab; tab++) v = std::max(v, std::fabs(w.lo[((size_t)c * n_tab + tab) * M + r]));
        return v > drop;
    };
    for (int c = 0; c < M; c++)
        for (int m = 0; m < nm; m++)
            for (int r = 0; r < M; r++)
                at[(size_t)r * nm + m + 1] += w.keep[((size_t)c * nm + m) * M + r] + (m == 0 && keeps_low(c, r));
    std::partial_sum(at.begin(), at.end(), at.begin());
    const size_t ne = at.back();
    ps.ent.resize(ne);
    ps.val.resize(ne * n_tab);
    for (int c = 0; c < M; c++)
        for (int m = 0; m < nm; m++)
            for (int r = 0; r < M; r++) {
                size_t& k = at[(size_t)r * nm + m];
                if (m == 0 && keeps_low(c, r)) {
                    ps.ent[k] = {r, c, 0};
                    for (int tab = 0; tab < n_tab; tab++) ps.val[tab * ne + k] = w.lo[((size_t)c * n_tab + tab) * M + r];
                    k++;
                }
                if (w.keep[((size_t)c * nm + m) * M + r]) {
                    ps.ent[k] = {r, c, m};
                    for (int tab = 0; tab < n_tab; tab++)
                        ps.val[tab * ne + k] = w.C[(((size_t)c * n_tab + tab) * nm + m) * M + r];
                    k++;
                }
            }
    return true;
}

// A group's program.
//
// 16 or 32 lanes (k_batch_power): L lanes of E slots, run as NS interleaved
// sequences (two from 12 slots on, of ceil(E/2) and floor(E/2): two
// independent FMA chains; slot q of sequence s is slot q NS + s of the lane).
// The entries of a row that share a monomial form a list; the lists are laid
// end to end over the sequences and cut where a sequence ends, so no slot is
// padding until the last ones.  Every piece of a list is a partial sum; the
// merge adds a row's partial sums, each times its monomial, and the sum to
// the state.  A group of twice its rows or more merges each row on W
// neighbouring lanes (partial sum j on lane j mod W), summed by shuffles.  In
// a narrower group lane k merges row k and the lanes past the last row help
// the rows with the most partial sums, which add the helper's sum (one
// shuffle): at 32 lanes the 19 rows of the 7-level NV have up to 10 partial
// sums and 13 lanes to spare (31 -> 28 FP64 instructions per exponential,
// 32.7 -> 30.0 ms on the sweep of 1024).
//
// 64 to 128 lanes (k_batch_power_rows): a row has W_r neighbouring lanes, a
// power of two with W_r E >= its entries, dealt round-robin; the entries read
// copies of the state scaled by each monomial, which the row's lanes write.
struct PowLayout {
    int L = 0, E = 0, NS = 1, RM = 0, W = 1;
    bool rows = false;
    int ctas = 0;                           // CTAs of a cluster (power_pack_big), 0: not one
    std::vector<int> order, first_row;      // its rows in the layout's order, each CTA's together
    int copies = 1;                         // row-aligned: copies written per lane
    std::vector<std::vector<int>> mono;     // ring values: exponents of each monomial, by degree
    int p1[kPowMaxMono] = {}, p2[kPowMaxMono] = {};   // value i = value p1 * coefficient p2
    int n_part = 0;
    std::vector<int> entry;                 // [E][L] entry of each slot (-1: padding)
    std::vector<int> xoff;                  // [E][L] column (M: the zero word); row-aligned:
                                            // monomial * M + column (monomials * M: the zero word)
    std::vector<unsigned> mask;             // [NS][2][L] piece starts, piece ends; row-aligned: [L]
                                            // row | W_r << 16 | place among the row's lanes << 24
    std::vector<int> pbase;                 // [NS][L] first partial sum of each sequence
    std::vector<unsigned> merge;            // [RM][slots] partial sum | ring value << 16 (n_part: zero)
    std::vector<int> helper;                // [L] lane that helps this row's merge, or -1
    int log_w() const {
        int lg = 0;
        while ((1 << lg) < W) lg++;
        return lg;
    }
    // FP64 instructions of one exponential
    int cost() const { return ctas ? E + log_w() + 2 : rows ? E + log_w() + 1 + copies : E + RM + std::max(log_w(), 1) + 1; }
    // Cycles of one exponential of a group alone on its SM sub-partitions
    // (fitted to the spin-1 sweep of 64, one group per SM: 32 lanes, 15
    // instructions, 1,980 cycles; row-aligned at 96 lanes, 3 slots and 4
    // shuffles, 1,285; 64 lanes, 6 slots, 3 shuffles and 2 copies, 2,150)
    int chain_cycles() const {
        return rows ? 450 + 100 * E + 138 * log_w() + 500 * (copies - 1) : 300 + 110 * cost();
    }
};

inline int pow_sequences(int E) { return E >= 12 ? 2 : 1; }

// fine steps of the coefficient ring of a cluster of `ctas`
inline int pow_big_ring(int ctas) { return ctas == 1 ? kPowRing : kPowRowsRing; }

// Dynamic shared memory of one CTA of a layout on M rows: `groups` groups of
// state (or copies), partial sums and ring, for K exponentials of Q nodes on
// n_chan channels; and a cluster's coefficients and operand offsets.  Every
// layout is checked against kPowSmem when it is chosen, so that one that does
// not fit gives way to another.
constexpr size_t kPowSmem = 226 * 1024;   // 227 KB less the kernels' static arrays
inline size_t power_smem(const PowLayout& Ly, int M, int K, int Q, int n_chan, int groups) {
    const size_t nm = Ly.mono.size(), copies = 2 * (nm * M + 1);
    if (Ly.ctas)
        return sizeof(double) * (copies + (size_t)pow_big_ring(Ly.ctas) * (Q * n_chan + K * nm) + nm) +
               (sizeof(double) + sizeof(unsigned short)) * (size_t)Ly.E * Ly.L;
    const size_t ring = (size_t)(Ly.rows ? kPowRowsRing : kPowRing);
    const size_t per_group = ((Ly.rows ? copies : (size_t)(M + 1 + Ly.n_part + 1)) +
                              ring * (Q * n_chan + K * nm) + nm + ring * K / 2) | 1;
    return sizeof(double) * groups * per_group;
}

// The monomials in use and their factors, by degree; at_mono: the value of
// each of the series' monomials.  False when the ring cannot hold them.
inline bool pow_monomials(const PowSeries& ps, PowLayout& Ly, std::vector<int>* at_mono) {
    auto degree = [](const std::vector<int>& a) { return std::accumulate(a.begin(), a.end(), 0); };
    auto less_one = [](std::vector<int> a, int* v) {
        *v = 0;
        while (!a[*v]) ++*v;
        a[*v]--;
        return a;
    };
    std::vector<std::vector<int>>& val = Ly.mono;
    val.assign(1, std::vector<int>(ps.n_live, 0));
    for (const PowEntry& e : ps.ent)
        if (std::find(val.begin(), val.end(), ps.mono[e.mono]) == val.end()) val.push_back(ps.mono[e.mono]);
    for (size_t i = 1; i < val.size(); i++) {
        int v;
        const std::vector<int> a = less_one(val[i], &v);
        if (std::find(val.begin(), val.end(), a) == val.end()) val.push_back(a);
    }
    std::stable_sort(val.begin(), val.end(), [&](const std::vector<int>& x, const std::vector<int>& y) {
        return degree(x) < degree(y);
    });
    if ((int)val.size() > kPowMaxMono) return false;
    for (size_t i = 1; i < val.size(); i++) {
        const std::vector<int> a = less_one(val[i], &Ly.p2[i]);
        Ly.p1[i] = (int)(std::find(val.begin(), val.end(), a) - val.begin());
    }
    at_mono->assign(ps.mono.size(), 0);
    for (size_t m = 0; m < ps.mono.size(); m++)
        (*at_mono)[m] = (int)(std::find(val.begin(), val.end(), ps.mono[m]) - val.begin());
    return true;
}

// The row-aligned program at up to L lanes (a multiple of 32 above L/2).
inline bool power_pack_rows(const PowSeries& ps, int L, PowLayout* out) {
    const int M = ps.M, ne = (int)ps.ent.size();
    PowLayout best;
    std::vector<int> at_mono;
    if (!pow_monomials(ps, best, &at_mono)) return false;
    const int nm = (int)best.mono.size();
    if (nm * M > 8000) return false;
    std::vector<std::vector<int>> rows(M);
    for (int i = 0; i < ne; i++) rows[ps.ent[i].row].push_back(i);
    std::vector<int> w_best;
    int cost_best = 0;
    for (int E : kPowRowSlots) {
        std::vector<int> w(M, 1);
        int sum = 0, wmax = 1, copies = 1;
        for (int r = 0; r < M; r++) {
            while (w[r] * E < (int)rows[r].size() && w[r] <= kPowRowLanes) w[r] *= 2;
            sum += w[r];
            wmax = std::max(wmax, w[r]);
            copies = std::max(copies, (nm + w[r] - 1) / w[r]);
        }
        if (sum > L || wmax > kPowRowLanes) continue;
        PowLayout t = best;
        t.rows = true;
        t.E = E;
        t.W = wmax;
        t.copies = copies;
        t.L = std::max((sum + 31) / 32 * 32, L / 2 + 32);
        if (w_best.empty() || t.chain_cycles() < cost_best) {
            best = t;
            w_best = w;
            cost_best = t.chain_cycles();
        }
    }
    if (w_best.empty()) return false;
    const int Lb = best.L;
    best.entry.assign((size_t)best.E * Lb, -1);
    best.xoff.assign((size_t)best.E * Lb, nm * M);
    best.mask.assign(Lb, (unsigned)M | (1u << 16));
    std::vector<int> ord(M);   // widest rows first: every row's lanes are aligned
    std::iota(ord.begin(), ord.end(), 0);
    std::stable_sort(ord.begin(), ord.end(), [&](int x, int y) { return w_best[x] > w_best[y]; });
    int lane = 0;
    for (int r : ord) {
        const int w = w_best[r];
        for (int k = 0; k < w; k++) best.mask[lane + k] = (unsigned)r | ((unsigned)w << 16) | ((unsigned)k << 24);
        for (int i = 0; i < (int)rows[r].size(); i++) {
            const size_t slot = (size_t)(i / w) * Lb + lane + i % w;
            const PowEntry& e = ps.ent[rows[r][i]];
            best.entry[slot] = rows[r][i];
            best.xoff[slot] = at_mono[e.mono] * M + e.col;
        }
        lane += w;
    }
    *out = best;
    return true;
}

// The program of a series at L lanes (64 and 128: up to as many); false when
// no compiled kernel holds it.
inline bool power_pack(const PowSeries& ps, int L, PowLayout* out) {
    if (L > 32) return L <= 128 && power_pack_rows(ps, L, out);
    const int M = ps.M, ne = (int)ps.ent.size();
    if (M > L || (L != 16 && L != 32)) return false;
    PowLayout Ly;
    Ly.L = L;
    while (Ly.W < 8 && 2 * Ly.W * M <= L) Ly.W *= 2;
    Ly.E = pow_pick(kPowSlots[L == 32], std::max(1, (ne + L - 1) / L));
    if (!Ly.E) return false;
    std::vector<int> at_mono;
    if (!pow_monomials(ps, Ly, &at_mono)) return false;
    // lists: entries by row, then monomial (ps.ent is in that order already)
    Ly.NS = pow_sequences(Ly.E);
    const int seqs = L * Ly.NS;
    auto length = [&](int sq) { return (Ly.E + Ly.NS - 1 - sq % Ly.NS) / Ly.NS; };
    Ly.entry.assign((size_t)Ly.E * L, -1);
    Ly.xoff.assign((size_t)Ly.E * L, M);
    Ly.mask.assign((size_t)Ly.NS * 2 * L, 0u);
    Ly.pbase.assign((size_t)Ly.NS * L, 0);
    std::vector<std::vector<unsigned>> merge(M);
    // entries are spread evenly over the sequences' slots, so the padding is
    // too
    int at = 0, before = 0;
    for (int sq = 0; sq < seqs; sq++) {
        const int l = sq / Ly.NS, s = sq % Ly.NS;
        const int S = length(sq);
        before += S;
        const int end = (int)((long)ne * before / ((long)L * Ly.E));
        Ly.pbase[(size_t)s * L + l] = Ly.n_part;
        int q = 0, prow = -1, pm = -1;
        for (; at < end; at++, q++) {
            const PowEntry& e = ps.ent[at];
            const size_t slot = (size_t)(q * Ly.NS + s) * L + l;
            if (e.row != prow || e.mono != pm) {
                if (prow >= 0) Ly.mask[(size_t)(2 * s + 1) * L + l] |= 1u << (q - 1);
                Ly.mask[(size_t)(2 * s) * L + l] |= 1u << q;
                prow = e.row;
                pm = e.mono;
                merge[prow].push_back((unsigned)Ly.n_part++ | ((unsigned)at_mono[pm] << 16));
            }
            Ly.entry[slot] = at;
            Ly.xoff[slot] = e.col;
        }
        if (prow >= 0) Ly.mask[(size_t)(2 * s + 1) * L + l] |= 1u << (S - 1);
    }
    const int W = Ly.W, slots = W > 1 ? M * W : L;
    std::vector<std::vector<unsigned>> sl(slots);
    Ly.helper.assign(L, -1);
    if (W > 1) {
        for (int r = 0; r < M; r++)
            for (size_t j = 0; j < merge[r].size(); j++) sl[(size_t)r * W + j % W].push_back(merge[r][j]);
    } else {
        for (int r = 0; r < M; r++) sl[r] = merge[r];
        std::vector<int> ord(M);
        std::iota(ord.begin(), ord.end(), 0);
        std::stable_sort(ord.begin(), ord.end(), [&](int x, int y) { return merge[x].size() > merge[y].size(); });
        for (int k = M, i = 0; k < slots && i < M; k++, i++) {
            std::vector<unsigned>& m = sl[ord[i]];
            Ly.helper[ord[i]] = k;
            sl[k].assign(m.begin() + (m.size() + 1) / 2, m.end());
            m.resize((m.size() + 1) / 2);
        }
    }
    int rm = 1;
    for (const auto& m : sl) rm = std::max(rm, (int)m.size());
    Ly.RM = pow_pick(kPowMerges[L == 32], rm);
    if (!Ly.RM || Ly.n_part > 60000) return false;
    Ly.merge.assign((size_t)Ly.RM * slots, (unsigned)Ly.n_part);
    for (int k = 0; k < slots; k++)
        for (size_t j = 0; j < sl[k].size(); j++) Ly.merge[j * slots + k] = sl[k][j];
    *out = Ly;
    return true;
}

// Large systems (k_power_big): the rows dealt to `ctas` CTAs of `threads`
// lanes, largest first to the CTA with the fewest entries; a row has
// ceil(entries / E) neighbouring lanes of one warp, E the smallest that lets
// every CTA hold its rows; false when its tables then outgrow shared memory
// (K exponentials of Q nodes on n_chan channels).  Rows are numbered
// CTA by CTA (order, first_row).  entry, xoff [cta][E][threads]; mask
// [cta][threads] lane words.
constexpr int kPowBigMaxRows = 512, kPowBigMaxCtas = 8;
inline bool power_pack_big(const PowSeries& ps, int ctas, int threads, PowLayout* out, int K = 2, int Q = 2,
                           int n_chan = 1) {
    const int M = ps.M, ne = (int)ps.ent.size();
    PowLayout Ly;
    std::vector<int> at_mono;
    if (!pow_monomials(ps, Ly, &at_mono)) return false;
    const int nm = (int)Ly.mono.size();
    if (M > kPowBigMaxRows || nm * M >= 65535) return false;
    std::vector<std::vector<int>> rows(M);
    for (int i = 0; i < ne; i++) rows[ps.ent[i].row].push_back(i);
    std::vector<int> ord(M);
    std::iota(ord.begin(), ord.end(), 0);
    std::stable_sort(ord.begin(), ord.end(), [&](int x, int y) { return rows[x].size() > rows[y].size(); });
    std::vector<long> load(ctas, 0);
    std::vector<std::vector<int>> mine(ctas);    // rows of each CTA, largest first
    for (int r : ord) {
        const int c = (int)(std::min_element(load.begin(), load.end()) - load.begin());
        load[c] += (long)rows[r].size() + 4;     // a row costs its lanes' last slots too
        mine[c].push_back(r);
    }
    const int warps = threads / 32;
    for (int E = std::max(1, (ne + ctas * threads - 1) / (ctas * threads));; E++) {
        Ly.ctas = ctas;
        Ly.L = threads;
        Ly.E = E;
        if (power_smem(Ly, M, K, Q, n_chan, 1) > kPowSmem) return false;
        std::vector<int> first(M, -1);           // a row's first lane in its CTA
        bool ok = true;
        int wmax = 1;
        for (int c = 0; c < ctas && ok; c++) {
            std::vector<int> used(warps, 0);
            for (int r : mine[c]) {
                const int w = std::max(1, ((int)rows[r].size() + E - 1) / E);
                int k = 0;
                while (k < warps && used[k] + w > 32) k++;
                ok = ok && k < warps;
                if (!ok) break;
                first[r] = k * 32 + used[k];
                used[k] += w;
                wmax = std::max(wmax, w);
            }
        }
        if (!ok) continue;
        Ly.rows = true;
        Ly.W = wmax;
        Ly.first_row.assign(1, 0);
        for (int c = 0; c < ctas; c++) {
            Ly.order.insert(Ly.order.end(), mine[c].begin(), mine[c].end());
            Ly.first_row.push_back((int)Ly.order.size());
        }
        std::vector<int> pos(M);
        for (int k = 0; k < M; k++) pos[Ly.order[k]] = k;
        Ly.entry.assign((size_t)ctas * E * threads, -1);
        Ly.xoff.assign((size_t)ctas * E * threads, nm * M);
        Ly.mask.assign((size_t)ctas * threads, (unsigned)M | (1u << 16));
        for (int c = 0; c < ctas; c++)
            for (int r : mine[c]) {
                const int w = std::max(1, ((int)rows[r].size() + E - 1) / E);
                for (int k = 0; k < w; k++)
                    Ly.mask[(size_t)c * threads + first[r] + k] =
                        (unsigned)pos[r] | ((unsigned)w << 16) | ((unsigned)k << 24);
                for (int i = 0; i < (int)rows[r].size(); i++) {
                    const size_t slot = ((size_t)c * E + i / w) * threads + first[r] + i % w;
                    const PowEntry& e = ps.ent[rows[r][i]];
                    Ly.entry[slot] = rows[r][i];
                    Ly.xoff[slot] = at_mono[e.mono] * M + pos[e.col];
                }
            }
        *out = Ly;
        return true;
    }
}

// Lanes per CTA for a cluster of `ctas`: enough warps to issue, few enough
// that the reduction and the barrier stay short (21 levels, 2,000 exponentials:
// clusters of 4 take 5.8 ms at 256 lanes and 6.9 at 512).
inline int power_big_threads(int ctas) { return ctas == 1 ? 1024 : ctas <= 2 ? 512 : 256; }

// Entries that the series of a large system has at least: the patterns of its
// Taylor terms up to third order, each counted while its bound (norms A_norm of
// the constant part and b of the varying one) is well above what is dropped.
// 0.42 to 0.83 of the entries for the 21-level NV (field on and off its axis, 5
// to 30 ps); 0.1 ms at 171 rows where the series takes 2 to 7 ms of all cores.
inline long power_least_entries(int M, const std::vector<int>& row_ptr, const std::vector<int>& col,
                                const std::vector<double>& A, const std::vector<double>* G, double A_norm,
                                double b) {
    const int words = (M + 63) / 64;
    using Bits = std::vector<uint64_t>;
    const double drop = std::min(kPowDrop, kPowDropSmall * std::pow(A_norm + b, 1.5));
    auto multiply = [&](const std::vector<double>& X, const Bits& Y, Bits* out) {
        for (int r = 0; r < M; r++)
            for (int q = row_ptr[r]; q < row_ptr[r + 1]; q++)
                if (X[q] != 0.0)
                    for (int w = 0; w < words; w++) (*out)[(size_t)r * words + w] |= Y[(size_t)col[q] * words + w];
    };
    // P[i][k]: the terms with i factors of the constant part and k of the varying one
    Bits P[4][4];
    P[0][0].assign((size_t)M * words, 0);
    for (int r = 0; r < M; r++) P[0][0][(size_t)r * words + r / 64] |= (uint64_t)1 << (r % 64);
    long n = 0;
    for (int k = 0; k <= (G ? 3 : 0); k++) {
        Bits all((size_t)M * words, 0);
        for (int i = 0; i + k <= 3; i++) {
            if (i + k == 0) continue;
            P[i][k].assign((size_t)M * words, 0);
            double bound = 1.0;
            for (int j = 1; j <= i; j++) bound *= A_norm / j;
            for (int j = 1; j <= k; j++) bound *= b / j;
            if (bound < 1024.0 * drop) continue;
            if (i) multiply(A, P[i - 1][k], &P[i][k]);
            if (k) multiply(*G, P[i][k - 1], &P[i][k]);
            for (size_t w = 0; w < all.size(); w++) all[w] |= P[i][k][w];
        }
        for (uint64_t w : all) n += __builtin_popcountll(w);
    }
    return n;
}

// Cycles of one exponential of a cluster (one CTA per SM): issue of the busiest
// sub-partition, reduction, and the rest as measured (operand loads of 32 warps
// for a single CTA, the exchange for the others; 16,100 cycles for 1 CTA, 9,400
// for 2, 6,000 for 4, 4,900 for 8).
inline int power_big_cycles(const PowLayout& Ly) {
    return Ly.L / 128 * Ly.E * 64 + 138 * Ly.log_w() + (Ly.ctas > 1 ? 2700 : 4700);
}

}  // namespace sss
