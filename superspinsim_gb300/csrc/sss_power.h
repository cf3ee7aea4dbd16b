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
#include <cmath>
#include <cstdint>
#include <numeric>
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
    const size_t MM = (size_t)M * M;
    std::vector<std::vector<double>> C((size_t)n_tab * nm, std::vector<double>(MM, 0.0));
    std::vector<std::vector<double>> C0lo(n_tab, std::vector<double>(MM, 0.0));
    std::vector<std::vector<double>> T(nm, std::vector<double>(MM)), Nx(nm, std::vector<double>(MM));
    std::vector<dd> D(MM), Dn(MM), Cd(MM);
    for (int tab = 0; tab < n_tab; tab++) {
        for (auto& t : T) std::fill(t.begin(), t.end(), 0.0);
        std::fill(D.begin(), D.end(), dd{0.0, 0.0});
        std::fill(Cd.begin(), Cd.end(), dd{0.0, 0.0});
        for (int i = 0; i < M; i++) {
            D[(size_t)i * M + i] = {1.0, 0.0};
            T[0][(size_t)i * M + i] = 1.0;
        }
        std::vector<std::vector<double>*> Ct(nm);
        for (int m = 0; m < nm; m++) Ct[m] = &C[(size_t)tab * nm + m];
        const std::vector<double>&ah = A_hi[tab], &al = A_lo[tab];
        for (int j = 1; j <= 60; j++) {
            double big = 0.0;
            for (int r = 0; r < M; r++) {
                dd* dn = &Dn[(size_t)r * M];
                std::fill(dn, dn + M, dd{0.0, 0.0});
                for (int q = row_ptr[r]; q < row_ptr[r + 1]; q++) {
                    if (ah[q] == 0.0) continue;
                    const dd* dc = &D[(size_t)col[q] * M];
                    const dd a{ah[q], al[q]};
                    for (int c = 0; c < M; c++)
                        if (dc[c].hi != 0.0) dn[c] = dd_add(dn[c], dd_mul(a, dc[c]));
                }
                for (int c = 0; c < M; c++) {
                    if (dn[c].hi == 0.0) continue;
                    dn[c] = dd_div(dn[c], j);
                    Cd[(size_t)r * M + c] = dd_add(Cd[(size_t)r * M + c], dn[c]);
                    big = std::max(big, std::fabs(dn[c].hi));
                }
            }
            for (int m = nm - 1; m >= 1; m--) {
                for (int r = 0; r < M; r++) {
                    double* n = &Nx[m][(size_t)r * M];
                    std::fill(n, n + M, 0.0);
                    for (int q = row_ptr[r]; q < row_ptr[r + 1]; q++) {
                        if (ah[q] != 0.0) {
                            const double a = ah[q], *t = &T[m][(size_t)col[q] * M];
                            for (int c = 0; c < M; c++) n[c] += a * t[c];
                        }
                        for (int g = 0; g < n_live; g++) {
                            if (lower[m][g] < 0 || G[g][q] == 0.0) continue;
                            const double a = G[g][q], *t = &T[lower[m][g]][(size_t)col[q] * M];
                            for (int c = 0; c < M; c++) n[c] += a * t[c];
                        }
                    }
                    double* cm = &(*Ct[m])[(size_t)r * M];
                    for (int c = 0; c < M; c++) {
                        n[c] /= j;
                        cm[c] += n[c];
                        big = std::max(big, std::fabs(n[c]));
                    }
                }
            }
            D.swap(Dn);
            for (size_t i = 0; i < MM; i++) T[0][i] = D[i].hi;
            for (int m = 1; m < nm; m++) T[m].swap(Nx[m]);
            if (big < 1e-26) break;
        }
        for (size_t i = 0; i < MM; i++) {
            (*Ct[0])[i] = Cd[i].hi;
            C0lo[tab][i] = Cd[i].lo;
        }
    }
    // keep, per column, all but the smallest entries (by their largest value
    // over the tables) whose sum stays below the bound
    std::vector<char> keep((size_t)nm * MM, 0);
    std::vector<std::pair<double, size_t>> colv;
    std::vector<double> size(nm, 1.0);   // largest value of each monomial
    for (int m = 0; m < nm; m++)
        for (int g = 0; g < n_live; g++) size[m] *= std::pow(rho[g], ps.mono[m][g]);
    for (int c = 0; c < M; c++) {
        colv.clear();
        for (int m = 0; m < nm; m++)
            for (int r = 0; r < M; r++) {
                double v = 0.0;
                for (int tab = 0; tab < n_tab; tab++)
                    v = std::max(v, std::fabs(C[(size_t)tab * nm + m][(size_t)r * M + c]));
                v *= size[m];
                if (v > 0.0) colv.push_back({v, (size_t)m * MM + (size_t)r * M + c});
            }
        std::sort(colv.begin(), colv.end());
        double s = 0.0;
        for (const auto& e : colv) {
            s += e.first;
            if (s > drop) keep[e.second] = 1;
        }
    }
    ps.ent.clear();
    std::vector<std::pair<size_t, bool>> src;   // matrix entry, low part
    for (int r = 0; r < M; r++)
        for (int m = 0; m < nm; m++)
            for (int c = 0; c < M; c++) {
                const size_t i = (size_t)r * M + c;
                if (m == 0) {
                    double lo = 0.0;
                    for (int tab = 0; tab < n_tab; tab++) lo = std::max(lo, std::fabs(C0lo[tab][i]));
                    if (lo > drop) {
                        ps.ent.push_back({r, c, 0});
                        src.push_back({i, true});
                    }
                }
                if (keep[(size_t)m * MM + i]) {
                    ps.ent.push_back({r, c, m});
                    src.push_back({i, false});
                }
            }
    const size_t ne = ps.ent.size();
    ps.val.assign(ne * n_tab, 0.0);
    for (int tab = 0; tab < n_tab; tab++)
        for (size_t k = 0; k < ne; k++)
            ps.val[tab * ne + k] = src[k].second ? C0lo[tab][src[k].first]
                                                 : C[(size_t)tab * nm + ps.ent[k].mono][src[k].first];
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

// Cycles of one exponential of a cluster (one CTA per SM): issue of the busiest
// sub-partition, reduction, and the rest as measured (operand loads of 32 warps
// for a single CTA, the exchange for the others; 16,100 cycles for 1 CTA, 9,400
// for 2, 6,000 for 4, 4,900 for 8).
inline int power_big_cycles(const PowLayout& Ly) {
    return Ly.L / 128 * Ly.E * 64 + 138 * Ly.log_w() + (Ly.ctas > 1 ? 2700 : 4700);
}

}  // namespace sss
