// Power-series batched kernels (variant 8): one multiplication by a constant
// sparse matrix per exponential (sss_power.h explains the form and holds the
// host side), included by the sss_power_*.cu units that instantiate them.
//
// k_batch_power, groups of 16 or 32 lanes.  Per exponential a group runs
//   1. E FMA slots per lane over its constant coefficients (registers) and
//      the state in shared memory, parking a partial sum wherever a piece of
//      a row ends;
//   2. a warp barrier;
//   3. the merge: the lanes that own a row add its partial sums, each times
//      its monomial, and add the sum to the row (in registers for the whole
//      trajectory, written to shared memory for the next exponential);
//   4. a warp barrier.
// It issues the fewest FP64 instructions (every slot but the last ones holds
// an entry), which is what bounds a batch that fills the SM sub-partitions.
//
// k_batch_power_rows, groups of 64 to 128 lanes (one trajectory per CTA) for
// batches that do not.  There the chain of one exponential bounds it: a row
// has a power-of-two number of neighbouring lanes to itself, whose E entries
// read the copies of the state scaled by each monomial, so its sum needs only
// shuffles, and one CTA barrier per exponential (the copies alternate
// between two buffers).  Spin-1 sweep of 64 x 20,000 steps: 27.1 ms with
// parked partial sums at 128 lanes (122 instructions per exponential).
//
// The ring of coefficients, the work queue and the readouts are the
// slot-programmed kernels'; the ring holds the monomial values of every
// exponential in place of its weights.
#pragma once
#include "sss_batch_args.cuh"
#include "sss_device.cuh"
#include "sss_power.h"

namespace sss {
namespace {

static_assert(kRing == kPowRing, "power_smem counts the ring");

// A trajectory taken from the queue: its program's index, output samples and,
// for propagator columns, the column.
struct PowTrajectory {
    int b = -1, T_b = 0, t = 0, col = -1;
    size_t bt = 0;
    const double* prog = nullptr;

    __device__ __forceinline__ void set(const BatchArgs& a, int taken) {
        b = a.order ? __ldg(a.order + taken) : taken;
        if (a.cols) {
            // column `col` of the propagators of a run of samples
            const int run = b / a.cols;
            col = b - run * a.cols;
            bt = run / a.col_runs;
            t = a.t_begin + (run - (int)bt * a.col_runs) * a.col_len;
            T_b = min(t + a.col_len, a.t_end);
        } else {
            bt = b;
            T_b = min(a.samples ? a.samples[b] : a.T_max, a.t_end);
            t = a.t_begin;
        }
        prog = a.prog ? a.prog + bt * a.nch * a.nseg * 5 : nullptr;
    }
};

// Refills the ring with R fine steps from step r of sample t on: node values,
// then the monomials of every exponential and its coefficient table.
template <int R, class Sync>
__device__ __forceinline__ void pow_fill_ring(const BatchArgs& a, const PowTrajectory& tr, int r, int li,
                                              int L, double* ringc, double* ring_m, int* ring_t,
                                              Sync gsync) {
    const int NC = a.n_lch, K = a.K, Q = a.Q, NM = a.pw_mono;
    for (int i = li; i < R * Q * NC; i += L) {
        const int s = i / (Q * NC), rem = i - s * Q * NC, k = rem / NC, ci = rem - k * NC;
        const int rr = r + s, ts = tr.t + rr / a.F, rs = rr % a.F;
        const int ch = a.lch_chan[ci];
        double val = 0.0;
        if (a.tab) {
            if (ts < a.T_max)
                val = __ldg(a.tab + ((tr.bt * a.F + rs) * a.T_max + ts) * (size_t)(Q * a.tab_G) +
                            (size_t)k * a.tab_G + ch);
        } else if (ch < a.nch) {
            const double tn = __dadd_rn(__dadd_rn(__dadd_rn(a.t0, __ldg(a.toff + rs)),
                                                  __dmul_rn(a.dt, (double)ts)),
                                        __ldg(a.noff + k));
            val = channel_value(tr.prog, a.nseg, ch, tn);
        }
        ringc[i] = val;
    }
    gsync();
    // rows in execution order (exponential K-1 first); every monomial is an
    // earlier one times a coefficient; the table follows the switched
    // channel's values
    for (int i = li; i < R * K; i += L) {
        const int s = i / K, e = K - 1 - (i - s * K);
        double cv[kPowMaxLive];
#pragma unroll
        for (int g = 0; g < kPowMaxLive; g++) {
            cv[g] = 0.0;
            if (g < a.n_live) {
                double w = 0.0;
                for (int k = 0; k < Q; k++)
                    w = fma(__ldg(a.W + e * Q + k), ringc[(s * Q + k) * NC + a.live_ch[g]], w);
                cv[g] = w * a.pw_scale[g];
            }
        }
        double* mv = ring_m + (size_t)i * NM;
        mv[0] = 1.0;
        for (int m = 1; m < NM; m++) mv[m] = mv[a.pw_p1[m]] * (a.pw_p2[m] == 0 ? cv[0] : cv[1]);
        if (a.pw_multi) {
            int code = 0;
            if (a.pw_sel_ch >= 0)
                for (int k = 0; k < Q; k++)
                    if (ringc[(s * Q + k) * NC + a.pw_sel_ch] == a.pw_sel_v) code |= 1 << k;
            ring_t[i] = a.pw_tab[(e << kMaxQ) + code];
        }
    }
    gsync();
}

// A predicated store of a partial sum (no branch around it).
__device__ __forceinline__ void park(unsigned addr, double x, unsigned yes) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p st.shared.f64 [%0], %1;\n\t}"
                 :: "r"(addr), "d"(x), "r"(yes));
}

template <int L, int E, int RM>
__global__ void __launch_bounds__(128, 1) k_batch_power(const BatchArgs a) {
    extern __shared__ double smem[];
    constexpr int NS = E >= 12 ? 2 : 1, R = kRing;
    static_assert(L <= 32, "a group lives in one warp");
    const int M = a.M, K = a.K, NM = a.pw_mono, W = a.pw_w;
    const int slot = threadIdx.x / L, li = threadIdx.x % L;
    const int n_x = M + 1, n_p = a.npart + 1;
    const size_t per_slot = ((size_t)n_x + n_p + (size_t)R * (a.Q * a.n_lch + K * NM) + NM + (size_t)R * K / 2) | 1;
    double* X = smem + slot * per_slot;            // state, zero word
    double* part = X + n_x;                        // partial sums, zero word
    double* ringc = part + n_p;                    // [s][k][channel] node values
    double* ring_m = ringc + R * a.Q * a.n_lch;    // [s][e][value] monomials
    int* ring_t = reinterpret_cast<int*>(ring_m + R * K * NM);  // [s][e] coefficient table
    const unsigned part_s = (unsigned)__cvta_generic_to_shared(part);
    if (li == 0) {
        X[M] = 0.0;
        part[a.npart] = 0.0;
    }
    // the lane's program
    int xo[E];
    double cf[E];
    unsigned start[NS], end[NS];
    int pb[NS];
#pragma unroll
    for (int q = 0; q < E; q++) {
        xo[q] = __ldg(a.pw_x + q * L + li);
        cf[q] = __ldg(a.pw_coef + (size_t)q * L + li);
    }
#pragma unroll
    for (int s = 0; s < NS; s++) {
        start[s] = __ldg(a.cw + (2 * s) * L + li);
        end[s] = __ldg(a.cw + (2 * s + 1) * L + li);
        pb[s] = __ldg(a.pcol + s * L + li);
    }
    // the lane's row: li / W, the row's lane that keeps it sub = 0
    const int sub = li & (W - 1), row = li / W < M ? li / W : 0;
    const bool own = li / W < M, keep = own && sub == 0;
    double v = 0.0, acc = 0.0;
    const double rw = keep && a.rw ? __ldg(a.rw + row) : 0.0;
    unsigned mw[RM];
#pragma unroll
    for (int m = 0; m < RM; m++)
        mw[m] = W > 1 ? (own ? __ldg(a.pw_merge + (size_t)m * M * W + li) : (unsigned)a.npart)
                      : __ldg(a.pw_merge + (size_t)m * L + li);
    const int help = __ldg(a.rbeg + li);   // lane that helps this row's merge, -1: none
    int cur_tab = 0;
    const bool extra = a.pw_multi || a.states;
    const unsigned leader = (threadIdx.x & 31) / L * L;
    const unsigned gmask = (L >= 32) ? 0xffffffffu : (((1u << L) - 1u) << leader);
    auto gsync = [&]() { __syncwarp(gmask); };
    gsync();

    PowTrajectory tr;
    int r = 0, rp = R;
    while (true) {
        if (r == 0 && tr.t >= tr.T_b) {
            if (tr.b >= 0 && a.fin && !a.cols && keep) {
                a.fin[(size_t)tr.b * a.N + __ldg(a.row_orig + row)] = v;
                note_nonfinite(a, v, tr.b, a.t_end);
            }
            if (tr.b >= 0 && a.readout)
                for (int tt = max(tr.T_b, a.t_begin) + li; tt < a.t_end; tt += L)
                    a.readout[(size_t)tr.b * a.T_max + tt] = 0.0;
            int nb = 0;
            if (li == 0) nb = atomicAdd(a.queue, 1);
            nb = __shfl_sync(gmask, nb, leader);
            if (nb >= a.ntraj) break;
            tr.set(a, nb);
            rp = R;
            acc = 0.0;
            if (a.cols)
                v = row == tr.col ? 1.0 : 0.0;
            else if (own)
                v = a.rho0[(size_t)tr.b * a.N + __ldg(a.row_orig + row)];
            if (keep) X[row] = v;
            if (tr.t >= tr.T_b) continue;
        }
        const int cset = a.n_const && r == 0 ? constant_set(a, tr.prog, tr.t) : -1;
        if (cset >= 0) {
            // the whole sample by its map; the ring starts afresh after it
            gsync();
            const double d = own ? constant_row(a, cset, X, row) : 0.0;
            gsync();
            v += d;
            if (keep) X[row] = v;
            gsync();
            rp = R;
            r = a.F - 1;
        } else if (rp == R) {
            pow_fill_ring<R>(a, tr, r, li, L, ringc, ring_m, ring_t, gsync);
            rp = 0;
        }
        for (int i = 0; i < K && cset < 0; i++) {
            const int re = rp * K + i;
            if (extra) {
                const int tab = a.pw_multi ? ring_t[re] : 0;
                if (tab != cur_tab) {
                    cur_tab = tab;
#pragma unroll
                    for (int q = 0; q < E; q++)
                        cf[q] = __ldg(a.pw_coef + ((size_t)tab * E + q) * L + li);
                }
                if (a.states && keep)
                    a.states[(((size_t)tr.b * a.st_steps + (size_t)(tr.t - a.t_begin) * a.F + r) * K + K - 1 - i) * M +
                             row] = v;
            }
            {
                double x[E], s[NS];
#pragma unroll
                for (int q = 0; q < E; q++) x[q] = X[xo[q]];
                unsigned pp[NS];
#pragma unroll
                for (int i = 0; i < NS; i++) {
                    s[i] = 0.0;
                    pp[i] = part_s + (unsigned)pb[i] * 8u;
                }
#pragma unroll
                for (int q = 0; q < E; q++) {
                    const int i = q % NS, k = q / NS;   // sequence, its slot
                    const double base = ((start[i] >> k) & 1u) ? 0.0 : s[i];
                    s[i] = fma(cf[q], x[q], base);
                    const unsigned ends = (end[i] >> k) & 1u;
                    park(pp[i], s[i], ends);
                    pp[i] += ends * 8u;
                }
            }
            gsync();
            const double* mv = ring_m + (size_t)re * NM;
            double d;
            {
                double g[RM], ps[RM];
#pragma unroll
                for (int m = 0; m < RM; m++) {
                    g[m] = mv[mw[m] >> 16];
                    ps[m] = part[mw[m] & 0xffffu];
                }
                d = g[0] * ps[0];
#pragma unroll
                for (int m = 1; m < RM; m++) d = fma(g[m], ps[m], d);
            }
            if (W > 1) {
                for (int o = W >> 1; o > 0; o >>= 1) d += __shfl_xor_sync(gmask, d, o);
            } else {
                const double x = __shfl_sync(gmask, d, (int)leader + max(help, 0));
                d += help >= 0 ? x : 0.0;
            }
            if (a.cols) {
                // residual form: the column minus its unit vector
                acc += d;
                v = acc + (row == tr.col ? 1.0 : 0.0);
            } else {
                v += d;
            }
            if (keep) X[row] = v;
            gsync();
        }
        if (cset < 0) rp++;
        if (++r == a.F) {
            r = 0;
            const int t = tr.t;
            if (a.cols && keep)
                a.prop[((tr.bt * (a.t_end - a.t_begin) + t - a.t_begin) * (size_t)M + tr.col) * M + row] = acc;
            if (a.trace && keep) a.trace[((size_t)tr.b * a.T_max + t) * a.N + __ldg(a.row_orig + row)] = v;
            if (a.readout) {
                double s = rw * v;
#pragma unroll
                for (int o = L / 2; o > 0; o >>= 1) s += __shfl_xor_sync(gmask, s, o);
                if (li == 0) {
                    a.readout[(size_t)tr.b * a.T_max + t] = s;
                    note_nonfinite(a, s, tr.b, t);
                }
            }
            tr.t++;
        }
    }
}

// One CTA per trajectory; L = blockDim.x lanes (64, 96 or 128), rows of up to
// 2^LG lanes.  Cols: propagator columns.  The body of an exponential is kept
// to the loads, the sums and one barrier, with no branch but the one on
// `extra` (several tables or stored states): at 9 FP64 instructions the other
// instructions -- 139 of them with run-time row widths, tables and ring
// direction -- took half the time.
template <int E, int LG, bool Cols>
__global__ void __launch_bounds__(128, 1) k_batch_power_rows(const BatchArgs a) {
    extern __shared__ double smem[];
    constexpr int R = kPowRowsRing;
    const int M = a.M, K = a.K, NM = a.pw_mono, L = blockDim.x, li = threadIdx.x;
    const int n_x = NM * M + 1;                    // copies [monomial][row], zero word
    double* X = smem;                              // two buffers of them
    double* ringc = X + 2 * n_x;
    double* ring_m = ringc + R * a.Q * a.n_lch;    // [s][exponential][value], and one row past the end
    int* ring_t = reinterpret_cast<int*>(ring_m + (R * K + 1) * NM);
    __shared__ int s_taken;
    __shared__ double s_red[4];
    if (li < 2) X[li * n_x + NM * M] = 0.0;
    if (li < NM) ring_m[R * K * NM + li] = 0.0;
    int xo[E];
    double cf[E];
#pragma unroll
    for (int q = 0; q < E; q++) {
        xo[q] = __ldg(a.pw_x + q * L + li);
        cf[q] = __ldg(a.pw_coef + (size_t)q * L + li);
    }
    // lane word: row (M: none), its lanes W_r and the lane's place among them
    const unsigned lw = __ldg(a.cw + li);
    const int row = (int)(lw & 0xffffu), Wr = (int)((lw >> 16) & 0xffu), sub = (int)(lw >> 24);
    const bool own = row < M, keep = own && sub == 0;
    const int copies = a.kc;                       // copies written per lane
    const bool copy1 = own && sub < NM;            // its first one, monomial `sub`
    const double* const m1 = ring_m + min(sub, NM - 1);
    double* const x1 = X + min(sub, NM - 1) * M + (own ? row : 0);
    double v = 0.0, acc = 0.0;
    const double rw = keep && a.rw ? __ldg(a.rw + row) : 0.0;
    const bool extra = a.pw_multi || a.states;
    int cur_tab = 0, xb = 0;                       // buffer offset: 0 or n_x
    auto gsync = [&]() { __syncthreads(); };
    // the lane's copies of its row, scaled by ring row j's monomials
    auto write_x = [&](int j) {
        const double x = m1[j * NM] * v;
        if (copy1) x1[xb] = x;
        if (copies > 1)
            for (int i = sub + Wr; i < NM; i += Wr) {
                const double y = ring_m[j * NM + i] * v;
                if (own) X[xb + i * M + row] = y;
            }
    };
    gsync();

    PowTrajectory tr;
    int r = 0, rp = R;
    while (true) {
        if (r == 0 && tr.t >= tr.T_b) {
            if (!Cols && tr.b >= 0 && a.fin && keep) {
                a.fin[(size_t)tr.b * a.N + __ldg(a.row_orig + row)] = v;
                note_nonfinite(a, v, tr.b, a.t_end);
            }
            if (tr.b >= 0 && a.readout)
                for (int tt = max(tr.T_b, a.t_begin) + li; tt < a.t_end; tt += L)
                    a.readout[(size_t)tr.b * a.T_max + tt] = 0.0;
            if (li == 0) s_taken = atomicAdd(a.queue, 1);
            __syncthreads();
            const int nb = s_taken;
            __syncthreads();
            if (nb >= a.ntraj) break;
            tr.set(a, nb);
            rp = R;
            acc = 0.0;
            if (Cols)
                v = row == tr.col ? 1.0 : 0.0;
            else if (own)
                v = a.rho0[(size_t)tr.b * a.N + __ldg(a.row_orig + row)];
            if (tr.t >= tr.T_b) continue;
        }
        const int cset = !Cols && a.n_const && r == 0 ? constant_set(a, tr.prog, tr.t) : -1;
        if (cset >= 0) {
            // the whole sample by its map; the ring starts afresh after it
            if (keep) X[xb + row] = v;
            gsync();
            v += own ? constant_row(a, cset, X + xb, row) : 0.0;
            gsync();
            rp = R;
            r = a.F - 1;
        } else if (rp == R) {
            pow_fill_ring<R>(a, tr, r, li, L, ringc, ring_m, ring_t, gsync);
            rp = 0;
            write_x(0);
            gsync();
        }
        for (int i = 0; i < K && cset < 0; i++) {
            const int re = rp * K + i;
            if (extra) {
                const int tab = a.pw_multi ? ring_t[re] : 0;
                if (tab != cur_tab) {
                    cur_tab = tab;
#pragma unroll
                    for (int q = 0; q < E; q++)
                        cf[q] = __ldg(a.pw_coef + ((size_t)tab * E + q) * L + li);
                }
                if (a.states && keep)
                    a.states[(((size_t)tr.b * a.st_steps + (size_t)(tr.t - a.t_begin) * a.F + r) * K + K - 1 - i) * M +
                             row] = v;
            }
            double x[E];
#pragma unroll
            for (int q = 0; q < E; q++) x[q] = X[xb + xo[q]];
            double d = cf[0] * x[0];
#pragma unroll
            for (int q = 1; q < E; q++) d = fma(cf[q], x[q], d);
#pragma unroll
            for (int o = 1; o < (1 << LG); o <<= 1) {
                const double y = __shfl_xor_sync(0xffffffffu, d, o);
                d += o < Wr ? y : 0.0;
            }
            if (Cols) {
                acc += d;
                v = acc + (row == tr.col ? 1.0 : 0.0);
            } else {
                v += d;
            }
            // the next exponential's copies, into the other buffer (past the
            // ring's end with its spare row: written again after the refill)
            xb ^= n_x;
            write_x(re + 1);
            gsync();
        }
        if (cset < 0) rp++;
        if (++r == a.F) {
            r = 0;
            const int t = tr.t;
            if (Cols && keep)
                a.prop[((tr.bt * (a.t_end - a.t_begin) + t - a.t_begin) * (size_t)M + tr.col) * M + row] = acc;
            if (a.trace && keep) a.trace[((size_t)tr.b * a.T_max + t) * a.N + __ldg(a.row_orig + row)] = v;
            if (a.readout) {
                double s = rw * v;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if ((li & 31) == 0) s_red[li >> 5] = s;
                __syncthreads();
                if (li == 0) {
                    for (int w = 1; w < L / 32; w++) s += s_red[w];
                    a.readout[(size_t)tr.b * a.T_max + t] = s;
                    note_nonfinite(a, s, tr.b, t);
                }
                __syncthreads();
            }
            tr.t++;
        }
    }
}

}  // namespace
}  // namespace sss

#define SSS_POWER(L, E, RM) \
    case E * 16 + RM: return launch(p, k_batch_power<L, E, RM>, a, threads, threads / L, smem, st);
