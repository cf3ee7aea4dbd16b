// Adjoint gradients of a time-integrated readout with respect to the
// parameters of one channel's segments (by default the x drive's
// amplitudes and phases).  No reference counterpart: the reference has no
// derivatives.  The forward model is the
// reference's integrator exactly as the batched kernel runs it
// (superspinsim/generate_simulator.py:1954-2015 step structure, CF weights
// :278-350, exponential K-1 first :1259-1294).
//
// Objective (per trajectory):  J = sum_t tw[t] * rw . rho(t0 + dt*(t+1)).
// Parameters: for every segment s of the differentiated channel c (channel
// 0, the x field, by default), its amplitude a_s and phase phi_s, and with
// four parameters also its offset o_s and frequency f_s
// (c(t) = o_s + a_s cos(tau f_s t + phi_s)).  Below, Gx stands for that
// channel's generator G_{c+1}.
//
// Every parameter enters a step's exponent Omega_e only through the scalar
// coefficient of Gx, so dOmega_e/dtheta = beta_e(theta) Gx with
// beta_e = h sum_k W[e,k] dc_x(t_k)/dtheta, and
//     dJ/dtheta = sum_steps sum_e beta_e * g_e,
//     g_e = mu_after^T L(Omega_e, Gx) rho_before,
// L the Frechet derivative of exp.  With the exponential truncated at
// degree d (as the forward pass evaluates it), L(Omega, G) is exactly
// sum_{a+b<=d-1} Omega^a G Omega^b / (a+b+1)!, so
//     g_e = sum_{a+b<=d-1} (u_a . z_b) / (a+b+1)!,
//     u_a = (Omega^T)^a mu,  z_b = G Omega^b rho,
// and the adjoint itself moves as mu <- sum_{a<=d} u_a / a!  (= E^T mu).
// Both come from one series: g_e = rho^T L(Omega^T, G^T) mu, and the
// block matrix [[Omega^T, G^T], [0, Omega^T]] applied to [0; mu] by Horner
// (degree d) gives L(Omega^T, G^T) mu on top and E^T mu below -- per term
// two transposed products with Omega and one with G, no dot products.
//
// Checkpointing: the forward pass keeps the state every C ~ sqrt(steps)
// steps; the backward sweep recomputes one interval at a time (storing the
// state before each exponential) and walks it in reverse.  Memory per
// trajectory in flight: (steps/C + C*K) * rows doubles.
//
// Layout and parallel structure are the batched kernel's shared-memory
// variant: a group of L lanes per trajectory, rows split across lanes,
// a device work queue.  The transposed products use a second per-lane entry
// list that points into the same assembled Omega.
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "sss_adjoint_ring.cuh"
#include "sss_adjoint_slots.cuh"
#include "sss_device.cuh"
#include "sss_internal.cuh"

namespace sss {
namespace {

constexpr int kAdjMaxTaylor = 24;

struct AdjArgs {
    int M, Ga, K, Q, F, nch, nseg, ntraj, degree, N, E, ET;
    int xg;          // position of Gx (the differentiated channel's generator) among the active ones
    int dch, npar;   // differentiated channel; parameters per segment (2 or 4)
    long n_steps;    // fine steps per trajectory
    int T, C, n_ck;
    double h, t0, dt;
    int gen_index[kMaxG];
    const double* toff;
    const double* noff;
    const double* W;
    const double* gv;       // Ga*E*L
    const unsigned* ent;    // E*L
    const int* cnt;         // L
    const int* rbeg;        // L+1 first row of each lane (lane order)
    const unsigned* tent;   // ET*L transposed words
    const int* tidx;        // ET*L index into Om (e*L + l), -1: zero
    const int* tcnt;        // L
    const int* row_orig;    // M
    const double* rw;       // M (compressed)
    const double* tw;       // T
    const double* rho0;     // ntraj*N
    const double* prog;     // ntraj*nch*nseg*5
    double* J;              // ntraj
    double* grad;           // ntraj*nseg*npar
    double* ck;             // slots*n_ck*M
    double* st;             // slots*C*K*M
    int* queue;
    double fact_inv[kAdjMaxTaylor + 2];
    double inv_j[kAdjMaxTaylor + 1];
};

__device__ __forceinline__ int wcol(unsigned w) { return (int)(w & 0xffffu); }
__device__ __forceinline__ int wend(unsigned w) { return (int)(w >> 16); }
// transposed-entry index flag: the differentiated generator is non-zero here
constexpr int kHasG = 1 << 30;


template <int L>
struct Group {
    int li;
    unsigned gmask;
    unsigned leader;
    int nE, nET, r0, r1;
    const unsigned* s_ent;
    const unsigned* s_tent;
    const int* s_tidx;
    __device__ void sync() const { __syncwarp(gmask); }
    __device__ double sum(double x) const {
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) x += __shfl_xor_sync(gmask, x, o);
        return x;
    }
    // out[row] = sum Om[e] in[col] over this lane's rows; optional Horner
    // form out = base + (.)*scale
    __device__ void fwd(const double* Om, const double* in, double* out, const double* base,
                        double scale) const {
        double s = 0.0;
        for (int e = 0; e < nE; e++) {
            unsigned w = s_ent[e * L + li];
            s = fma(Om[e * L + li], in[wcol(w)], s);
            if (wend(w)) {
                int row = wend(w) - 1;
                out[row] = base ? fma(s, scale, base[row]) : s;
                s = 0.0;
            }
        }
    }
    __device__ void trans(const double* Om, const double* in, double* out) const {
        double s = 0.0;
        for (int e = 0; e < nET; e++) {
            unsigned w = s_tent[e * L + li];
            int q = s_tidx[e * L + li];
            if (q >= 0) s = fma(Om[q & ~kHasG], in[wcol(w)], s);
            if (wend(w)) {
                out[wend(w) - 1] = s;
                s = 0.0;
            }
        }
    }
    // px_out = (Om^T px + G^T py)*scale, py_out = base + (Om^T py)*scale on
    // this lane's rows (G^T values read through the same entry indices)
    __device__ void trans_block(const double* Om, const double* Gv, const double* px,
                                const double* py, double* px_out, double* py_out,
                                const double* base, double scale) const {
        double s1 = 0.0, s2 = 0.0;
        for (int e = 0; e < nET; e++) {
            unsigned w = s_tent[e * L + li];
            int q = s_tidx[e * L + li];
            if (q >= 0) {
                const int c = wcol(w);
                const bool has_g = (q & kHasG) != 0;
                q &= ~kHasG;
                const double o = Om[q], pyc = py[c];
                s1 = fma(o, px[c], s1);
                if (has_g) s1 = fma(Gv[q], pyc, s1);
                s2 = fma(o, pyc, s2);
            }
            if (wend(w)) {
                const int row = wend(w) - 1;
                px_out[row] = s1 * scale;
                py_out[row] = fma(s2, scale, base[row]);
                s1 = 0.0;
                s2 = 0.0;
            }
        }
    }
    __device__ double dot(const double* a, const double* b) const {
        double s = 0.0;
        for (int i = r0; i < r1; i++) s = fma(a[i], b[i], s);
        return s;
    }
};

template <int L>
__global__ void __launch_bounds__(256) k_adjoint(const AdjArgs a) {
    extern __shared__ double smem[];
    const int M = a.M, Ga = a.Ga, E = a.E, ET = a.ET, d = a.degree, Q = a.Q, K = a.K;
    double* s_gv = smem;                                   // Ga*E*L
    double* s_rw = s_gv + (size_t)Ga * E * L;              // M
    unsigned* s_ent = reinterpret_cast<unsigned*>(s_rw + M);
    unsigned* s_tent = s_ent + (size_t)E * L;
    int* s_tidx = reinterpret_cast<int*>(s_tent + (size_t)ET * L);
    const size_t shared_words = (size_t)Ga * E * L + M + ((size_t)E * L + 2 * (size_t)ET * L + 1) / 2;
    const size_t per_slot = ((size_t)E * L + 7 * (size_t)M + kMaxQ * kMaxG + 4 * kMaxQ) | 1;
    const int slot = threadIdx.x / L, li = threadIdx.x % L;
    double* Om = smem + shared_words + slot * per_slot;
    double* v = Om + (size_t)E * L;      // state
    double* bA = v + M;                  // Horner / power buffers
    double* bB = bA + M;
    double* mu = bB + M;
    double* mun = mu + M;
    double* u0 = mun + M;
    double* u1 = u0 + M;
    double* coef = u1 + M;               // Q*Ga
    double* nd = coef + kMaxQ * kMaxG;   // per node: cos, -amp*sin, segment (as double), used

    for (int i = threadIdx.x; i < Ga * E * L; i += blockDim.x) s_gv[i] = a.gv[i];
    for (int i = threadIdx.x; i < M; i += blockDim.x) s_rw[i] = a.rw ? a.rw[i] : 0.0;
    for (int i = threadIdx.x; i < E * L; i += blockDim.x) s_ent[i] = a.ent[i];
    for (int i = threadIdx.x; i < ET * L; i += blockDim.x) {
        s_tent[i] = a.tent[i];
        s_tidx[i] = a.tidx[i];
    }
    __syncthreads();

    Group<L> grp;
    grp.li = li;
    const unsigned lane_in_warp = threadIdx.x & 31;
    grp.leader = lane_in_warp / L * L;
    grp.gmask = (L == 32) ? 0xffffffffu : (((1u << L) - 1u) << grp.leader);
    grp.nE = __ldg(a.cnt + li);
    grp.nET = __ldg(a.tcnt + li);
    grp.r0 = __ldg(a.rbeg + li);
    grp.r1 = __ldg(a.rbeg + li + 1);
    grp.s_ent = s_ent;
    grp.s_tent = s_tent;
    grp.s_tidx = s_tidx;
    const long gslot = (long)blockIdx.x * (blockDim.x / L) + slot;
    double* ck = a.ck + gslot * (long)a.n_ck * M;
    double* st = a.st + gslot * (long)a.C * K * M;

    // coefficients of step n at the Q nodes; with derivs, also the x
    // channel's segment and its derivative factors at each node
    auto coefficients = [&](const double* prog, long n, bool derivs) {
        const int t = (int)(n / a.F), r = (int)(n % a.F);
        for (int i = li; i < Q * Ga; i += L) {
            int k = i / Ga, g = a.gen_index[i - k * Ga];
            double val = 1.0;
            if (g > 0) {
                double tn = __dadd_rn(__dadd_rn(__dadd_rn(a.t0, __ldg(a.toff + r)),
                                                __dmul_rn(a.dt, (double)t)),
                                      __ldg(a.noff + k));
                val = (g - 1 < a.nch) ? channel_value(prog, a.nseg, g - 1, tn) : 0.0;
            }
            coef[i] = val;
        }
        if (derivs && li < Q) {
            const int k = li;
            double tn = __dadd_rn(__dadd_rn(__dadd_rn(a.t0, __ldg(a.toff + r)),
                                            __dmul_rn(a.dt, (double)t)),
                                  __ldg(a.noff + k));
            const double* dprog = prog + (size_t)a.dch * a.nseg * 5;
            int s = channel_segment(dprog, a.nseg, tn);
            double cs = 0.0, dph = 0.0;
            if (s >= 0) {
                const double* p = dprog + s * 5;
                double arg = __dadd_rn(__dmul_rn(__dmul_rn(6.283185307179586, p[3]), tn), p[4]);
                double sn, cn;
                sincos(arg, &sn, &cn);
                cs = cn;
                dph = -p[2] * sn;
            }
            nd[4 * k] = cs;
            nd[4 * k + 1] = dph;
            nd[4 * k + 2] = (double)s;
            nd[4 * k + 3] = dph * (6.283185307179586 * tn);  // d c / d frequency
        }
        grp.sync();
    };
    auto assemble = [&](int e) {
        double ag[kMaxG];
        for (int g = 0; g < Ga; g++) {
            double s = 0.0;
            for (int k = 0; k < Q; k++) s = fma(__ldg(a.W + e * Q + k), coef[k * Ga + g], s);
            ag[g] = s * a.h;
        }
        for (int q = 0; q < grp.nE; q++) {
            double o = 0.0;
            for (int g = 0; g < Ga; g++) o = fma(ag[g], s_gv[((size_t)g * E + q) * L + li], o);
            Om[q * L + li] = o;
        }
        grp.sync();
    };
    // v <- exp(Om) v, Horner
    auto expv = [&]() {
        const double* cur = v;
        double* nxt = bA;
        for (int j = d; j >= 1; j--) {
            grp.fwd(Om, cur, nxt, v, a.inv_j[j]);
            grp.sync();
            cur = nxt;
            nxt = (nxt == bA) ? bB : bA;
        }
        for (int i = grp.r0; i < grp.r1; i++) v[i] = cur[i];
        grp.sync();
    };

    while (true) {
        int nb = 0;
        if (li == 0) nb = atomicAdd(a.queue, 1);
        const int b = __shfl_sync(grp.gmask, nb, grp.leader);
        if (b >= a.ntraj) break;
        const double* prog = a.prog + (size_t)b * a.nch * a.nseg * 5;
        // ---- forward with checkpoints ----
        for (int i = grp.r0; i < grp.r1; i++) v[i] = a.rho0[(size_t)b * a.N + a.row_orig[i]];
        grp.sync();
        double Jacc = 0.0;
        for (long n = 0; n < a.n_steps; n++) {
            if (n % a.C == 0) {
                double* c = ck + (n / a.C) * M;
                for (int i = grp.r0; i < grp.r1; i++) c[i] = v[i];
            }
            coefficients(prog, n, false);
            for (int e = K - 1; e >= 0; e--) {
                assemble(e);
                expv();
            }
            if ((n + 1) % a.F == 0) {
                int t = (int)((n + 1) / a.F) - 1;
                Jacc = fma(a.tw[t], grp.sum(grp.dot(s_rw, v)), Jacc);
            }
        }
        if (li == 0) a.J[b] = Jacc;
        double* gb = a.grad + (size_t)b * a.nseg * a.npar;
        if (li == 0)
            for (int s = 0; s < a.npar * a.nseg; s++) gb[s] = 0.0;
        // ---- backward ----
        for (int i = grp.r0; i < grp.r1; i++) mu[i] = 0.0;
        grp.sync();
        for (long c = a.n_ck - 1; c >= 0; c--) {
            const long n0 = c * a.C, n1 = min(n0 + (long)a.C, a.n_steps);
            for (int i = grp.r0; i < grp.r1; i++) v[i] = ck[c * M + i];
            grp.sync();
            for (long n = n0; n < n1; n++) {
                coefficients(prog, n, false);
                for (int e = K - 1; e >= 0; e--) {
                    double* s = st + ((n - n0) * K + e) * M;
                    for (int i = grp.r0; i < grp.r1; i++) s[i] = v[i];
                    assemble(e);
                    expv();
                }
            }
            for (long n = n1 - 1; n >= n0; n--) {
                if ((n + 1) % a.F == 0) {
                    const double w = a.tw[(n + 1) / a.F - 1];
                    for (int i = grp.r0; i < grp.r1; i++) mu[i] = fma(w, s_rw[i], mu[i]);
                }
                coefficients(prog, n, true);
                for (int e = 0; e < K; e++) {
                    assemble(e);
                    const double* s = st + ((n - n0) * K + e) * M;
                    for (int i = grp.r0; i < grp.r1; i++) v[i] = s[i];
                    grp.sync();
                    // Transposed block series on [0; mu]:
                    //   px <- (Om^T px + G^T py)/j,  py <- mu + (Om^T py)/j,
                    // j = d..1; then py = E^T mu and px = L(Om^T, G^T) mu,
                    // so g = rho_before . px.
                    double* pxc = mun;   // zero on entry
                    double* pyc = mu;
                    double* pxn = u0;
                    double* pyn = u1;
                    for (int i = grp.r0; i < grp.r1; i++) mun[i] = 0.0;
                    grp.sync();
                    for (int j = d; j >= 1; j--) {
                        grp.trans_block(Om, s_gv + (size_t)a.xg * E * L, pxc, pyc, pxn, pyn, mu,
                                        a.inv_j[j]);
                        grp.sync();
                        if (j == d) {
                            // pxc/pyc were mun/mu; move to the ping-pong pair
                            pxc = pxn; pyc = pyn;
                            pxn = bA; pyn = bB;
                        } else {
                            double* t1 = pxc; pxc = pxn; pxn = t1;
                            double* t2 = pyc; pyc = pyn; pyn = t2;
                        }
                    }
                    const double g = grp.sum(grp.dot(v, pxc));
                    for (int i = grp.r0; i < grp.r1; i++) mu[i] = pyc[i];
                    grp.sync();
                    if (li == 0) {
                        for (int k = 0; k < Q; k++) {
                            int sgm = (int)nd[4 * k + 2];
                            if (sgm < 0) continue;
                            double hw = a.h * __ldg(a.W + e * Q + k);
                            double* gs = gb + (size_t)a.npar * sgm;
                            gs[0] = fma(hw * nd[4 * k], g, gs[0]);
                            gs[1] = fma(hw * nd[4 * k + 1], g, gs[1]);
                            if (a.npar == 4) {
                                gs[2] = fma(hw, g, gs[2]);
                                gs[3] = fma(hw * nd[4 * k + 3], g, gs[3]);
                            }
                        }
                    }
                    grp.sync();
                }
            }
        }
    }
}

template <int L>
int launch_adj(sss_plan* p, const AdjArgs& a, int threads, size_t smem, int grid, cudaStream_t st) {
    if (int rc = allow_smem(k_adjoint<L>)) return rc;
    k_adjoint<L><<<grid, threads, smem, st>>>(a);
    SSS_CUDA(cudaGetLastError());
    (void)p;
    return SSS_OK;
}

// ---------------------------------------------------------------------------
// Row-part adjoint.  The forward pass runs the row-part forward kernel and
// keeps the state before every exponential (no recomputation); this kernel
// then walks each trajectory backwards.  Per exponential it assembles Omega
// on the row-part layout of the transposed pattern (rows of Omega^T are the
// columns of Omega) and runs the transposed block series
//     px <- (Omega^T px + G^T py)/j,   py <- mu + (Omega^T py)/j,  j = d..1,
// from px = 0, py = mu: then py = E^T mu (the new adjoint) and
// g = rho_before . px = mu^T L(Omega, G) rho_before.  Per entry three FMAs
// (two chains share the gathered py value); G^T entries sit first in each
// part so that only the first `ngx` positions carry the third FMA.  The
// differentiated channel's coefficients and derivative factors (cos, -a sin,
// segment and -a sin tau t at every node) come from a ring filled kRing
// steps at a time, walking back.
// Gradient sums are kept per node and segment in registers of every lane
// (its share of g) and summed over the group and added to the output only
// when the node's segment changes.  The stored state before an exponential
// is loaded when the exponential starts, so its latency hides behind the
// series.
struct AdjPartsArgs {
    int M, K, Q, F, nch, nseg, ntraj, degree, T;
    long n_steps;
    double h, t0, dt;
    int n_live, x_live, kc, ngx;
    int dch, npar;          // differentiated channel; parameters per segment (2 or 4)
    int live[kMaxG];
    int gen_index[kMaxG];
    const int* pcol;        // C*P*L transposed entry columns [e][l]
    const unsigned* cw;     // kCloseMax*L close words [k][l]
    const double* om0;      // K*C*P*L constant part of Omega^T per exponential
    const double* gv;       // Ga*C*P*L transposed generator values [g][e][l]
    const double* gx;       // C*P*L  differentiated generator's values (the G of the series)
    const int* rbeg;        // L+1
    const int* fwdpos;      // M: index of each row in the stored forward states
    const double* rw;       // M
    const double* tw;       // T
    const double* toff;
    const double* noff;
    const double* W;
    const double* states;   // ntraj*n_steps*K*M
    const double* readout;  // ntraj*T
    const double* prog;
    double* J;
    double* grad;
    int* queue;
    double inv_j[kAdjMaxTaylor + 1];
};

template <int L, int C, int P>
__global__ void __launch_bounds__(256, 1) k_adjoint_parts(const AdjPartsArgs a) {
    extern __shared__ double smem[];
    constexpr int CP = C * P;
    const int M = a.M, NL = a.n_live, K = a.K, Q = a.Q, d = a.degree;
    const int Ms = M + 2;  // rows, the zero row M, the sink row M+1
    const int slot = threadIdx.x / L, li = threadIdx.x % L;
    const size_t per_slot =
        (6 * (size_t)Ms + 2 * (size_t)(L * C + 1) + (size_t)kRing * (Q * NL + K * NL + 4 * Q)) | 1;
    double* sb = smem + slot * per_slot;
    double* parts1 = sb + 6 * (size_t)Ms;
    double* parts2 = parts1 + L * C + 1;
    double* ringc = parts2 + L * C + 1;         // [s][k][live] node values
    double* ring_ag = ringc + kRing * Q * NL;   // [s][e][live] CF weights
    double* ring_d = ring_ag + kRing * K * NL;  // [s][k][4] cos, -a sin, segment, -a sin tau t
    double* s_rw = smem + (size_t)(blockDim.x / L) * per_slot;
    for (int i = threadIdx.x; i < M; i += blockDim.x) s_rw[i] = a.rw[i];
    for (int i = li; i < 6 * Ms; i += L) sb[i] = 0.0;
    for (int i = li; i < 2 * (L * C + 1); i += L) parts1[i] = 0.0;
    int col[CP];
    double gx[CP];
#pragma unroll
    for (int e = 0; e < CP; e++) {
        col[e] = __ldg(a.pcol + (size_t)e * L + li);
        gx[e] = __ldg(a.gx + (size_t)e * L + li);
    }
    unsigned cw[kCloseMax];
#pragma unroll
    for (int k = 0; k < kCloseMax; k++) cw[k] = __ldg(a.cw + (size_t)k * L + li);
    const int kc = a.kc, ngx = a.ngx;
    const int r0 = __ldg(a.rbeg + li), r1 = __ldg(a.rbeg + li + 1);
    // positions of this lane's first rows in the stored forward states: their
    // values are loaded when an exponential starts and used after its series
    constexpr int kPre = 4;
    int fpos[kPre];
#pragma unroll
    for (int i = 0; i < kPre; i++) fpos[i] = r0 + i < r1 ? __ldg(a.fwdpos + r0 + i) : 0;
    __syncthreads();

    // a group of L <= 32 lanes lives in one warp; a wider one is the CTA
    constexpr bool kCta = L > 32;
    const unsigned lane_in_warp = threadIdx.x & 31;
    const unsigned leader = kCta ? 0u : lane_in_warp / L * L;
    const unsigned gmask = (L >= 32) ? 0xffffffffu : (((1u << L) - 1u) << leader);
    __shared__ int s_bcast;
    __shared__ double s_red[kCta ? L / 32 : 1];
    auto gsync = [&]() {
        if (kCta) __syncthreads(); else __syncwarp(gmask);
    };
    // sum over the group, valid in lane 0
    auto gsum = [&](double v) {
#pragma unroll
        for (int o = (L < 32 ? L : 32) / 2; o > 0; o >>= 1) v += __shfl_xor_sync(gmask, v, o);
        if (kCta) {
            if (lane_in_warp == 0) s_red[threadIdx.x >> 5] = v;
            __syncthreads();
            if (threadIdx.x == 0)
                for (int w = 1; w < L / 32; w++) v += s_red[w];
            __syncthreads();
        }
        return v;
    };
    const double* zb = sb;    // stays zero
    double* mu = sb + Ms;
    double* yA = mu + Ms;
    double* yB = yA + Ms;
    double* xA = yB + Ms;
    double* xB = xA + Ms;
    double om[CP];

    while (true) {
        int nb = 0;
        if (li == 0) nb = atomicAdd(a.queue, 1);
        if (kCta) {
            if (li == 0) s_bcast = nb;
            __syncthreads();
            nb = s_bcast;
            __syncthreads();
        } else {
            nb = __shfl_sync(gmask, nb, leader);
        }
        const int b = nb;
        if (b >= a.ntraj) break;
        const double* prog = a.prog + (size_t)b * a.nch * a.nseg * 5;
        // objective from the forward readouts
        {
            double s = 0.0;
            for (int t = li; t < a.T; t += L) s = fma(a.tw[t], a.readout[(size_t)b * a.T + t], s);
            s = gsum(s);
            if (li == 0) a.J[b] = s;
        }
        const double* dprog = prog + (size_t)a.dch * a.nseg * 5;
        double* gb = a.grad + (size_t)b * a.nseg * a.npar;
        // every lane: its share of the running gradient sums per node, for
        // segment cur_seg[k] (the same in every lane); summed over the group
        // only when the node's segment changes
        int cur_seg[kMaxQ];
        double acc_a[kMaxQ], acc_p[kMaxQ], acc_o[kMaxQ], acc_f[kMaxQ];
#pragma unroll
        for (int k = 0; k < kMaxQ; k++) {
            cur_seg[k] = -1;
            acc_a[k] = 0.0;
            acc_p[k] = 0.0;
            acc_o[k] = 0.0;
            acc_f[k] = 0.0;
        }
        // node k's sums over the group into its segment's gradient entries,
        // then zero (every lane calls it together)
        auto flush = [&](int k) {
            const double ta = gsum(acc_a[k]), tp = gsum(acc_p[k]);
            double to = 0.0, tf = 0.0;
            if (a.npar == 4) {
                to = gsum(acc_o[k]);
                tf = gsum(acc_f[k]);
            }
            if (li == 0) {
                double* gs = gb + (size_t)a.npar * cur_seg[k];
                gs[0] += ta;
                gs[1] += tp;
                if (a.npar == 4) {
                    gs[2] += to;
                    gs[3] += tf;
                }
            }
            acc_a[k] = acc_p[k] = acc_o[k] = acc_f[k] = 0.0;
        };
        for (int row = r0; row < r1; row++) mu[row] = 0.0;
        gsync();
        const double* st_b = a.states + (size_t)b * a.n_steps * K * M;
        int rp = kRing;
        for (long n = a.n_steps - 1; n >= 0; n--) {
            if ((n + 1) % a.F == 0) {
                const double w = a.tw[(n + 1) / a.F - 1];
                for (int row = r0; row < r1; row++) mu[row] = fma(w, s_rw[row], mu[row]);
                gsync();
            }
            if (rp == kRing) {
                // steps n, n-1, ..., n-kRing+1: node values of the live channels;
                // for the differentiated channel also cos, -a sin, the segment
                // and -a sin tau t
                adjoint_ring_nodes(a, prog, dprog, n, li, L, ringc, ring_d);
                gsync();
                adjoint_ring_weights(a, li, L, ringc, ring_ag);
                gsync();
                rp = 0;
            }
            for (int e_exp = 0; e_exp < K; e_exp++) {
                const double* rb = st_b + ((size_t)n * K + e_exp) * M;
                double rbv[kPre];
#pragma unroll
                for (int i = 0; i < kPre; i++) rbv[i] = r0 + i < r1 ? __ldg(rb + fpos[i]) : 0.0;
                const double* o0 = a.om0 + (size_t)e_exp * CP * L + li;
#pragma unroll
                for (int e = 0; e < CP; e++) om[e] = __ldg(o0 + (size_t)e * L);
                for (int gi = 0; gi < NL; gi++) {
                    const double c = ring_ag[(rp * K + e_exp) * NL + gi];
                    if (is_zero(c)) continue;
                    const double* gv = a.gv + (size_t)a.live[gi] * CP * L + li;
#pragma unroll
                    for (int e = 0; e < CP; e++) om[e] = fma(c, __ldg(gv + (size_t)e * L), om[e]);
                }
                const double* pxc = zb;
                const double* pyc = mu;
                double* pxn = xA;
                double* pyn = yA;
                for (int j = d; j >= 1; j--) {
                    const double ij = a.inv_j[j];
                    // three independent chains per part: Omega^T px, G^T py
                    // (the first ngx entries) and Omega^T py
                    double s1[C], s2[C], s3[C];
#pragma unroll
                    for (int c = 0; c < C; c++) {
                        s1[c] = 0.0;
                        s2[c] = 0.0;
                        s3[c] = 0.0;
                    }
#pragma unroll
                    for (int q = 0; q < P; q++)
#pragma unroll
                        for (int c = 0; c < C; c++) {
                            const int e = c * P + q;
                            const double yv = pyc[col[e]];
                            s2[c] = fma(om[e], yv, s2[c]);
                            s1[c] = fma(om[e], pxc[col[e]], s1[c]);
                            if (q < ngx) s3[c] = fma(gx[e], yv, s3[c]);
                        }
#pragma unroll
                    for (int c = 0; c < C; c++) {
                        parts1[li * C + c] = s1[c] + s3[c];
                        parts2[li * C + c] = s2[c];
                    }
                    gsync();
                    double a1 = 0.0, a2 = 0.0;
#pragma unroll
                    for (int k = 0; k < kCloseMax; k++) {
                        if (k >= kc) break;
                        const unsigned w = cw[k];
                        const int row = (int)(w & 0xffffu), pi = (int)((w >> 16) & 0x7fffu);
                        const bool first = (w >> 31) != 0;
                        a1 = fma(parts1[pi], ij, first ? 0.0 : a1);
                        a2 = fma(parts2[pi], ij, first ? mu[row] : a2);
                        pxn[row] = a1;
                        pyn[row] = a2;
                    }
                    gsync();
                    pxc = pxn;
                    pyc = pyn;
                    pxn = (pxn == xA) ? xB : xA;
                    pyn = (pyn == yA) ? yB : yA;
                }
                // this lane's share of g = rho_before . px;  mu <- E^T mu (the
                // buffer holding it)
                double g = 0.0;
#pragma unroll
                for (int i = 0; i < kPre; i++)
                    if (r0 + i < r1) g = fma(rbv[i], pxc[r0 + i], g);
                for (int row = r0 + kPre; row < r1; row++) g = fma(rb[__ldg(a.fwdpos + row)], pxc[row], g);
                double* newmu = const_cast<double*>(pyc);
                if (newmu == yA) yA = mu; else yB = mu;
                mu = newmu;
#pragma unroll
                for (int k = 0; k < kMaxQ; k++) {
                    if (k >= Q) break;
                    const double* rd = ring_d + (rp * Q + k) * 4;
                    const int sg = (int)rd[2];
                    if (sg != cur_seg[k]) {  // the same in every lane of the group
                        if (cur_seg[k] >= 0) flush(k);
                        cur_seg[k] = sg;
                    }
                    if (sg >= 0) {
                        const double hw = a.h * __ldg(a.W + e_exp * Q + k);
                        acc_a[k] = fma(hw * rd[0], g, acc_a[k]);
                        acc_p[k] = fma(hw * rd[1], g, acc_p[k]);
                        acc_o[k] = fma(hw, g, acc_o[k]);
                        acc_f[k] = fma(hw * rd[3], g, acc_f[k]);
                    }
                }
                gsync();
            }
            rp++;
        }
#pragma unroll
        for (int k = 0; k < kMaxQ; k++)
            if (k < Q && cur_seg[k] >= 0) flush(k);
        gsync();
    }
}

template <int L>
int launch_adj_parts(sss_plan* p, int C, int P, const AdjPartsArgs& a, int threads, size_t smem,
                     cudaStream_t st) {
    auto go = [&](auto kern) -> int {
        if (int rc = allow_smem(kern)) return rc;
        int per_sm = 0;
        SSS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem));
        if (per_sm < 1) return fail(SSS_EINVAL, "adjoint kernel does not fit on an SM");
        const int slots = threads / L;
        const int grid = std::max(1, std::min((a.ntraj + slots - 1) / slots, per_sm * p->num_sms));
        kern<<<grid, threads, smem, st>>>(a);
        SSS_CUDA(cudaGetLastError());
        return SSS_OK;
    };
    static_assert(sizeof(kPartShapes) / sizeof(kPartShapes[0]) == 4, "one case per part shape");
    if (C == 1 && P == 4) return go(k_adjoint_parts<L, 1, 4>);
    if (C == 2 && P == 4) return go(k_adjoint_parts<L, 2, 4>);
    if (C == 4 && P == 4) return go(k_adjoint_parts<L, 4, 4>);
    if (C == 2 && P == 8) return go(k_adjoint_parts<L, 2, 8>);
    return fail(SSS_EINVAL, "no adjoint kernel for this part shape");
}

// Row-part adjoint: forward with stored states, then the backward kernel,
// over trajectory chunks sized to the free device memory.  Returns
// SSS_EINVAL (with nothing launched) when the pattern does not fit the
// row-part kernels or the states of one trajectory do not fit in memory.
// The slot-programmed backward (sss_adjoint_slots.cu): the block matrix
// [[Omega^T, G^T], [0, Omega^T]] of the forward layout's rows, 2M block rows
// -- px of row c holds the Omega^T entries (Omega[r][c], column r) and the
// G^T entries (G[r][c], column M + r), py of row c the Omega^T entries
// (column M + r) -- laid out by the forward kernels' phased or slot-packed
// packer at 32 lanes, with bank-aware placement.  Builds the kernel's
// tables into p->w_adjb and its arguments (the per-chunk pointers are set at
// launch); SSS_EINVAL, with nothing uploaded, when the block fits neither
// program.
static int adjoint_slots_prepare(sss_plan* p, const BatchLayout& Ly, int ntraj, int gd, int xg,
                                 double t0, double dt, int T, int F, int nch, int nseg,
                                 const double* h_rw, const double* h_tw, int dch, int npar,
                                 AdjSlotArgs* out, BatchLayout* BLo, size_t* smem_out,
                                 int* threads_out, cudaStream_t st) {
    const SparseGenerators& sp = p->sparse;
    const int M = Ly.M, Ga = Ly.Ga, K = p->d.K, Q = p->d.Q;
    // lanes: as configured (32 or 64), else two warps per trajectory
    // (slot-packed, 64 lanes) while the batch leaves SM sub-partitions
    // without a warp at one warp per trajectory (measured on the C4 workload,
    // 256 shapes: 64 lanes 1.19x faster than 32, 128 lanes no better), else 32
    int Lw = p->batch_lanes;
    if (Lw != 32 && Lw != 64) Lw = (long)ntraj * 2 <= 4L * p->num_sms ? 64 : 32;
    const bool wide = Lw > 32;
    if (2 * M + 2 > (int)kSlotIdx) return fail(SSS_EINVAL, "block series too large for slot words");
    std::vector<std::vector<BatchLayout::Ent>> brows(2 * (size_t)M);
    p->slot_consts.clear();
    for (int r = 0; r < M; r++)
        for (const BatchLayout::Ent& en : Ly.row_ents[r]) {
            brows[en.col].push_back({r, en.q});
            brows[(size_t)M + en.col].push_back({M + r, en.q});
            const double gval = sp.val[(size_t)gd * sp.nnz + en.q];
            if (gval != 0.0) {
                brows[en.col].push_back({M + r, sp.nnz + (int)p->slot_consts.size()});
                p->slot_consts.push_back(gval);
            }
        }
    // generators assembled every exponential: the differentiated one and
    // those whose channel varies
    std::vector<char> varies(sp.G, 0);
    std::vector<int> live;
    int x_live = -1;
    for (int gi = 0; gi < Ga; gi++) {
        const int g = Ly.active[gi];
        if (g != 0 && (g == gd || !Ly.chan_const[g])) {
            varies[g] = 1;
            if (gi == xg) x_live = (int)live.size();
            live.push_back(gi);
        }
    }
    std::vector<int> brr(2 * (size_t)M);
    for (int i = 0; i < 2 * M; i++) brr[i] = i;
    BatchLayout& BL = *BLo;
    int rc = SSS_EINVAL;
    if (wide) {
        rc = phased_layout_rows(p, brows, 64, 64, 8, Ly.active, brr, varies, &BL);
        if (rc != SSS_OK) {
            set_error("");
            rc = slots_layout_rows(p, brows, 64, 64, 8, Ly.active, brr, &BL);
        }
        if (rc != SSS_OK) set_error("");
    }
    if (rc != SSS_OK) {
        rc = phased_layout_rows(p, brows, 32, 32, kSlotsMax, Ly.active, brr, varies, &BL);
        if (rc != SSS_OK) {
            set_error("");
            rc = slots_layout_rows(p, brows, 32, 32, kSlotsMax, Ly.active, brr, &BL);
        }
    }
    if (rc != SSS_OK) return rc;
    const int L = BL.L, threads = BL.threads;
    BL.M = 2 * M;
    BL.Ga = Ga;
    BL.active = Ly.active;
    if (int rc2 = place_banks(p, BL, Ly.active, varies)) return rc2;
    const int S = BL.S, Ms = 2 * M + 2 + BL.npart, NL = (int)live.size();
    if (NL > kMaxG) return fail(SSS_EINVAL, "too many live generators");
    // the constant part of the block per exponential: the folded generators,
    // 1 for partial adds, the G^T values for constant entries
    const double h = dt / F;
    const size_t SL = (size_t)S * L;
    std::vector<double> om0((size_t)K * SL, 0.0);
    for (int gi = 0; gi < Ga; gi++) {
        if (std::find(live.begin(), live.end(), gi) != live.end()) continue;
        const int g = Ly.active[gi];
        const double X = g == 0 ? 1.0 : Ly.chan_value[g];
        for (int e = 0; e < K; e++) {
            double s = 0.0;
            for (int k = 0; k < Q; k++) s = std::fma(p->W[e * Q + k], X, s);
            const double ag = s * h;
            for (size_t i = 0; i < SL; i++) {
                double& o = om0[(size_t)e * SL + i];
                o = std::fma(ag, BL.gv[(size_t)gi * SL + i], o);
            }
        }
    }
    for (int e = 0; e < K; e++)
        for (size_t i = 0; i < SL; i++) {
            if (BL.entry_q[i] == -2) om0[(size_t)e * SL + i] = 1.0;
            if (BL.entry_q[i] == -3) om0[(size_t)e * SL + i] = BL.cval[i];
        }
    std::vector<int> ppx(M), ppy(M), fpos(M);
    std::vector<double> rw(M, 0.0), tw(h_tw, h_tw + T), toff(F), noff(Q);
    for (int i = 0; i < M; i++) {
        ppx[i] = BL.newpos[i];
        ppy[i] = BL.newpos[(size_t)M + i];
        fpos[i] = Ly.newpos[i];
        if (h_rw) rw[i] = h_rw[Ly.row_orig[Ly.newpos[i]]];
    }
    for (int r = 0; r < F; r++) toff[r] = ((double)r * dt) / F;
    for (int k = 0; k < Q; k++) noff[k] = (dt * p->nodes[k]) / F;
    // blob: gv | om0 | rw | tw | toff | noff | cw | ppx | ppy | fpos
    std::vector<double> dbl(BL.gv);
    const size_t o_om0 = dbl.size();
    dbl.insert(dbl.end(), om0.begin(), om0.end());
    const size_t o_rw = dbl.size();
    dbl.insert(dbl.end(), rw.begin(), rw.end());
    const size_t o_tw = dbl.size();
    dbl.insert(dbl.end(), tw.begin(), tw.end());
    const size_t o_toff = dbl.size();
    dbl.insert(dbl.end(), toff.begin(), toff.end());
    const size_t o_noff = dbl.size();
    dbl.insert(dbl.end(), noff.begin(), noff.end());
    std::vector<int> ints(BL.cw.begin(), BL.cw.end());
    const size_t o_px = ints.size();
    ints.insert(ints.end(), ppx.begin(), ppx.end());
    const size_t o_py = ints.size();
    ints.insert(ints.end(), ppy.begin(), ppy.end());
    const size_t o_fp = ints.size();
    ints.insert(ints.end(), fpos.begin(), fpos.end());
    const size_t bytes = sizeof(double) * dbl.size() + sizeof(int) * ints.size();
    if (int rc2 = p->w_adjb.ensure(bytes + 64)) return rc2;
    {
        std::vector<char> blob(bytes);
        memcpy(blob.data(), dbl.data(), sizeof(double) * dbl.size());
        memcpy(blob.data() + sizeof(double) * dbl.size(), ints.data(), sizeof(int) * ints.size());
        SSS_CUDA(cudaMemcpyAsync(p->w_adjb.p, blob.data(), bytes, cudaMemcpyHostToDevice, st));
        SSS_CUDA(cudaStreamSynchronize(st));  // the host blob goes out of scope
    }
    const double* dv = p->w_adjb.as<double>();
    const int* di = reinterpret_cast<const int*>(dv + dbl.size());
    AdjSlotArgs a{};
    a.M = M;
    a.M2 = 2 * M;
    a.Ms = Ms;
    a.K = K; a.Q = Q; a.F = F; a.nch = nch; a.nseg = nseg; a.degree = Ly.degree; a.T = T;
    a.n_steps = (long)T * F;
    a.h = h; a.t0 = t0; a.dt = dt;
    a.n_live = NL;
    a.x_live = x_live;
    a.dch = dch;
    a.npar = npar;
    for (int i = 0; i < NL; i++) a.live[i] = live[i];
    for (int gi = 0; gi < Ga; gi++) a.gen_index[gi] = Ly.active[gi];
    for (int i = 0; i < NL; i++) {
        unsigned m = 0;
        for (int q = 0; q < S; q++)
            for (int l = 0; l < L; l++)
                if (BL.gv[((size_t)live[i] * S + q) * L + l] != 0.0) m |= 1u << q;
        a.amask[i] = m;
    }
    a.cw = reinterpret_cast<const unsigned*>(di);
    a.gv = dv;
    a.om0 = dv + o_om0;
    a.rw = dv + o_rw;
    a.tw = dv + o_tw;
    a.toff = dv + o_toff;
    a.noff = dv + o_noff;
    a.ppx = di + o_px;
    a.ppy = di + o_py;
    a.fpos = di + o_fp;
    a.W = p->d_gens.as<double>() + p->gens.size();
    for (int j = 0; j <= kMaxTaylor; j++) a.cfac[j] = 0.0;
    for (int j = 1; j <= Ly.degree; j++) {
        double c = 1.0;
        for (int k = j; k <= Ly.degree; k++) c *= k;
        a.cfac[j] = c;
    }
    a.inv_dfact = 1.0 / a.cfac[1];
    const size_t per_slot = ((3 * (size_t)Ms + (size_t)kRing * (Q * NL + K * NL + 4 * Q)) | 1);
    const size_t smem = sizeof(double) * (per_slot * (threads / L) + M);
    if (smem > 227 * 1024) return fail(SSS_EINVAL, "slot adjoint kernel: shared memory per CTA too large");
    *out = a;
    *smem_out = smem;
    *threads_out = threads;
    return SSS_OK;
}

int adjoint_run_parts(sss_plan* p, int ntraj, const double* d_rho0, int nch, int nseg,
                      const double* d_prog, double t0, double dt, int T, int F,
                      const double* h_rw, const double* h_tw, int dch, int npar, double* d_J,
                      double* d_grad, cudaStream_t st) {
    const int N = p->d.N, K = p->d.K, Q = p->d.Q;
    const int gd = dch + 1;  // the differentiated channel's generator
    BatchLayout Ly;
    if (int rc = build_layout(p, ntraj, d_rho0, nch, nseg, d_prog, dt, F, {gd}, true, &Ly, st, true))
        return rc;
    if (Ly.M == 0) return fail(SSS_EINVAL, "empty pattern");
    if (Ly.substeps != 1) return fail(SSS_EINVAL, "the adjoint needs one sub-step per exponential");
    if (Ly.degree > kAdjMaxTaylor) return fail(SSS_EINVAL, "Taylor degree too large for the adjoint");
    int xg = -1;
    for (int gi = 0; gi < Ly.Ga; gi++)
        if (Ly.active[gi] == gd) xg = gi;
    if (xg < 0)
        return fail(SSS_EINVAL, "the generator of channel " + std::to_string(dch) +
                                    " is zero on the reachable rows");
    const int M = Ly.M, Ga = Ly.Ga;
    const long n_steps = (long)T * F;
    const size_t per_traj = sizeof(double) * (size_t)n_steps * K * M;
    size_t free_b = 0, total_b = 0;
    SSS_CUDA(cudaMemGetInfo(&free_b, &total_b));
    const size_t budget = p->adj_max_bytes ? p->adj_max_bytes : free_b / 2;
    if (per_traj > budget) return fail(SSS_EINVAL, "adjoint states of one trajectory exceed memory");
    const int chunk = (int)std::min<size_t>((size_t)ntraj, budget / per_traj);

    // ---- the forward pass on the power series where that layout fits (its
    // rows in its own order, which the backward passes read the states in):
    // the row-part forward of 256 pulse shapes takes as many dependent Horner
    // terms as a sweep, and every exponential's state is stored either way ----
    BatchLayout FL;
    if (p->batch_variant == 0 || p->batch_variant == 8) {
        struct Flag {
            sss_plan* p;
            int variant;
            explicit Flag(sss_plan* q) : p(q), variant(q->batch_variant) {
                p->adj_forward = true;
                p->batch_variant = 0;
            }
            ~Flag() {
                p->adj_forward = false;
                p->batch_variant = variant;
            }
        } flag(p);
        const int rc = build_layout(p, ntraj, d_rho0, nch, nseg, d_prog, dt, F, {gd}, true, &FL, st);
        if (rc == SSS_OK && FL.power && FL.M == M) {
            Ly.newpos = FL.newpos;
            Ly.row_orig = FL.row_orig;
        } else if (rc != SSS_OK && rc != SSS_EINVAL) {
            return rc;
        } else {
            FL = BatchLayout();
            set_error("");
        }
    }
    const BatchLayout& forward = FL.power ? FL : Ly;

    // ---- the slot-programmed backward, where the block series fits ----
    if (p->batch_variant != 4 && p->batch_variant != 5 && Ly.degree <= kMaxTaylor) {
        AdjSlotArgs sa{};
        BatchLayout BL;
        size_t smem = 0;
        int threads = 0;
        const int rc = adjoint_slots_prepare(p, Ly, ntraj, gd, xg, t0, dt, T, F, nch, nseg, h_rw,
                                             h_tw, dch, npar, &sa, &BL, &smem, &threads, st);
        if (rc == SSS_OK) {
            PartsForward fw;
            if (int rc2 = parts_forward_prepare(p, forward, ntraj, nch, nseg, dt, F, h_rw, {gd},
                                                p->w_adjf, &fw, st))
                return rc2;
            if (int rc2 = p->w_states.ensure(per_traj * chunk)) return rc2;
            if (int rc2 = p->w_adjro.ensure(sizeof(double) * (size_t)chunk * T)) return rc2;
            if (int rc2 = p->w_adjst.ensure(sizeof(double) * (size_t)chunk * N)) return rc2;
            if (int rc2 = p->w_queue.ensure(sizeof(int) * 4)) return rc2;
            SSS_CUDA(cudaMemsetAsync(d_J, 0, sizeof(double) * ntraj, st));
            SSS_CUDA(cudaMemsetAsync(d_grad, 0, sizeof(double) * (size_t)ntraj * nseg * npar, st));
            if (!p->ev_begin) {
                SSS_CUDA(cudaEventCreate(&p->ev_begin));
                SSS_CUDA(cudaEventCreate(&p->ev_end));
            }
            SSS_CUDA(cudaEventRecord(p->ev_begin, st));
            int launches = 0;
            for (int b0 = 0; b0 < ntraj; b0 += chunk) {
                const int nb = std::min(chunk, ntraj - b0);
                double* state = p->w_adjst.as<double>();
                const double* prog = d_prog + (size_t)b0 * nch * nseg * 5;
                SSS_CUDA(cudaMemcpyAsync(state, d_rho0 + (size_t)b0 * N, sizeof(double) * (size_t)nb * N,
                                         cudaMemcpyDeviceToDevice, st));
                if (int rc2 = parts_forward_launch(p, fw, nb, state, prog, t0, T, p->w_adjro.as<double>(),
                                                   p->w_states.as<double>(), st))
                    return rc2;
                AdjSlotArgs ab = sa;
                ab.ntraj = nb;
                ab.states = p->w_states.as<double>();
                ab.readout = p->w_adjro.as<double>();
                ab.prog = prog;
                ab.J = d_J + b0;
                ab.grad = d_grad + (size_t)b0 * nseg * npar;
                ab.queue = p->w_queue.as<int>();
                SSS_CUDA(cudaMemsetAsync(ab.queue, 0, sizeof(int), st));
                if (int rc2 = launch_adjoint_slots(p, BL.L, BL.phased, BL.shape, BL.S, ab, threads, smem, st))
                    return rc2;
                launches += 2;
            }
            SSS_CUDA(cudaEventRecord(p->ev_end, st));
            p->ev_recorded = true;
            p->last_launches = launches;
            p->last_batch_lanes = BL.L;
            p->last_degree = Ly.degree;
            p->last_substeps = 1;
            p->last_rows = M;
            p->last_nnz = (int)Ly.nnz;
            p->last_variant = BL.phased ? 7 : 6;
            return SSS_OK;
        }
        if (rc != SSS_EINVAL) return rc;
        set_error("");
    }

    // ---- backward layout: the transposed pattern, x-generator entries first ----
    std::vector<int> rows_reached(M);
    for (int i = 0; i < M; i++) rows_reached[i] = Ly.row_orig[Ly.newpos[i]];
    const SparseGenerators& sp = p->sparse;
    std::vector<std::vector<BatchLayout::Ent>> rowsT(M);
    std::vector<std::vector<char>> prioT(M);
    for (int i = 0; i < M; i++)
        for (const BatchLayout::Ent& en : Ly.row_ents[i]) {
            rowsT[en.col].push_back({i, en.q});
            prioT[en.col].push_back(sp.val[(size_t)gd * sp.nnz + en.q] != 0.0);
        }
    BatchLayout TL;
    // lanes of the backward groups: the narrowest that fits and gives every
    // SM sub-partition a warp, else the widest that fits (no wider than twice
    // the 4-entry parts); one trajectory per CTA above 32 lanes
    int Lb = 0, ngx = 0;
    {
        long parts4 = 0;
        for (const auto& re : rowsT) parts4 += std::max<long>(1, ((long)re.size() + 3) / 4);
        for (int Lc : {16, 32, 64, 128, 256}) {
            if (p->batch_lanes > 0 && Lc != p->batch_lanes) continue;  // configured lanes
            if (Lb && Lc > 2 * parts4) break;
            BatchLayout trial;
            if (parts_layout_rows(p, rowsT, prioT, Lc, Lc > 32 ? Lc : 32, 3, 2, Ly.active,
                                  rows_reached, &trial, nullptr) != SSS_OK)
                continue;
            Lb = Lc;
            if ((long)ntraj * Lc >= 4L * 32 * p->num_sms) break;
        }
        if (!Lb) return fail(SSS_EINVAL, "the transposed pattern fits no row-part shape");
    }
    const int threads = Lb > 32 ? Lb : 32;
    if (int rc = parts_layout_rows(p, rowsT, prioT, Lb, threads, 3, 2, Ly.active, rows_reached, &TL, &ngx))
        return rc;
    const int CP = TL.C * TL.P;

    // ---- forward tables (the differentiated channel kept live) ----
    PartsForward fw;
    if (int rc = parts_forward_prepare(p, forward, ntraj, nch, nseg, dt, F, h_rw, {gd}, p->w_adjf, &fw, st))
        return rc;

    // ---- backward tables ----
    const double h = dt / F;
    std::vector<int> live;
    std::vector<double> om0((size_t)K * CP * Lb, 0.0);
    for (int gi = 0; gi < Ga; gi++) {
        const int g = Ly.active[gi];
        if (g != 0 && (g == gd || !Ly.chan_const[g])) {
            live.push_back(gi);
            continue;
        }
        const double X = g == 0 ? 1.0 : Ly.chan_value[g];
        for (int e = 0; e < K; e++) {
            double s = 0.0;
            for (int k = 0; k < Q; k++) s = std::fma(p->W[e * Q + k], X, s);
            const double ag = s * h;
            for (int i = 0; i < CP * Lb; i++) {
                double& o = om0[(size_t)e * CP * Lb + i];
                o = std::fma(ag, TL.gv[(size_t)gi * CP * Lb + i], o);
            }
        }
    }
    int x_live = -1;
    for (size_t i = 0; i < live.size(); i++)
        if (live[i] == xg) x_live = (int)i;
    std::vector<double> rwb(M, 0.0), tw(h_tw, h_tw + T), toff(F), noff(Q);
    for (int k = 0; k < M; k++) rwb[k] = h_rw ? h_rw[TL.row_orig[k]] : 0.0;
    for (int r = 0; r < F; r++) toff[r] = ((double)r * dt) / F;
    for (int k = 0; k < Q; k++) noff[k] = (dt * p->nodes[k]) / F;
    std::vector<int> fwdpos(M), rbeg(Lb + 1, 0);
    for (int i = 0; i < M; i++) fwdpos[TL.newpos[i]] = Ly.newpos[i];
    for (int l = 0; l < Lb; l++) rbeg[l + 1] = rbeg[l] + (int)TL.lane_of[l].size();
    // blob: gv | gx | om0 | rw | tw | toff | noff | pcol | cw | rbeg | fwdpos
    std::vector<double> dbl(TL.gv);
    const size_t o_gx = dbl.size();
    dbl.insert(dbl.end(), TL.gv.begin() + (size_t)xg * CP * Lb, TL.gv.begin() + (size_t)(xg + 1) * CP * Lb);
    const size_t o_om0 = dbl.size();
    dbl.insert(dbl.end(), om0.begin(), om0.end());
    const size_t o_rw = dbl.size();
    dbl.insert(dbl.end(), rwb.begin(), rwb.end());
    const size_t o_tw = dbl.size();
    dbl.insert(dbl.end(), tw.begin(), tw.end());
    const size_t o_toff = dbl.size();
    dbl.insert(dbl.end(), toff.begin(), toff.end());
    const size_t o_noff = dbl.size();
    dbl.insert(dbl.end(), noff.begin(), noff.end());
    std::vector<int> ints(TL.pcol);
    const size_t o_cw = ints.size();
    ints.insert(ints.end(), TL.cw.begin(), TL.cw.end());
    const size_t o_rbeg = ints.size();
    ints.insert(ints.end(), rbeg.begin(), rbeg.end());
    const size_t o_fwd = ints.size();
    ints.insert(ints.end(), fwdpos.begin(), fwdpos.end());
    const size_t bytes = sizeof(double) * dbl.size() + sizeof(int) * ints.size();
    if (int rc = p->w_adjb.ensure(bytes + 64)) return rc;
    {
        std::vector<char> blob(bytes);
        memcpy(blob.data(), dbl.data(), sizeof(double) * dbl.size());
        memcpy(blob.data() + sizeof(double) * dbl.size(), ints.data(), sizeof(int) * ints.size());
        SSS_CUDA(cudaMemcpyAsync(p->w_adjb.p, blob.data(), bytes, cudaMemcpyHostToDevice, st));
        SSS_CUDA(cudaStreamSynchronize(st));  // the host blob goes out of scope
    }
    const double* dv = p->w_adjb.as<double>();
    const int* di = reinterpret_cast<const int*>(dv + dbl.size());

    AdjPartsArgs a{};
    a.M = M; a.K = K; a.Q = Q; a.F = F; a.nch = nch; a.nseg = nseg; a.degree = Ly.degree; a.T = T;
    a.n_steps = n_steps; a.h = h; a.t0 = t0; a.dt = dt;
    a.n_live = (int)live.size();
    a.x_live = x_live;
    a.dch = dch;
    a.npar = npar;
    a.kc = TL.kc;
    a.ngx = ngx;
    for (size_t i = 0; i < live.size(); i++) a.live[i] = live[i];
    for (int gi = 0; gi < Ga; gi++) a.gen_index[gi] = Ly.active[gi];
    a.gv = dv;
    a.gx = dv + o_gx;
    a.om0 = dv + o_om0;
    a.rw = dv + o_rw;
    a.tw = dv + o_tw;
    a.toff = dv + o_toff;
    a.noff = dv + o_noff;
    a.pcol = di;
    a.cw = reinterpret_cast<const unsigned*>(di + o_cw);
    a.rbeg = di + o_rbeg;
    a.fwdpos = di + o_fwd;
    a.W = p->d_gens.as<double>() + p->gens.size();
    for (int j = 0; j <= kAdjMaxTaylor; j++) a.inv_j[j] = j ? 1.0 / j : 0.0;
    const size_t smem = sizeof(double) *
        (((6 * (size_t)(M + 2) + 2 * (size_t)(Lb * TL.C + 1) +
           (size_t)kRing * (Q * live.size() + K * live.size() + 4 * Q)) | 1) * (threads / Lb) + M);
    if (smem > 227 * 1024) return fail(SSS_EINVAL, "adjoint kernel: shared memory per CTA too large");

    // ---- buffers and chunks ----
    if (int rc = p->w_states.ensure(per_traj * chunk)) return rc;
    if (int rc = p->w_adjro.ensure(sizeof(double) * (size_t)chunk * T)) return rc;
    if (int rc = p->w_adjst.ensure(sizeof(double) * (size_t)chunk * N)) return rc;
    if (int rc = p->w_queue.ensure(sizeof(int) * 4)) return rc;
    SSS_CUDA(cudaMemsetAsync(d_J, 0, sizeof(double) * ntraj, st));
    SSS_CUDA(cudaMemsetAsync(d_grad, 0, sizeof(double) * (size_t)ntraj * nseg * npar, st));
    if (!p->ev_begin) {
        SSS_CUDA(cudaEventCreate(&p->ev_begin));
        SSS_CUDA(cudaEventCreate(&p->ev_end));
    }
    SSS_CUDA(cudaEventRecord(p->ev_begin, st));
    int launches = 0;
    for (int b0 = 0; b0 < ntraj; b0 += chunk) {
        const int nb = std::min(chunk, ntraj - b0);
        double* state = p->w_adjst.as<double>();
        const double* prog = d_prog + (size_t)b0 * nch * nseg * 5;
        SSS_CUDA(cudaMemcpyAsync(state, d_rho0 + (size_t)b0 * N, sizeof(double) * (size_t)nb * N,
                                 cudaMemcpyDeviceToDevice, st));
        if (int rc = parts_forward_launch(p, fw, nb, state, prog, t0, T, p->w_adjro.as<double>(),
                                          p->w_states.as<double>(), st))
            return rc;
        AdjPartsArgs ab = a;
        ab.ntraj = nb;
        ab.states = p->w_states.as<double>();
        ab.readout = p->w_adjro.as<double>();
        ab.prog = prog;
        ab.J = d_J + b0;
        ab.grad = d_grad + (size_t)b0 * nseg * npar;
        ab.queue = p->w_queue.as<int>();
        SSS_CUDA(cudaMemsetAsync(ab.queue, 0, sizeof(int), st));
        int rc;
        switch (Lb) {
            case 16: rc = launch_adj_parts<16>(p, TL.C, TL.P, ab, threads, smem, st); break;
            case 32: rc = launch_adj_parts<32>(p, TL.C, TL.P, ab, threads, smem, st); break;
            case 64: rc = launch_adj_parts<64>(p, TL.C, TL.P, ab, threads, smem, st); break;
            case 128: rc = launch_adj_parts<128>(p, TL.C, TL.P, ab, threads, smem, st); break;
            default: rc = launch_adj_parts<256>(p, TL.C, TL.P, ab, threads, smem, st); break;
        }
        if (rc) return rc;
        launches += 2;
    }
    SSS_CUDA(cudaEventRecord(p->ev_end, st));
    p->ev_recorded = true;
    p->last_launches = launches;
    p->last_batch_lanes = Lb;
    p->last_degree = Ly.degree;
    p->last_substeps = 1;
    p->last_rows = M;
    p->last_nnz = (int)Ly.nnz;
    p->last_variant = 4;
    return SSS_OK;
}

}  // namespace

int adjoint_run(sss_plan* p, int ntraj, const double* d_rho0, int nch, int nseg,
                const double* d_prog, double t0, double dt, int T, int F, const double* h_rw,
                const double* h_tw, int dch, int npar, double* d_J, double* d_grad,
                cudaStream_t st) {
    if (dch < 0 || dch >= nch || dch + 1 >= p->d.G)
        return fail(SSS_EINVAL, "the differentiated channel must be a program channel with a "
                                "generator (0 <= channel < nch, channel + 1 < G)");
    if (npar != 2 && npar != 4) return fail(SSS_EINVAL, "parameters per segment must be 2 or 4");
    if (p->batch_variant == 0 || p->batch_variant == 4 || p->batch_variant == 5 || p->batch_variant == 8) {
        const int rc = adjoint_run_parts(p, ntraj, d_rho0, nch, nseg, d_prog, t0, dt, T, F, h_rw,
                                         h_tw, dch, npar, d_J, d_grad, st);
        if (rc != SSS_EINVAL || p->batch_variant == 4 || p->batch_variant == 5) return rc;
        set_error("");
    }
    const int N = p->d.N, K = p->d.K, Q = p->d.Q;
    const int gd = dch + 1;
    BatchLayout Ly;
    if (int rc = build_layout(p, ntraj, d_rho0, nch, nseg, d_prog, dt, F, {gd}, false, &Ly, st))
        return rc;
    SSS_CUDA(cudaMemsetAsync(d_J, 0, sizeof(double) * ntraj, st));
    SSS_CUDA(cudaMemsetAsync(d_grad, 0, sizeof(double) * (size_t)ntraj * nseg * npar, st));
    if (Ly.M == 0) return SSS_OK;
    if (Ly.substeps != 1)
        return fail(SSS_EINVAL, "the adjoint needs one sub-step per exponential (use a smaller dt/F)");
    int xg = -1;
    for (int gi = 0; gi < Ly.Ga; gi++)
        if (Ly.active[gi] == gd) xg = gi;
    if (xg < 0)
        return fail(SSS_EINVAL, "the generator of channel " + std::to_string(dch) +
                                    " is zero on the reachable rows");
    const int M = Ly.M, L = Ly.L, E = Ly.E, d = Ly.degree;
    if (d > kAdjMaxTaylor) return fail(SSS_EINVAL, "Taylor degree too large for the adjoint");
    // lane row ranges (lane order) and owner of each row
    std::vector<int> rbeg(L + 1, 0), owner(M, 0);
    for (int l = 0; l < L; l++) rbeg[l + 1] = rbeg[l] + (int)Ly.lane_of[l].size();
    for (int l = 0; l < L; l++)
        for (int k = rbeg[l]; k < rbeg[l + 1]; k++) owner[k] = l;
    // transposed entries: for each forward entry (row r, col c) at Om index
    // e*L + l, an entry (row c, col r) of the owner of c
    std::vector<std::vector<std::pair<int, std::pair<int, int>>>> trows(M);  // row c -> (col r, q)
    for (int l = 0; l < L; l++) {
        int e = 0;
        for (int i : Ly.lane_of[l]) {
            const auto& ents = Ly.row_ents[i];
            int n = std::max<int>(1, (int)ents.size());
            for (int j = 0; j < (int)ents.size(); j++) {
                int r = Ly.newpos[i], c = Ly.newpos[ents[j].col];
                trows[c].push_back({r, {e + j, l}});
            }
            e += n;
        }
    }
    std::vector<int> tcnt(L, 0);
    for (int l = 0; l < L; l++)
        for (int k = rbeg[l]; k < rbeg[l + 1]; k++) tcnt[l] += std::max<int>(1, (int)trows[k].size());
    const int ET = *std::max_element(tcnt.begin(), tcnt.end());
    std::vector<unsigned> tent((size_t)ET * L, 0u);
    std::vector<int> tidx((size_t)ET * L, -1);
    for (int l = 0; l < L; l++) {
        int e = 0;
        for (int k = rbeg[l]; k < rbeg[l + 1]; k++) {
            auto& lst = trows[k];
            std::sort(lst.begin(), lst.end());
            int n = std::max<int>(1, (int)lst.size());
            for (int j = 0; j < n; j++) {
                unsigned w = j < (int)lst.size() ? (unsigned)lst[j].first : (unsigned)k;
                if (j == n - 1) w |= (unsigned)(k + 1) << 16;
                tent[(size_t)(e + j) * L + l] = w;
                if (j < (int)lst.size()) {
                    const int fe = lst[j].second.first, fl = lst[j].second.second;
                    int q = fe * L + fl;
                    if (Ly.gv[((size_t)xg * E + fe) * L + fl] != 0.0) q |= kHasG;
                    tidx[(size_t)(e + j) * L + l] = q;
                }
            }
            e += n;
        }
    }
    const long n_steps = (long)T * F;
    int C = (int)std::ceil(std::sqrt((double)n_steps));
    C = std::max(C, 1);
    const int n_ck = (int)((n_steps + C - 1) / C);
    std::vector<double> rw(M, 0.0), tw(h_tw, h_tw + T);
    for (int k = 0; k < M; k++) rw[k] = h_rw ? h_rw[Ly.row_orig[k]] : 0.0;
    std::vector<double> toff(F), noff(Q);
    for (int r = 0; r < F; r++) toff[r] = ((double)r * dt) / F;
    for (int k = 0; k < Q; k++) noff[k] = (dt * p->nodes[k]) / F;
    // device blob: gv | rw | tw | toff | noff | ent | tent | tidx | cnt | tcnt | rbeg | row_orig
    std::vector<double> dbl(Ly.gv);
    const size_t o_rw = dbl.size();
    dbl.insert(dbl.end(), rw.begin(), rw.end());
    const size_t o_tw = dbl.size();
    dbl.insert(dbl.end(), tw.begin(), tw.end());
    const size_t o_toff = dbl.size();
    dbl.insert(dbl.end(), toff.begin(), toff.end());
    const size_t o_noff = dbl.size();
    dbl.insert(dbl.end(), noff.begin(), noff.end());
    std::vector<int> ints;
    auto put = [&](const int* b, size_t n) {
        size_t o = ints.size();
        ints.insert(ints.end(), b, b + n);
        return o;
    };
    const size_t o_ent = put(reinterpret_cast<const int*>(Ly.words.data()), Ly.words.size());
    const size_t o_tent = put(reinterpret_cast<const int*>(tent.data()), tent.size());
    const size_t o_tidx = put(tidx.data(), tidx.size());
    const size_t o_cnt = put(Ly.cnt.data(), Ly.cnt.size());
    const size_t o_tcnt = put(tcnt.data(), tcnt.size());
    const size_t o_rbeg = put(rbeg.data(), rbeg.size());
    const size_t o_rorig = put(Ly.row_orig.data(), Ly.row_orig.size());
    const size_t bytes = sizeof(double) * dbl.size() + sizeof(int) * ints.size();
    if (int rc = p->w_aux.ensure(bytes + 64)) return rc;
    std::vector<char> blob(bytes);
    memcpy(blob.data(), dbl.data(), sizeof(double) * dbl.size());
    memcpy(blob.data() + sizeof(double) * dbl.size(), ints.data(), sizeof(int) * ints.size());
    SSS_CUDA(cudaMemcpyAsync(p->w_aux.p, blob.data(), bytes, cudaMemcpyHostToDevice, st));
    const double* dv = p->w_aux.as<double>();
    const int* di = reinterpret_cast<const int*>(dv + dbl.size());

    const int threads = p->batch_threads > 0 ? p->batch_threads : 64;
    if (threads % L) return fail(SSS_EINVAL, "CTA size must be a multiple of the lanes per trajectory");
    const int slots_per_cta = threads / L;
    const size_t shared_words = (size_t)Ly.Ga * E * L + M + ((size_t)E * L + 2 * (size_t)ET * L + 1) / 2;
    const size_t per_slot = ((size_t)E * L + 7 * (size_t)M + kMaxQ * kMaxG + 4 * kMaxQ) | 1;
    const size_t smem = sizeof(double) * (shared_words + slots_per_cta * per_slot);
    if (smem > 227 * 1024) return fail(SSS_EINVAL, "adjoint kernel: shared memory per CTA too large");
    int grid = std::max(1, (ntraj + slots_per_cta - 1) / slots_per_cta);
    grid = std::min(grid, p->num_sms * 8);
    const long slots = (long)grid * slots_per_cta;
    const size_t scratch = sizeof(double) * (size_t)slots * ((size_t)n_ck * M + (size_t)C * K * M);
    if (int rc = p->w_prop.ensure(scratch)) return rc;
    if (int rc = p->w_queue.ensure(sizeof(int) * 4)) return rc;
    SSS_CUDA(cudaMemsetAsync(p->w_queue.p, 0, sizeof(int) * 4, st));

    AdjArgs a{};
    a.M = M; a.Ga = Ly.Ga; a.K = K; a.Q = Q; a.F = F; a.nch = nch; a.nseg = nseg;
    a.ntraj = ntraj; a.degree = d; a.N = N; a.E = E; a.ET = ET; a.xg = xg;
    a.dch = dch; a.npar = npar;
    a.n_steps = n_steps; a.T = T; a.C = C; a.n_ck = n_ck;
    a.h = dt / F; a.t0 = t0; a.dt = dt;
    for (int gi = 0; gi < Ly.Ga; gi++) a.gen_index[gi] = Ly.active[gi];
    a.toff = dv + o_toff;
    a.noff = dv + o_noff;
    a.W = p->d_gens.as<double>() + p->gens.size();
    a.gv = dv;
    a.rw = dv + o_rw;
    a.tw = dv + o_tw;
    a.ent = reinterpret_cast<const unsigned*>(di + o_ent);
    a.tent = reinterpret_cast<const unsigned*>(di + o_tent);
    a.tidx = di + o_tidx;
    a.cnt = di + o_cnt;
    a.tcnt = di + o_tcnt;
    a.rbeg = di + o_rbeg;
    a.row_orig = di + o_rorig;
    a.rho0 = d_rho0;
    a.prog = d_prog;
    a.J = d_J;
    a.grad = d_grad;
    a.ck = p->w_prop.as<double>();
    a.st = a.ck + (size_t)slots * n_ck * M;
    a.queue = p->w_queue.as<int>();
    double f = 1.0;
    for (int j = 0; j < kAdjMaxTaylor + 2; j++) {
        if (j > 0) f /= j;
        a.fact_inv[j] = f;
    }
    for (int j = 0; j <= kAdjMaxTaylor; j++) a.inv_j[j] = j ? 1.0 / j : 0.0;
    if (!p->ev_begin) {
        SSS_CUDA(cudaEventCreate(&p->ev_begin));
        SSS_CUDA(cudaEventCreate(&p->ev_end));
    }
    SSS_CUDA(cudaEventRecord(p->ev_begin, st));
    int rc;
    switch (L) {
        case 1: rc = launch_adj<1>(p, a, threads, smem, grid, st); break;
        case 2: rc = launch_adj<2>(p, a, threads, smem, grid, st); break;
        case 4: rc = launch_adj<4>(p, a, threads, smem, grid, st); break;
        case 8: rc = launch_adj<8>(p, a, threads, smem, grid, st); break;
        case 16: rc = launch_adj<16>(p, a, threads, smem, grid, st); break;
        default: rc = launch_adj<32>(p, a, threads, smem, grid, st); break;
    }
    if (rc) return rc;
    SSS_CUDA(cudaEventRecord(p->ev_end, st));
    p->ev_recorded = true;
    p->last_launches = 1;
    p->last_batch_lanes = L;
    p->last_degree = d;
    p->last_substeps = 1;
    p->last_rows = M;
    p->last_nnz = (int)Ly.nnz;
    return SSS_OK;
}

}  // namespace sss
