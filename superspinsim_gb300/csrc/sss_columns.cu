// Drop-in runs from host buffers by propagator columns (reference
// superspinsim/generate_simulator.py:1954-2038: the fine-step loop, the chain
// and the frame sandwich).
//
// The reference builds the propagator of every output sample, all samples in
// parallel, and chains them.  A propagator's column c is the trajectory that
// starts from the unit vector e_c, so the batched kernels build it: column c
// of a run of samples is one of their trajectories (BatchArgs::cols), on the
// rows reachable from the initial state and the generators' non-zeros, with
// the Taylor action or the power series in place of dense matrix products.
// For the 7-level NV 19 columns of 19 rows take about 20 kFLOP per step, the
// dense 49 x 49 products of k_step_propagators 3.3 MFLOP (500 samples of 200
// steps: 340.8 ms there).  Columns are kept in residual form (minus their unit
// vector), as the dense path keeps propagators.
//
// The chain over T samples, serial, would take 0.5 us a sample; it runs over
// blocks of kBlock samples instead (product of each block's propagators, all
// blocks in parallel; chain over the blocks; states inside each block, all
// blocks in parallel).
//
// sss_simulate comes here for plans with the Taylor exponential; plans with
// the reference's own exponential, unitary mode, sss_simulate_device (which
// must not read its inputs on the host) and what no layout fits keep the
// dense path.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "sss_batch_args.cuh"
#include "sss_device.cuh"
#include "sss_internal.cuh"

namespace sss {

int batch_columns_args(sss_plan* p, const BatchLayout& Ly, int ntraj, int nch, int nseg, double dt, int F,
                       DevBuf& tables, BatchArgs* a, size_t* smem, cudaStream_t st);
int batch_columns_launch(sss_plan* p, const BatchLayout& Ly, const BatchArgs& a, size_t smem, cudaStream_t st);

namespace {

constexpr int kBlock = kColBlock;   // runs per block of the chain
constexpr int kSmallSamples = 32, kSmallExps = 5;   // samples and exponentials per sample of a small call
constexpr int kMaxTerms = 256;      // Taylor terms per exponential (dense products cost about 400)
constexpr int kLanesPerRow = 8;     // lanes of a matrix row in the chain kernels

struct ChainArgs {
    int M, N, n_full, T, len, t_begin;   // samples in this chunk, per run; global first sample
    const double* prop;                  // [trajectory][sample][column][row], minus the identity
    const int* row_orig;
    const double* rho0;                  // ntraj * (n_full or N)
    const double *V, *Vinv, *P;
    double* state;                       // ntraj * 2M: the state at the chunk's first sample, low part
    double* block;                       // ntraj * blocks * M * M: block products minus the identity
    double* vstart;                      // ntraj * blocks * 2M: the state at each block's first sample and
                                         // its low part
    double* y;                           // ntraj * T * M: states (V or P given), else unused
    double* out;                         // ntraj * T_all * (n_full or N), sample t_begin on
    int T_all;
};

// the state vector x0 = P^T rho0 (or rho0), in the eigenbasis where there is
// one, on the kept rows: run by one CTA
__device__ void initial_rows(const ChainArgs& a, int b, double* x0, double* v) {
    const int nio = a.P ? a.n_full : a.N;
    for (int i = threadIdx.x; i < a.N; i += blockDim.x) {
        double acc = 0.0;
        if (a.P)
            for (int k = 0; k < a.n_full; k++)
                acc = fma(a.P[(size_t)k * a.N + i], a.rho0[(size_t)b * nio + k], acc);
        else
            acc = a.rho0[(size_t)b * nio + i];
        x0[i] = acc;
    }
    __syncthreads();
    for (int r = threadIdx.x; r < a.M; r += blockDim.x) {
        const int i = a.row_orig[r];
        double acc = x0[i];
        if (a.Vinv) {
            acc = 0.0;
            for (int k = 0; k < a.N; k++) acc = fma(a.Vinv[(size_t)i * a.N + k], x0[k], acc);
        }
        v[r] = acc;
    }
    __syncthreads();
}

__device__ __forceinline__ bool ends_run(const ChainArgs& a, int t) {
    return (t + 1) % a.len == 0 || t + 1 == a.T;
}

// R <- (I + S)(I + R) - I over the runs of a block: one CTA per (block, trajectory)
__global__ void __launch_bounds__(256) k_block_product(const ChainArgs a) {
    extern __shared__ double sm[];
    const int M = a.M, MM = M * M, b = blockIdx.y, nb = gridDim.x;
    double *R = sm, *Q = sm + MM, *S = Q + MM;
    const int t0 = blockIdx.x * kBlock * a.len, t1 = min(a.T, t0 + kBlock * a.len);
    bool first = true;
    for (int t = t0; t < t1; t++) {
        if (!ends_run(a, t)) continue;
        const double* St = a.prop + ((size_t)b * a.T + t) * MM;   // [column][row]
        if (first) {
            for (int i = threadIdx.x; i < MM; i += blockDim.x) R[i] = St[i];
            first = false;
            __syncthreads();
            continue;
        }
        for (int i = threadIdx.x; i < MM; i += blockDim.x) S[i] = St[i];
        __syncthreads();
        for (int i = threadIdx.x; i < MM; i += blockDim.x) {
            const int c = i / M, r = i - c * M;
            double acc = S[i] + R[i];
            for (int k = 0; k < M; k++) acc = fma(S[k * M + r], R[c * M + k], acc);
            Q[i] = acc;
        }
        __syncthreads();
        double* tmp = R;
        R = Q;
        Q = tmp;
    }
    double* dst = a.block + ((size_t)b * nb + blockIdx.x) * MM;
    for (int i = threadIdx.x; i < MM; i += blockDim.x) dst[i] = R[i];
}

// d = S v for S [column][row] in global memory, kLanesPerRow lanes per row;
// every lane of a row returns d
__device__ __forceinline__ double row_product(const double* S, const double* v, int M, int row, int sub,
                                              bool own) {
    double d = 0.0;
    if (own)
        for (int c = sub; c < M; c += kLanesPerRow) d = fma(__ldg(S + (size_t)c * M + row), v[c], d);
#pragma unroll
    for (int o = kLanesPerRow / 2; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
    return d;
}

// hi + lo <- hi + lo + d: the states keep their low part through the chain, so
// a sample's state is rounded once, as the dense path's serial chain rounds it
// once a sample
__device__ __forceinline__ void add_low(double& hi, double& lo, double d) {
    const double x = d + lo, s = hi + x, z = s - hi;
    lo = (hi - (s - z)) + (x - z);
    hi = s;
}

// the state at every block's first sample (more: and past the last block):
// one CTA per trajectory
__global__ void __launch_bounds__(512) k_block_chain(const ChainArgs a, int blocks, int more) {
    __shared__ double v[kPlainMaxN], x0[kPlainMaxN];
    const int M = a.M, b = blockIdx.x;
    const int row = threadIdx.x / kLanesPerRow, sub = threadIdx.x % kLanesPerRow;
    const bool own = row < M;
    if (a.t_begin == 0) {
        initial_rows(a, b, x0, v);
    } else {
        for (int r = threadIdx.x; r < M; r += blockDim.x) v[r] = a.state[(size_t)b * 2 * M + r];
        __syncthreads();
    }
    double mine = own ? v[row] : 0.0, low = own && a.t_begin ? a.state[((size_t)b * 2 + 1) * M + row] : 0.0;
    for (int k = 0; k < blocks; k++) {
        if (own && sub == 0) {
            double* o = a.vstart + ((size_t)b * blocks + k) * 2 * M + row;
            o[0] = mine;
            o[M] = low;
        }
        if (k + 1 == blocks && !more) break;
        const double d = row_product(a.block + ((size_t)b * blocks + k) * M * M, v, M, row, sub, own);
        add_low(mine, low, d);
        __syncthreads();
        if (own && sub == 0) v[row] = mine;
        __syncthreads();
    }
    if (own && sub == 0) {
        a.state[(size_t)b * 2 * M + row] = mine;
        a.state[((size_t)b * 2 + 1) * M + row] = low;
    }
}

// every sample's state inside a block, from the block's first: one CTA per
// (block, trajectory).  Lab frame without a projection: written to the output
// (rows outside the kept ones are zero); else to y for k_lab_states.
__global__ void __launch_bounds__(512) k_block_states(const ChainArgs a, int blocks) {
    __shared__ double v[kPlainMaxN];
    __shared__ int pos[kPlainMaxN];
    const int M = a.M, b = blockIdx.y, k = blockIdx.x;
    const int row = threadIdx.x / kLanesPerRow, sub = threadIdx.x % kLanesPerRow;
    const bool own = row < M, direct = !a.V && !a.P;
    for (int i = threadIdx.x; i < a.N; i += blockDim.x) pos[i] = -1;
    __syncthreads();
    for (int r = threadIdx.x; r < M; r += blockDim.x) {
        v[r] = a.vstart[((size_t)b * blocks + k) * 2 * M + r];
        pos[a.row_orig[r]] = r;
    }
    __syncthreads();
    double mine = own ? v[row] : 0.0, low = own ? a.vstart[((size_t)b * blocks + k) * 2 * M + M + row] : 0.0;
    const int orig = own ? a.row_orig[row] : 0;
    const int t0 = k * kBlock * a.len, t1 = min(a.T, t0 + kBlock * a.len);
    for (int t = t0; t < t1; t++) {
        double y = mine, ylow = low;
        add_low(y, ylow, row_product(a.prop + ((size_t)b * a.T + t) * M * M, v, M, row, sub, own));
        if (direct) {
            double* o = a.out + ((size_t)b * a.T_all + a.t_begin + t) * a.N;
            if (own && sub == 0) o[orig] = y;
            for (int i = threadIdx.x; i < a.N; i += blockDim.x)
                if (pos[i] < 0) o[i] = 0.0;
        } else if (own && sub == 0) {
            a.y[((size_t)b * a.T + t) * M + row] = y;
        }
        if (ends_run(a, t)) {
            mine = y;
            low = ylow;
            __syncthreads();
            if (own && sub == 0) v[row] = mine;
            __syncthreads();
        }
    }
}

// lab-basis states V y, and in the equivalence-class mode rho0 + P (V y - x0)
// (k_chain in sss_plain.cu): one CTA per (sample, trajectory)
__global__ void __launch_bounds__(64) k_lab_states(const ChainArgs a) {
    __shared__ double x0[kPlainMaxN], w[kPlainMaxN], ys[kPlainMaxN];
    const int b = blockIdx.y, t = blockIdx.x;
    const double* y = a.y + ((size_t)b * a.T + t) * a.M;
    if (threadIdx.x < a.M) ys[threadIdx.x] = y[threadIdx.x];
    if (threadIdx.x < a.N) w[threadIdx.x] = 0.0;
    __syncthreads();
    if (a.V) {
        if (threadIdx.x < a.N) {
            double o = 0.0;
            for (int r = 0; r < a.M; r++) o = fma(a.V[(size_t)threadIdx.x * a.N + a.row_orig[r]], ys[r], o);
            w[threadIdx.x] = o;
        }
    } else if (threadIdx.x < a.M) {
        w[a.row_orig[threadIdx.x]] = ys[threadIdx.x];
    }
    const int nio = a.P ? a.n_full : a.N;
    double* out = a.out + ((size_t)b * a.T_all + a.t_begin + t) * nio;
    if (!a.P) {
        if (threadIdx.x < a.N) out[threadIdx.x] = w[threadIdx.x];
        return;
    }
    if (threadIdx.x < a.N) {
        double acc = 0.0;
        for (int k = 0; k < a.n_full; k++)
            acc = fma(a.P[(size_t)k * a.N + threadIdx.x], a.rho0[(size_t)b * nio + k], acc);
        x0[threadIdx.x] = acc;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < a.n_full; i += blockDim.x) {
        double acc = a.rho0[(size_t)b * nio + i];
        for (int k = 0; k < a.N; k++) acc = fma(a.P[(size_t)i * a.N + k], w[k] - x0[k], acc);
        out[i] = acc;
    }
}

}  // namespace

int columns_run(sss_plan* p, int ntraj, const double* h_rho0, const double* d_rho0, int nch, int nseg,
                const double* h_prog, const double* d_prog, const double* d_tab, double t0, double dt,
                int T, int F, double* d_out, cudaStream_t st) {
    const int N = p->d.N;
    if (N > kPlainMaxN || p->u_n || p->d.expm != SSS_EXPM_TAYLOR || p->d.taylor_degree > 0)
        return fail(SSS_EINVAL, "not a run by columns");
    // and the smallest calls, whose host analysis takes longer than their dense
    // products (one trajectory, N = 4 to 9, columns against dense: F K = 1, 1 sample
    // 98 to 132 us against 48 to 60; F K = 5, 20 samples 118 to 161 against 98 to
    // 147; from F K = 10 on, or 40 samples in the rotating frame and 80 in the lab
    // frame, the columns are faster)
    if (ntraj == 1 && N <= 9 && T <= kSmallSamples && F * p->d.K <= kSmallExps)
        return fail(SSS_EINVAL, "a call too small for columns");
    // a coefficient that is not finite is the dense path's: it reports the NaN
    // that its generator makes of every state, also of the rows it does not move
    // (1e100: the cosine's argument then stays finite)
    for (size_t i = 0, n = h_prog ? (size_t)ntraj * nch * nseg * 5 : 0; i < n; i++)
        if (i % 5 && !(std::fabs(h_prog[i]) <= 1e100)) return fail(SSS_EINVAL, "a coefficient is not finite");
    // the plan's batched configuration and report stay as they are
    struct Saved {
        sss_plan* p;
        int lanes, threads, variant, bb, ba, nl, ln;
        double cost[kLaneCounts], chain[kLaneCounts];
        explicit Saved(sss_plan* q)
            : p(q), lanes(q->batch_lanes), threads(q->batch_threads), variant(q->batch_variant),
              bb(q->last_bank_before), ba(q->last_bank_after), nl(q->mk_n_live), ln(q->mk_live_nnz) {
            memcpy(cost, q->auto_cost, sizeof(cost));
            memcpy(chain, q->auto_chain, sizeof(chain));
            q->batch_lanes = q->batch_threads = q->batch_variant = 0;
            std::swap(q->w_queue, q->w_cols_queue);
        }
        ~Saved() {
            p->batch_lanes = lanes;
            p->batch_threads = threads;
            p->batch_variant = variant;
            p->last_bank_before = bb;
            p->last_bank_after = ba;
            p->mk_n_live = nl;
            p->mk_live_nnz = ln;
            memcpy(p->auto_cost, cost, sizeof(cost));
            memcpy(p->auto_chain, chain, sizeof(chain));
            std::swap(p->w_queue, p->w_cols_queue);
            p->cols_samples = 0;
            p->auto_lanes_ntraj = 0;
            p->host_rho0 = p->host_prog = nullptr;
        }
    } saved(p);
    p->cols_samples = (long)ntraj * T;
    p->host_rho0 = p->n_full ? nullptr : h_rho0;
    p->host_prog = h_prog;
    BatchLayout Ly;
    if (int rc = build_layout(p, ntraj, d_rho0, nch, nseg, d_prog, dt, F, {}, true, &Ly, st, false, d_tab, T))
        return rc;
    const int M = Ly.M;
    if (M == 0 || !(Ly.slots || Ly.power)) return fail(SSS_EINVAL, "no column layout");
    // an exponent so large that the Taylor action takes hundreds of terms (its
    // sub-steps end at 1,024) is the dense path's: scaling and squaring
    if (Ly.slots && (long)Ly.degree * Ly.substeps > kMaxTerms)
        return fail(SSS_EINVAL, "the exponent is too large for the Taylor action");
    BatchArgs a{};
    size_t smem = 0;
    if (int rc = batch_columns_args(p, Ly, ntraj, nch, nseg, dt, F, p->w_cols_tables, &a, &smem, st)) return rc;
    // launches of whole blocks of samples, or of whole trajectories
    const int len = p->cols.len, step = kBlock * len, Tc = std::min(T, p->cols.samples), nb = p->cols.traj;
    const size_t per_sample = sizeof(double) * (size_t)M * M;
    const int blocks_c = (Tc + step - 1) / step;
    const bool direct = !p->rotating && !p->n_full;
    if (int rc = p->w_prop.ensure(per_sample * Tc * nb)) return rc;
    const size_t n_state = (size_t)nb * 2 * M, n_block = (size_t)nb * blocks_c * M * M,
                 n_vs = (size_t)nb * blocks_c * 2 * M, n_y = direct ? 0 : (size_t)nb * Tc * M;
    if (int rc = p->w_aux.ensure(sizeof(double) * (n_state + n_block + n_vs + n_y))) return rc;
    ChainArgs c{};
    c.M = M;
    c.N = N;
    c.n_full = p->n_full;
    c.len = len;
    c.prop = p->w_prop.as<double>();
    c.row_orig = a.row_orig;
    c.V = p->rotating ? p->d_V.as<double>() : nullptr;
    c.Vinv = p->rotating ? p->d_Vinv.as<double>() : nullptr;
    c.P = p->n_full ? p->d_P.as<double>() : nullptr;
    c.state = p->w_aux.as<double>();
    c.block = c.state + n_state;
    c.vstart = c.block + n_block;
    c.y = c.vstart + n_vs;
    c.T_all = T;
    const int nio = p->state_in();
    const int threads = (M * kLanesPerRow + 31) / 32 * 32;
    const size_t psmem = 3 * per_sample;
    if (int rc = allow_smem(k_block_product)) return rc;
    int launches = 0;
    for (int b = 0; b < ntraj; b += nb) {
        const int n = std::min(nb, ntraj - b);
        for (int t = 0; t < T; t += Tc) {
            const int Tn = std::min(Tc, T - t), runs = (Tn + len - 1) / len, blocks = (Tn + step - 1) / step;
            a.cols = M;
            a.col_len = len;
            a.col_runs = runs;
            a.ntraj = n * runs * M;
            a.t_begin = t;
            a.t_end = t + Tn;
            a.T_max = T;
            a.t0 = t0;
            a.prog = d_prog ? d_prog + (size_t)b * nch * nseg * 5 : nullptr;
            a.tab = d_tab ? d_tab + (size_t)b * F * T * p->d.Q * p->d.G : nullptr;
            a.prop = p->w_prop.as<double>();
            SSS_CUDA(cudaMemsetAsync(a.queue, 0, sizeof(int), st));
            if (int rc = batch_columns_launch(p, Ly, a, smem, st)) return rc;
            c.T = Tn;
            c.t_begin = t;
            c.rho0 = d_rho0 + (size_t)b * nio;
            c.out = d_out + (size_t)b * T * nio;
            const int more = t + Tn < T;
            if (blocks > 1 || more) {
                k_block_product<<<dim3(blocks, n), 256, psmem, st>>>(c);
                launches++;
            }
            k_block_chain<<<n, threads, 0, st>>>(c, blocks, more);
            k_block_states<<<dim3(blocks, n), threads, 0, st>>>(c, blocks);
            launches += 3;   // the columns, the chain, the states
            if (!direct) {
                k_lab_states<<<dim3(Tn, n), 64, 0, st>>>(c);
                launches++;
            }
            SSS_CUDA(cudaGetLastError());
        }
    }
    p->last_launches = launches;
    return SSS_OK;
}

}  // namespace sss
