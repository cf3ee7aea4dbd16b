// Power-series batched kernel for large systems (more than 64 reachable rows):
// one trajectory per thread-block cluster (sss_power.h explains the form and
// holds the packing, power_pack_big).
//
// The 21-level NV's series at 5 ps has 18,800 entries on 171 rows, too many
// for one CTA's registers.  The rows are dealt to the C CTAs of a cluster; a
// CTA keeps its coefficients and operand offsets in shared memory (10 bytes an
// entry: 215 KB for C = 1) beside the state's copies scaled by each monomial.
// Per exponential every row's lanes sum their entries, reduce by shuffles, add
// to the row and write its copies, which the CTA's warps carry into every other
// CTA's shared memory (two alternating buffers), then one cluster barrier.
//
// What bounds it: FP64 issue for C = 1 (8 warps per SM sub-partition x 21
// slots x 64 cycles), and from C = 4 on the exchange as well.  The Taylor action
// of the same trajectory on one CTA is 9 terms with a chain of 13 to 16 slots and
// two barriers each, 19,900 cycles per exponential at 128 lanes whatever the
// batch leaves idle.
#include <cooperative_groups.h>

#include "sss_power.cuh"

namespace cg = cooperative_groups;

namespace sss {
namespace {

// R: fine steps of the coefficient ring (16 where the tables fill shared memory)
template <int R>
__global__ void __launch_bounds__(1024, 1) k_power_big(const BatchArgs a) {
    extern __shared__ double smem[];
    cg::cluster_group cluster = cg::this_cluster();
    const int C = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int M = a.M, K = a.K, NM = a.pw_mono, E = a.E, T = blockDim.x, li = threadIdx.x;
    const int n_x = NM * M + 1;                       // copies [monomial][row], zero word
    double* X = smem;                                 // two buffers of them
    double* ringc = X + 2 * n_x;
    double* ring_m = ringc + R * a.Q * a.n_lch;       // [s][exponential][value], and one row past the end
    double* coef = ring_m + (R * K + 1) * NM;         // [q][lane]
    unsigned short* xo = reinterpret_cast<unsigned short*>(coef + (size_t)E * T);
    __shared__ double s_red[32], s_part[kPowBigMaxCtas];
    if (li < 2) X[li * n_x + NM * M] = 0.0;
    for (int i = li; i < NM; i += T) ring_m[R * K * NM + i] = 0.0;
    for (int q = 0; q < E; q++) {
        const size_t at = ((size_t)rank * E + q) * T + li;
        coef[q * T + li] = __ldg(a.pw_coef + at);
        xo[q * T + li] = (unsigned short)__ldg(a.pw_x + at);
    }
    // lane word: row (M: none), its lanes W and the lane's place among them
    const unsigned lw = __ldg(a.cw + (size_t)rank * T + li);
    const int row = (int)(lw & 0xffffu), W = (int)((lw >> 16) & 0xffu), sub = (int)(lw >> 24);
    const bool own = row < M, keep = own && sub == 0;
    const int wmax = a.pw_w, lane = li & 31;
    const double rw = keep && a.rw ? __ldg(a.rw + row) : 0.0;
    double v = 0.0;
    int xb = 0;
    auto gsync = [&]() { __syncthreads(); };
    auto csync = [&]() {
        if (C > 1) cluster.sync(); else __syncthreads();
    };
    // The rows' copies scaled by ring row j's monomials, in every CTA.  The
    // row's lanes write them here; then each warp carries this CTA's rows, which
    // are neighbours in the copies, to one other CTA.  (Remote stores by the
    // rows' own lanes, eight CTAs each, made 5,730 cycles per exponential;
    // spread over CTAs within a warp, 11,100.)
    const int r0 = __ldg(a.rbeg + rank), nr = __ldg(a.rbeg + rank + 1) - r0;
    const int warps = T / 32, parts = max(1, warps / C);   // warps per destination
    auto write_x = [&](int j) {
        if (own)
            for (int m = sub; m < NM; m += W) X[xb + m * M + row] = ring_m[j * NM + m] * v;
        if (C == 1) return;
        __syncthreads();
        for (int unit = li / 32; unit < C * parts; unit += warps) {
            const int to = unit % C;
            if (to == rank) continue;
            double* const X_to = cluster.map_shared_rank(X, to);
            for (int i = unit / C * 32 + lane; i < NM * nr; i += parts * 32) {
                const int m = i / nr, at = xb + m * M + r0 + (i - m * nr);
                X_to[at] = X[at];
            }
        }
    };
    csync();

    const int n_clusters = gridDim.x / C;
    for (int taken = blockIdx.x / C; taken < a.ntraj; taken += n_clusters) {
        PowTrajectory tr;
        tr.set(a, taken);
        if (own) v = a.rho0[(size_t)tr.b * a.N + __ldg(a.row_orig + row)];
        int r = 0, rp = R;
        while (tr.t < tr.T_b) {
            if (rp == R) {
                pow_fill_ring<R>(a, tr, r, li, T, ringc, ring_m, nullptr, gsync);
                rp = 0;
                write_x(0);
                csync();
            }
            for (int i = 0; i < K; i++) {
                if (a.states && keep)
                    a.states[(((size_t)tr.b * a.st_steps + (size_t)(tr.t - a.t_begin) * a.F + r) * K + K - 1 - i) * M +
                             row] = v;
                const double* Xb = X + xb;
                const double* cf = coef + li;
                const unsigned short* xq = xo + li;
                double d = 0.0;
#pragma unroll 4
                for (int q = 0; q < E; q++) d = fma(cf[q * T], Xb[xq[q * T]], d);
                // the sum over the row's lanes, to its first one and back
                for (int o = 1; o < wmax; o <<= 1) {
                    const double y = __shfl_down_sync(0xffffffffu, d, o);
                    if ((sub & (2 * o - 1)) == 0 && sub + o < W) d += y;
                }
                v += __shfl_sync(0xffffffffu, d, lane - sub);
                xb ^= n_x;
                write_x(rp * K + i + 1);
                csync();
            }
            rp++;
            if (++r < a.F) continue;
            r = 0;
            const int t = tr.t++;
            if (a.trace && keep) a.trace[((size_t)tr.b * a.T_max + t) * a.N + __ldg(a.row_orig + row)] = v;
            if (a.readout) {
                double s = rw * v;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if (lane == 0) s_red[li >> 5] = s;
                __syncthreads();
                if (li == 0) {
                    for (int w = 1; w < T / 32; w++) s += s_red[w];
                    if (C > 1) *cluster.map_shared_rank(&s_part[rank], 0) = s;
                }
                csync();
                if (li == 0 && rank == 0) {
                    for (int c = 1; c < C; c++) s += s_part[c];
                    a.readout[(size_t)tr.b * a.T_max + t] = s;
                    note_nonfinite(a, s, tr.b, t);
                }
            }
        }
        if (a.fin && keep) {
            a.fin[(size_t)tr.b * a.N + __ldg(a.row_orig + row)] = v;
            note_nonfinite(a, v, tr.b, a.t_end);
        }
        if (a.readout && rank == 0)
            for (int tt = max(tr.T_b, a.t_begin) + li; tt < a.t_end; tt += T)
                a.readout[(size_t)tr.b * a.T_max + tt] = 0.0;
        csync();   // the ring and the copies are the next trajectory's
    }
    csync();       // no CTA leaves while another may still write to it
}

}  // namespace

// Clusters of `ctas` CTAs the GPU holds at once with one CTA per SM (its GPCs
// need not divide into them: 16 of 8 CTAs on 152 SMs), 0 on error.
int power_big_resident(int ctas) {
    const auto kernel = pow_big_ring(ctas) == kRing ? k_power_big<kRing> : k_power_big<kPowRowsRing>;
    const int smem = 180 * 1024;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = ctas;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3((unsigned)power_big_threads(ctas));
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int active = 0;
    if (allow_smem(kernel) ||
        cudaOccupancyMaxActiveClusters(&active, kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return active;
}

int launch_power_big(sss_plan* p, int ctas, const BatchArgs& a, int threads, size_t smem, cudaStream_t st) {
    const auto kernel = pow_big_ring(ctas) == kRing ? k_power_big<kRing> : k_power_big<kPowRowsRing>;
    if (int rc = allow_smem(kernel)) return rc;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = ctas;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    const int n_work = p->launch_active > 0 ? std::min(p->launch_active, a.ntraj) : a.ntraj;
    cfg.gridDim = dim3((unsigned)(ctas * n_work));
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int active = 0;
    SSS_CUDA(cudaOccupancyMaxActiveClusters(&active, kernel, &cfg));
    if (active < 1) return fail(SSS_EINVAL, "no cluster of the power-series kernel fits on the GPU");
    const int grid = ctas * std::max(1, std::min(n_work, active));
    cfg.gridDim = dim3((unsigned)grid);
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    SSS_CUDA(cudaStreamIsCapturing(st, &cap));
    const bool timed = cap == cudaStreamCaptureStatusNone && !p->cols_samples;
    if (timed && !p->ev_begin) {
        SSS_CUDA(cudaEventCreate(&p->ev_begin));
        SSS_CUDA(cudaEventCreate(&p->ev_end));
    }
    if (timed && !p->ev_keep_begin) SSS_CUDA(cudaEventRecord(p->ev_begin, st));
    SSS_CUDA(cudaLaunchKernelEx(&cfg, kernel, a));
    if (timed) {
        SSS_CUDA(cudaEventRecord(p->ev_end, st));
        p->ev_recorded = true;
    }
    if (!p->cols_samples) p->last_grid = grid;
    return SSS_OK;
}

}  // namespace sss
