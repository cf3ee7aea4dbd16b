// Launches of the power-series kernels for groups wider than a warp (one CTA per
// trajectory), for sss_power_rows.cu (trajectories) and sss_power_rows_cols.cu
// (propagator columns): two units, so that they compile side by side.
#pragma once
#include "sss_power.cuh"

namespace sss {
namespace {

template <int E, bool Cols>
int launch_rows(sss_plan* p, int W, const BatchArgs& a, int threads, size_t smem, cudaStream_t st) {
    switch (W) {
        case 1:
        case 2: return launch(p, k_batch_power_rows<E, 1, Cols>, a, threads, 1, smem, st);
        case 4: return launch(p, k_batch_power_rows<E, 2, Cols>, a, threads, 1, smem, st);
        case 8: return launch(p, k_batch_power_rows<E, 3, Cols>, a, threads, 1, smem, st);
        default: return launch(p, k_batch_power_rows<E, 4, Cols>, a, threads, 1, smem, st);
    }
}

template <bool Cols>
int launch_any_rows(sss_plan* p, int E, int W, const BatchArgs& a, int threads, size_t smem, cudaStream_t st) {
    switch (E) {
        case 1: return launch_rows<1, Cols>(p, W, a, threads, smem, st);
        case 2: return launch_rows<2, Cols>(p, W, a, threads, smem, st);
        case 3: return launch_rows<3, Cols>(p, W, a, threads, smem, st);
        case 4: return launch_rows<4, Cols>(p, W, a, threads, smem, st);
        case 5: return launch_rows<5, Cols>(p, W, a, threads, smem, st);
        case 6: return launch_rows<6, Cols>(p, W, a, threads, smem, st);
        case 7: return launch_rows<7, Cols>(p, W, a, threads, smem, st);
        case 8: return launch_rows<8, Cols>(p, W, a, threads, smem, st);
        case 9: return launch_rows<9, Cols>(p, W, a, threads, smem, st);
        case 10: return launch_rows<10, Cols>(p, W, a, threads, smem, st);
        case 12: return launch_rows<12, Cols>(p, W, a, threads, smem, st);
        case 14: return launch_rows<14, Cols>(p, W, a, threads, smem, st);
        case 16: return launch_rows<16, Cols>(p, W, a, threads, smem, st);
        case 20: return launch_rows<20, Cols>(p, W, a, threads, smem, st);
        default: return fail(SSS_EINVAL, "no power-series kernel for this layout");
    }
}

}  // namespace
}  // namespace sss
