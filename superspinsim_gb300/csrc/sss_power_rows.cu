// Power-series kernels for groups wider than a warp (one CTA per trajectory).
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

}  // namespace

int launch_power_rows(sss_plan* p, int E, int W, const BatchArgs& a, int threads, size_t smem,
                      cudaStream_t st) {
    switch (E) {
        case 1: return launch_rows<1, false>(p, W, a, threads, smem, st);
        case 2: return launch_rows<2, false>(p, W, a, threads, smem, st);
        case 3: return launch_rows<3, false>(p, W, a, threads, smem, st);
        case 4: return launch_rows<4, false>(p, W, a, threads, smem, st);
        case 5: return launch_rows<5, false>(p, W, a, threads, smem, st);
        case 6: return launch_rows<6, false>(p, W, a, threads, smem, st);
        case 7: return launch_rows<7, false>(p, W, a, threads, smem, st);
        case 8: return launch_rows<8, false>(p, W, a, threads, smem, st);
        case 9: return launch_rows<9, false>(p, W, a, threads, smem, st);
        case 10: return launch_rows<10, false>(p, W, a, threads, smem, st);
        case 12: return launch_rows<12, false>(p, W, a, threads, smem, st);
        case 14: return launch_rows<14, false>(p, W, a, threads, smem, st);
        case 16: return launch_rows<16, false>(p, W, a, threads, smem, st);
        case 20: return launch_rows<20, false>(p, W, a, threads, smem, st);
        default: return fail(SSS_EINVAL, "no power-series kernel for this layout");
    }
}

}  // namespace sss
