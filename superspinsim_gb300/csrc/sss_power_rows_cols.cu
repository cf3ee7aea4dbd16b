// Power-series kernels for groups wider than a warp, propagator columns.
#include "sss_power_rows.cuh"

namespace sss {

int launch_power_rows_cols(sss_plan* p, int E, int W, const BatchArgs& a, int threads, size_t smem,
                           cudaStream_t st) {
    return launch_any_rows<true>(p, E, W, a, threads, smem, st);
}

}  // namespace sss
