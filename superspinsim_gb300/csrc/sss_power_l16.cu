// Power-series kernels for groups of 16 lanes.
#include "sss_power.cuh"

namespace sss {

int launch_power_l16(sss_plan* p, int E, int RM, const BatchArgs& a, int threads, size_t smem,
                     cudaStream_t st) {
    switch (E * 16 + RM) {
        SSS_POWER(16, 8, 3)
        SSS_POWER(16, 8, 4)
        SSS_POWER(16, 8, 5)
        SSS_POWER(16, 8, 6)
        SSS_POWER(16, 8, 8)
        SSS_POWER(16, 10, 3)
        SSS_POWER(16, 10, 4)
        SSS_POWER(16, 10, 5)
        SSS_POWER(16, 10, 6)
        SSS_POWER(16, 10, 8)
        SSS_POWER(16, 12, 3)
        SSS_POWER(16, 12, 4)
        SSS_POWER(16, 12, 5)
        SSS_POWER(16, 12, 6)
        SSS_POWER(16, 12, 8)
        SSS_POWER(16, 14, 3)
        SSS_POWER(16, 14, 4)
        SSS_POWER(16, 14, 5)
        SSS_POWER(16, 14, 6)
        SSS_POWER(16, 14, 8)
        SSS_POWER(16, 16, 3)
        SSS_POWER(16, 16, 4)
        SSS_POWER(16, 16, 5)
        SSS_POWER(16, 16, 6)
        SSS_POWER(16, 16, 8)
        SSS_POWER(16, 20, 3)
        SSS_POWER(16, 20, 4)
        SSS_POWER(16, 20, 5)
        SSS_POWER(16, 20, 6)
        SSS_POWER(16, 20, 8)
        SSS_POWER(16, 24, 3)
        SSS_POWER(16, 24, 4)
        SSS_POWER(16, 24, 5)
        SSS_POWER(16, 24, 6)
        SSS_POWER(16, 24, 8)
        default: return fail(SSS_EINVAL, "no power-series kernel for this layout");
    }
}

}  // namespace sss
