// Power-series kernels for groups of 32 lanes, 2, 3, 4, 6, 8, 10, 12, 14 slots.
#include "sss_power.cuh"

namespace sss {

int launch_power_l32a(sss_plan* p, int E, int RM, const BatchArgs& a, int threads, size_t smem,
                      cudaStream_t st) {
    switch (E * 16 + RM) {
        SSS_POWER(32, 2, 3)
        SSS_POWER(32, 2, 4)
        SSS_POWER(32, 2, 5)
        SSS_POWER(32, 2, 6)
        SSS_POWER(32, 2, 7)
        SSS_POWER(32, 2, 8)
        SSS_POWER(32, 3, 3)
        SSS_POWER(32, 3, 4)
        SSS_POWER(32, 3, 5)
        SSS_POWER(32, 3, 6)
        SSS_POWER(32, 3, 7)
        SSS_POWER(32, 3, 8)
        SSS_POWER(32, 4, 3)
        SSS_POWER(32, 4, 4)
        SSS_POWER(32, 4, 5)
        SSS_POWER(32, 4, 6)
        SSS_POWER(32, 4, 7)
        SSS_POWER(32, 4, 8)
        SSS_POWER(32, 6, 3)
        SSS_POWER(32, 6, 4)
        SSS_POWER(32, 6, 5)
        SSS_POWER(32, 6, 6)
        SSS_POWER(32, 6, 7)
        SSS_POWER(32, 6, 8)
        SSS_POWER(32, 8, 3)
        SSS_POWER(32, 8, 4)
        SSS_POWER(32, 8, 5)
        SSS_POWER(32, 8, 6)
        SSS_POWER(32, 8, 7)
        SSS_POWER(32, 8, 8)
        SSS_POWER(32, 10, 3)
        SSS_POWER(32, 10, 4)
        SSS_POWER(32, 10, 5)
        SSS_POWER(32, 10, 6)
        SSS_POWER(32, 10, 7)
        SSS_POWER(32, 10, 8)
        SSS_POWER(32, 12, 3)
        SSS_POWER(32, 12, 4)
        SSS_POWER(32, 12, 5)
        SSS_POWER(32, 12, 6)
        SSS_POWER(32, 12, 7)
        SSS_POWER(32, 12, 8)
        SSS_POWER(32, 14, 3)
        SSS_POWER(32, 14, 4)
        SSS_POWER(32, 14, 5)
        SSS_POWER(32, 14, 6)
        SSS_POWER(32, 14, 7)
        SSS_POWER(32, 14, 8)
        default: return fail(SSS_EINVAL, "no power-series kernel for this layout");
    }
}

}  // namespace sss
