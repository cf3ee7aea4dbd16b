// Power-series kernels for groups of 32 lanes, 16 to 20, 22, 24 and 28 slots.
#include "sss_power.cuh"

namespace sss {

int launch_power_l32b(sss_plan* p, int E, int RM, const BatchArgs& a, int threads, size_t smem,
                      cudaStream_t st) {
    switch (E * 16 + RM) {
        SSS_POWER(32, 16, 3)
        SSS_POWER(32, 16, 4)
        SSS_POWER(32, 16, 5)
        SSS_POWER(32, 16, 6)
        SSS_POWER(32, 16, 7)
        SSS_POWER(32, 16, 8)
        SSS_POWER(32, 18, 3)
        SSS_POWER(32, 18, 4)
        SSS_POWER(32, 18, 5)
        SSS_POWER(32, 18, 6)
        SSS_POWER(32, 18, 7)
        SSS_POWER(32, 18, 8)
        SSS_POWER(32, 20, 3)
        SSS_POWER(32, 20, 4)
        SSS_POWER(32, 20, 5)
        SSS_POWER(32, 20, 6)
        SSS_POWER(32, 20, 7)
        SSS_POWER(32, 20, 8)
        SSS_POWER(32, 22, 3)
        SSS_POWER(32, 22, 4)
        SSS_POWER(32, 22, 5)
        SSS_POWER(32, 22, 6)
        SSS_POWER(32, 22, 7)
        SSS_POWER(32, 22, 8)
        SSS_POWER(32, 24, 3)
        SSS_POWER(32, 24, 4)
        SSS_POWER(32, 24, 5)
        SSS_POWER(32, 24, 6)
        SSS_POWER(32, 24, 7)
        SSS_POWER(32, 24, 8)
        SSS_POWER(32, 28, 3)
        SSS_POWER(32, 28, 4)
        SSS_POWER(32, 28, 5)
        SSS_POWER(32, 28, 6)
        SSS_POWER(32, 28, 7)
        SSS_POWER(32, 28, 8)
        SSS_POWER(32, 17, 3)
        SSS_POWER(32, 17, 4)
        SSS_POWER(32, 17, 5)
        SSS_POWER(32, 17, 6)
        SSS_POWER(32, 17, 7)
        SSS_POWER(32, 17, 8)
        SSS_POWER(32, 19, 3)
        SSS_POWER(32, 19, 4)
        SSS_POWER(32, 19, 5)
        SSS_POWER(32, 19, 6)
        SSS_POWER(32, 19, 7)
        SSS_POWER(32, 19, 8)
        default: return fail(SSS_EINVAL, "no power-series kernel for this layout");
    }
}

}  // namespace sss
