// How a drop-in run by propagator columns (sss_columns.cu) is cut into launches
// (host code).
//
// The columns of a launch's samples are its trajectories: run after run of `len`
// samples, M columns each.  Their propagators stay below a bound of memory, so
// long runs take several launches, of whole blocks of the chain; each should
// still have as many columns as fill the SM sub-partitions with four warps of
// 8-lane groups, and longer runs past that (the states inside a run need no
// chain).
#pragma once
#include <algorithm>
#include <cstddef>

namespace sss {

constexpr int kColBlock = 16;                  // runs per block of the chain
constexpr int kColMaxTraj = 65535;             // trajectories of a launch: blocks in a grid's y dimension
constexpr size_t kColBytes = 2ull << 30;       // propagators of a launch

struct ColumnsCut {
    int len = 1;      // samples per run
    int samples = 0;  // per launch and trajectory: all T, or whole blocks of one trajectory
    int traj = 1;     // trajectories per launch
    long runs = 0;    // runs of a full launch, all trajectories
};

inline ColumnsCut columns_cut(int ntraj, int T, int M, int num_sms, size_t bytes = kColBytes) {
    const size_t per_sample = sizeof(double) * (size_t)M * M;
    const long cap = (long)std::max<size_t>(1, bytes / per_sample);
    ColumnsCut c;
    c.samples = (int)std::min<long>(T, cap);
    c.traj = c.samples < T ? 1 : (int)std::min<long>(std::min(ntraj, kColMaxTraj), std::max(1L, cap / T));
    const long want = 16L * 4 * num_sms, n = (long)c.samples * c.traj;
    c.len = (int)std::max(1L, (n * M + want - 1) / want);
    if (c.samples < T) {
        c.len = (int)std::max(1L, std::min<long>(c.len, cap / kColBlock));
        c.samples = std::max(1, c.samples / (kColBlock * c.len)) * kColBlock * c.len;
    }
    c.runs = (long)c.traj * ((std::min(T, c.samples) + c.len - 1) / c.len);
    return c;
}

}  // namespace sss
