// fl_launch.h -- launchers of the single-mode stepper, one per built grid size
// and precision; each is compiled in its own translation unit.
#pragma once
#include <algorithm>

#include <cuda_runtime.h>

#include "fl_types.h"

namespace fl {

struct LaunchArgs {
    const void* desc;      // SlotDesc<R>[]
    SlotState* state;      // SlotState[]
    const int* active;     // slot indices, one CTA or cluster each
    int nactive;
    int max_evals;         // RHS evaluations per slot in this launch
    cudaStream_t stream;
    int cluster = 1;       // CTAs per slot (a size of sm_cluster_built, else 1)
};

// cluster sizes built for a grid
constexpr bool sm_cluster_built(int logn, int c) {
    return logn == 12 ? c == 2 || c == 4
         : logn == 13 ? c == 2 || c == 4 || c == 8
         : logn == 14 ? c == 4 || c == 8 : false;
}

// CTAs per slot for a launch of this many slots: the size whose waves take
// the least time.  A C-CTA solve takes a fraction of a one-CTA solve (column
// rel), and the clusters in flight are bounded by the SMs of a GPC: 74 of two
// CTAs, 32 of four, 14 of eight on 148 SMs.  Measured per gradient batch
// (ms, 0.3 m; 1 / 2 / 4 / 8 CTAs): Nt = 2^13, 8 slots 8.9 / 5.9 / 4.7 / 4.5,
// 24 slots 9.0 / 6.0 / 4.8 / 8.7, 60 slots 9.6 / 6.5 / 9.5 / 17.7, 148 slots
// 11.6 / 13.7 / 23 / 44; 2^12, 8 slots 4.9 / 4.2 / 4.0, 36 slots 5.4 / 4.6 /
// 7.9; 2^14, 8 slots 23.8 / - / 9.1 / 8.1, 40 slots 26.6 / - / 18.5 / 24.1.
inline int sm_cluster(int sm_count, int logn, int slots) {
    static const struct {
        int c, per148;
        double rel[3];  // 2^12, 2^13, 2^14
    } size[] = {{1, 148, {1.0, 1.0, 1.0}},
                {2, 74, {0.86, 0.66, 1.0}},
                {4, 32, {0.82, 0.54, 0.38}},
                {8, 14, {1.0, 0.50, 0.34}}};
    int best = 1;
    double least = 1e300;
    for (const auto& z : size) {
        if (z.c > 1 && !sm_cluster_built(logn, z.c)) continue;
        const int cap = std::max(1, z.per148 * sm_count / 148);
        const double t = ((slots + cap - 1) / cap) * (z.c == 1 ? 1.0 : z.rel[logn - 12]);
        if (t < least) {
            least = t;
            best = z.c;
        }
    }
    return best;
}

using LaunchFn = cudaError_t (*)(const LaunchArgs&);

struct RhsArgs {
    const void* desc;      // one SlotDesc<R> (tables and scratch)
    int adjoint;
    double z;
    const double* in;      // N complex doubles: ũ or λ̃
    const double* ufwd;    // N complex doubles: forward field (adjoint)
    double* out;           // N complex doubles
    cudaStream_t stream;
};
using RhsFn = cudaError_t (*)(const RhsArgs&);
RhsFn rhs_launcher(int fp64, int logn);

// returns nullptr when (precision, log2 Nt) is not built
LaunchFn sm_launcher(int fp64, int logn);

// pump-gain forward solve of one single-mode problem (FP32 right-hand side,
// FP64 state and error norm), run to completion in one launch; false / an
// error when log2 Nt is not built (2^6..2^13)
bool gain_built(int logn);
cudaError_t launch_gain(int logn, const GainDesc* desc, GainOut* out, cudaStream_t stream);

}  // namespace fl
