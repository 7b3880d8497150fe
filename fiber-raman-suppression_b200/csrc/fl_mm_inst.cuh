// fl_mm_inst.cuh -- instantiation helper of the multimode evaluation round.
#pragma once
#include <nvtx3/nvToolsExt.h>

#include "fl_evidence.cuh"
#include "fl_mm.cuh"
#include "fl_mm_launch.h"

namespace fl {

// which: 0 prologue, 1 pairs, 2 epilogue; CL CTAs (one cluster) per transform
template <bool MIX, int LOGN, int LOGE, int CL>
cudaError_t mm_launch_tasks(const MmRound& a, int which) {
    using G = MmTasks<MIX, LOGN, LOGE, CL>;
    const size_t smem = G::SMEM;
    void (*k)(const MmDesc*, const MmState*, const int*) =
        which == 0   ? mm_prologue_kernel<MIX, LOGN, LOGE, CL>
        : which == 1 ? mm_pairs_kernel<MIX, LOGN, LOGE, CL>
                     : mm_epilogue_kernel<MIX, LOGN, LOGE, CL>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int fields = a.adjoint && mm_adj_mixed(a.M, a.N, a.fp64) ? 2 : 1;
    const int units = which == 0   ? fields * a.M
                      : which == 1 ? (a.adjoint ? 2 : 1) * ((a.NP + 1) / 2)
                                   : a.M;
    return mm_chain_launch(k, dim3(units * CL, a.nactive), G::T, smem, a.stream, CL,
                           which != 0 || a.chained, static_cast<const MmDesc*>(a.desc),
                           static_cast<const MmState*>(a.state), a.active);
}

// one evaluation round; each stage's launches sit in a named NVTX range
// (host-side: under graph capture the ranges mark the capture)
template <int LOGN, int LOGE, int CL>
cudaError_t mm_round(const MmRound& a) {
    cudaError_t e;
#define FL_TRY(name, x)             \
    nvtxRangePushA("fl: mm " name); \
    e = (x);                        \
    nvtxRangePop();                 \
    if (e != cudaSuccess) return e;
    auto tasks = [&](int which) {
        return a.fp64 ? mm_launch_tasks<false, LOGN, LOGE, CL>(a, which)
                      : mm_launch_tasks<true, LOGN, LOGE, CL>(a, which);
    };
    FL_TRY("prologue", tasks(0))
    if (a.adjoint) {
        FL_TRY("Im X contraction", mm_launch_contract(a, 1))
    }
    FL_TRY("low-rank reduction", mm_launch_contract(a, 3))
    FL_TRY("pairs", tasks(1))
    FL_TRY("contraction", mm_launch_contract(a, 0))
    if (a.adjoint) {
        FL_TRY("adjoint contraction", mm_launch_contract(a, 2))
    }
    FL_TRY("epilogue", tasks(2))
    if (a.control) {
        FL_TRY("control", mm_launch_control(a, 1))
    }
#undef FL_TRY
    return cudaSuccess;
}

}  // namespace fl

#define FL_MM_INSTANCE(LOGN, LOGE, CL)                                                     \
    namespace fl {                                                                         \
    cudaError_t mm_round_##LOGN(const MmRound& a) { return mm_round<LOGN, LOGE, CL>(a); } \
    cudaError_t mm_evidence_##LOGN(const EvidenceArgs& a) {                                \
        return launch_evidence<LOGN, LOGE, CL>(a);                                         \
    }                                                                                      \
    }
