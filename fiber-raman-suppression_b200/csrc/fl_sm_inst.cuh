// fl_sm_inst.cuh -- instantiation helper for the single-mode stepper.
#pragma once
#include "fl_launch.h"
#include "fl_sm.cuh"

namespace fl {

// one CTA (CL = 1) or a cluster of CL CTAs per slot
template <typename RF, typename RA, int LOGN, int CL>
cudaError_t launch_sm_c(const LaunchArgs& a) {
    auto kern = sm_advance_kernel<RF, RA, LOGN, CL>;
    const size_t smem = SmShared<RA, LOGN, CL>::BYTES;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return e;
    const int T = XShape<LOGN, CL>::TC;
    if constexpr (CL == 1) {
        kern<<<a.nactive, T, smem, a.stream>>>(static_cast<const SlotDesc*>(a.desc), a.state,
                                               a.active, a.max_evals);
        return cudaGetLastError();
    } else {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(a.nactive * CL);
        cfg.blockDim = dim3(T);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = a.stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = CL;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        return cudaLaunchKernelEx(&cfg, kern, static_cast<const SlotDesc*>(a.desc), a.state,
                                  a.active, a.max_evals);
    }
}

template <typename RF, typename RA, int LOGN>
cudaError_t launch_sm(const LaunchArgs& a) {
    if constexpr (sm_cluster_built(LOGN, 8))
        if (a.cluster == 8) return launch_sm_c<RF, RA, LOGN, 8>(a);
    if constexpr (sm_cluster_built(LOGN, 4))
        if (a.cluster == 4) return launch_sm_c<RF, RA, LOGN, 4>(a);
    if constexpr (sm_cluster_built(LOGN, 2))
        if (a.cluster == 2) return launch_sm_c<RF, RA, LOGN, 2>(a);
    return launch_sm_c<RF, RA, LOGN, 1>(a);
}

template <typename RF, typename RA, int LOGN>
cudaError_t launch_rhs(const RhsArgs& a) {
    auto kern = sm_rhs_kernel<RF, RA, LOGN>;
    const size_t smem = SmShared<RA, LOGN, 1>::BYTES;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return e;
    kern<<<1, XShape<LOGN, 1>::T, smem, a.stream>>>(static_cast<const SlotDesc*>(a.desc), a.adjoint,
                                                    a.z, a.in, a.ufwd, a.out);
    return cudaGetLastError();
}

}  // namespace fl

// NAME is the forward precision (float: FP32 forward with FP64 adjoint;
// double: FP64 throughout)
#define FL_SM_INSTANCE(NAME, RF, RA, LOGN)                                      \
    namespace fl {                                                              \
    cudaError_t launch_sm_##NAME##_##LOGN(const LaunchArgs& a) {                \
        return launch_sm<RF, RA, LOGN>(a);                                      \
    }                                                                           \
    cudaError_t launch_rhs_##NAME##_##LOGN(const RhsArgs& a) {                  \
        return launch_rhs<RF, RA, LOGN>(a);                                     \
    }                                                                           \
    }
