// fl_check.cu -- the stepper's own math routines, evaluated one by one (the
// checked build only; the default library has no such entry point).
#ifdef FL_CHECKED
#include "fl_sm.cuh"

namespace fl {
// which: 0 sqrt_nb(a), 1 rcp_nb(a), 2 phasor<double>(a, b), 3 phasor<float>(a, b)
__global__ void check_math_kernel(int which, int n, const double* __restrict__ a,
                                  const double* __restrict__ b, double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (which == 0) out[i] = sqrt_nb(a[i]);
    else if (which == 1) out[i] = rcp_nb(a[i]);
    else st2(out, i, which == 2 ? phasor<double>(a[i], b[i]) : up(phasor<float>(a[i], b[i])));
}
}  // namespace fl

// host arrays of n values (out: 2 n for the phasors); 0 or the CUDA error
extern "C" int fl_check_math(int which, int n, const double* a, const double* b, double* out) {
    const size_t in = sizeof(double) * (size_t)n, res = which < 2 ? in : 2 * in;
    double* d = nullptr;
    cudaError_t e = cudaMalloc(&d, 4 * in);
    if (e != cudaSuccess) return e;
    e = cudaMemcpy(d, a, in, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d + n, b, in, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        fl::check_math_kernel<<<(n + 255) / 256, 256>>>(which, n, d, d + n, d + 2 * (size_t)n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d + 2 * (size_t)n, res, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e;
}
#endif
