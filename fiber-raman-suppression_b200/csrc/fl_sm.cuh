// fl_sm.cuh -- single-mode GMMNLSE stepper: one CTA, or a cluster of CTAs
// when few problems run at once, owns one problem (slot)
// and runs its whole adaptive Tsit5 solve, the checkpoint-replay recompute
// and the adjoint solve as a state machine whose state lives in global
// memory, so a launch can advance a slot by a bounded number of attempted
// steps (serving) or run it to completion (plain drop-in).
//
// Reference path: forward RHS src/simulation/simulate_disp_mmf.jl:25-60,
// adjoint RHS src/simulation/sensitivity_disp_mmf.jl:32-79 (with the helper
// terms :93-215), drivers simulate_disp_mmf.jl:183-207 and
// sensitivity_disp_mmf.jl:309-332, band objective
// src/fiberlab/physics_helpers.jl:222-232, phase gradient
// src/fiberlab/physics_models.jl:1042.
//
// For M = 1 the RHS is evaluated in an algebraically identical form with
// fewer transforms (4 forward, 5 adjoint instead of 4 and 14):
//   forward  dũ = i e^{-iDz} τ F⁻¹[((1-fR) I + h∗I) u_t],  I = γ|u_t|²
//   adjoint  dλ̃ = i e^{-iDz} F⁻¹[ λ_t (2(1-fR) I + h∗I) - (1-fR) γ λ_t* u_t²
//                                 + 2i (h̃⋆Y) u_t ],  Y = γ Im(λ_t u_t*)
// where u_t = F(e^{iDz} ũ), λ_t = F(e^{iDz} τ λ̃), h∗ is the Raman convolution
// with the fftshift folded into Heff = hR (-1)^k, and h̃⋆ the correlation
// (conj(Heff)).  The two Raman terms of the reference adjoint (:93-132) are
// complex conjugates of each other and combine into the single real
// correlation of Y; h∗I and h̃⋆Y share one complex transform pair.
//
// Precision (FP32 mode, RF = float): states, phase arguments, transforms of
// the field, stage sums, error norm and reductions in FP64; the forward's
// stage vectors and the dense interpolant are stored in RF, and on the grids
// up to 2^11 its Raman convolution runs in RF (see SmSolver).  The adjoint
// integration (the gradient accumulation along z) is FP64 throughout, stage
// vectors included: an FP32 adjoint amplifies its round-off through the
// modulation-instability gain of the anomalous-dispersion fiber and misses
// 1e-3 gradient accuracy (measured 2e-3..7e-3 on the Nt = 2^13 band-objective
// problem).  The FP64 mode stores everything in FP64.
#pragma once
#include <type_traits>

#include "fl_fft.cuh"
#include "fl_types.h"
#include "fl_xfft.cuh"

namespace fl {

// Tsitouras (2011) 5(4) pair, as used by OrdinaryDiffEq's Tsit5.
static __device__ __constant__ double kT5c[7] = {0.0, 0.161, 0.327, 0.9, 0.9800255409045097, 1.0, 1.0};
static __device__ __constant__ double kT5a[7][6] = {
    {0, 0, 0, 0, 0, 0},
    {0.161, 0, 0, 0, 0, 0},
    {-0.008480655492356989, 0.335480655492357, 0, 0, 0, 0},
    {2.897153057105493, -6.359448489975075, 4.3622954328695815, 0, 0, 0},
    {5.325864828439257, -11.748883564062828, 7.4955393428898365, -0.09249506636175525, 0, 0},
    {5.86145544294642, -12.92096931784711, 8.159367898576159, -0.071584973281401,
     -0.028269050394068383, 0},
    {0.09646076681806523, 0.01, 0.4798896504144996, 1.379008574103742, -3.290069515436081,
     2.324710524099774}};
static __device__ __constant__ double kT5bt[7] = {-0.00178001105222577714, -0.0008164344596567469,
                                           0.007880878010261995,    -0.1447110071732629,
                                           0.5823571654525552,      -0.45808210592918697,
                                           0.015151515151515152};
// free 4th-order interpolant b_i(θ) = Σ_p r[i][p] θ^(p+1)
static __device__ __constant__ double kT5r[7][4] = {
    {1.0, -2.763706197274826, 2.9132554618219126, -1.0530884977290216},
    {0.0, 0.13169999999999998, -0.2234, 0.1017},
    {0.0, 3.9302962368947516, -5.941033872131505, 2.490627285651253},
    {0.0, -12.411077166933676, 30.33818863028232, -16.548102889244902},
    {0.0, 37.50931341651104, -88.1789048947664, 47.37952196281928},
    {0.0, -27.896526289197286, 65.09189467479366, -34.87065786149661},
    {0.0, 1.5, -4.0, 2.5}};

// PI controller defaults of OrdinaryDiffEq for a 5th-order method
constexpr double kBeta1 = 7.0 / 50.0, kBeta2 = 2.0 / 25.0, kGamma = 0.9;
constexpr double kQmin = 0.2, kQmax = 10.0, kQoldInit = 1e-4;
constexpr double kEps = 2.220446049250313e-16;

// Square root and reciprocal without the library's branches (sixteen of
// each per step sit on one warp's critical path, and a call in the slow path
// keeps the compiler from interleaving them): the hardware's approximation
// (about 2^-20) and two Newton steps each.  The root's first step is coupled
// (Goldschmidt's iteration: g -> sqrt(m), h -> 1 / (2 sqrt(m))), its second
// adds the residual m - g g, so one rounding is left.
// Both hold to an ulp where argument and result are normal numbers (measured
// 0.50).  Outside: sqrt_nb of zero and of subnormal m is 0, rcp_nb above 2^1022
// is 0; infinity, and for rcp_nb zero and subnormal w, give no finite value (a
// field whose square overflows has no finite derivative either).
__device__ __forceinline__ double sqrt_nb(double m) {
    double r;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(m));
    double g = m * r, h = 0.5 * r;
    const double e = fma(-g, h, 0.5);
    g = fma(g, e, g);
    h = fma(h, e, h);
    g = fma(fma(-g, g, m), h, g);
    return fabs(m) < 2.2250738585072014e-308 ? 0.0 : g;
}
__device__ __forceinline__ double rcp_nb(double w) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(w));
#pragma unroll
    for (int i = 0; i < 2; i++) r = fma(r, fma(-w, r, 1.0), r);
    return r;
}

// exp(+i D z) from the FP64 phase in turns, reduced mod 1 by adding and
// subtracting 1.5 2^52 (the nearest integer for |D z| < 2^51 turns).
// The turns split into a quadrant q and a rest |r| <= 1/8; cos and sin of
// 2 pi r by their Taylor series (to x^16 and x^15 in FP64: the first term
// left out is 5e-17 at pi/4; to x^10 and x^9 in FP32: 2e-9), then a quarter
// turn per q.  Straight-line, so the values of a chunk interleave: the
// library's FP64 sincospi took 330 cycles per value on one warp.
template <typename R>
__device__ __forceinline__ cx<R> quarter_turns(R c, R s, int q) {
    const bool odd = q & 1;
    const R a = odd ? s : c, b = odd ? c : s;
    return mk((q + 1) & 2 ? -a : a, q & 2 ? -b : b);
}
template <typename R>
__device__ __forceinline__ cx<R> phasor(double dturn, double z);
__device__ __forceinline__ double turn_split(double dturn, double z, int& q) {
    const double big = 6755399441055744.0;
    const double t = __dmul_rn(dturn, z), f = t - ((t + big) - big);  // [-1/2, 1/2]
    const double k = fma(f, 4.0, big);                                // nearest quarter
    q = __double2loint(k);
    return fma(k - big, -0.25, f);
}
template <>
__device__ __forceinline__ cx<float> phasor<float>(double dturn, double z) {
    int q;
    const float x = 6.2831853071795864769f * (float)turn_split(dturn, z, q), y = x * x;
    const float s = fmaf(x * y, fmaf(y, fmaf(y, fmaf(y, 1.0f / 362880.0f, -1.0f / 5040.0f),
                                             1.0f / 120.0f), -1.0f / 6.0f), x);
    const float c = fmaf(y, fmaf(y, fmaf(y, fmaf(y, fmaf(y, -1.0f / 3628800.0f, 1.0f / 40320.0f),
                                                 -1.0f / 720.0f), 1.0f / 24.0f), -0.5f), 1.0f);
    return quarter_turns(c, s, q);
}
template <>
__device__ __forceinline__ cx<double> phasor<double>(double dturn, double z) {
    int q;
    const double x = 6.2831853071795864769 * turn_split(dturn, z, q), y = x * x;
    double s = -1.0 / 1307674368000.0, c = 1.0 / 20922789888000.0;
    s = fma(s, y, 1.0 / 6227020800.0);
    c = fma(c, y, -1.0 / 87178291200.0);
    s = fma(s, y, -1.0 / 39916800.0);
    c = fma(c, y, 1.0 / 479001600.0);
    s = fma(s, y, 1.0 / 362880.0);
    c = fma(c, y, -1.0 / 3628800.0);
    s = fma(s, y, -1.0 / 5040.0);
    c = fma(c, y, 1.0 / 40320.0);
    s = fma(s, y, 1.0 / 120.0);
    c = fma(c, y, -1.0 / 720.0);
    s = fma(s, y, -1.0 / 6.0);
    c = fma(c, y, 1.0 / 24.0);
    s = fma(x * y, s, x);
    c = fma(c, y, -0.5);
    c = fma(c, y, 1.0);
    return quarter_turns(c, s, q);
}

__device__ __forceinline__ cx<double> ld2(const double* p, int b) {
    const double2 v = reinterpret_cast<const double2*>(p)[b];
    return mk(v.x, v.y);
}
__device__ __forceinline__ void st2(double* p, int b, cx<double> v) {
    reinterpret_cast<double2*>(p)[b] = make_double2(v.re, v.im);
}
// |x|² rounded the same way wherever it is evaluated (no contraction choice
// left to the compiler), so energies of one field compare exactly
__device__ __forceinline__ double energy(cx<double> x) {
    return __fma_rn(x.re, x.re, __dmul_rn(x.im, x.im));
}
template <typename R>
__device__ __forceinline__ cx<double> up(cx<R> a) {
    return mk((double)a.re, (double)a.im);
}
template <typename R>
__device__ __forceinline__ cx<R> down(cx<double> a) {
    return mk((R)a.re, (R)a.im);
}

// deterministic block reductions (fixed shuffle tree, fixed warp order)
template <int T>
__device__ __forceinline__ double block_sum(double v, double* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < T / 32; w++) s += red[w];
    return s;
}
template <int T>
__device__ __forceinline__ double block_max(double v, double* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < T / 32; w++) s = fmax(s, red[w]);
    return s;
}

// Shared-memory layout of the stepper: [transform buffers][64 reduction
// doubles][transform tables][tensor-memory slot].
template <typename RMAX, int LOGN, int C>
struct SmShared {
    static constexpr size_t RED = XPlan<RMAX, RMAX, LOGN, C>::BYTES;
    static constexpr size_t TAB = RED + 64 * sizeof(double);
    static constexpr size_t TAB32 = TAB + sizeof(cx<RMAX>) * XTables<RMAX, LOGN, C>::SIZE;
    // FP64 arithmetic with E = 4 or 8: the tables of the forward's FP32
    // transforms (SmSolver)
    static constexpr bool BOTH =
        sizeof(RMAX) == 8 && XShape<LOGN, C>::E >= 4 && XShape<LOGN, C>::SMALL;
    using X32 = XTables<float, LOGN, C, x_loge(LOGN), true>;
    static constexpr size_t SLOT =
        (TAB32 + (BOTH ? sizeof(cx<float>) * X32::SIZE : 0) + 15) & ~size_t(15);
    // a cluster's CTAs hold tensor memory until their siblings finish: at
    // most one such CTA fits an SM, so that no two clusters wait for each
    // other's columns
    static constexpr size_t BYTES = C > 1 && SLOT + 16 < 116 * 1024 ? 116 * 1024 : SLOT + 16;
    static_assert(BYTES <= 227 * 1024, "shared memory of one CTA");
};
template <typename R, int LOGN, int C>
__device__ __forceinline__ cx<R>* smem_tables(unsigned char* smraw) {
    return reinterpret_cast<cx<R>*>(smraw + SmShared<R, LOGN, C>::TAB);
}

// Fill the transform tables and wait for the group.
template <typename R, int LOGN, int C>
__device__ __forceinline__ void load_tables(const SlotDesc& d, unsigned char* smraw, int rank) {
    using SH = SmShared<R, LOGN, C>;
    x_fill<R, LOGN, C>(smem_tables<R, LOGN, C>(smraw), (const cx<R>*)d.tw[sizeof(R) == 8], rank);
    if constexpr (SH::BOTH)
        x_fill<float, LOGN, C, x_loge(LOGN), true>(reinterpret_cast<cx<float>*>(smraw + SH::TAB32),
                                                   (const cx<float>*)d.tw[0], rank);
    XForm<R, R, LOGN, C>::sync();
}

// ---------------------------------------------------------------------------
// Tensor memory as the right-hand side's per-thread scratch (sm_100a).
//
// Each RHS evaluation parks two fields between its transforms -- u_t in the
// forward, λ_t and u_t in the adjoint -- and, where there is room, its
// phasors, and every thread only ever reads back the bins it wrote.  The
// transforms leave the SM's 256 KB of tensor memory unused: the CTA
// allocates columns once (tcgen05.alloc) and threads move their own values
// with tcgen05.st / tcgen05.ld (32x32b shape: a warp addresses the 32 lanes
// of its lane quarter, warp % 4, and each thread its own lane's columns), in
// place of per-slot fields in global memory (five 128 KB round trips per FP64
// adjoint evaluation at Nt = 2^13).  Layout: lane 32 (w % 4) + (t % 32),
// columns (w / 4) COLS_WARP + f 4E + [0, 4E) for field f of warp w.
constexpr uint32_t kNoTmem = 0xFFFFFFFFu;

template <int LOGN, int C>
struct TmLayout {
    using S = XShape<LOGN, C>;
    static constexpr int E = S::E, T = S::TC;
    static constexpr int WARPS = T / 32;
    static constexpr int PER_Q = (WARPS + 3) / 4;      // warps sharing a lane quarter
    // FP64 fields (4 words per value); the third holds the evaluation's
    // phasors where the columns of the CTAs that fit an SM allow it.  At 2^14
    // one FP64 field on one CTA is the whole tensor memory: it takes slot 0
    // (u_t, λ_t and, around the transforms, the phasors), slot 1 stays in
    // global memory.  148 gradients there, 0.1 m: 16.9 ms with all of them in
    // global memory (38 MB a field over the SMs), 12.9 so.
    static constexpr int FIELDS = C > 1 || LOGN <= 11 ? 3 : LOGN <= 13 ? 2 : 1;
    static constexpr int COLS_WARP = FIELDS * 4 * E;
    static constexpr int NEED = COLS_WARP * PER_Q;
    // allocation: a power of two >= 32 columns
    static constexpr int COLS = NEED <= 32 ? 32 : NEED <= 64 ? 64 : NEED <= 128 ? 128
                              : NEED <= 256 ? 256 : 512;
    // one CTA per problem: the grids whose registers admit no more CTAs per
    // SM than the columns do (sm_min_ctas: 2^7 and 2^8 eight of 64 columns,
    // 2^9 four of 64, 2^10 two of 128, 2^11 two of 256, 2^12 one of 256, 2^13
    // and 2^14 one of 512), so an allocation waits for no CTA of its own kernel;
    // clusters: always (one CTA per SM, SmShared)
    static constexpr bool ENABLED = NEED <= 512 && E >= 4;
    static_assert(C == 1 || ENABLED, "clusters keep their scratch in tensor memory");
    template <typename R>
    static constexpr bool phasors() { return ENABLED && (FIELDS == 3 || (FIELDS == 2 && sizeof(R) == 4)); }
};

__device__ __forceinline__ void tm_st16(uint32_t a, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, "
        "%11, %12, %13, %14, %15, %16};" ::"r"(a),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
        "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tm_ld16(uint32_t a, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, "
        "%11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(a)
        : "memory");
}
__device__ __forceinline__ void tm_st8(uint32_t a, const uint32_t (&r)[8]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(a),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
        : "memory");
}
__device__ __forceinline__ void tm_ld8(uint32_t a, uint32_t (&r)[8]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7])
        : "r"(a)
        : "memory");
}
__device__ __forceinline__ void tm_st(uint32_t a, const uint32_t (&r)[16]) { tm_st16(a, r); }
__device__ __forceinline__ void tm_st(uint32_t a, const uint32_t (&r)[8]) { tm_st8(a, r); }
__device__ __forceinline__ void tm_ld(uint32_t a, uint32_t (&r)[16]) { tm_ld16(a, r); }
__device__ __forceinline__ void tm_ld(uint32_t a, uint32_t (&r)[8]) { tm_ld8(a, r); }
__device__ __forceinline__ void tm_wait_st() {
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tm_wait_ld() {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void pack_words(cx<float> v, uint32_t* w) {
    w[0] = __float_as_uint(v.re);
    w[1] = __float_as_uint(v.im);
}
__device__ __forceinline__ void pack_words(cx<double> v, uint32_t* w) {
    w[0] = (uint32_t)__double2loint(v.re);
    w[1] = (uint32_t)__double2hiint(v.re);
    w[2] = (uint32_t)__double2loint(v.im);
    w[3] = (uint32_t)__double2hiint(v.im);
}
__device__ __forceinline__ void unpack_words(const uint32_t* w, cx<float>& v) {
    v.re = __uint_as_float(w[0]);
    v.im = __uint_as_float(w[1]);
}
__device__ __forceinline__ void unpack_words(const uint32_t* w, cx<double>& v) {
    v.re = __hiloint2double((int)w[1], (int)w[0]);
    v.im = __hiloint2double((int)w[3], (int)w[2]);
}

// This thread's scratch fields (its own E bins) in precision R, in chunks of
// VPC values.
template <typename R, int LOGN, int C>
struct TmScratch {
    using L = TmLayout<LOGN, C>;
    static constexpr int E = L::E;
    static constexpr int WPV = (int)(2 * sizeof(R) / 4);  // words per complex value
    // values per chunk: the loads of a chunk have to fit the registers
    // (FP64 with fewer than 16 values per thread: half as many)
    static constexpr int VPC = E < 4 ? E : sizeof(R) == 8 && E < 16 ? 2 : 4;
    static constexpr int CH = E / VPC;                    // chunks per field
    static constexpr int W = VPC * WPV < 8 ? 8 : VPC * WPV;  // words per chunk
    static_assert(!L::ENABLED || W == VPC * WPV, "a field is whole chunks");
    uint32_t a0;  // this warp's field 0, column 0
    __device__ explicit TmScratch(uint32_t tm) {
        const int w = threadIdx.x >> 5;
        a0 = tm + ((uint32_t)(32 * (w & 3)) << 16) + (uint32_t)((w >> 2) * L::COLS_WARP);
    }
    __device__ __forceinline__ uint32_t addr(int f, int c) const {
        return a0 + (uint32_t)(f * 4 * E + c * W);
    }
    __device__ __forceinline__ void put_chunk(int f, int c, const cx<R> (&v)[VPC]) const {
        uint32_t w[W];
#pragma unroll
        for (int j = 0; j < VPC; j++) pack_words(v[j], w + j * WPV);
        tm_st(addr(f, c), w);
    }
    __device__ __forceinline__ void get(int f, int c, cx<R> (&o)[VPC]) const {
        uint32_t w[W];
        tm_ld(addr(f, c), w);
        tm_wait_ld();
#pragma unroll
        for (int j = 0; j < VPC; j++) unpack_words(w + j * WPV, o[j]);
    }
    __device__ __forceinline__ void get2(int c, cx<R> (&o0)[VPC], cx<R> (&o1)[VPC]) const {
        uint32_t w0[W], w1[W];
        tm_ld(addr(0, c), w0);
        tm_ld(addr(1, c), w1);
        tm_wait_ld();
#pragma unroll
        for (int j = 0; j < VPC; j++) {
            unpack_words(w0 + j * WPV, o0[j]);
            unpack_words(w1 + j * WPV, o1[j]);
        }
    }
};

// Allocate the CTA's scratch columns (warp 0) and publish the address through
// the shared-memory slot; every thread of the CTA calls it.  The caller frees
// them with tm_free before the CTA exits.
template <int LOGN, int C>
__device__ __forceinline__ uint32_t tm_alloc(uint32_t* slot) {
    using L = TmLayout<LOGN, C>;
    if constexpr (!L::ENABLED) {
        return kNoTmem;
    } else {
        if ((threadIdx.x >> 5) == 0) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                             (uint32_t)__cvta_generic_to_shared(slot)),
                         "r"(L::COLS));
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        return *slot;
    }
}
template <int LOGN, int C>
__device__ __forceinline__ void tm_free(uint32_t tm) {
    using L = TmLayout<LOGN, C>;
    if constexpr (L::ENABLED) {
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        if ((threadIdx.x >> 5) == 0)
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tm),
                         "r"(L::COLS));
    }
}

struct NoLoad {  // the forward reads no stored field
    struct Raw {};
};

// What a run of right-hand-side evaluations starts from: the stages
// [stage, stage + count) of one attempt, or (stage 0) one evaluation of a
// given field.  Each stage's input is built in the registers its first
// transform starts from; the derivative of the stage before it is still there.
struct StageRun {
    int stage, count;
    const double* x;     // FP64 state (workspace order; stage 0 with xbin: bin order)
    int xbin;
    const void* k1;      // stage 0: x + c k1 (null: x); with x null: the field itself
    double c;
    double* copy;        // stage 0: x also goes here (nullable)
    void* out;           // stage 0: where the derivative goes
    double z, zload;     // stage 0: position, and that of the forward field (adjoint)
    char* kb;            // stage vectors, ks bytes apart, and their FSAL permutation
    size_t ks;
    int perm;
    // logical stage i: the permutation swaps stages 0 and 6 (an index, not a
    // table of pointers: a pointer load in front of every stage's data loads
    // cost as much as the data, 1.7 k of 5.4 k cycles per chunk at 2^10)
    __device__ __forceinline__ char* stage_vec(int i) const {
        const int p = perm && (i == 0 || i == 6) ? 6 - i : i;
        return kb + (size_t)p * ks;
    }
    double cz, dt;       // stage i is evaluated at cz + c_i dt
    double* xnew;        // stage 7: the new state
    int want_err;        // stage 7: also the error partial, weights and norm
    double at, rt;
    // adjoint: the stored steps [seg_lo, seg_hi) of the forward, or a field
    int seg_lo, seg_hi;
    const double* ufwd;
};

// Pieces of one problem's solve in RHS precision R over a group of C CTAs.
// Workspace fields (states, stages, scratch, checkpoints, interpolants) are
// private to the thread that owns their bins and lie in thread order
// (own(s)), tables and caller arrays in bin order (bin(s)).
//
// Code size is a first-order cost here: with one to four warps per scheduler
// nothing hides an instruction-cache miss, and every evaluation runs the
// whole body once.  So only the transforms and the pointwise terms between
// them are unrolled over the thread's values; the stage input and the
// derivative's way out are rolled loops over chunks of VPC values that pass
// through the scratch slots (tensor memory).  Unrolling those as well made
// the forward evaluation 147 KB of code instead of 44 KB and every part of
// it slower (Nt = 2^10: radix-16 pass with twiddles 711 against 474 cycles).
//
// Arithmetic runs in R, the stage vectors are stored in K.  The FP32 mode
// stores its forward stages and interpolants in FP32 but transforms in FP64:
// of the forward solve's error against FP64 nearly all comes from the two
// transforms of the field itself (rounding each to FP32 costs 0.5e-6 ..
// 2.5e-6 at the fiber's end, amplified by the modulation-instability gain;
// every other rounding 0.2e-6 together), and on an FP64 pipe at half the FP32
// rate the solves stay latency-bound: error 2e-7 instead of 1e-6 .. 2e-6.
template <typename R, typename K, int LOGN, int CL>
struct SmSolver {
    using XF = XForm<R, R, LOGN, CL>;
    static constexpr int N = XF::N, E = XF::E;
    static constexpr int P = sizeof(R) == 8 ? 1 : 0;  // table precision index
    using C = cx<R>;
    using CK = cx<K>;
    using TM = TmLayout<LOGN, CL>;
    using TMS = TmScratch<R, LOGN, CL>;
    static constexpr int VPC = TMS::VPC, CH = TMS::CH;
    static constexpr bool REGS = E == 2;  // slots in registers (2^6)
    // The forward's Raman convolution in FP32: on the grids of 4 or 8 values
    // per thread its two transforms are a third of an evaluation's FP64
    // latency (one solve at Nt = 2^10: 3.2 -> 2.7 ms).  On the larger ones
    // two more transform bodies cost more instruction fetch than they save
    // arithmetic (forward body at 2^13 105 KB; one solve at 2^14 9.4 -> 12.1
    // ms, 592 gradients at 2^13 unchanged).
    static constexpr bool CONV32 = sizeof(K) < sizeof(R) && SmShared<R, LOGN, CL>::BOTH;
    static constexpr bool PHC = REGS || TM::template phasors<R>();  // phasors kept in a slot
    static constexpr int PHF = sizeof(R) == 8 || REGS ? 2 : 1;       // ... this one

    const SlotDesc& d;
    XF xf;
    const C* __restrict__ Heff;
    const R* __restrict__ ss;
    const double* __restrict__ Dturns;
    C* scr0;
    C* scr1;
    uint32_t tm;  // tensor-memory scratch of the CTA, or kNoTmem: scr0 / scr1 in global memory
    mutable C slot_[REGS ? 3 : 1][E];

    __device__ SmSolver(const SlotDesc& dd, unsigned char* smem, int rank, uint32_t tmaddr = kNoTmem)
        : d(dd), xf(smem, smem_tables<R, LOGN, CL>(smem), rank),
          Heff((const C*)dd.Heff[P]), ss((const R*)dd.ss[P]), Dturns(dd.Dturns),
          scr0((C*)dd.scr[0]), scr1((C*)dd.scr[1]), tm(tmaddr) {}

    __device__ __forceinline__ int bin(int s) const { return xf.bin(s); }
    __device__ __forceinline__ int own(int s) const { return xf.own(s); }
    __device__ __forceinline__ bool tmem() const { return TM::ENABLED && tm != kNoTmem; }

    // ---- scratch slots: chunk c (values c VPC ..) of slot f ----
    __device__ __forceinline__ void put(int f, int c, const C (&v)[VPC]) const {
        if constexpr (REGS) {
#pragma unroll
            for (int j = 0; j < VPC; j++) slot_[f][j] = v[j];
        } else if (f < TM::FIELDS && tmem()) {
            TMS(tm).put_chunk(f, c, v);
        } else {
            C* s = f ? scr1 : scr0;
#pragma unroll
            for (int j = 0; j < VPC; j++) s[own(c * VPC + j)] = v[j];
        }
    }
    __device__ __forceinline__ void get(int f, int c, C (&v)[VPC]) const {
        if constexpr (REGS) {
#pragma unroll
            for (int j = 0; j < VPC; j++) v[j] = slot_[f][j];
        } else if (f < TM::FIELDS && tmem()) {
            TMS(tm).get(f, c, v);
        } else {
            const C* s = f ? scr1 : scr0;
#pragma unroll
            for (int j = 0; j < VPC; j++) v[j] = s[own(c * VPC + j)];
        }
    }
    __device__ __forceinline__ void wait_put() const {
        if (tmem()) tm_wait_st();
    }
    __device__ __forceinline__ void put_all(int f, const C (&v)[E]) const {
#pragma unroll
        for (int c = 0; c < CH; c++) {
            C t[VPC];
#pragma unroll
            for (int j = 0; j < VPC; j++) t[j] = v[c * VPC + j];
            put(f, c, t);
        }
        wait_put();
    }
    __device__ __forceinline__ void get_all(int f, C (&v)[E]) const {
#pragma unroll
        for (int c = 0; c < CH; c++) {
            C t[VPC];
            get(f, c, t);
#pragma unroll
            for (int j = 0; j < VPC; j++) v[c * VPC + j] = t[j];
        }
    }

    // The transforms of one right-hand side, forward (adj = false) or
    // adjoint, from the input in v (ũ e^{iDz}, or λ̃ e^{iDz} τ with
    // ũ(z) e^{iDz} in slot 1) to the nonlinear term back in frequency, as a
    // runtime loop over the transforms so the kernel holds one
    // copy of each direction (inverse transforms run as conj∘F∘conj):
    //   forward  f0: -F-> u_t                 f1: (γ|u_t|², 0) -F->
    //            f2: ·Heff -F⁻¹-> N h∗I       f3: ((1-fR)I + h∗I) u_t -F⁻¹->
    //   adjoint  f0: -F-> λ_t                 f1: -F-> u_t
    //            f2: (I, Y) -F-> X            f3: split X into Î, Ŷ;
    //                Heff Î + i conj(Heff) Ŷ -F⁻¹-> N (h∗I + i h̃⋆Y)
    //            f4: η -F⁻¹->
    __device__ __forceinline__ void transforms(const bool adj, C (&v)[E]) const {
        const R g = (R)d.gamma, ofr = (R)d.one_m_fR, invn = R(1) / R(N);
        if constexpr (CONV32) {
            if (!adj) {
                forward32(v, g, ofr, invn);
                return;
            }
        }
        const int nfft = adj ? 5 : 4;
#pragma unroll 1
        for (int f = 0; f < nfft; f++) {
            bool inv = false, to_a = false, presync = false;
            const int op = adj ? 8 + f : f;
            if (op == 1) {
                put_all(0, v);
#pragma unroll
                for (int s = 0; s < E; s++) v[s] = mk(g * abs2(v[s]), R(0));
                to_a = true;
            } else if (op == 2) {
#pragma unroll
                for (int s = 0; s < E; s++) v[s] = cmul(v[s], Heff[bin(s)]);
                inv = true;
            } else if (op == 3) {
#pragma unroll
                for (int c = 0; c < CH; c++) {
                    C u[VPC];
                    get(0, c, u);
#pragma unroll
                    for (int j = 0; j < VPC; j++) {
                        const int s = c * VPC + j;
                        const R fac = ofr * (g * abs2(u[j])) + v[s].re * invn;
                        v[s] = scale(u[j], fac);
                    }
                }
                inv = to_a = true;
            } else if (op == 9) {
                put_all(0, v);
                get_all(1, v);
                presync = true;  // f0's warps may still be in the region buffer
            } else if (op == 10) {
                put_all(1, v);
#pragma unroll
                for (int c = 0; c < CH; c++) {
                    C l[VPC];
                    get(0, c, l);
#pragma unroll
                    for (int j = 0; j < VPC; j++) {
                        const int s = c * VPC + j;
                        const R I = g * abs2(v[s]);
                        const R Y = g * (l[j].im * v[s].re - l[j].re * v[s].im);  // γ Im(λ u*)
                        v[s] = mk(I, Y);
                    }
                }
                to_a = true;
            } else if (op == 11) {
                // split the two real spectra (I and Y) with X[k] and conj(X[-k]):
                // Î = (X[k] + conj(X[-k]))/2, i Ŷ = (X[k] - conj(X[-k]))/2;
                // Heff Î + i conj(Heff) Ŷ = Re Heff X[k] + i Im Heff conj(X[-k])
                xf.mirror_apply(v, Heff);
                inv = true;
            } else if (op == 12) {
                // η = λ_t (2(1-fR) I + h∗I) - (1-fR) γ λ_t* u_t² + 2i (h̃⋆Y) u_t
#pragma unroll
                for (int c = 0; c < CH; c++) {
                    C l[VPC], u[VPC];
                    if (TM::FIELDS > 1 && tmem()) {
                        TMS(tm).get2(c, l, u);
                    } else {
                        get(0, c, l);
                        get(1, c, u);
                    }
#pragma unroll
                    for (int j = 0; j < VPC; j++) {
                        const C lt = l[j], ut = u[j], x = v[c * VPC + j];
                        const R I = g * abs2(ut);
                        const R Rr = x.re * invn, Ri = x.im * invn;
                        const C t1 = scale(lt, R(2) * ofr * I + Rr);
                        const C t2 = scale(cmulc(cmul(ut, ut), lt), ofr * g);    // (1-fR)γ λ* u²
                        const C t3 = mk(-R(2) * Ri * ut.im, R(2) * Ri * ut.re);  // 2i Ri u
                        v[c * VPC + j] = t1 - t2 + t3;
                    }
                }
                inv = to_a = true;
            }
            if (inv) conj_all(v);
            xf.transform(v, to_a, presync);
            if (inv) conj_all(v);
        }
    }

    // The forward with its Raman convolution (f1, f2) in FP32
    __device__ __forceinline__ void forward32(C (&v)[E], const R g, const R ofr, const R invn) const {
        using F = cx<float>;
        const F* __restrict__ H = (const F*)d.Heff[0];
        XForm<float, R, LOGN, CL> xc(
            xf.sm, reinterpret_cast<const F*>(xf.sm + SmShared<R, LOGN, CL>::TAB32), xf.rank);
        xf.transform(v, false, false);
        put_all(0, v);
        F w[E];
#pragma unroll
        for (int s = 0; s < E; s++) w[s] = mk((float)(g * abs2(v[s])), 0.f);
        xc.flip = xf.flip;
        xc.transform(w, true, false);
#pragma unroll
        for (int s = 0; s < E; s++) w[s] = conjc(cmul(w[s], H[bin(s)]));
        xc.transform(w, false, false);  // real: its conjugate is not needed
        xf.flip = xc.flip;
#pragma unroll
        for (int c = 0; c < CH; c++) {
            C u[VPC];
            get(0, c, u);
#pragma unroll
            for (int j = 0; j < VPC; j++) {
                const int s = c * VPC + j;
                // (which product the compiler fuses would depend on the instance)
                const R fac = fma((R)w[s].re, invn, ofr * (g * abs2(u[j])));
                v[s] = conjc(scale(u[j], fac));
            }
        }
        xf.transform(v, true, false);
        conj_all(v);
    }

    // ---- stage helpers ---------------------------------------------------
    // logical stage i -> physical buffer; perm swaps stages 0 and 6 (FSAL)
    __device__ __forceinline__ static CK* kp(void* const* k, int perm, int i) {
        int p = (perm && (i == 0 || i == 6)) ? 6 - i : i;
        return (CK*)k[p];
    }

    // The input field of stage st, with its phasors, into the slots: stages
    // 1..5 ũ_n + dt Σ_{j<st} a[st][j] k_j (FP64 accumulation, stage 0
    // first); 6 the new state, written to xnew in FP64, and the partial error
    // dt Σ_{j<6} b̃_j k_j; 0 the probe field x + c k1.  All stage loads of a chunk are issued
    // before the first is used: one L2 latency per chunk, where a loop over
    // the stages waited for each.
    template <bool ADJ, class Load>
    __device__ __forceinline__ void input(const StageRun& in, const int st, const double z,
                                          const Load& ld) const {
        const CK* k[6];
        double a[6];
#pragma unroll
        for (int j = 0; j < 6; j++) {
            k[j] = (const CK*)in.stage_vec(j);
            a[j] = kT5a[st][j];
        }
        const double dt = in.dt;
#pragma unroll 1
        for (int c = 0; c < CH; c++) {
            const int s0 = c * VPC;
            C y[VPC], ph[VPC];
            double Dt[VPC];
            R tau[VPC];
            cx<double> un[VPC];
            typename Load::Raw raw;
            if (st > 0) {
                CK x[6][VPC];
#pragma unroll
                for (int j = 0; j < 6; j++)
                    if (j < st) {
#pragma unroll
                        for (int i = 0; i < VPC; i++) x[j][i] = k[j][own(s0 + i)];
                    }
#pragma unroll
                for (int i = 0; i < VPC; i++) un[i] = ld2(in.x, own(s0 + i));
#pragma unroll
                for (int i = 0; i < VPC; i++) Dt[i] = Dturns[bin(s0 + i)];
                if constexpr (ADJ) {
#pragma unroll
                    for (int i = 0; i < VPC; i++) tau[i] = ss[bin(s0 + i)];
                    ld.fetch(s0, raw);
                }
                double ar[VPC], ai[VPC];
#pragma unroll
                for (int i = 0; i < VPC; i++) ar[i] = ai[i] = 0.0;
#pragma unroll
                for (int j = 0; j < 6; j++)
                    if (j < st) {
#pragma unroll
                        for (int i = 0; i < VPC; i++) {
                            ar[i] += a[j] * (double)x[j][i].re;
                            ai[i] += a[j] * (double)x[j][i].im;
                        }
                    }
#pragma unroll
                for (int i = 0; i < VPC; i++)
                    y[i] = mk((R)(un[i].re + dt * ar[i]), (R)(un[i].im + dt * ai[i]));
                if (st == 6) {
                    double er[VPC], ei[VPC];
#pragma unroll
                    for (int i = 0; i < VPC; i++) er[i] = ei[i] = 0.0;
#pragma unroll
                    for (int j = 0; j < 6; j++) {
                        const double bt = kT5bt[j];
#pragma unroll
                        for (int i = 0; i < VPC; i++) {
                            er[i] += bt * (double)x[j][i].re;
                            ei[i] += bt * (double)x[j][i].im;
                        }
                    }
#pragma unroll
                    for (int i = 0; i < VPC; i++) {
                        const int b = own(s0 + i);
                        const cx<double> u1 = mk(un[i].re + dt * ar[i], un[i].im + dt * ai[i]);
                        st2(in.xnew, b, u1);
                        if (in.want_err) st2(d.esv, b, mk(dt * er[i], dt * ei[i]));
                    }
                }
            } else {
                const CK* k1 = (const CK*)in.k1;
#pragma unroll
                for (int i = 0; i < VPC; i++) {
                    const int s = s0 + i;
                    Dt[i] = Dturns[bin(s)];
                    if constexpr (ADJ) tau[i] = ss[bin(s)];
                    const CK f0 = k1 ? k1[own(s)] : mk(K(0), K(0));
                    const cx<double> x = in.x ? ld2(in.x, in.xbin ? bin(s) : own(s)) : up(f0);
                    if (in.copy) st2(in.copy, own(s), x);
                    y[i] = k1 && in.x
                               ? mk((R)(x.re + in.c * (double)f0.re), (R)(x.im + in.c * (double)f0.im))
                               : down<R>(x);
                }
                if constexpr (ADJ) ld.fetch(s0, raw);
            }
#pragma unroll
            for (int i = 0; i < VPC; i++) {
                ph[i] = phasor<R>(Dt[i], z);
                y[i] = cmul(y[i], ph[i]);
                if constexpr (ADJ) y[i] = scale(y[i], tau[i]);
            }
            put(0, c, y);
            if constexpr (ADJ) {
                C u[VPC];
                ld.eval(raw, s0, u);
#pragma unroll
                for (int i = 0; i < VPC; i++) u[i] = cmul(u[i], ph[i]);
                put(1, c, u);
            }
            if constexpr (PHC) put(PHF, c, ph);
        }
        wait_put();
    }

    // slot 0 -> the derivative i e^{-iDz} (τ) x / N, stored in out; the
    // thread's part of the error norm when the derivative is k7 of an attempt
    template <bool ADJ>
    __device__ __forceinline__ double output(const StageRun& in, const int st, const double z,
                                             CK* out) const {
        const R invn = R(1) / R(N);
#pragma unroll 1
        for (int c = 0; c < CH; c++) {
            const int s0 = c * VPC;
            C v[VPC], ph[VPC];
            R sc[VPC];
            if constexpr (!PHC) {
                double Dt[VPC];
#pragma unroll
                for (int i = 0; i < VPC; i++) Dt[i] = Dturns[bin(s0 + i)];
#pragma unroll
                for (int i = 0; i < VPC; i++) ph[i] = phasor<R>(Dt[i], z);
            } else {
                get(PHF, c, ph);
            }
#pragma unroll
            for (int i = 0; i < VPC; i++) sc[i] = ADJ ? invn : ss[bin(s0 + i)] * invn;
            get(0, c, v);
#pragma unroll
            for (int i = 0; i < VPC; i++) {
                const C y = cmulc(v[i], ph[i]);  // e^{-iDz} x
                out[own(s0 + i)] = mk((K)(-y.im * sc[i]), (K)(y.re * sc[i]));
            }
        }
        return st == 6 && in.want_err ? error_norm(in, out) : 0.0;
    }
    // the thread's part of the error norm, k7 in k: Σ |dt Σ b̃_j k_j|² / w²,
    // w = abstol + reltol max(|u_n|, |u_{n+1}|)
    __device__ __forceinline__ double error_norm(const StageRun& in, const CK* k) const {
        const double dt = in.dt, bt = kT5bt[6];
        // (four values in flight; two beside the unrolled evaluations, where four
        // cost 592 gradients at 2^13 135.5 ms for 134.7)
        constexpr int NC = WIDE ? 2 : E < 4 ? E : 4;
        double acc = 0.0;
#pragma unroll 1
        for (int s0 = 0; s0 < E; s0 += NC) {
            CK v[NC];
            cx<double> e6[NC], un[NC], u1[NC];
#pragma unroll
            for (int i = 0; i < NC; i++) {
                const int b = own(s0 + i);
                v[i] = k[b];
                e6[i] = ld2(d.esv, b);
                un[i] = ld2(in.x, b);
                u1[i] = ld2(in.xnew, b);
            }
#pragma unroll
            for (int i = 0; i < NC; i++) {
                const double m0 = un[i].re * un[i].re + un[i].im * un[i].im;
                const double m1 = u1[i].re * u1[i].re + u1[i].im * u1[i].im;
                const double w = rcp_nb(in.at + sqrt_nb(fmax(m0, m1)) * in.rt);
                // (w * w would leave the range where the tolerances are below 1e-154)
                const double er = (e6[i].re + dt * bt * (double)v[i].re) * w;
                const double ei = (e6[i].im + dt * bt * (double)v[i].im) * w;
                acc += er * er + ei * ei;
            }
        }
        return acc;
    }

    // The same with the thread's values unrolled, in registers from the input
    // to the stored derivative, for CTAs of 8 warps and more (2^12 to 2^14 on
    // one CTA, 2^13 on two).  There the warps hide
    // one another's latencies and instruction fetches, and the loads in
    // flight per thread decide: at Nt = 2^13 on one CTA the rolled loops
    // above took 27.6 ms per gradient, this form 22.5.
    static constexpr bool WIDE = XF::TC >= 256 && E >= 16;
    static constexpr int SC = E < 8 ? E : 8;
    template <bool ADJ, class Load>
    __device__ __forceinline__ void input_wide(const StageRun& in, const int st, const double z,
                                               const Load& ld, C (&v)[E]) const {
        const double dt = in.dt;
        if (st > 0 && st < 6) {
#pragma unroll
            for (int s0 = 0; s0 < E; s0 += SC) {
                double ar[SC], ai[SC];
#pragma unroll
                for (int c = 0; c < SC; c++) ar[c] = ai[c] = 0.0;
#pragma unroll 1
                for (int j = 0; j < st; j++) {
                    const CK* __restrict__ kj = (const CK*)in.stage_vec(j);
                    const double a = kT5a[st][j];
                    CK x[SC];
#pragma unroll
                    for (int c = 0; c < SC; c++) x[c] = kj[own(s0 + c)];
#pragma unroll
                    for (int c = 0; c < SC; c++) {
                        ar[c] += a * (double)x[c].re;
                        ai[c] += a * (double)x[c].im;
                    }
                }
#pragma unroll
                for (int c = 0; c < SC; c++) {
                    const cx<double> un = ld2(in.x, own(s0 + c));
                    v[s0 + c] = mk((R)(un.re + dt * ar[c]), (R)(un.im + dt * ai[c]));
                }
            }
        } else if (st == 6) {
            constexpr int SC7 = sizeof(R) == 8 ? 4 : 8;  // two sums per point
#pragma unroll
            for (int s0 = 0; s0 < E; s0 += SC7) {
                double ar[SC7], ai[SC7], er[SC7], ei[SC7];
#pragma unroll
                for (int c = 0; c < SC7; c++) ar[c] = ai[c] = er[c] = ei[c] = 0.0;
#pragma unroll 1
                for (int j = 0; j < 6; j++) {
                    const CK* __restrict__ kj = (const CK*)in.stage_vec(j);
                    const double a = kT5a[6][j], bt = kT5bt[j];
                    CK x[SC7];
#pragma unroll
                    for (int c = 0; c < SC7; c++) x[c] = kj[own(s0 + c)];
#pragma unroll
                    for (int c = 0; c < SC7; c++) {
                        ar[c] += a * (double)x[c].re;
                        ai[c] += a * (double)x[c].im;
                        er[c] += bt * (double)x[c].re;
                        ei[c] += bt * (double)x[c].im;
                    }
                }
#pragma unroll
                for (int c = 0; c < SC7; c++) {
                    const int b = own(s0 + c);
                    const cx<double> un = ld2(in.x, b);
                    const cx<double> u1 = mk(un.re + dt * ar[c], un.im + dt * ai[c]);
                    st2(in.xnew, b, u1);
                    if (in.want_err) st2(d.esv, b, mk(dt * er[c], dt * ei[c]));
                    v[s0 + c] = down<R>(u1);
                }
            }
        } else {
            const CK* k1 = (const CK*)in.k1;
#pragma unroll 4
            for (int s = 0; s < E; s++) {
                const CK f0 = k1 ? k1[own(s)] : mk(K(0), K(0));
                const cx<double> x = in.x ? ld2(in.x, in.xbin ? bin(s) : own(s)) : up(f0);
                if (in.copy) st2(in.copy, own(s), x);
                scr0[own(s)] = k1 && in.x
                                   ? mk((R)(x.re + in.c * (double)f0.re), (R)(x.im + in.c * (double)f0.im))
                                   : down<R>(x);
            }
#pragma unroll
            for (int s = 0; s < E; s++) v[s] = scr0[own(s)];
        }
        phasors_and_field<ADJ>(z, ld);
#pragma unroll
        for (int c = 0; c < CH; c++) {
            C ph[VPC];
            get(PHS, c, ph);
#pragma unroll
            for (int i = 0; i < VPC; i++) {
                const int s = c * VPC + i;
                v[s] = cmul(v[s], ph[i]);
                if constexpr (ADJ) v[s] = scale(v[s], ss[bin(s)]);
            }
        }
    }
    // the evaluation's phasors into a slot -- the one they stay in, or slot 0
    // before and after the transforms need it -- and ũ(z) e^{iDz} into slot 1
    static constexpr int PHS = PHC ? PHF : 0;
    template <bool ADJ, class Load>
    __device__ __forceinline__ void phasors_and_field(const double z, const Load& ld) const {
#pragma unroll 1
        for (int c = 0; c < CH; c++) {
            typename Load::Raw raw;
            C u[VPC], ph[VPC];
            double Dt[VPC];
#pragma unroll
            for (int i = 0; i < VPC; i++) Dt[i] = Dturns[bin(c * VPC + i)];
            if constexpr (ADJ) ld.fetch(c * VPC, raw);
#pragma unroll
            for (int i = 0; i < VPC; i++) ph[i] = phasor<R>(Dt[i], z);
            put(PHS, c, ph);
            if constexpr (ADJ) {
                ld.eval(raw, c * VPC, u);
#pragma unroll
                for (int i = 0; i < VPC; i++) u[i] = cmul(u[i], ph[i]);
                put(1, c, u);
            }
        }
        wait_put();
    }
    template <bool ADJ>
    __device__ __forceinline__ double output_wide(const StageRun& in, const int st, const double z,
                                                  C (&v)[E], CK* out) const {
        const R invn = R(1) / R(N);
        if constexpr (!PHC) phasors_and_field<false>(z, NoLoad{});
#pragma unroll
        for (int c = 0; c < CH; c++) {
            C ph[VPC];
            get(PHS, c, ph);
#pragma unroll
            for (int i = 0; i < VPC; i++) {
                const int s = c * VPC + i;
                const C y = cmulc(v[s], ph[i]);  // e^{-iDz} x
                const R sc = ADJ ? invn : ss[bin(s)] * invn;
                out[own(s)] = mk((K)(-y.im * sc), (K)(y.re * sc));
            }
        }
        return st == 6 && in.want_err ? error_norm(in, out) : 0.0;
    }

    // The run's evaluations; make_load(z) prepares the forward field's
    // loader.  Returns the thread's part of the error norm after stage 6.
    template <bool ADJ, class MakeLoad>
    __device__ __forceinline__ double run(const StageRun& in, MakeLoad&& make_load) {
        double acc = 0.0;
        const int end = in.stage == 0 ? 1 : in.stage + in.count;
        // E <= 8: the run starts at the first exchange buffer, which the run
        // before may still be reading
        if constexpr (XF::S::SMALL) XF::sync();
#pragma unroll 1
        for (int st = in.stage; st < end; st++) {
            const double z = st == 0 ? in.z : in.cz + kT5c[st] * in.dt;
            const auto ld = make_load(*this, st == 0 ? in.zload : z);
            CK* out = (CK*)(st == 0 ? (char*)in.out : in.stage_vec(st));
            C v[E];
            if constexpr (WIDE) {
                input_wide<ADJ>(in, st, z, ld, v);
            } else {
                input<ADJ>(in, st, z, ld);
                get_all(0, v);
            }
            transforms(ADJ, v);
            if constexpr (WIDE) {
                acc = output_wide<ADJ>(in, st, z, v, out);
            } else {
                put_all(0, v);
                acc = output<ADJ>(in, st, z, out);
            }
        }
        return acc;
    }
};

// PI controller: returns q and q11 (OrdinaryDiffEqCore stepsize_controller!)
__device__ __forceinline__ double pi_q(double EEst, double qold, double& q11) {
    if (EEst == 0.0) {
        q11 = 0.0;
        return 1.0 / kQmax;
    }
    q11 = pow(EEst, kBeta1);
    double q = q11 / pow(qold, kBeta2);
    q = q / kGamma;
    return fmax(1.0 / kQmax, fmin(1.0 / kQmin, q));
}

// Hairer initial step from the norms of the launch, f0 and the probe f1
// (OrdinaryDiffEqCore ode_determine_initdt; 5 = the method order).
__device__ __forceinline__ double initdt_first(double d0, double d1, double span) {
    double dt0 = (d0 < 1e-5 || d1 < 1e-5) ? 1e-6 : (d0 / d1) / 100.0;
    return fmin(dt0, span);
}
__device__ __forceinline__ double initdt_final(double dt0, double d1, double d2, double nd,
                                               double dtmin, double span) {
    if (nd == 0.0) return fmax(dtmin, 100 * dt0);  // constant derivative over the probe
    const double mx = fmax(d1, d2);
    const double dt1 = mx <= 1e-15 ? fmax(1e-6, dt0 * 1e-3) : pow(10.0, -(2.0 + log10(mx)) / 5.0);
    return fmax(dtmin, fmin(fmin(100 * dt0, dt1), span));
}

// Forward field for the adjoint RHS: the dense interpolant (precision RF) of
// the stored step of the current segment that holds zz, or an FP64 field
// given directly (bin order).
template <typename RF>
struct SegNode {
    int n = -1;              // the stored step found last, its start and length,
    double z0, dt, z1;       // and the start of the next one
    // the last stored step in [lo, hi) starting at or before zz (the logged
    // step starts increase).  Successive evaluations mostly stay in one step
    // or move to a neighbour, so the search starts from the last one found
    // and reads the log only when it moves.
    __device__ __forceinline__ void find(const double* lg, int lo, int hi, double zz) {
        if (n < lo || n >= hi) {  // by bisection
            int a = lo, b = hi - 1;
            while (a < b) {
                const int mid = (a + b + 1) >> 1;
                if (lg[2 * mid] <= zz) a = mid;
                else b = mid - 1;
            }
            set(lg, a, hi);
            return;
        }
        while (n > lo && z0 > zz) set(lg, n - 1, hi);
        while (n < hi - 1 && z1 <= zz) set(lg, n + 1, hi);
    }
    __device__ __forceinline__ void set(const double* lg, int i, int hi) {
        n = i;
        z0 = lg[2 * i];
        dt = lg[2 * i + 1];
        z1 = i + 1 < hi ? lg[2 * i + 2] : INFINITY;
    }
};
template <typename RF, class Sol>
struct SegLoader {
    static constexpr int N = Sol::N, VPC = Sol::VPC;
    const Sol& S;
    const double* direct;
    const cx<RF>* sg;
    double th, dtn;
    // the stored values of a chunk
    struct Raw {
        cx<RF> c[5][VPC];
    };
    __device__ __forceinline__ void fetch(int s0, Raw& w) const {
        if (!direct) {
#pragma unroll
            for (int q = 0; q < 5; q++)
#pragma unroll
                for (int j = 0; j < VPC; j++) w.c[q][j] = sg[(size_t)q * N + S.own(s0 + j)];
        }
    }
    // ũ at values s0 .. s0 + VPC - 1 of this thread
    __device__ __forceinline__ void eval(const Raw& r, int s0, typename Sol::C (&w)[VPC]) const {
        if (direct) {
#pragma unroll
            for (int j = 0; j < VPC; j++) {
                const cx<double> x = ld2(direct, S.bin(s0 + j));
                w[j].re = x.re;
                w[j].im = x.im;
            }
            return;
        }
        const double t2 = th * th, t3 = t2 * th, t4 = t3 * th;
#pragma unroll
        for (int j = 0; j < VPC; j++) {
            w[j].re = (double)r.c[0][j].re +
                      dtn * (th * (double)r.c[1][j].re + t2 * (double)r.c[2][j].re +
                             t3 * (double)r.c[3][j].re + t4 * (double)r.c[4][j].re);
            w[j].im = (double)r.c[0][j].im +
                      dtn * (th * (double)r.c[1][j].im + t2 * (double)r.c[2][j].im +
                             t3 * (double)r.c[3][j].im + t4 * (double)r.c[4][j].im);
        }
    }
};
// Out-of-line runs of RHS evaluations: the transform bodies get the full
// register budget of the CTA instead of sharing it with the state machine's
// live values.
template <typename R, typename K, int LOGN, int CL>
__device__ __noinline__ double rhs_fwd_call(const SlotDesc* d, unsigned char* sm, int rank,
                                            const StageRun* in, uint32_t tm = kNoTmem) {
    using Sol = SmSolver<R, K, LOGN, CL>;
    Sol S(*d, sm, rank, tm);
    return S.template run<false>(*in, [](const Sol&, double) { return NoLoad{}; });
}

template <typename RF, typename R, int LOGN, int CL>
__device__ __noinline__ double rhs_adj_call(const SlotDesc* d, unsigned char* sm, int rank,
                                            const StageRun* in, uint32_t tm = kNoTmem) {
    using Sol = SmSolver<R, R, LOGN, CL>;
    Sol S(*d, sm, rank, tm);
    SegNode<RF> node;
    return S.template run<true>(*in, [&](const Sol& sol, double zz) {
        SegLoader<RF, Sol> ld{sol, in->ufwd, nullptr, 0.0, 0.0};
        if (!in->ufwd) {
            node.find(d->steplog, in->seg_lo, in->seg_hi, zz);
            ld.dtn = node.dt;
            ld.th = (zz - node.z0) / node.dt;
            ld.sg = (const cx<RF>*)d->seg + (size_t)(node.n - in->seg_lo) * 5 * Sol::N;
        }
        return ld;
    });
}

// the shared-memory word tcgen05.alloc writes the tensor-memory address to
template <typename RMAX, int LOGN, int CL>
__device__ __forceinline__ uint32_t* tm_slot(unsigned char* smraw) {
    return reinterpret_cast<uint32_t*>(smraw + SmShared<RMAX, LOGN, CL>::SLOT);
}

// One RHS evaluation on one CTA (unit parity of the right-hand sides):
// in/ufwd/out are N complex doubles; forward in RF, adjoint in RA.
template <typename RF, typename RA, int LOGN>
__global__ void __launch_bounds__(XShape<LOGN, 1>::T, 1)
    sm_rhs_kernel(const SlotDesc* __restrict__ d, int adjoint, double z,
                  const double* __restrict__ in, const double* __restrict__ ufwd,
                  double* __restrict__ out) {
    using XF = XForm<RA, RA, LOGN, 1>;
    extern __shared__ __align__(16) unsigned char smraw[];
    const uint32_t tm = tm_alloc<LOGN, 1>(tm_slot<RA, LOGN, 1>(smraw));
    load_tables<RA, LOGN, 1>(*d, smraw, 0);
    StageRun si{};
    si.x = in;
    si.xbin = 1;
    si.z = si.zload = z;
    si.ufwd = ufwd;
    si.out = adjoint ? d->ka[0] : d->kf[0];
    const XF xf(smraw, nullptr, 0);
    if (adjoint) {
        rhs_adj_call<RF, RA, LOGN, 1>(d, smraw, 0, &si, tm);
        const cx<RA>* k = (const cx<RA>*)d->ka[0];
#pragma unroll
        for (int s = 0; s < XF::E; s++) st2(out, xf.bin(s), up(k[xf.own(s)]));
    } else {
        rhs_fwd_call<RA, RF, LOGN, 1>(d, smraw, 0, &si, tm);
        const cx<RF>* k = (const cx<RF>*)d->kf[0];
#pragma unroll
        for (int s = 0; s < XF::E; s++) st2(out, xf.bin(s), up(k[xf.own(s)]));
    }
    tm_free<LOGN, 1>(tm);
}

// Steps [lo, hi) of the current sub-segment: the segment of checkpoint seg
// (ck_stride steps) is replayed and integrated backward in sub-segments of at
// most seg_cap steps, last first.  Each sub-segment replays the segment from
// its checkpoint; the steps before the sub-segment are recomputed without
// storing their interpolant, so a solve of any length fits the K checkpoints
// and the seg_cap-step interpolant buffer (at the cost of recomputation that
// grows with ck_stride / seg_cap) instead of failing for capacity.
// (Shared by the single-mode and the multimode steppers: Desc / State are
// SlotDesc / SlotState or MmDesc / MmState.)
struct SubSeg {
    int seg_lo, seg_hi, lo, hi;
};
template <class Desc, class State>
__device__ __forceinline__ SubSeg sub_segment(const Desc& d, const State& st) {
    SubSeg r;
    if (st.dense) {  // the forward kept the interpolant of every step: one range
        r.seg_lo = r.lo = 0;
        r.seg_hi = r.hi = st.nsteps;
        return r;
    }
    r.seg_lo = st.seg * st.ck_stride;
    r.seg_hi = min(r.seg_lo + st.ck_stride, st.nsteps);
    r.lo = r.seg_lo + st.sub * d.seg_cap;
    r.hi = min(r.lo + d.seg_cap, r.seg_hi);
    return r;
}
// index of the last sub-segment of segment seg
template <class Desc, class State>
__device__ __forceinline__ int last_sub(const Desc& d, const State& st, int seg) {
    const int lo = seg * st.ck_stride, hi = min(lo + st.ck_stride, st.nsteps);
    return (hi - lo - 1) / d.seg_cap;
}

// Dense interpolant of an accepted step into sg (5 fields): c0 = ũ_n,
// c_p = Σ_i r_ip k_i (Tsit5's free 4th-order interpolant); all stage loads
// of a chunk of points in flight together, as in SmSolver::input.
template <typename RF, class Sol>
__device__ __forceinline__ void store_interp(const Sol& S, const double* u, int kperm,
                                             cx<RF>* sg) {
    using CF = cx<RF>;
    const SlotDesc& d = S.d;
    constexpr int N = Sol::N, E = Sol::E;
    constexpr int RC = E < 4 ? E : 4;
    static_assert(E % RC == 0, "chunks tile the thread's points");
    const CF* k[7];
    const size_t kfs = (CF*)d.kf[1] - (CF*)d.kf[0];
#pragma unroll
    for (int i = 0; i < 7; i++)
        k[i] = (const CF*)d.kf[0] + (size_t)(kperm && (i == 0 || i == 6) ? 6 - i : i) * kfs;
#pragma unroll 1
    for (int s0 = 0; s0 < E; s0 += RC) {
        CF x[7][RC];
        cx<double> un[RC];
#pragma unroll
        for (int i = 0; i < 7; i++)
#pragma unroll
            for (int c = 0; c < RC; c++) x[i][c] = k[i][S.own(s0 + c)];
#pragma unroll
        for (int c = 0; c < RC; c++) un[c] = ld2(u, S.own(s0 + c));
#pragma unroll
        for (int c = 0; c < RC; c++) {
            const int b = S.own(s0 + c);
            sg[b] = down<RF>(un[c]);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                double cr = 0.0, ci = 0.0;
#pragma unroll
                for (int i = 0; i < 7; i++) {
                    cr += kT5r[i][q] * (double)x[i][c].re;
                    ci += kT5r[i][q] * (double)x[i][c].im;
                }
                sg[(size_t)(q + 1) * N + b] = mk((RF)cr, (RF)ci);
            }
        }
    }
}

// Checked build (-DFL_CHECKED): before each step of the state machine, the
// indices a step will use -- stage, buffer parities, the step count against
// the step log, the checkpoint segment and sub-segment against the
// checkpoint slots and the interpolant buffer, the save position -- are
// checked against their buffers.  A violation ends the slot with ST_CHECK
// (FL_ECHECK) before any access, instead of trapping.  The default build
// compiles the check away.  Shared by both steppers (SlotDesc / SlotState,
// MmDesc / MmState).
template <class Desc, class State>
__device__ __forceinline__ bool state_in_bounds(const Desc& d, const State& st) {
    bool ok = st.stage >= 0 && st.stage <= 6 && (st.cur | st.kperm | st.acur | st.akperm) >= 0 &&
              (st.cur | st.kperm | st.acur | st.akperm) <= 1 && st.save_idx >= 0 &&
              st.save_idx <= d.nsave && st.nsteps >= 0 &&
              (d.step_cap == 0 || st.nsteps <= d.step_cap);
    const int ph = st.phase;
    if (ok && (ph == PH_REC || ph == PH_ADJ_INIT || ph == PH_ADJ)) {
        const SubSeg sb = sub_segment(d, st);
        // a replay has steps left in its sub-segment; the adjoint follows a
        // finished replay (rec_pos at the sub-segment's end)
        const int rec_end = sb.seg_lo + st.rec_pos;
        ok = d.step_cap > 0 && st.nsteps >= 1 && sb.lo >= 0 && sb.lo < sb.hi &&
             sb.hi <= st.nsteps && sb.hi - sb.lo <= d.seg_cap && st.rec_pos >= 0 &&
             (st.dense || (st.seg >= 0 && st.seg < d.ck_cap && st.ck_stride >= 1 &&
                           (ph == PH_REC ? rec_end < sb.hi : rec_end <= sb.hi)));
    }
    return ok;
}

template <typename RF, class Sol>
__device__ __forceinline__ void restore_checkpoint(const Sol& S, int seg, SlotState& st) {
    const SlotDesc& d = S.d;
    constexpr int N = Sol::N, E = Sol::E;
#pragma unroll 4
    for (int s = 0; s < E; s++) {
        const int b = S.own(s);
        reinterpret_cast<double2*>(d.u[0])[b] =
            reinterpret_cast<const double2*>(d.ck_u)[(size_t)seg * N + b];
        ((cx<RF>*)d.kf[0])[b] = ((const cx<RF>*)d.ck_k1)[(size_t)seg * N + b];
    }
    st.cur = 0;
    st.kperm = 0;
    st.rec_pos = 0;
    st.stage = 0;
}

// Hairer initial step, part 1 (after f0, in k1): the probe step dt0 (> 0)
// or, when no probe is needed, -dtinit.  x0 in bin order for the launch.
template <typename K, class Sol, class SumF>
__device__ __forceinline__ double init_after_f0(const Sol& S, const double* x0, bool xbin,
                                                const cx<K>* k1, double at, double rt, double L,
                                                double dtmin, SumF&& sum, double& d1_out) {
    constexpr int N = Sol::N, E = Sol::E;
    double s0 = 0.0, s1 = 0.0;
#pragma unroll 4
    for (int s = 0; s < E; s++) {
        const cx<double> x = ld2(x0, xbin ? S.bin(s) : S.own(s));
        const double ax = sqrt(x.re * x.re + x.im * x.im);
        const double sk = at + ax * rt;
        s0 += (ax / sk) * (ax / sk);
        const double af = sqrt(abs2(up(k1[S.own(s)])));
        s1 += (af / sk) * (af / sk);
    }
    const double d0 = sqrt(sum(s0) / N);
    const double d1 = sqrt(sum(s1) / N);
    d1_out = d1;
    const double dt0 = initdt_first(d0, d1, L);
    if (!isfinite(d1)) return -dtmin;
    if (dt0 < 10 * kEps) return -fmax(1e-6, dtmin);
    return dt0;
}

// Hairer initial step, part 2 (after the probe f1 at x0 ± dt0 f0, in kp)
template <typename K, class Sol, class SumF>
__device__ __forceinline__ double init_after_f1(const Sol& S, const double* x0, bool xbin,
                                                const cx<K>* k1, const cx<K>* kp, double at,
                                                double rt, double dt0, double d1, double L,
                                                double dtmin, SumF&& sum) {
    constexpr int N = Sol::N, E = Sol::E;
    double s2 = 0.0, ndiff = 0.0;
#pragma unroll 4
    for (int s = 0; s < E; s++) {
        const cx<double> x = ld2(x0, xbin ? S.bin(s) : S.own(s));
        const double sk = at + sqrt(x.re * x.re + x.im * x.im) * rt;
        const cx<K> f0 = k1[S.own(s)], f1 = kp[S.own(s)];
        const double dr = (double)f1.re - (double)f0.re;
        const double di = (double)f1.im - (double)f0.im;
        s2 += (dr * dr + di * di) / (sk * sk);
        ndiff += (dr != 0.0 || di != 0.0) ? 1.0 : 0.0;
    }
    const double d2 = sqrt(sum(s2) / N) / dt0;
    const double nd = sum(ndiff);
    return initdt_final(dt0, d1, d2, nd, dtmin, L);
}

// The state machine.  Each loop iteration performs at most one RHS
// evaluation (forward in RF, adjoint in RA) plus the bookkeeping around it,
// so the FFT code exists once per precision in the kernel.
// CTAs per SM the registers must admit: 128 per thread at 2^8..2^11 (512
// threads per SM), up to 255 on the other grids of less than 512 threads.
// FP64 stage vectors (wide) need more than 128 at 2^8 and 2^11, where the cap
// spilled 700 to 1100 bytes per adjoint evaluation: 592 gradients 1.61 ->
// 1.32 ms at 2^8 and 6.90 -> 5.81 at 2^11, one 1.26 -> 1.02 and 3.42 -> 2.20.
// At 2^7 the tensor memory admits eight (TmLayout), so a cap for sixteen
// bought nothing: 592 gradients 1.35 -> 1.07 ms without, one 1.09 -> 0.90.
constexpr int sm_min_ctas(int logn, bool wide) {
    return logn <= 7 ? 8 : logn == 8 && wide ? 4 : logn <= 10 ? 1 << (11 - logn)
         : logn == 11 && !wide ? 2 : 1;
}
template <typename RF, typename RA, int LOGN, int CL>
__global__ void __launch_bounds__(XShape<LOGN, CL>::TC, sm_min_ctas(LOGN, sizeof(RF) == 8))
    sm_advance_kernel(const SlotDesc* __restrict__ descs, SlotState* __restrict__ states,
                      const int* __restrict__ active, int max_evals) {
    using SolF = SmSolver<RA, RF, LOGN, CL>;
    using SolA = SmSolver<RA, RA, LOGN, CL>;
    using CF = cx<RF>;
    using CA = cx<RA>;
    constexpr int N = SolF::N, E = SolF::E, T = SolF::XF::T;
    static_assert(!TmLayout<LOGN, CL>::ENABLED || CL > 1 ||
                      TmLayout<LOGN, CL>::COLS * sm_min_ctas(LOGN, sizeof(RF) == 8) <= 512,
                  "a CTA that the registers admit finds its columns");
    extern __shared__ __align__(16) unsigned char smraw[];
    double* red = reinterpret_cast<double*>(smraw + SmShared<RA, LOGN, CL>::RED);

    const int slot = active[blockIdx.x / CL], rank = blockIdx.x % CL;
    const SlotDesc& d = descs[slot];
    SlotState st = states[slot];  // group-uniform copy
    if (st.phase == PH_DONE) return;
    const uint32_t tm = tm_alloc<LOGN, CL>(tm_slot<RA, LOGN, CL>(smraw));
    load_tables<RA, LOGN, CL>(d, smraw, rank);
    SolF SF(d, smraw, rank);
    const bool lead = rank == 0 && threadIdx.x == 0;
    const double L = d.L, dtmin = kEps * L;
    int flip = 0;
    auto sum = [&](double v) { return x_reduce<T, CL, false>(v, red, flip, rank); };
    auto maxv = [&](double v) { return x_reduce<T, CL, true>(v, red, flip, rank); };
    // the stage vectors of a slot lie one stride apart (work_create)
    const size_t kfs = (char*)d.kf[1] - (char*)d.kf[0], kas = (char*)d.ka[1] - (char*)d.ka[0];
    int evals = 0;

    while (st.phase != PH_DONE && evals < max_evals) {
#ifdef FL_CHECKED
        if (!state_in_bounds(d, st)) {
            st.status = ST_CHECK;
            st.phase = PH_DONE;
            continue;
        }
#endif
        // ------------------------------------------------ phases without an RHS
        if (st.phase == PH_SEED) {
            // terminal seed λ̃(L) (interaction frame) into lam[0]
            const double* uf = d.u[st.cur];
            double* lam = d.lam[0];
            if (d.mode == MODE_BAND_GRADIENT) {
                // Band objective (physics_helpers.jl:222-232).  With one mode
                // the fundamental-mode and worst-mode objectives are the same
                // (:234-286: one active mode, log-sum-exp = its fraction,
                // weight 1).  The peak objective (:288-302) puts the strongest
                // in-band bin (lowest index among equals) in place of the band.
                const bool peak = d.objective == OBJ_RAMAN_PEAK;
                double et = 0.0, eb = 0.0, emax = -1.0;
#pragma unroll 4
                for (int s = 0; s < E; s++) {
                    const int b = SF.bin(s);
                    const double e = energy(ld2(uf, SF.own(s)));
                    et += e;
                    if (d.mask[b]) {
                        eb += e;
                        emax = fmax(emax, e);
                    }
                }
                const double tot = sum(et);
                double band = sum(eb);
                int pk = -1;
                if (peak) {
                    band = maxv(emax);
                    // lowest index as the largest key N - b (the maximum folds from 0)
                    double key = 0.0;
#pragma unroll 4
                    for (int s = 0; s < E; s++) {
                        const int b = SF.bin(s);
                        if (d.mask[b] && energy(ld2(uf, SF.own(s))) == band) key = fmax(key, (double)(N - b));
                    }
                    pk = N - (int)maxv(key);
                }
                const double cost = band / tot;
                double sc = 1.0 / tot;
                st.J = cost;
                if (d.log_cost) {  // physics_helpers.jl:320-326
                    st.J = 10.0 * log10(fmax(cost, 1e-15));
                    sc *= cost <= 1e-15 ? 0.0 : 10.0 / (log(10.0) * cost);
                }
                // e^{-iDL} (u_L (sel - J)/E) = ũ(L) (sel - J)/E, sel the band or peak bin
#pragma unroll 4
                for (int s = 0; s < E; s++) {
                    const int b = SF.bin(s);
                    const cx<double> x = ld2(uf, SF.own(s));
                    const double sel = peak ? (b == pk ? 1.0 : 0.0) : (d.mask[b] ? 1.0 : 0.0);
                    const double f = (sel - cost) * sc;
                    st2(lam, SF.own(s), mk(x.re * f, x.im * f));
                }
            } else {
                st.J = 0.0;
#pragma unroll 4
                for (int s = 0; s < E; s++) {
                    const int b = SF.bin(s);
                    const cx<double> x = ld2(d.lamL, b);
                    const cx<double> p = phasor<double>(d.Dturns[b], L);
                    st2(lam, SF.own(s), mk(x.re * p.re + x.im * p.im, x.im * p.re - x.re * p.im));
                }
            }
            double mx = 0.0;
            bool finite = true;
#pragma unroll 4
            for (int s = 0; s < E; s++) {
                const cx<double> x = ld2(lam, SF.own(s));
                const double a = sqrt(x.re * x.re + x.im * x.im);
                if (!isfinite(a)) finite = false;
                mx = fmax(mx, a);
            }
            const double scl = maxv(finite ? mx : INFINITY);
            if (!isfinite(scl)) {
                st.status = ST_NONFINITE;
                st.phase = PH_DONE;
                continue;
            }
            st.abstol_adj = scl == 0.0 ? d.abstol : d.abstol * scl;  // sensitivity_disp_mmf.jl:324-325
            st.acur = 0;
            st.akperm = 0;
            st.a_naccept = st.a_nreject = st.a_nf = st.a_iters = 0;
            st.nrec = 0;
            // every step's interpolant is in the buffer when the forward fit it
            // (kept by the forward; an earlier adjoint of this solve then did
            // not overwrite it)
            st.dense = st.nsteps <= d.seg_cap ? 1 : 0;
            if (st.dense) {
                st.seg = 0;
                st.sub = 0;
                st.phase = PH_ADJ_INIT;
                continue;
            }
            st.seg = (st.nsteps + st.ck_stride - 1) / st.ck_stride - 1;
            st.sub = last_sub(d, st, st.seg);
            restore_checkpoint<RF>(SF, st.seg, st);
            st.phase = PH_REC;
            continue;
        }
        if (st.phase == PH_FINAL) {
            // λ(0) = λ̃(0); ∂J/∂φ = 2 Re(conj(λ0) i u_shaped) (physics_models.jl:1042)
            const double* lam = d.lam[st.acur];
#pragma unroll 4
            for (int s = 0; s < E; s++) {
                const int b = SF.bin(s);
                const cx<double> l = ld2(lam, SF.own(s));
                if (d.lam0_out) st2(d.lam0_out, b, l);
                if (d.grad_out) {
                    const cx<double> us = ld2(d.u0, b);
                    d.grad_out[b] = 2.0 * (l.im * us.re - l.re * us.im);
                }
            }
            st.phase = PH_DONE;
            continue;
        }

        // ------------------------------------------------ build the stage input
        const bool adj = st.phase == PH_ADJ_INIT || st.phase == PH_ADJ;
        StageRun in{};
        if (st.phase == PH_FWD_INIT) {
            in.x = d.u0;
            in.xbin = 1;
            in.copy = st.stage == 0 ? d.u[0] : nullptr;
            in.k1 = st.stage == 0 ? nullptr : d.kf[0];
            in.c = st.cdt;
            in.out = d.kf[st.stage == 0 ? 0 : 1];
            in.z = st.stage == 0 ? 0.0 : st.cdt;
        } else if (st.phase == PH_FWD || st.phase == PH_REC) {
            if (st.stage == 0) {
                if (st.phase == PH_REC) {
                    const int n = st.seg * st.ck_stride + st.rec_pos;
                    st.cz = d.steplog[2 * n];
                    st.cdt = d.steplog[2 * n + 1];
                } else {
                    if (++st.iters > d.max_iters) {
                        st.status = ST_MAXITERS;
                        st.phase = PH_DONE;
                        continue;
                    }
                    // fix_dt_at_bounds!, modify_dt_for_tstops!
                    double adt = fmax(fmin(fabs(st.dt), L), dtmin);
                    const double rem = L - st.z;
                    if (adt > rem) adt = rem;
                    if (adt <= dtmin && rem > dtmin) {
                        st.status = ST_DT_UNDERFLOW;
                        st.phase = PH_DONE;
                        continue;
                    }
                    st.cz = st.z;
                    st.cdt = adt;
                }
                st.stage = 1;
            }
            in.x = d.u[st.cur];
            in.kb = (char*)d.kf[0];
            in.ks = kfs;
            in.perm = st.kperm;
            in.xnew = d.u[st.cur ^ 1];
            in.want_err = st.phase == PH_FWD;
            in.at = d.abstol;
            in.rt = d.reltol;
        } else if (st.phase == PH_ADJ_INIT) {
            in.x = d.lam[0];
            in.k1 = st.stage == 0 ? nullptr : d.ka[0];
            in.c = -st.cdt;
            in.out = d.ka[st.stage == 0 ? 0 : 1];
            in.z = st.stage == 0 ? L : L - st.cdt;
            in.zload = st.stage == 0 ? L : fmax(in.z, d.steplog[2 * sub_segment(d, st).lo]);
        } else {  // PH_ADJ
            const double zlo = d.steplog[2 * sub_segment(d, st).lo];
            if (st.stage == 0) {
                if (++st.a_iters > d.max_iters) {
                    st.status = ST_MAXITERS;
                    st.phase = PH_DONE;
                    continue;
                }
                // Segment starts are stopping points of this implementation only
                // (the reference integrates the adjoint without them), so they
                // are made transparent to the controller: no sliver step before
                // one (the last two steps are split evenly) and the proposal
                // from before the clip is restored after it.
                const double prop = fmax(fmin(fabs(st.adt), L), dtmin);
                const double rem = st.az - zlo;
                double adt = prop;
                if (adt >= rem) adt = rem;
                else if (adt > 0.5 * rem) adt = 0.5 * rem;
                st.aprop = prop;
                st.cz = st.az;
                st.cdt = -adt;
                st.stage = 1;
            }
            in.x = d.lam[st.acur];
            in.kb = (char*)d.ka[0];
            in.ks = kas;
            in.perm = st.akperm;
            in.xnew = d.lam[st.acur ^ 1];
            in.want_err = 1;
            in.at = st.abstol_adj;
            in.rt = d.reltol;
        }

        // ------------------------- the probe's evaluation, or the attempt's stages
        const bool probe = st.phase == PH_FWD_INIT || st.phase == PH_ADJ_INIT;
        in.stage = probe ? 0 : st.stage;
        in.count = probe ? 1 : min(7 - st.stage, max_evals - evals);
        in.cz = st.cz;
        in.dt = st.cdt;
        double acc;
        if (adj) {
            const SubSeg sb = sub_segment(d, st);
            in.seg_lo = sb.lo;
            in.seg_hi = sb.hi;
            acc = rhs_adj_call<RF, RA, LOGN, CL>(&d, smraw, rank, &in, tm);
        } else {
            acc = rhs_fwd_call<RA, RF, LOGN, CL>(&d, smraw, rank, &in, tm);
        }
        evals += in.count;

        // ------------------------------------------------ consume the derivative
        if (st.phase == PH_FWD_INIT || st.phase == PH_ADJ_INIT) {
            const bool fw = st.phase == PH_FWD_INIT;
            if (st.stage == 0) {
                double d1;
                const double r =
                    fw ? init_after_f0<RF>(SF, d.u0, true, (const CF*)d.kf[0], d.abstol, d.reltol, L,
                                           dtmin, sum, d1)
                       : init_after_f0<RA>(SF, d.lam[0], false, (const CA*)d.ka[0], st.abstol_adj,
                                           d.reltol, L, dtmin, sum, d1);
                if (r > 0.0) {  // probe step
                    st.cdt = r;
                    st.cz = d1;
                    st.stage = 1;
                    continue;
                }
                st.cdt = -r;
            } else {
                st.cdt =
                    fw ? init_after_f1<RF>(SF, d.u0, true, (const CF*)d.kf[0], (const CF*)d.kf[1],
                                           d.abstol, d.reltol, st.cdt, st.cz, L, dtmin, sum)
                       : init_after_f1<RA>(SF, d.lam[0], false, (const CA*)d.ka[0],
                                           (const CA*)d.ka[1], st.abstol_adj, d.reltol, st.cdt,
                                           st.cz, L, dtmin, sum);
            }
            st.stage = 0;
            if (fw) {
                st.z = 0.0;
                st.dt = st.cdt;
                st.qold = kQoldInit;
                st.cur = 0;
                st.kperm = 0;
                st.nsteps = 0;
                st.ck_stride = 1;
                st.naccept = st.nreject = st.iters = 0;
                st.nf = 3;
                if (d.ck_cap > 0) {
                    const CF* k1 = (const CF*)d.kf[0];
#pragma unroll 4
                    for (int s = 0; s < E; s++) {
                        const int b = SF.own(s);
                        reinterpret_cast<double2*>(d.ck_u)[b] =
                            reinterpret_cast<const double2*>(d.u0)[SF.bin(s)];
                        ((CF*)d.ck_k1)[b] = k1[b];
                    }
                }
                st.save_idx = 0;
                while (st.save_idx < d.nsave && d.zsave[st.save_idx] == 0.0) {
                    double* o = d.save_out + (size_t)st.save_idx * 2 * N;
#pragma unroll 4
                    for (int s = 0; s < E; s++) st2(o, SF.bin(s), ld2(d.u0, SF.bin(s)));
                    st.save_idx++;
                }
                st.phase = PH_FWD;
            } else {
                st.az = L;
                st.adt = -st.cdt;
                st.aqold = kQoldInit;
                st.a_nf = 3;
                st.acur = 0;
                st.akperm = 0;
                st.phase = PH_ADJ;
            }
            continue;
        }

        if (st.phase == PH_FWD || st.phase == PH_REC) {
            const bool rec = st.phase == PH_REC;
            st.stage += in.count;
            if (st.stage < 7) continue;
            st.stage = 0;
            const double z = st.cz, dt = st.cdt;
            const double* u = d.u[st.cur];
            if (rec) {
                // interpolant of this step, kept only for the steps of the
                // current sub-segment
                const SubSeg sb = sub_segment(d, st);
                const int n = sb.seg_lo + st.rec_pos;
                if (n >= sb.lo)
                    store_interp<RF>(SF, u, st.kperm,
                                     (CF*)d.seg + (size_t)(n - sb.lo) * 5 * N);
                st.cur ^= 1;
                st.kperm ^= 1;
                st.rec_pos++;
                st.nrec++;
                if (n + 1 >= sb.hi) st.phase = st.a_nf == 0 ? PH_ADJ_INIT : PH_ADJ;
                continue;
            }
            const double EEst = sqrt(sum(acc) / (double)N);
            if (!isfinite(EEst)) {
                st.status = ST_NONFINITE;
                st.phase = PH_DONE;
                continue;
            }
            double q11;
            const double q = pi_q(EEst, st.qold, q11);
            st.nf += 6;
            if (EEst > 1.0) {
                st.nreject++;
                st.dt = dt / fmin(1.0 / kQmin, q11 / kGamma);
                continue;
            }
            st.naccept++;
            if (d.step_cap > 0) {  // step_cap 0: forward only, nothing kept for an adjoint
                if (st.nsteps >= d.step_cap) {
                    st.status = ST_CAPACITY;
                    st.phase = PH_DONE;
                    continue;
                }
                if (lead) {
                    d.steplog[2 * st.nsteps] = z;
                    d.steplog[2 * st.nsteps + 1] = dt;
                }
                // while the solve fits the interpolant buffer, keep each
                // step's interpolant now: the adjoint then needs no recompute
                if (st.nsteps < d.seg_cap)
                    store_interp<RF>(SF, u, st.kperm,
                                     (CF*)d.seg + (size_t)st.nsteps * 5 * N);
            }
            double znew = z + dt;
            if (fabs(znew - L) < 100.0 * kEps * fmax(z, L)) znew = L;  // snap to the tstop
            // save positions in (z, znew) and on an interior step end: dense
            // output (positions at L take the final state below)
            while (st.save_idx < d.nsave && d.zsave[st.save_idx] > z &&
                   (d.zsave[st.save_idx] < znew || (d.zsave[st.save_idx] == znew && znew < L))) {
                const double zs = d.zsave[st.save_idx];
                const double th = (zs - z) / dt;
                double* o = d.save_out + (size_t)st.save_idx * 2 * N;
#pragma unroll 4
                for (int s = 0; s < E; s++) {
                    const int b = SF.own(s), f = SF.bin(s);
                    double xr = 0.0, xi = 0.0;
                    for (int i = 0; i < 7; i++) {
                        double bi = 0.0, tp = th;
                        for (int qq = 0; qq < 4; qq++) {
                            bi += kT5r[i][qq] * tp;
                            tp *= th;
                        }
                        const CF ki = SolF::kp(d.kf, st.kperm, i)[b];
                        xr += bi * (double)ki.re;
                        xi += bi * (double)ki.im;
                    }
                    const cx<double> un = ld2(u, b);
                    const cx<double> x = mk(un.re + dt * xr, un.im + dt * xi);
                    const cx<double> p = phasor<double>(d.Dturns[f], zs);
                    st2(o, f, mk(x.re * p.re - x.im * p.im, x.re * p.im + x.im * p.re));
                }
                st.save_idx++;
            }
            st.nsteps++;
            st.z = znew;
            st.cur ^= 1;
            st.kperm ^= 1;
            st.qold = fmax(EEst, kQoldInit);
            st.dt = fmin(fmax((q == 1.0) ? dt : dt / q, dtmin), L);
            // z-checkpoints with thinning: K slots at steps j*stride
            if (d.ck_cap > 0 && (st.nsteps % st.ck_stride) == 0) {
                int slotc = st.nsteps / st.ck_stride;
                if (slotc >= d.ck_cap) {
                    for (int j = 1; j < d.ck_cap / 2; j++) {
#pragma unroll 4
                        for (int s = 0; s < E; s++) {
                            const int b = SF.own(s);
                            reinterpret_cast<double2*>(d.ck_u)[(size_t)j * N + b] =
                                reinterpret_cast<double2*>(d.ck_u)[(size_t)2 * j * N + b];
                            ((CF*)d.ck_k1)[(size_t)j * N + b] =
                                ((CF*)d.ck_k1)[(size_t)2 * j * N + b];
                        }
                    }
                    st.ck_stride *= 2;
                    slotc = st.nsteps / st.ck_stride;
                }
#ifdef FL_CHECKED
                if (slotc < 0 || slotc >= d.ck_cap) {
                    st.status = ST_CHECK;
                    st.phase = PH_DONE;
                    continue;
                }
#endif
                const double* un = d.u[st.cur];
                const CF* k1 = SolF::kp(d.kf, st.kperm, 0);
#pragma unroll 4
                for (int s = 0; s < E; s++) {
                    const int b = SF.own(s);
                    reinterpret_cast<double2*>(d.ck_u)[(size_t)slotc * N + b] =
                        reinterpret_cast<const double2*>(un)[b];
                    ((CF*)d.ck_k1)[(size_t)slotc * N + b] = k1[b];
                }
            }
            if (st.z == L) {
                const double* uf = d.u[st.cur];
#pragma unroll 4
                for (int s = 0; s < E; s++) {
                    const int b = SF.bin(s);
                    const cx<double> x = ld2(uf, SF.own(s));
                    const cx<double> p = phasor<double>(d.Dturns[b], L);
                    const cx<double> y = mk(x.re * p.re - x.im * p.im, x.re * p.im + x.im * p.re);
                    for (int si = st.save_idx; si < d.nsave; si++)
                        st2(d.save_out + (size_t)si * 2 * N, b, y);
                    if (d.uL_out) st2(d.uL_out, b, y);
                }
                st.save_idx = d.nsave;
                st.phase = d.mode == MODE_FORWARD ? PH_DONE : PH_SEED;
            }
            continue;
        }

        // PH_ADJ
        {
            st.stage += in.count;
            if (st.stage < 7) continue;
            st.stage = 0;
            const double z = st.cz, dt = st.cdt;
            const double zlo = d.steplog[2 * sub_segment(d, st).lo];
            const double EEst = sqrt(sum(acc) / (double)N);
            if (!isfinite(EEst)) {
                st.status = ST_NONFINITE;
                st.phase = PH_DONE;
                continue;
            }
            double q11;
            const double q = pi_q(EEst, st.aqold, q11);
            st.a_nf += 6;
            if (EEst > 1.0) {
                st.a_nreject++;
                st.adt = st.adt / fmin(1.0 / kQmin, q11 / kGamma);
                continue;
            }
            st.a_naccept++;
            double znew = z + dt;
            if (fabs(znew - zlo) < 100.0 * kEps * fmax(z, zlo)) znew = zlo;
            st.az = znew;
            st.acur ^= 1;
            st.akperm ^= 1;
            st.aqold = fmax(EEst, kQoldInit);
            const double adt = -dt;
            double dtn = fmin(fmax((q == 1.0) ? adt : adt / q, dtmin), L);
            if (adt < st.aprop) dtn = fmax(dtn, st.aprop);  // shortened for a segment start
            st.adt = -dtn;
            if (st.az == zlo) {
                if (st.sub > 0) {  // the previous sub-segment of this segment
                    st.sub--;
                    restore_checkpoint<RF>(SF, st.seg, st);
                    st.phase = PH_REC;
                } else if (st.seg == 0) {
                    st.phase = PH_FINAL;
                } else {
                    st.seg--;
                    st.sub = last_sub(d, st, st.seg);
                    restore_checkpoint<RF>(SF, st.seg, st);
                    st.phase = PH_REC;
                }
            }
        }
    }
    SolF::XF::sync();  // no CTA leaves while another still writes into it
    if (lead) states[slot] = st;
    tm_free<LOGN, CL>(tm);
}

}  // namespace fl
