// fl_xfft.cuh -- transforms of one problem over the warps of a CTA or of a
// thread-block cluster, with a single group-wide exchange per transform.
//
// A spectral field in layout A holds, per thread, E bins of one or two
// "columns" (bins x + s N/16, s = 0..15).  A field in layout B (time) holds
// the values the transform leaves there; every pointwise operation on it
// reads and writes the same slots, so the order inside B never matters.
//
//   to_b  (A -> B, decimation in frequency)  radix 16 over s in the thread,
//         W_N^{xq}, exchange: column element q goes to region q; each region
//         is an independent transform of N/16 points owned by at most one
//         warp, which finishes it with warp-local exchanges only.
//   to_a  (B -> A, decimation in time)       the same steps mirrored.
//
// Both are unnormalised, exponent sign -1 (inverses run as conj F conj).
// Against a Stockham transform, whose every exchange is a CTA-wide pass with
// two barriers, the warps drift apart inside their regions, so one warp's
// shared-memory phase overlaps another's arithmetic: one gradient at
// Nt = 2^13 on one CTA 24.3 ms with the Stockham transform, 22.5 with this
// one, 11.3 on a cluster of eight.
//
// Region transform of N/16 = 16 L points (L lanes per region, E = 16):
// radix 16 over j (x = l + L j), W_{N/16}^{lr}, then L points per r: L <= 16
// in one thread after a transposition inside the warp; L = 32 (Nt = 2^13)
// takes its radix-2 step between lanes l and l + 16 by shuffles first.
// Nt = 2^14 (E = 32): regions of 1024 points, 32 per lane, 32 x 32.
//
// Columns are dealt so that bin -k is reached without shared memory: with
// E = 16, lane i < 16 of warp w holds column 16 w + i and lane 16 + i holds
// column N/16 - (16 w + i) (lane 16 of warp 0: N/32, its own mirror); with
// E = 32 a thread holds columns g and N/16 - g itself.
//
// C > 1: the group is a cluster of C CTAs; regions and columns are split
// over the CTAs in thread order.  Exchanges push into the owning CTA's shared
// memory and a cluster barrier follows; two buffers (regions B, columns A)
// leave one barrier per transform.  The arithmetic per value is that of
// C = 1, so results do not depend on C.
#pragma once
#include "fl_fft.cuh"

namespace fl {

__host__ __device__ constexpr int x_loge(int logn) {
    return logn <= 6 ? 1 : logn <= 10 ? 2 : logn <= 11 ? 3 : logn <= 13 ? 4 : 5;
}

// exp(-2 pi i k / 16) times a, 0 <= k <= 9
template <typename R>
__device__ __forceinline__ cx<R> tw16(cx<R> a, int k) {
    if (k == 0) return a;
    if (k == 4) return mk(a.im, -a.re);
    cx<R> w = w32<R>(2 * (k & 7));
    if (k >= 8) w = mk(-w.re, -w.im);
    return cmul(a, w);
}

// radix-4 DFT of a[base + STRIDE i]
template <int STRIDE, typename R, int E>
__device__ __forceinline__ void dft4(cx<R> (&a)[E], int base) {
    const cx<R> x0 = a[base], x1 = a[base + STRIDE], x2 = a[base + 2 * STRIDE],
                x3 = a[base + 3 * STRIDE];
    const cx<R> t0 = x0 + x2, t1 = x0 - x2, t2 = x1 + x3, d = x1 - x3;
    const cx<R> t3 = mk(d.im, -d.re);
    a[base] = t0 + t2;
    a[base + STRIDE] = t1 + t3;
    a[base + 2 * STRIDE] = t0 - t2;
    a[base + 3 * STRIDE] = t1 - t3;
}

// radix-16 DFT of a[base + STRIDE n] as 4 x 4, natural order in and out
template <int STRIDE, typename R, int E>
__device__ __forceinline__ void dft16(cx<R> (&a)[E], int base) {
#pragma unroll
    for (int b = 0; b < 4; b++) dft4<4 * STRIDE>(a, base + STRIDE * b);
#pragma unroll
    for (int c = 1; c < 4; c++)
#pragma unroll
        for (int b = 1; b < 4; b++)
            a[base + STRIDE * (4 * c + b)] = tw16(a[base + STRIDE * (4 * c + b)], b * c);
#pragma unroll
    for (int c = 0; c < 4; c++) dft4<STRIDE>(a, base + STRIDE * 4 * c);
    // a[4c + d] = X[c + 4d]: transpose by renaming
#pragma unroll
    for (int c = 0; c < 4; c++)
#pragma unroll
        for (int d = c + 1; d < 4; d++) {
            const cx<R> t = a[base + STRIDE * (4 * c + d)];
            a[base + STRIDE * (4 * c + d)] = a[base + STRIDE * (4 * d + c)];
            a[base + STRIDE * (4 * d + c)] = t;
        }
}

// radix-32 DFT of the whole array, natural order in and out
template <typename R>
__device__ __forceinline__ void dft32(cx<R> (&a)[32]) {
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const cx<R> u = a[i], v = a[i + 16];
        a[i] = u + v;
        a[i + 16] = tw32<false>(u - v, i);
    }
    dft16<1>(a, 0);   // even outputs
    dft16<1>(a, 16);  // odd outputs
    cx<R> t[32];
#pragma unroll
    for (int i = 0; i < 32; i++) t[i] = a[i];
#pragma unroll
    for (int k = 0; k < 16; k++) {
        a[2 * k] = t[k];
        a[2 * k + 1] = t[16 + k];
    }
}

// DFT of RAD points a[base + STRIDE n] (natural order)
template <int RAD, int STRIDE, typename R, int E>
__device__ __forceinline__ void dft_small(cx<R> (&a)[E], int base) {
    if constexpr (RAD == 16) dft16<STRIDE>(a, base);
    else if constexpr (RAD == 4) dft4<STRIDE>(a, base);
    else dft_inreg<RAD, false, STRIDE>(a, base);
}

// v[BASE + r] *= w1^r for r in [1, CNT): products of at most two powers deep
// per group of four (short chains, rounding a few ulp)
template <int CNT, int BASE, typename R, int E>
__device__ __forceinline__ void mul_powers(cx<R> (&v)[E], const cx<R> w1) {
    const cx<R> w2 = cmul(w1, w1), w3 = cmul(w2, w1), w4 = cmul(w2, w2);
    v[BASE + 1] = cmul(v[BASE + 1], w1);
    v[BASE + 2] = cmul(v[BASE + 2], w2);
    v[BASE + 3] = cmul(v[BASE + 3], w3);
    cx<R> x = w4;
#pragma unroll
    for (int a = 4; a < CNT; a += 4) {
        v[BASE + a] = cmul(v[BASE + a], x);
        v[BASE + a + 1] = cmul(v[BASE + a + 1], cmul(x, w1));
        v[BASE + a + 2] = cmul(v[BASE + a + 2], cmul(x, w2));
        v[BASE + a + 3] = cmul(v[BASE + a + 3], cmul(x, w3));
        if (a + 4 < CNT) x = cmul(x, w4);
    }
}

// ---- cluster primitives ----------------------------------------------------
__device__ __forceinline__ uint32_t x_smem(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ uint32_t x_mapa(uint32_t a, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void x_st(uint32_t a, cx<float> v) {
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.re), "f"(v.im)
                 : "memory");
}
__device__ __forceinline__ void x_st(uint32_t a, cx<double> v) {
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.re), "d"(v.im)
                 : "memory");
}
__device__ __forceinline__ void x_st(uint32_t a, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void x_cluster_sync() {
    asm volatile(
        "barrier.cluster.arrive.release.aligned;\n\t"
        "barrier.cluster.wait.acquire.aligned;" ::
            : "memory");
}

__device__ __forceinline__ cx<float> x_shfl(cx<float> v, int src) {
    return mk(__shfl_sync(0xffffffffu, v.re, src), __shfl_sync(0xffffffffu, v.im, src));
}
__device__ __forceinline__ cx<double> x_shfl(cx<double> v, int src) {
    return mk(__shfl_sync(0xffffffffu, v.re, src), __shfl_sync(0xffffffffu, v.im, src));
}

// ---------------------------------------------------------------------------
// Geometry of a group of C CTAs for one problem of 2^LOGN points.
// ---------------------------------------------------------------------------
template <int LOGN, int C, int LE = x_loge(LOGN)>
struct XShape {
    static constexpr int LOGE = LE;
    static constexpr int N = 1 << LOGN, E = 1 << LOGE;
    static constexpr int T = N / E;      // threads of the group
    static constexpr int TC = T / C;     // threads per CTA
    static constexpr bool SMALL = LE <= 3;  // E <= 8: Stockham
    static constexpr int TT = N / 16;    // columns; points of a region
    static constexpr int L = E == 32 ? 32 : TT / 16;  // lanes per region
    // region stride in elements: room for the warp-local transposition
    // (rows of L + 1, L = 32: 32 rows of 17 or 33), offset so that the
    // regions a warp touches at once fall into different banks
    static constexpr int RS = E == 32 ? 1056 : L == 32 ? 544 : 272;
    static constexpr int REG = SMALL ? 0 : 16 / C;   // regions per CTA
    static constexpr int BUF = SMALL ? N + N / 8 : REG * RS;  // elements of one buffer
    static_assert(C == 1 || (!SMALL && TC >= 32 && C <= 16), "cluster split");
};

// Shared-memory plan.  The FP64 buffers bound the size; FP32 transforms use
// the same bytes.  One CTA: one FP64 buffer (two would halve the CTAs per SM
// or not fit), two FP32 ones where they fit in it; clusters: two of each.
// FP64 at 2^14 points on one CTA exchanges real and imaginary parts in turn.
template <typename R, typename RMAX, int LOGN, int C, int LE = x_loge(LOGN)>
struct XPlan {
    using S = XShape<LOGN, C, LE>;
    static constexpr bool SPLIT = C == 1 && 2 * sizeof(R) * (size_t)S::BUF > 200 * 1024;
    static constexpr size_t ONE = (SPLIT ? sizeof(R) : 2 * sizeof(R)) * (size_t)S::BUF;
    static constexpr bool SPLITM = C == 1 && 2 * sizeof(RMAX) * (size_t)S::BUF > 200 * 1024;
    static constexpr size_t ONEM = (SPLITM ? sizeof(RMAX) : 2 * sizeof(RMAX)) * (size_t)S::BUF;
    static constexpr size_t BYTES = ((C > 1 || S::SMALL ? 2 * ONEM : ONEM) + 15) & ~size_t(15);
    static constexpr bool TWO = 2 * ONE <= BYTES;  // separate A and B buffers
    static_assert((C == 1 && !S::SMALL) || TWO, "clusters and small grids need both buffers");
};

// Twiddle tables in shared memory, filled once per kernel from the full
// table W_N^k.  E >= 16: first-pass columns (FP32: two-level products
// W^e = hi[e >> 6] lo[e & 63]; FP64: W_N^x, powers by products), second pass
// (FP32: W_{N/16}^{lr}; FP64: W_{N/16}^l), W_32^i.  LEAN: the FP32 transforms
// of an FP64 solve, whose tables come on top.
template <typename R, int LOGN, int C, int LE = x_loge(LOGN), bool LEAN = false>
struct XTables {
    using S = XShape<LOGN, C, LE>;
    static constexpr bool F32 = sizeof(R) == 4;
    static constexpr bool TWO_LEVEL = F32 && S::E >= 16;
    static constexpr int R2 = S::E == 32 ? 32 : 16;
    static constexpr int N1 = S::SMALL ? 0
                              : F32 ? 64 + S::N / 64 : S::TC * (S::E / 16);
    static constexpr int N2 = S::SMALL ? 0 : (F32 ? R2 * S::L : S::L);
    static constexpr int N3 = !S::SMALL && S::L == 32 && S::E == 16 ? 16 : 0;
    // E <= 8: W_{E ns}^{m r}, m < ns, of each radix-E pass (ns = its stride)
    // after the first pass, r = 1..E-1 (FP64 with E = 8 and LEAN: r = 1, the others by
    // products); a pass's table starts at (ns - FIRST) NR / (E - 1)
    static constexpr int RE = S::E < 4 ? 4 : S::E;
    static constexpr int LRE = RE == 4 ? 2 : 3;
    static constexpr int FIRST = LOGN % LRE ? 1 << (LOGN % LRE) : RE;
    static constexpr int NR = LEAN || (!F32 && RE == 8) ? 1 : RE - 1;
    static constexpr int SIZE = S::SMALL ? (S::N - FIRST) / (RE - 1) * NR : N1 + N2 + N3;
};

template <int LOGN, int C>
__device__ __forceinline__ int x_col(int g, int half) {
    using S = XShape<LOGN, C>;
    if constexpr (S::E == 32) {
        if (half == 0) return g;
        return g == 0 ? S::TT / 2 : S::TT - g;
    } else {
        const int w = g >> 5, i = g & 15;
        if (!(g & 16)) return 16 * w + i;
        return g == 16 ? S::TT / 2 : S::TT - 16 * w - i;
    }
}
// thread of the group holding column x (E = 32: and which of its halves)
template <int LOGN, int C>
__device__ __forceinline__ int x_owner(int x, int& half) {
    using S = XShape<LOGN, C>;
    half = 0;
    if constexpr (S::E == 32) {
        if (x < S::TT / 2) return x;
        half = 1;
        return x == S::TT / 2 ? 0 : S::TT - x;
    } else {
        if (x < S::TT / 2) return 32 * (x >> 4) + (x & 15);
        if (x == S::TT / 2) return 16;
        const int y = S::TT - x;
        return 32 * (y >> 4) + 16 + (y & 15);
    }
}

template <typename R, int LOGN, int C, int LE = x_loge(LOGN), bool LEAN = false>
__device__ __forceinline__ void x_fill(cx<R>* dst, const cx<R>* __restrict__ full, int rank) {
    using S = XShape<LOGN, C, LE>;
    using X = XTables<R, LOGN, C, LE, LEAN>;
    if constexpr (S::SMALL) {
        for (int ns = X::FIRST; ns < S::N; ns *= X::RE)
            for (int i = threadIdx.x; i < X::NR * ns; i += S::TC)
                dst[(ns - X::FIRST) / (X::RE - 1) * X::NR + i] =
                    full[(i % ns) * (i / ns + 1) * (S::N / (X::RE * ns))];
    } else {
        const int tid = threadIdx.x, g = rank * S::TC + tid;
        if constexpr (X::TWO_LEVEL) {
            for (int i = tid; i < X::N1; i += S::TC) dst[i] = i < 64 ? full[i] : full[(i - 64) * 64];
        } else {
#pragma unroll
            for (int h = 0; h < S::E / 16; h++) dst[h * S::TC + tid] = full[x_col<LOGN, C>(g, h)];
        }
        // W_{N/16}^{l r} = W_N^{16 l r}
        for (int i = tid; i < X::N2; i += S::TC)
            dst[X::N1 + i] = full[X::F32 ? (16 * (i % S::L) * (i / S::L)) & (S::N - 1) : 16 * i];
        for (int i = tid; i < X::N3; i += S::TC) dst[X::N1 + X::N2 + i] = full[i * (S::N / 32)];
    }
}

// One group's transform engine in precision R.  An FP32 engine beside an FP64
// one (RMAX) uses the same bytes for the same region, column buffer and flip
// side, so transforms of both precisions may follow one another.
template <typename R, typename RMAX, int LOGN, int C, int LE = x_loge(LOGN)>
struct XForm {
    using S = XShape<LOGN, C, LE>;
    using P = XPlan<R, RMAX, LOGN, C, LE>;
    using X = XTables<R, LOGN, C, LE, (sizeof(R) < sizeof(RMAX))>;
    using V = cx<R>;
    static constexpr int N = S::N, E = S::E, T = S::T, TC = S::TC, TT = S::TT, L = S::L;
    // region stride in elements, the larger precision's in bytes
    static constexpr int RS = S::RS * (int)(P::ONEM / P::ONE);

    unsigned char* sm;        // the buffers
    const cx<R>* tab;         // XTables in shared memory
    int rank, g;              // CTA in the group, thread in the group
    mutable int flip;         // E <= 8: buffer of the next exchange

    __device__ __forceinline__ XForm(unsigned char* smem, const cx<R>* t, int rk)
        : sm(smem), tab(t), rank(rk), g(rk * TC + (int)threadIdx.x), flip(0) {}

    // workspace slot and bin of value s of this thread
    __device__ __forceinline__ int own(int s) const { return g + T * s; }
    __device__ __forceinline__ int bin(int s) const {
        if constexpr (S::SMALL) return g + T * s;
        else return x_col<LOGN, C>(g, s >> 4) + TT * (s & 15);
    }
    __device__ __forceinline__ static void sync() {
        if constexpr (C > 1) x_cluster_sync();
        else if constexpr (E == 2) __syncwarp();  // one warp
        else __syncthreads();
    }

    // ---- exchanges ----
    // A -> B: element q of column x to region q; then region element l + L j
    __device__ __forceinline__ void columns_to_regions(V (&v)[E], bool pre) const {
        const int q0 = g / L, l = g % L;
        if constexpr (C > 1) {
            if (pre) sync();
            const uint32_t base = x_smem(sm);
#pragma unroll
            for (int h = 0; h < E / 16; h++) {
                const int x = x_col<LOGN, C>(g, h);
#pragma unroll
                for (int q = 0; q < 16; q++)
                    x_st(x_mapa(base, q / S::REG) + (uint32_t)sizeof(V) * ((q % S::REG) * RS + x),
                         v[16 * h + q]);
            }
            sync();
            const V* b = reinterpret_cast<const V*>(sm) + (q0 % S::REG) * RS;
#pragma unroll
            for (int j = 0; j < E; j++) v[j] = b[l + L * j];
        } else {
            constexpr int PARTS = P::SPLIT ? 2 : 1;
#pragma unroll
            for (int part = 0; part < PARTS; part++) {
                if (pre || !P::TWO) sync();
#pragma unroll
                for (int h = 0; h < E / 16; h++) {
                    const int x = x_col<LOGN, C>(g, h);
#pragma unroll
                    for (int q = 0; q < 16; q++) put(q * RS + x, v[16 * h + q], part);
                }
                sync();
#pragma unroll
                for (int j = 0; j < E; j++) take(q0 * RS + l + L * j, v[j], part);
            }
        }
    }
    // B -> A: region element l + L j to its column; then element q of the column
    __device__ __forceinline__ void regions_to_columns(V (&v)[E]) const {
        const int q0 = g / L, l = g % L;
        if constexpr (C > 1) {
            const uint32_t base = x_smem(sm + P::ONEM);
#pragma unroll
            for (int j = 0; j < E; j++) {
                int half;
                const int o = x_owner<LOGN, C>(l + L * j, half);
                x_st(x_mapa(base, o / TC) +
                         (uint32_t)sizeof(V) * ((16 * half + q0) * TC + o % TC),
                     v[j]);
            }
            sync();
            const V* a = reinterpret_cast<const V*>(sm + P::ONEM);
#pragma unroll
            for (int s = 0; s < E; s++) v[s] = a[s * TC + threadIdx.x];
        } else {
            constexpr int PARTS = P::SPLIT ? 2 : 1;
            constexpr int AB = P::TWO ? S::RS : 0;  // the column buffer: the regions' second halves
            V w[E];
#pragma unroll
            for (int part = 0; part < PARTS; part++) {
                if (part) sync();
                else __syncwarp();
#pragma unroll
                for (int j = 0; j < E; j++) put(AB + q0 * RS + l + L * j, v[j], part);
                sync();
#pragma unroll
                for (int h = 0; h < E / 16; h++) {
                    const int x = x_col<LOGN, C>(g, h);
#pragma unroll
                    for (int q = 0; q < 16; q++) take(AB + q * RS + x, w[16 * h + q], part);
                }
            }
#pragma unroll
            for (int s = 0; s < E; s++) v[s] = w[s];
        }
    }
    // whole values, or (SPLIT) one part of them, at element i of the buffer
    __device__ __forceinline__ void put(int i, const V& x, int part) const {
        if constexpr (P::SPLIT) reinterpret_cast<R*>(sm)[i] = part ? x.im : x.re;
        else reinterpret_cast<V*>(sm)[i] = x;
    }
    __device__ __forceinline__ void take(int i, V& x, int part) const {
        if constexpr (!P::SPLIT) x = reinterpret_cast<const V*>(sm)[i];
        else if (part) x.im = reinterpret_cast<const R*>(sm)[i];
        else x.re = reinterpret_cast<const R*>(sm)[i];
    }
    // warp-local exchange inside this thread's region: value s to wr(s), from rd(s)
    template <class WR, class RD>
    __device__ __forceinline__ void in_region(V (&v)[E], WR&& wr, RD&& rd) const {
        const int b = (g / L) % S::REG * RS;
        constexpr int PARTS = P::SPLIT ? 2 : 1;
#pragma unroll
        for (int part = 0; part < PARTS; part++) {
            __syncwarp();
#pragma unroll
            for (int s = 0; s < E; s++) put(b + wr(s), v[s], part);
            __syncwarp();
#pragma unroll
            for (int s = 0; s < E; s++) take(b + rd(s), v[s], part);
        }
    }

    // ---- twiddles ----
    // v[16 h + q] *= W_N^{x_h q}
    __device__ __forceinline__ void tw_columns(V (&v)[E]) const {
        if constexpr (X::TWO_LEVEL) {
#pragma unroll
            for (int h = 0; h < E / 16; h++) {
                const int x = x_col<LOGN, C>(g, h);
#pragma unroll
                for (int q = 1; q < 16; q++) {
                    const int e = (x * q) & (N - 1);
                    v[16 * h + q] = cmul(v[16 * h + q], cmul(tab[64 + (e >> 6)], tab[e & 63]));
                }
            }
        } else {
            mul_powers<16, 0>(v, tab[threadIdx.x]);
            if constexpr (E == 32) mul_powers<16, 16>(v, tab[TC + threadIdx.x]);
        }
    }
    // v[r] *= W_{N/16}^{l r}
    __device__ __forceinline__ void tw_region(V (&v)[E]) const {
        const int l = g % L;
        if constexpr (X::F32) {
#pragma unroll
            for (int r = 1; r < E; r++) v[r] = cmul(v[r], tab[X::N1 + r * L + l]);
        } else {
            mul_powers<E, 0>(v, tab[X::N1 + l]);
        }
    }
    // lanes l < 16 keep the values r = 0..7 of lanes l and l + 16, the others
    // r = 8..15: on return a[u] is lane (l & 15)'s value and b[u] lane
    // (l & 15) + 16's, r = u + 8 [l >= 16]
    __device__ __forceinline__ static void pair_split(const V (&v)[E], V (&a)[8], V (&b)[8]) {
        const int lane = threadIdx.x & 31;
        const bool hi = lane & 16;
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const V keep = hi ? v[u + 8] : v[u], send = hi ? v[u] : v[u + 8];
            const V got = x_shfl(send, lane ^ 16);
            a[u] = hi ? got : keep;
            b[u] = hi ? keep : got;
        }
    }
    // the reverse: a[u] belongs to lane l & 15, b[u] to lane (l & 15) + 16
    __device__ __forceinline__ static void pair_join(V (&v)[E], const V (&a)[8], const V (&b)[8]) {
        const int lane = threadIdx.x & 31;
        const bool hi = lane & 16;
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const V keep = hi ? b[u] : a[u], send = hi ? a[u] : b[u];
            const V got = x_shfl(send, lane ^ 16);
            v[u] = hi ? got : keep;
            v[u + 8] = hi ? keep : got;
        }
    }

    // ---- transforms ----
    // ---- E = 4, 8: Stockham radix E, natural order on both sides ----
    // One butterfly per thread and pass (the bits that log2 E leaves over go
    // into a first pass of a smaller radix), unrolled, twiddles from the
    // correctly rounded table.  Exchanges alternate between two buffers, so
    // each costs one barrier.  On these grids many warps with few values each
    // beat few warps with sixteen: one problem's evaluation is a chain of
    // latencies (an FP64 FMA 37 cycles, an L2 load 530) that only other warps
    // hide.  Nt = 2^10, one forward solve: 4.25 ms with 64 threads of 16
    // values, 3.2 ms with 256 threads of 4 (2.7 with the convolution in FP32).
    static __device__ __forceinline__ int pad4(int i) { return i + (i >> (sizeof(R) == 8 ? 3 : 4)); }
    __device__ __forceinline__ V* flip_buffer() const {
        V* b = reinterpret_cast<V*>(sm + (flip ? P::ONEM : 0));
        flip ^= 1;
        return b;
    }
    template <int NS>
    __device__ __forceinline__ void passes(V (&v)[E]) const {
        const int t = threadIdx.x, m = t & (NS - 1);
        if constexpr (NS > 1) {
            const V* w = tab + (NS - X::FIRST) / (E - 1) * X::NR + m;
            if constexpr (X::NR == 1) {
                mul_powers<E, 0>(v, w[0]);
            } else {
#pragma unroll
                for (int q = 1; q < E; q++) v[q] = cmul(v[q], w[(q - 1) * NS]);
            }
        }
        dft_small<E, 1>(v, 0);
        if constexpr (NS * E < N) {
            V* b = flip_buffer();
#pragma unroll
            for (int q = 0; q < E; q++) b[pad4((t - m) * E + m + q * NS)] = v[q];
            sync();
#pragma unroll
            for (int s = 0; s < E; s++) v[s] = b[pad4(t + T * s)];
            passes<NS * E>(v);
        }
    }
    // 2^6 on one warp: six radix-2 passes, unrolled, so that each one's strides
    // and its choice of twiddle are constants (as a loop over the strides with
    // CTA barriers one forward solve took 0.68 ms, so 0.39, and 0.31 without
    // the cap of 128 registers)
    template <int NS>
    __device__ __forceinline__ void passes2(V (&v)[E]) const {
        const int t = threadIdx.x, m = t & (NS - 1);
        const V y = NS > 1 ? cmul(v[1], w2(m * (N / (2 * NS)))) : v[1];
        const V a = v[0] + y, d = v[0] - y;
        if constexpr (NS * 2 < N) {
            V* b = flip_buffer();
            b[pad4((t - m) * 2 + m)] = a;
            b[pad4((t - m) * 2 + m + NS)] = d;
            sync();
            v[0] = b[pad4(t)];
            v[1] = b[pad4(t + T)];
            passes2<NS * 2>(v);
        } else {
            v[0] = a;
            v[1] = d;
        }
    }
    __device__ __forceinline__ void stockham(V (&v)[E]) const {
        const int t = threadIdx.x;
        if constexpr (E == 2) {
            passes2<1>(v);
        } else if constexpr (X::FIRST < E) {
            constexpr int F = X::FIRST, M = E / F;  // M butterflies of radix F, stride 1
            V* b = flip_buffer();
#pragma unroll
            for (int q = 0; q < M; q++) {
                dft_small<F, M>(v, q);
#pragma unroll
                for (int k = 0; k < F; k++) b[pad4(F * (t + T * q) + k)] = v[q + M * k];
            }
            sync();
#pragma unroll
            for (int s = 0; s < E; s++) v[s] = b[pad4(t + T * s)];
            passes<F>(v);
        } else {
            passes<1>(v);
        }
    }
    // W_N^e, e < N/2, from the table of the last radix-4 pass (r = 1); a
    // quarter turn is exact
    __device__ __forceinline__ V w2(int e) const {
        const V w = tab[(N / 4 - X::FIRST) + (e & (N / 4 - 1))];
        return e < N / 4 ? w : mk(w.im, -w.re);
    }

    // Transform v, to B or to A.  pre: another thread of the group may still
    // be using the region buffer.
    __device__ __forceinline__ void transform(V (&v)[E], const bool to_a, const bool pre) const {
        if constexpr (S::SMALL) {
            stockham(v);
        } else if (to_a) {
            regions_back(v);
            regions_to_columns(v);
            tw_columns(v);
#pragma unroll
            for (int h = 0; h < E; h += 16) dft16<1>(v, h);
        } else {
#pragma unroll
            for (int h = 0; h < E; h += 16) dft16<1>(v, h);
            tw_columns(v);
            columns_to_regions(v, pre);
            regions_out(v);
        }
    }
    // the N/16-point transforms of the regions, decimation in frequency
    __device__ __forceinline__ void regions_out(V (&v)[E]) const {
        const int l = g % L;
        if constexpr (E == 32) {
            dft32(v);
            tw_region(v);
            in_region(v, [=](int r) { return 33 * r + l; }, [=](int i) { return 33 * l + i; });
            dft32(v);
        } else if constexpr (L == 16) {
            dft16<1>(v, 0);
            tw_region(v);
            in_region(v, [=](int r) { return 17 * r + l; }, [=](int i) { return 17 * l + i; });
            dft16<1>(v, 0);
        } else {
            dft16<1>(v, 0);
            tw_region(v);
            V a[8], b[8];
            pair_split(v, a, b);
            const V w = tab[X::N1 + X::N2 + (l & 15)];  // W_32^i
#pragma unroll
            for (int u = 0; u < 8; u++) {
                v[2 * u] = a[u] + b[u];
                v[2 * u + 1] = cmul(a[u] - b[u], w);
            }
            // value 2u + p: sequence (r, p), r = u + 8 [l >= 16], point i = l & 15
            const int wb = 17 * (l & 16) + (l & 15);
            in_region(v, [=](int s) { return wb + 17 * s; }, [=](int i) { return 17 * l + i; });
            dft16<1>(v, 0);
        }
    }
    // ... and decimation in time
    __device__ __forceinline__ void regions_back(V (&v)[E]) const {
        const int l = g % L;
        if constexpr (E == 32) {
            dft32(v);
            in_region(v, [=](int i) { return 33 * l + i; }, [=](int r) { return 33 * r + l; });
            tw_region(v);
            dft32(v);
        } else if constexpr (L == 16) {
            dft16<1>(v, 0);
            in_region(v, [=](int i) { return 17 * l + i; }, [=](int r) { return 17 * r + l; });
            tw_region(v);
            dft16<1>(v, 0);
        } else {
            dft16<1>(v, 0);
            const int wb = 17 * (l & 16) + (l & 15);
            in_region(v, [=](int i) { return 17 * l + i; }, [=](int s) { return wb + 17 * s; });
            const V w = tab[X::N1 + X::N2 + (l & 15)];
            V a[8], b[8];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const V y = cmul(v[2 * u + 1], w);
                a[u] = v[2 * u] + y;
                b[u] = v[2 * u] - y;
            }
            pair_join(v, a, b);
            tw_region(v);
            dft16<1>(v, 0);
        }
    }

    // v[k] <- Re H[k] v[k] + i Im H[k] conj(v[-k])
    __device__ __forceinline__ static V blend(V h, V x, V m) {
        return mk(h.re * x.re + h.im * m.im, h.re * x.im + h.im * m.re);
    }
    __device__ __forceinline__ void mirror_apply(V (&v)[E], const V* __restrict__ H) const {
        if constexpr (S::SMALL) {
            V h[E];
#pragma unroll
            for (int s = 0; s < E; s++) h[s] = H[bin(s)];
            V* b = flip_buffer();
#pragma unroll
            for (int s = 0; s < E; s++) b[pad4(bin(s))] = v[s];
            sync();
#pragma unroll
            for (int s = 0; s < E; s++) v[s] = blend(h[s], v[s], b[pad4((N - bin(s)) & (N - 1))]);
        } else {
            // Slot s of a column pairs with slot 15 - s of its mirror column:
            // the partner lane's (E = 16) or the thread's other column
            // (E = 32).  N/32 mirrors itself; column 0 (thread 0) pairs s
            // with -s mod 16.
            const bool z = g == 0;
            const int lane = threadIdx.x & 31, src = (g == 0 || g == 16) ? lane : lane ^ 16;
            const V v0 = v[0], v8 = v[8];
            V up = v0;  // column 0: the value one slot up, v[16 - s] beside v[15 - s]
#pragma unroll
            for (int s = 0; s < 8; s++) {
                const V a = v[s], b = v[15 - s];
                V ma, mb;  // mirrors of a and b
                if constexpr (E == 32) {
                    const V c = v[16 + s], e = v[31 - s];
                    ma = e;
                    mb = c;
                    v[16 + s] = blend(H[bin(16 + s)], c, z ? e : b);
                    v[31 - s] = blend(H[bin(31 - s)], e, z ? c : a);
                } else {
                    ma = x_shfl(b, src);
                    mb = x_shfl(a, src);
                }
                // column 0: a = v[s] mirrors v[16 - s] (up), b = v[15 - s] mirrors v[s + 1]
                const V nx = s < 7 ? v[s + 1] : v8;
                v[s] = blend(H[bin(s)], a, z ? up : ma);
                v[15 - s] = blend(H[bin(15 - s)], b, z ? nx : mb);
                up = b;
            }
        }
    }
};

// ---- reductions over the group ---------------------------------------------
// Fixed shuffle tree per warp, then the group's warps in order: the result
// does not depend on C.  red: 2 x (T / 32) doubles (alternating halves, so
// one barrier per reduction orders it against the next); flip is uniform.
template <int T, int C, bool MAX>
__device__ __forceinline__ double x_reduce(double v, double* red, int& flip, int rank) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double w = __shfl_xor_sync(0xffffffffu, v, o);
        v = MAX ? fmax(v, w) : v + w;
    }
    constexpr int W = T / 32, WC = W / C;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double* r = red + (flip ? 32 : 0);
    flip ^= 1;
    if constexpr (C == 1) {
        if (lane == 0) r[warp] = v;
        __syncthreads();
    } else {
        if (lane < C) x_st(x_mapa(x_smem(r + rank * WC + warp), lane), v);
        x_cluster_sync();
    }
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < W; w++) s = MAX ? fmax(s, r[w]) : s + r[w];
    return s;
}

}  // namespace fl
