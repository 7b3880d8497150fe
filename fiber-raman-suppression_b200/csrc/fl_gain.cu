// fl_gain.cu -- pump-gain single-mode forward stepper (disp_gain_smf!).
//
// Reference: the right-hand side src/simulation/simulate_disp_gain_mmf.jl:
// 21-66 (disp_mmf!'s nonlinear term plus g(ω)ũ/2, and dP/dz = g_P P), the
// gain models :68-102 with calculate_gain_YDFA (src/gain_simulation/gain.jl:
// 150-166), and the solver :204-239 (Tsit5 over the state [P; ũ]).
//
// One CTA integrates one problem to z = L in one launch.  The nonlinear term
// is the single-mode stepper's forward right-hand side (its transforms).  The
// gain of a stage is computed from the stage input before them: two block sums
// give the rate-equation terms W12 and W21 of the stage's spectrum (|ũ|² =
// |e^{iDz}ũ|²), the inversion n2 follows, and each thread keeps g_b ũ_b / 2
// of its own bins in scratch and adds it to the derivative.  The
// pump power and its seven stage derivatives are block-uniform FP64 scalars;
// the RMS error norm runs over the Nt + 1 components of the state, as the
// reference's does over [P; ũ].  FP32 right-hand side, FP64 state, stage
// accumulation and error norm, as the main stepper.
#include "fl_launch.h"
#include "fl_sm.cuh"

namespace fl {

// One evaluation at z, the field in registers from the stage sum to the stored
// derivative k[to]: the field is u + dt Σ_{j<n} a_j k_j (FP64 accumulation;
// a_j the coefficients of stage n, or 1 for the probe), the pump power there
// pp; stage 6 also leaves the new state in un, the partial error and the
// weights.  Returns dP/dz.
// Out of line: one body for the launch, the probe and the stages.  All loads
// of a chunk of points are in flight for one stage vector after the other
// (Nt = 2^12, 0.2 m, one solve: 2.07 ms with the stages inside the points and
// the field handed over through global memory, 1.37 so; 2^13 2.96 and 2.09).
template <int LOGN>
__device__ __noinline__ double gain_eval(const GainDesc& g, unsigned char* smraw, double* red,
                                         int& flip, int n, int to, bool probe, double z, double dt,
                                         double pp, const double* u, double* un) {
    using Sol = SmSolver<float, float, LOGN, 1>;
    using CF = cx<float>;
    constexpr int N = Sol::N, E = Sol::E, T = Sol::XF::T, SC = E < 8 ? E : 8;
    const SlotDesc& d = g.s;
    const Sol S(d, smraw, 0);
    auto sum = [&](double v) { return x_reduce<T, 1, false>(v, red, flip, 0); };
    CF v[E];
#pragma unroll
    for (int s0 = 0; s0 < E; s0 += SC) {
        double ar[SC], ai[SC], er[SC], ei[SC];
#pragma unroll
        for (int c = 0; c < SC; c++) ar[c] = ai[c] = er[c] = ei[c] = 0.0;
#pragma unroll 1
        for (int j = 0; j < n; j++) {
            const CF* kj = static_cast<const CF*>(d.kf[j]);
            const double a = probe ? 1.0 : kT5a[n][j];
            CF x[SC];
#pragma unroll
            for (int c = 0; c < SC; c++) x[c] = kj[S.own(s0 + c)];
#pragma unroll
            for (int c = 0; c < SC; c++) {
                ar[c] += a * (double)x[c].re;
                ai[c] += a * (double)x[c].im;
            }
            if (n == 6) {
                const double bt = kT5bt[j];
#pragma unroll
                for (int c = 0; c < SC; c++) {
                    er[c] += bt * (double)x[c].re;
                    ei[c] += bt * (double)x[c].im;
                }
            }
        }
#pragma unroll
        for (int c = 0; c < SC; c++) {
            const int b = S.own(s0 + c);
            const cx<double> x0 = ld2(u, b);
            const cx<double> u1 = mk(x0.re + dt * ar[c], x0.im + dt * ai[c]);
            v[s0 + c] = down<float>(u1);
            if (n == 6) {
                st2(un, b, u1);
                st2(d.esv, b, mk(dt * er[c], dt * ei[c]));
                const double m0 = x0.re * x0.re + x0.im * x0.im;
                const double m1 = u1.re * u1.re + u1.im * u1.im;
                d.skv[b] = d.abstol + sqrt(fmax(m0, m1)) * d.reltol;
            }
        }
    }
    // g(ω)ũ/2, kept for the way out
    CF* gb = static_cast<CF*>(d.ka[1]);
    double gP = -1.0;
    if (g.kind == 0) {
#pragma unroll
        for (int s = 0; s < E; s++) gb[S.own(s)] = scale(v[s], (float)(0.5 * g.g_const));
    } else {
        double w12 = 0.0, w21 = 0.0;
#pragma unroll
        for (int s = 0; s < E; s++) {
            const int b = S.bin(s);
            const double e = abs2(up(v[s]));
            w12 += g.wa[b] * e;
            w21 += g.we[b] * e;
        }
        w12 = sum(w12);
        w21 = sum(w21);
        const double r12 = g.r12c * pp, r21 = g.r21c * pp;
        const double n2 = (r12 + w12) / (r12 + r21 + w12 + w21 + g.inv_tau), n1 = 1.0 - n2;
#pragma unroll
        for (int s = 0; s < E; s++) {
            const int b = S.bin(s);
            gb[S.own(s)] = scale(v[s], (float)(0.5 * (g.sE[b] * n2 - g.sA[b] * n1)));
        }
        gP = g.gpe * n2 - g.gpa * n1;
    }
#pragma unroll
    for (int s = 0; s < E; s++) v[s] = cmul(v[s], phasor<float>(d.Dturns[S.bin(s)], z));
    // (the run before may still be reading the first exchange buffer)
    if constexpr (Sol::XF::S::SMALL) Sol::XF::sync();
    S.transforms(false, v);
    CF* out = static_cast<CF*>(d.kf[to]);
    const float invn = 1.0f / N;
#pragma unroll
    for (int s = 0; s < E; s++) {
        const int f = S.bin(s), b = S.own(s);
        const CF y = cmulc(v[s], phasor<float>(d.Dturns[f], z));  // e^{-iDz} x
        const float sc = S.ss[f] * invn;
        out[b] = mk(-y.im * sc, y.re * sc) + gb[b];
    }
    return gP * pp;
}

template <int LOGN>
__global__ void __launch_bounds__(XShape<LOGN, 1>::T, 1)
    gain_forward_kernel(const GainDesc* __restrict__ gdp, GainOut* __restrict__ out) {
    using Sol = SmSolver<float, float, LOGN, 1>;
    using CF = cx<float>;
    constexpr int N = Sol::N, E = Sol::E, T = Sol::XF::T;
    extern __shared__ __align__(16) unsigned char smraw[];
    double* red = reinterpret_cast<double*>(smraw + SmShared<float, LOGN, 1>::RED);
    const GainDesc& g = *gdp;
    const SlotDesc& d = g.s;
    load_tables<float, LOGN, 1>(d, smraw, 0);
    const Sol S(d, smraw, 0);
    int flip = 0;
    auto sum = [&](double v) { return x_reduce<T, 1, false>(v, red, flip, 0); };
    CF* k[7];
#pragma unroll
    for (int i = 0; i < 7; i++) k[i] = static_cast<CF*>(d.kf[i]);
    double* u = d.u[0];
    double* un = d.u[1];
    const double L = d.L, dtmin = kEps * L, at = d.abstol, rt = d.reltol;
    auto eval = [&](int n, int to, bool probe, double z, double dt, double pp) -> double {
        return gain_eval<LOGN>(g, smraw, red, flip, n, to, probe, z, dt, pp, u, un);
    };

    // ---- launch and f0
#pragma unroll
    for (int s = 0; s < E; s++) {
        const cx<double> x = ld2(d.u0, S.bin(s));
        st2(u, S.own(s), x);
    }
    double pp = g.pump0;
    // save positions at z = 0: the launch (the lab frame equals the interaction frame there)
    int save_idx = 0;
    while (save_idx < d.nsave && d.zsave[save_idx] == 0.0) {
        double* o = d.save_out + (size_t)save_idx * 2 * N;
#pragma unroll
        for (int s = 0; s < E; s++) st2(o, S.bin(s), ld2(d.u0, S.bin(s)));
        if (threadIdx.x == 0) g.pump_save[save_idx] = pp;
        save_idx++;
    }
    long nf = 0, naccept = 0, nreject = 0;
    int status = ST_OK;
    double kp[7];
    kp[0] = eval(0, 0, false, 0.0, 0.0, pp);
    nf++;

    // ---- initial step (OrdinaryDiffEqCore ode_determine_initdt), P one more
    // component of the norms; weights from the launch
    const double skp = at + fabs(pp) * rt;
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int s = 0; s < E; s++) {
        const cx<double> x = ld2(u, S.own(s));
        const double ax = sqrt(x.re * x.re + x.im * x.im), sk = at + ax * rt;
        const double af = sqrt(abs2(up(k[0][S.own(s)])));
        s0 += (ax / sk) * (ax / sk);
        s1 += (af / sk) * (af / sk);
    }
    s0 = sum(s0) + (pp / skp) * (pp / skp);
    s1 = sum(s1) + (kp[0] / skp) * (kp[0] / skp);
    const double d0 = sqrt(s0 / (N + 1)), d1 = sqrt(s1 / (N + 1));
    double dt;
    if (isnan(d1)) {
        dt = dtmin;
    } else {
        const double dt0 = fmin((d0 < 1e-5 || d1 < 1e-5) ? 1e-6 : (d0 / d1) / 100.0, L);
        if (dt0 < 10.0 * kEps) {
            dt = fmax(1e-6, dtmin);
        } else {
            const double kp1 = eval(1, 1, true, dt0, dt0, pp + dt0 * kp[0]);
            nf++;
            double s2 = 0.0, nd = 0.0;
#pragma unroll
            for (int s = 0; s < E; s++) {
                const int b = S.own(s);
                const cx<double> x = ld2(u, b);
                const double sk = at + sqrt(x.re * x.re + x.im * x.im) * rt;
                const CF f0 = k[0][b], f1 = k[1][b];
                const double dr = (double)f1.re - (double)f0.re;
                const double di = (double)f1.im - (double)f0.im;
                s2 += (dr * dr + di * di) / (sk * sk);
                nd += (dr != 0.0 || di != 0.0) ? 1.0 : 0.0;
            }
            const double dp = kp1 - kp[0];
            s2 = sum(s2) + (dp / skp) * (dp / skp);
            nd = sum(nd) + (dp != 0.0 ? 1.0 : 0.0);
            const double d2 = sqrt(s2 / (N + 1)) / dt0;
            dt = initdt_final(dt0, d1, d2, nd, dtmin, L);
        }
    }
    nf++;  // the reference evaluates f0 once more after the initial step

    // ---- Tsit5 with the PI controller, FSAL (k0 <- k6 on accept)
    double z = 0.0, qold = kQoldInit;
    long iters = 0;
    while (z < L) {
        if (++iters > d.max_iters) {
            status = ST_MAXITERS;
            break;
        }
        double adt = fmax(fmin(fabs(dt), L), dtmin);
        const double rem = L - z;
        if (adt > rem) adt = rem;
        if (adt <= dtmin && rem > dtmin) {
            status = ST_DT_UNDERFLOW;
            break;
        }
        dt = adt;
        double pnew = pp;
        for (int st = 1; st < 7; st++) {
            double acc = 0.0;
            for (int j = 0; j < st; j++) acc += kT5a[st][j] * kp[j];
            const double pps = pp + dt * acc;
            if (st == 6) pnew = pps;
            kp[st] = eval(st, st, false, z + kT5c[st] * dt, dt, pps);
            nf++;
        }
        // error dt Σ b̃_j k_j over the Nt + 1 components
        double acc = 0.0;
#pragma unroll
        for (int s = 0; s < E; s++) {
            const int b = S.own(s);
            const cx<double> e6 = ld2(d.esv, b);
            const CF k6 = k[6][b];
            const double er = e6.re + dt * kT5bt[6] * (double)k6.re;
            const double ei = e6.im + dt * kT5bt[6] * (double)k6.im;
            const double w = d.skv[b];
            acc += (er * er + ei * ei) / (w * w);
        }
        acc = sum(acc);
        double ep = 0.0;
        for (int j = 0; j < 7; j++) ep += kT5bt[j] * kp[j];
        ep *= dt;
        const double wp = at + fmax(fabs(pp), fabs(pnew)) * rt;
        const double EEst = sqrt((acc + (ep / wp) * (ep / wp)) / (N + 1));
        if (!isfinite(EEst)) {
            status = ST_NONFINITE;
            break;
        }
        double q11;
        const double q = pi_q(EEst, qold, q11);
        if (EEst > 1.0) {
            nreject++;
            dt = dt / fmin(1.0 / kQmin, q11 / kGamma);
            continue;
        }
        naccept++;
        double znew = z + dt;
        if (fabs(znew - L) < 100.0 * kEps * fmax(z, L)) znew = L;  // snap to the tstop
        // save positions in (z, znew) and on an interior step end: Tsit5's
        // free interpolant u_n + dt Σ_i b_i(θ) k_i for the field and the pump
        // power (positions at L take the final state below)
        while (save_idx < d.nsave && d.zsave[save_idx] > z &&
               (d.zsave[save_idx] < znew || (d.zsave[save_idx] == znew && znew < L))) {
            const double zs = d.zsave[save_idx], th = (zs - z) / dt;
            double bi[7];
            for (int i = 0; i < 7; i++) {
                double b = 0.0, tp = th;
                for (int q = 0; q < 4; q++) {
                    b += kT5r[i][q] * tp;
                    tp *= th;
                }
                bi[i] = b;
            }
            double* o = d.save_out + (size_t)save_idx * 2 * N;
#pragma unroll
            for (int s = 0; s < E; s++) {
                const int b = S.own(s), f = S.bin(s);
                double xr = 0.0, xi = 0.0;
                for (int i = 0; i < 7; i++) {
                    const CF ki = k[i][b];
                    xr += bi[i] * (double)ki.re;
                    xi += bi[i] * (double)ki.im;
                }
                const cx<double> un0 = ld2(u, b);
                const cx<double> x = mk(un0.re + dt * xr, un0.im + dt * xi);
                const cx<double> p = phasor<double>(d.Dturns[f], zs);
                st2(o, f, mk(x.re * p.re - x.im * p.im, x.re * p.im + x.im * p.re));
            }
            if (threadIdx.x == 0) {
                double pk = 0.0;
                for (int i = 0; i < 7; i++) pk += bi[i] * kp[i];
                g.pump_save[save_idx] = pp + dt * pk;
            }
            save_idx++;
        }
        z = znew;
#pragma unroll
        for (int s = 0; s < E; s++) {
            const int b = S.own(s);
            st2(u, b, ld2(un, b));
            k[0][b] = k[6][b];
        }
        pp = pnew;
        kp[0] = kp[6];
        qold = fmax(EEst, kQoldInit);
        dt = fmin(fmax((q == 1.0) ? dt : dt / q, dtmin), L);
    }

    // ---- lab-frame spectrum at the end (and the save positions at L), pump
    // power and counters
#pragma unroll
    for (int s = 0; s < E; s++) {
        const int b = S.bin(s);
        const cx<double> x = ld2(u, S.own(s));
        const cx<double> p = phasor<double>(d.Dturns[b], z);
        const cx<double> y = mk(x.re * p.re - x.im * p.im, x.re * p.im + x.im * p.re);
        st2(d.uL_out, b, y);
        if (status == ST_OK)
            for (int si = save_idx; si < d.nsave; si++) st2(d.save_out + (size_t)si * 2 * N, b, y);
    }
    if (threadIdx.x == 0 && status == ST_OK)
        for (int si = save_idx; si < d.nsave; si++) g.pump_save[si] = pp;
    if (threadIdx.x == 0) {
        out->naccept = naccept;
        out->nreject = nreject;
        out->nf = nf;
        out->status = status;
        out->z_end = z;
        out->pump_L = pp;
    }
}

template <int LOGN>
cudaError_t launch_gain_t(const GainDesc* desc, GainOut* out, cudaStream_t stream) {
    auto kern = gain_forward_kernel<LOGN>;
    const size_t smem = SmShared<float, LOGN, 1>::BYTES;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return e;
    kern<<<1, XShape<LOGN, 1>::T, smem, stream>>>(desc, out);
    return cudaGetLastError();
}

bool gain_built(int logn) { return logn >= 6 && logn <= 13; }

cudaError_t launch_gain(int logn, const GainDesc* desc, GainOut* out, cudaStream_t stream) {
    switch (logn) {
        case 6: return launch_gain_t<6>(desc, out, stream);
        case 7: return launch_gain_t<7>(desc, out, stream);
        case 8: return launch_gain_t<8>(desc, out, stream);
        case 9: return launch_gain_t<9>(desc, out, stream);
        case 10: return launch_gain_t<10>(desc, out, stream);
        case 11: return launch_gain_t<11>(desc, out, stream);
        case 12: return launch_gain_t<12>(desc, out, stream);
        case 13: return launch_gain_t<13>(desc, out, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace fl
