"""Timed cases of the stepper: what a program asks of it, over the range it is asked for.

A case is one call (or one pair of calls) through the public Python binding of
the C-ABI, from one short propagation to the batched multimode inverse-design
launch.  `listed()` are fixed points of the ranges, `draw()` takes others.

FP32-mode outputs are handed on in single precision (the mode's accuracy);
FP64-mode outputs stay in double.

`exact()` integrates the same problem in FP64 with plain torch / numpy: the
interaction-picture right-hand sides, Tsit5 with its free interpolant and PI
step control, stop-free adjoint, at the case's tolerances.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "fiber-raman-suppression_b200"))

C0, N2 = 2.99792458e8, 2.3e-20
BETAS = (-2.17e-26, 1.2e-40)
REP = 80e6
FWHM = 185e-15

# kind: forward    GPUProblem.forward on host arrays, nsave positions
#       propagate  solve.propagate from a resolved problem (tables uploaded in
#                  the call) with the device evidence sums
#       adjoint    GPUProblem.forward, a seed made from its output, .adjoint
#       gradient   phase_gradient_batch on host arrays
#       gradient_device  the same on device buffers
#       mode_gradient    mode_phase_gradient_batch_device (a phase per mode and bin)
#       serve      a burst of requests through the continuous-batching server
_DEFAULT = dict(order=-1, batch=1, nsave=2, precision="fp32", log_cost=False, band=-13.0)


def _case(name, kind, nt, window, length, power, **kw):
    return dict(_DEFAULT, name=name, kind=kind, nt=nt, window=float(window), length=float(length),
                power=float(power), **kw)


def listed():
    return [
        # the smallest useful call: one short fibre on a small grid, host arrays
        _case("forward 2^10", "forward", 1024, 10.0, 0.5, 0.1),
        # the reference's plain double-precision propagation
        _case("forward 2^13 fp64", "forward", 8192, 10.0, 0.5, 0.1, precision="fp64"),
        # a long window on the largest single-CTA grid
        _case("forward 2^14", "forward", 16384, 45.0, 0.7, 0.08),
        # the drop-in call of a script: tables built and uploaded, five saved
        # positions along the fibre, evidence sums
        _case("propagate 2^12 saves", "propagate", 4096, 12.0, 0.6, 0.07, nsave=5),
        # the adjoint contract (an rrule): forward, the program's own seed, adjoint
        _case("adjoint pair 2^11", "adjoint", 2048, 8.0, 0.4, 0.06),
        # one inverse-design gradient, one problem per call
        _case("gradient 2^13", "gradient", 8192, 10.0, 0.5, 0.1),
        # one optimiser's line search: a few trial phases, cost in dB
        _case("gradient 2^12 x 4", "gradient", 4096, 11.0, 0.5, 0.08, batch=4, log_cost=True,
              band=-5.0),
        # the batched inverse-design step on resident buffers
        _case("gradient 2^13 x 592", "gradient_device", 8192, 10.0, 0.5, 0.1, batch=592),
        # a burst of mixed requests through the server
        _case("serve 2^11..2^13 x 72", "serve", 8192, 10.0, 0.5, 0.1, batch=72, band=-5.0),
        # few modes in double precision
        _case("forward 3 modes fp64", "forward", 2048, 8.0, 0.3, 0.1, order=1, precision="fp64"),
        # six modes, one forward + adjoint per call
        _case("gradient 6 modes", "gradient", 4096, 5.0, 1.0, 0.16, order=2,
              band=-2.0),
        # multimode inverse design: ten modes, 64 launch-phase candidates
        _case("mode gradient 10 modes x 64", "mode_gradient", 16384, 10.0, 0.4, 0.4, order=3,
              batch=64, band=-2.0),
    ]


def draw(rng):
    """One more case of the same ranges (sizes over their logarithm)."""
    kind = rng.choice(["forward", "forward", "propagate", "adjoint", "gradient", "gradient_device",
                       "mode_gradient", "serve"])
    length = math.exp(rng.uniform(math.log(0.05), math.log(0.7)))
    power = rng.uniform(0.02, 0.1)
    kw = dict(precision="fp64" if rng.random() < 0.2 else "fp32")
    step = rng.uniform(2.7e-3, 8e-3)  # ps per sample: positive frequencies, >= 20 samples per pulse
    if kind == "serve":
        nt, step, kw = 8192, 10.0 / 8192, dict(batch=rng.randint(9, 70), band=-5.0)
        length = min(length, 0.5)
    elif kind == "mode_gradient":
        kw.update(order=rng.randint(1, 3), band=-2.0, batch=int(math.exp(rng.uniform(0.0, math.log(24.5)))))
        nt = 2 ** rng.randint(9, 12)
        power = rng.uniform(0.1, 0.3)
    else:
        if rng.random() < 0.25:
            kw["order"] = rng.randint(1, 2)
        top = 13 if kw.get("order") else (15 if kind in ("forward", "propagate") else 14)
        nt = 2 ** rng.randint(9, top)
        if kind in ("forward", "propagate"):
            kw["nsave"] = rng.randint(2, 7)
        elif kind.startswith("gradient"):
            most = 2 ** 22 // nt if not kw.get("order") else 2 ** 16 // nt
            kw.update(batch=max(1, int(math.exp(rng.uniform(0.0, math.log(max(most, 2)))))),
                      log_cost=rng.random() < 0.5, band=-rng.choice([2.0, 3.0, 5.0]))
    window = round(nt * max(step, 3.0 / nt), 3)
    c = _case("", kind, nt, window, round(length, 4), round(power, 4), **kw)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# what the program holds before the call
# ---------------------------------------------------------------------------

def _modes(c):
    return (c["order"] + 1) * (c["order"] + 2) // 2 if c["order"] >= 0 else 1


def _requests(c, seed):
    """The burst of a serve case: (nt, length, power, is_gradient) per request;
    lengths and powers come from the seed."""
    kind, r = np.random.default_rng(c["batch"]), np.random.default_rng(seed)
    return [(1 << int(kind.integers(11, 14)), float(r.uniform(0.2, 1.0) * c["length"]),
             float(r.uniform(0.3, 1.0) * c["power"]), bool(kind.integers(0, 2)))
            for _ in range(c["batch"])]


def _phases(c, seed):
    r = np.random.default_rng(seed + 77)
    if c["kind"] == "mode_gradient":
        return r.standard_normal((c["batch"], _modes(c), c["nt"])) * 0.5
    return 0.5 * r.standard_normal((c["batch"], c["nt"]))


def _problem(c, seed, nt=None):
    from fiberlab_gpu import problem as P
    nt = nt or c["nt"]
    if c["order"] < 0:
        fp = P.single_mode_problem(nt=nt, time_window_ps=c["window"], L=c["length"],
                                   power_w=c["power"], fwhm_s=FWHM, rep_rate_hz=REP,
                                   raman_threshold_thz=c["band"],
                                   validate_grid=c["kind"] == "propagate")
        fp.uw0 = _launch(c, fp.uw0, nt, c["window"], seed)
        return fp
    return P.multimode_problem(c["order"], 64, nt, c["window"], c["length"], c["power"] / REP,
                               200e-15, seed, raman_threshold_thz=c["band"])


def _launch(c, uw0, nt, window, seed):
    """The program's pulse.  Gradients shape the flat-phase pulse by their own
    phases; the others take a slightly chirped one (the seed's chirp)."""
    if c["kind"] not in ("forward", "propagate", "adjoint"):
        return uw0
    w = 2 * np.pi * np.fft.fftfreq(nt, window / nt)
    gdd = np.random.default_rng(seed + 5).uniform(-0.002, 0.002)  # ps^2
    return uw0 * np.exp(0.5j * gdd * w * w)[None, :]


def prepare(case, seed):
    c = case
    from fiberlab_gpu._capi import Context, GPUProblem
    s = dict(c=c)
    many = c["kind"] == "mode_gradient"
    s["ctx"] = ctx = Context(0, checkpoints=8, segment_steps=48) if many else Context(0)
    if c["kind"] == "serve":
        from fiberlab_gpu.serving import Server
        s["gp"] = {n: GPUProblem(ctx, _problem(c, seed, n)) for n in (2048, 4096, 8192)}
        s["server"] = Server(ctx, checkpoints=32, segment_steps=64)
        s["reqs"] = []
        for i, (nt, length, power, grad) in enumerate(_requests(c, seed)):
            u0 = s["gp"][nt].fp.uw0 * math.sqrt(power / c["power"])
            ph = 0.5 * np.random.default_rng(seed + 100 + i).standard_normal(nt) if grad else None
            s["reqs"].append((nt, length, u0, ph))
        return s
    s["fp"] = fp = _problem(c, seed)
    if c["kind"] == "propagate":
        s["z"] = np.linspace(0.0, fp.L, c["nsave"])
        s["z"][-1] = fp.L
        return s
    s["gp"] = GPUProblem(ctx, fp, c["precision"])
    if c["kind"] == "forward":
        s["z"] = np.linspace(0.0, fp.L, c["nsave"])
        s["z"][-1] = fp.L
    elif c["kind"] == "adjoint":
        s["w"] = np.linspace(0.2, 1.8, fp.nt)[None, :]
    else:
        ph = _phases(c, seed)
        if c["kind"] == "gradient":
            s["ph"] = ph
        else:
            s["u0"] = torch.from_numpy(np.ascontiguousarray(fp.uw0)).cuda()
            s["ph"] = torch.from_numpy(ph).cuda()
            s["mask"] = torch.from_numpy(fp.mask.astype(np.uint8)).cuda()
            s["J"] = torch.empty(c["batch"], dtype=torch.float64, device="cuda")
            s["g"] = torch.empty_like(s["ph"])
    return s


def _out(c, *arrays):
    """The outputs at the accuracy of the case's precision mode."""
    if c["precision"] == "fp64":
        return list(arrays)
    return [a.float() if isinstance(a, torch.Tensor) else
            a.astype(np.complex64 if a.dtype.kind == "c" else np.float32) for a in arrays]


def run(state):
    s, c = state, state["c"]
    kind = c["kind"]
    if kind == "forward":
        return _out(c, s["gp"].forward(s["fp"].uw0, s["z"])[0])
    if kind == "propagate":
        from fiberlab_gpu import solve
        r = solve.propagate(s["fp"], s["z"], precision=c["precision"], ctx=s["ctx"])
        return _out(c, r.spectra, r.device_evidence)
    if kind == "adjoint":
        u, _ = s["gp"].forward()
        lam, _ = s["gp"].adjoint(u[-1] * s["w"])
        return _out(c, u, lam)
    if kind == "gradient":
        J, g, _ = s["gp"].phase_gradient_batch(s["ph"], log_cost=c["log_cost"])
        return _out(c, J, g)
    if kind in ("gradient_device", "mode_gradient"):
        f = s["gp"].phase_gradient_batch_device if kind == "gradient_device" else \
            s["gp"].mode_phase_gradient_batch_device
        f(s["u0"].data_ptr(), c["batch"], s["ph"].data_ptr(), s["mask"].data_ptr(),
          s["J"].data_ptr(), s["g"].data_ptr(), log_cost=c["log_cost"], with_stats=False)
        return _out(c, s["J"], s["g"])
    live = []
    for nt, length, u0, ph in s["reqs"]:
        gp = s["gp"][nt]
        live.append(s["server"].submit_forward(gp, u0, length) if ph is None else
                    s["server"].submit_band_gradient(gp, ph, u0=u0, L=length))
    done = [s["server"].wait(r) for r in live]
    fields = [r.out_field.ravel() for r in done if r.out_field is not None]
    grads = [r.out_grad / np.linalg.norm(r.out_grad) for r in done if r.out_grad is not None]
    return _out(c, np.concatenate(fields) if fields else np.zeros(1, complex),
                np.concatenate(grads) if grads else np.zeros(1),
                np.array([r.J for r in done if r.out_grad is not None]))


def _attempts(c):
    """Attempted Tsit5 steps of one solve (an estimate from solves of these ranges)."""
    return 8.0 + 90.0 * c["length"] * math.sqrt(c["power"] / 0.1)


def work(case):
    """Launch, tables and outputs once; the transforms and pointwise terms of
    six right-hand sides per attempted step, forward and (where it has one)
    adjoint."""
    c, M = case, _modes(case)
    n = c["nt"] * M * c["batch"]
    adj = c["kind"] not in ("forward", "propagate")
    fft = 5.0 * math.log2(c["nt"])
    pairs = M * (M + 1) / 2
    fwd = (2 + 2 * pairs / M / 2) * fft + 60 + 8.0 * M * pairs
    bwd = (3 + 4 * pairs / M / 2) * fft + 90 + 24.0 * M * pairs
    flops = 6 * n * _attempts(c) * (fwd + 40 + (bwd + 40 if adj else 0))
    out = 16 * c["nsave"] if not adj else 8 if c["kind"] != "adjoint" else 48
    return {"bytes": n * (16.0 + out) + c["nt"] * (8.0 * M + 33) + 8.0 * M ** 4, "flops": flops}


# ---------------------------------------------------------------------------
# the same in FP64, in plain torch and numpy
# ---------------------------------------------------------------------------

_A = ((), (0.161,), (-0.008480655492356989, 0.335480655492357),
      (2.897153057105493, -6.359448489975075, 4.3622954328695815),
      (5.325864828439257, -11.748883564062828, 7.4955393428898365, -0.09249506636175525),
      (5.86145544294642, -12.92096931784711, 8.159367898576159, -0.071584973281401,
       -0.028269050394068383),
      (0.09646076681806523, 0.01, 0.4798896504144996, 1.379008574103742, -3.290069515436081,
       2.324710524099774))
_C = (0.0, 0.161, 0.327, 0.9, 0.9800255409045097, 1.0, 1.0)
_BT = (-0.00178001105222577714, -0.0008164344596567469, 0.007880878010261995, -0.1447110071732629,
       0.5823571654525552, -0.45808210592918697, 0.015151515151515152)
_R = ((1.0, -2.763706197274826, 2.9132554618219126, -1.0530884977290216),
      (0.0, 0.13169999999999998, -0.2234, 0.1017),
      (0.0, 3.9302962368947516, -5.941033872131505, 2.490627285651253),
      (0.0, -12.411077166933676, 30.33818863028232, -16.548102889244902),
      (0.0, 37.50931341651104, -88.1789048947664, 47.37952196281928),
      (0.0, -27.896526289197286, 65.09189467479366, -34.87065786149661), (0.0, 1.5, -4.0, 2.5))


def _setup(c, seed, nt, power, length):
    """Grid tables, Kerr tensor and launch in numpy."""
    M, T = _modes(c), c["window"]
    dt, f0 = T / nt, C0 / 1550e-9 / 1e12
    f = np.fft.fftfreq(nt, dt)
    w = 2 * np.pi * f
    d, r = 1e3 / 32.0, 1e3 / 12.2
    h = np.exp(-1j * w * T / 2) * 0.18 * (d * d + r * r) / ((d + 1j * w) ** 2 + r * r)
    h[nt // 2] = h[nt // 2].real
    D = sum(((w * 1e12) ** (n + 2) / math.factorial(n + 2)) * b for n, b in enumerate(BETAS))
    t = 1e-12 * (-T / 2 + np.arange(nt) * dt)
    if M == 1:
        gam, D = np.full((1, 1, 1, 1), 1.1e-3), D[None, :]
        env, ppk, amp = 1 / np.cosh(t * 1.7627 / FWHM), 0.881374 * power / FWHM / REP, np.ones(1)
    else:
        from numpy.polynomial.hermite import hermval
        nx, w0 = 64, 15e-6
        dx = 8 * w0 / nx
        X, Y = np.meshgrid(*2 * [(np.arange(nx) - (nx - 1) / 2) * dx], indexing="ij")
        idx = [(g - n, n) for g in range(c["order"] + 1) for n in range(g + 1)]
        ps = [hermval(math.sqrt(2) * X / w0, np.eye(m + 1)[m]) *
              hermval(math.sqrt(2) * Y / w0, np.eye(n + 1)[n]) * np.exp(-(X ** 2 + Y ** 2) / w0 ** 2)
              for m, n in idx]
        ps = np.stack([(p / np.linalg.norm(p)).ravel() for p in ps], 1)
        gam = np.einsum("pi,pj,pk,pl->ijkl", ps, ps, ps, ps, optimize=True) / dx ** 2 * \
            N2 * 2 * np.pi * f0 * 1e12 / C0
        D = np.stack([D + (0, 50, 100, 150)[m + n] + (0.0, 1e-13, -1e-13, 1e-13)[m + n] * w * 1e12
                      for m, n in idx])
        rng = np.random.default_rng(seed)
        wt = rng.dirichlet(np.ones(M))
        amp = np.sqrt(wt) * np.exp(1j * rng.uniform(0, 2 * math.pi, M))
        amp = amp / np.linalg.norm(amp)
        env, ppk = 1 / np.cosh(t * 1.7627 / 200e-15), 0.881374 * power / REP / 200e-15
    ut = env[None, :] * np.conj(amp)[:, None]
    u0 = np.fft.ifft(ut / math.sqrt(np.max(np.sum(np.abs(ut) ** 2, 0))) * math.sqrt(ppk), axis=1)
    if M == 1:
        u0 = _launch(c, u0, nt, T, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    tt = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    return dict(D=tt(D), g=tt(gam.reshape(M * M, M * M)), H=tt(h * (-1.0) ** np.arange(nt)), M=M,
                ss=tt((f0 + f) / f0), u0=u0, mask=f < c["band"], L=length, nt=nt, dev=dev, tt=tt)


def _rhs(p, z, u):
    M = p["M"]
    ph = torch.polar(torch.ones_like(p["D"]), p["D"] * z[:, None, None])
    ut = torch.fft.fft(u * ph)
    P = (ut[:, :, None] * ut[:, None].conj()).real.flatten(1, 2)
    P = torch.matmul(p["g"], P)
    S = 0.82 * P + torch.fft.ifft(p["H"] * torch.fft.fft(P)).real
    eta = (S.view(-1, M, M, p["nt"]) * ut[:, None]).sum(2)
    return 1j * p["ss"] * ph.conj() * torch.fft.ifft(eta)


def _rhs_adj(p, z, lam, u):
    M, g, sh = p["M"], p["g"], (-1, p["M"], p["M"], p["nt"])
    ph = torch.polar(torch.ones_like(p["D"]), p["D"] * z[:, None, None])
    lt, ut = torch.fft.fft(lam * ph * p["ss"]), torch.fft.fft(u * ph)
    P = torch.matmul(g, (ut[:, :, None] * ut[:, None].conj()).real.flatten(1, 2))
    S = 1.64 * P + torch.fft.ifft(p["H"] * torch.fft.fft(P)).real
    X = torch.matmul(g, (lt[:, :, None] * ut[:, None].conj()).imag.flatten(1, 2))
    Cq = torch.fft.ifft(p["H"].conj() * torch.fft.fft(X)).real
    W = torch.matmul(g.to(ut.dtype), (ut[:, :, None] * ut[:, None]).flatten(1, 2))
    eta = (S.view(sh) * lt[:, None] - 0.82 * W.view(sh) * lt[:, None].conj() +
           2j * Cq.view(sh) * ut[:, None]).sum(2)
    return 1j * ph.conj() * torch.fft.ifft(eta)


def _norm(x):
    return torch.sqrt(torch.mean(torch.abs(x) ** 2, dim=(1, 2)))


def _integrate(p, f, x, L, back, atol, accept):
    """Tsit5 over [0, L] (or L -> 0) for every sample at once, each with its
    own steps; accept(which, z, dt, x, k) sees the accepted ones."""
    rtol, eps, B = 1e-8, 2.220446049250313e-16, x.shape[0]
    sg, dtmin = (-1.0 if back else 1.0), eps * L
    z = torch.full((B,), L if back else 0.0, dtype=torch.float64, device=x.device)
    col = lambda v: v[:, None, None]  # noqa: E731
    k1 = f(z, x)
    sk = col(atol) + torch.abs(x) * rtol
    d0, d1 = _norm(x / sk), _norm(k1 / sk)
    dt0 = torch.where((d0 < 1e-5) | (d1 < 1e-5), torch.full_like(d0, 1e-6), d0 / d1 / 100).clamp(max=L)
    d2 = _norm((f(z + sg * dt0, x + col(sg * dt0) * k1) - k1) / sk) / dt0
    mx = torch.maximum(d1, d2)
    dt1 = torch.where(mx <= 1e-15, (dt0 * 1e-3).clamp(min=1e-6), 10 ** (-(2 + torch.log10(mx)) / 5))
    dt = torch.minimum(100 * dt0, dt1).clamp(dtmin, L)
    qold = torch.full_like(dt, 1e-4)
    live = torch.ones_like(dt, dtype=torch.bool)
    while bool(live.any()):
        rem = z if back else L - z
        h = torch.where(live, torch.minimum(dt.clamp(dtmin, L), rem), torch.zeros_like(dt))
        k = [k1]
        for i in range(1, 7):
            y = x + col(sg * h) * sum(a * kk for a, kk in zip(_A[i], k))
            k.append(f(z + sg * h * _C[i], y))
        e = col(h) * sum(b * kk for b, kk in zip(_BT, k))
        E = _norm(e / (col(atol) + torch.maximum(torch.abs(x), torch.abs(y)) * rtol))
        q11 = E ** 0.14
        q = (q11 / qold ** 0.08 / 0.9).clamp(0.1, 5.0)
        ok = live & (E <= 1.0)
        accept(ok, z, sg * h, x, k)
        zn = z + sg * h
        end = torch.abs(zn) < 100 * eps * L if back else torch.abs(zn - L) < 100 * eps * L
        zn = torch.where(end, torch.full_like(zn, 0.0 if back else L), zn)
        x = torch.where(col(ok), y, x)
        k1 = torch.where(col(ok), k[6], k1)
        dt = torch.where(ok, h / q, torch.where(live, h / (q11 / 0.9).clamp(max=5.0), dt))
        qold = torch.where(ok, E.clamp(min=1e-4), qold)
        z = torch.where(ok, zn, z)
        live = live & ~(ok & end)
    return x


def _solve(p, u0, saves=None, seed=None, stop=None):
    """Forward solve of launches u0 (B, M, Nt); with seed(uL) also the adjoint
    from its terminal field.  Returns (saved lab spectra, J, λ(0))."""
    B, M, N = u0.shape
    L, dev = p["L"], p["dev"]
    # each sample's accepted steps (start, length) and interpolant coefficients
    store = dict(z=torch.full((B, 32), math.inf, dtype=torch.float64, device=dev),
                 h=torch.ones((B, 32), dtype=torch.float64, device=dev),
                 a=torch.zeros((B, 32 if seed else 0, 5, M, N), dtype=u0.dtype, device=dev))
    count = torch.zeros(B, dtype=torch.long, device=dev)
    saved = {}

    def accept(ok, z, h, x, k):
        if saves is not None:
            for i, zs in enumerate(saves):
                m = ok & (z < zs) & (z + h >= zs) & (zs > 0)
                if bool(m.any()):
                    th = (zs - z) / h
                    b = sum(kk * sum(_R[j][q] * th ** (q + 1) for q in range(4))[:, None, None]
                            for j, kk in enumerate(k))
                    saved[i] = torch.where(m[:, None, None], x + h[:, None, None] * b,
                                           saved.get(i, torch.zeros_like(x)))
        if seed is not None:
            if int(count.max()) + 1 >= store["z"].shape[1]:
                store["z"] = torch.cat([store["z"], torch.full_like(store["z"], math.inf)], 1)
                store["h"] = torch.cat([store["h"], torch.ones_like(store["h"])], 1)
                store["a"] = torch.cat([store["a"], torch.zeros_like(store["a"])], 1)
            b = torch.nonzero(ok).flatten()
            store["z"][b, count[b]], store["h"][b, count[b]] = z[b], h[b]
            store["a"][b, count[b], 0] = x[b]
            for q in range(4):
                store["a"][b, count[b], q + 1] = sum(_R[j][q] * kk[b] for j, kk in enumerate(k))
            count.add_(ok)

    atol = torch.full((B,), 1e-6, dtype=torch.float64, device=dev)
    x = _integrate(p, lambda z, y: _rhs(p, z, y), u0, L, False, atol, accept)
    lab = lambda v, z: v * torch.polar(torch.ones_like(p["D"]), p["D"] * z)  # noqa: E731
    uL = lab(x, L)
    spectra = None
    if saves is not None:
        spectra = torch.stack([u0 if zs == 0 else uL if zs == L else lab(saved[i], zs)
                               for i, zs in enumerate(saves)], 1)
    if seed is None:
        return spectra, None, None
    J, lam = seed(uL)
    lam = lam * torch.polar(torch.ones_like(p["D"]), -p["D"] * L)

    def field(z):
        n = ((store["z"] <= z[:, None]).sum(1) - 1).clamp(min=0)
        every = torch.arange(B, device=dev)
        a, h = store["a"][every, n], store["h"][every, n]
        th = (z - store["z"][every, n]) / h
        return a[:, 0] + h[:, None, None] * sum((th ** q)[:, None, None] * a[:, q]
                                                for q in range(1, 5))

    scale = torch.abs(lam).amax(dim=(1, 2))
    lam0 = _integrate(p, lambda z, y: _rhs_adj(p, z, y, field(z)), lam, L, True,
                      1e-6 * torch.where(scale == 0, torch.ones_like(scale), scale),
                      lambda *a: None)
    return spectra, J, lam0


def _band_seed(mask, log_cost):
    def seed(uL):
        e = torch.abs(uL) ** 2
        tot = e.sum(dim=(1, 2))
        J = (e * mask).sum(dim=(1, 2)) / tot
        s = uL * ((mask - J[:, None, None]) / tot[:, None, None])
        if log_cost:
            s = s * (10 / (math.log(10) * J))[:, None, None]
            J = 10 * torch.log10(J)
        return J, s
    return seed


def _gradient(p, c, ph):
    """J and dJ/dphase of phases (B, Nt) or (B, M, Nt), a few samples at a time."""
    u0, mask = p["tt"](p["u0"]), p["tt"](p["mask"]).double()
    per = ph.ndim == 3
    Js, gs, n = [], [], max(1, 2 ** 21 // (p["M"] ** 2 * p["nt"]))
    for b in range(0, len(ph), n):
        q = p["tt"](ph[b:b + n])
        u = u0[None] * torch.polar(torch.ones_like(q), q).reshape(len(q), -1, p["nt"])
        _, J, lam = _solve(p, u, seed=_band_seed(mask, c["log_cost"]))
        g = 2 * (lam.conj() * 1j * u).real
        Js.append(J.cpu())
        gs.append((g if per else g.sum(1)).cpu())
    return torch.cat(Js).numpy(), torch.cat(gs).numpy()


def exact(case, seed):
    c = case
    if c["kind"] == "serve" or _modes(c) ** 2 * c["nt"] * c["batch"] > 2 ** 23:
        return None
    p = _setup(c, seed, c["nt"], c["power"], c["length"])
    u0 = p["tt"](p["u0"])[None]
    if c["kind"] in ("forward", "propagate"):
        z = np.linspace(0.0, c["length"], c["nsave"])
        z[-1] = c["length"]
        out = _solve(p, u0, saves=z.tolist())[0][0].cpu().numpy()
        return [out] if c["kind"] == "forward" else [out, None]
    if c["kind"] == "adjoint":
        w = p["tt"](np.linspace(0.2, 1.8, c["nt"]))
        s, _, lam = _solve(p, u0, saves=[0.0, c["length"]], seed=lambda u: (None, u * w))
        return [s[0].cpu().numpy(), lam[0].cpu().numpy()]
    J, g = _gradient(p, c, _phases(c, seed))
    return [J, g]
