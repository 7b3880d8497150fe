"""The steppers over their transform plans: every grid size against the
FP64 oracle, and the same bits whatever number of CTAs a solve runs on."""
import numpy as np
import pytest

from fiberlab_gpu import problem as P
from fiberlab_gpu._capi import Context, GPUProblem
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def _problem(nt, L=0.2):
    return P.single_mode_problem(nt=nt, time_window_ps=max(3.0, nt * 3e-3), L=L, power_w=0.08,
                                 rep_rate_hz=80e6, raman_threshold_thz=-3.0, validate_grid=False)


# 2^6: radix 2; 2^7, 2^8, 2^9, 2^10: radix 4 with and without a first radix-2
# pass; 2^11: radix 8 after radix 4; 2^12, 2^13: radix 16 with 16- and
# 32-point regions; 2^14: radix 16 and 32
@pytest.mark.parametrize("logn", [6, 7, 8, 9, 10, 11, 12, 13, 14])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_rhs_every_grid(gpu_ctx, logn, precision):
    fp = _problem(1 << logn)
    rng = np.random.default_rng(logn)
    u = fp.uw0 * np.exp(0.3j * rng.standard_normal(fp.nt))[None, :]
    lam = (rng.standard_normal(fp.nt) + 1j * rng.standard_normal(fp.nt))[None, :] * 1e-3
    gp = GPUProblem(gpu_ctx, fp, precision)
    z = 0.1307
    # forward in the mode's precision (2e-6, the bound of the suite's other
    # right-hand-side checks); adjoint FP64, up to the rounding of the phase D z
    floor = 2 * np.finfo(float).eps * float(np.max(np.abs(fp.D))) * z
    assert rel(gp.rhs(z, u), O.rhs_forward(fp, z, u)) < (2e-6 if precision == "fp32" else
                                                         max(1e-10, floor))
    assert rel(gp.rhs(z, lam, u), O.rhs_adjoint(fp, z, lam, u)) < max(1e-10, floor)


# 1 slot: 4 or 8 CTAs each; 20: 4 (2^14: 4); 40: 2; 80: one CTA each
@pytest.mark.parametrize("nt", [4096, 8192, 16384])
def test_same_bits_on_any_number_of_ctas(gpu_ctx, nt):
    fp = _problem(nt, L=0.03)
    phis = 0.3 * np.random.default_rng(nt).standard_normal((80, nt))
    gp = GPUProblem(gpu_ctx, fp)
    J, g, st = gp.phase_gradient_batch(phis)
    assert all(s["status"] == 0 for s in st)
    for n in (1, 20, 40):
        Jn, gn, _ = gp.phase_gradient_batch(phis[80 - n:])
        assert np.array_equal(Jn, J[80 - n:]) and np.array_equal(gn, g[80 - n:])
    Jo, go, _ = O.phase_gradient(fp, phis[79])
    assert abs(J[79] - Jo) < 1e-5 * Jo and rel(g[79], go) < 1e-3


# every transform of the multimode kernels (2^15: clusters of four CTAs), with
# and without the tensor-core contractions (M >= 6 in FP32), beside the FP32
# and FP64 tasks of one launch
@pytest.mark.parametrize("logn", [6, 7, 8, 9, 10, 11, 12, 13, 14, 15])
@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_multimode_rhs_every_grid(gpu_ctx, logn, order, precision):
    nt = 1 << logn
    fp = P.multimode_problem(order, 32, nt, max(3.0, nt * 1.5e-3), 0.2, 2e-9, 200e-15, 1,
                             raman_threshold_thz=-3.0)
    rng = np.random.default_rng(logn)
    u = fp.uw0 * np.exp(0.3j * rng.standard_normal((fp.M, nt)))
    lam = (rng.standard_normal((fp.M, nt)) + 1j * rng.standard_normal((fp.M, nt))) * 1e-3
    gp = GPUProblem(gpu_ctx, fp, precision)
    z = 0.1307
    # the bounds of the suite's other right-hand-side checks, FP64 up to the
    # rounding of the phase D z; the adjoint of FP32 solves with M >= 6 and
    # whole 128-point tiles is mixed
    floor = max(1e-10, 2 * np.finfo(float).eps * float(np.max(np.abs(fp.D))) * z)
    mixed = precision == "fp32" and fp.M >= 6 and nt % 128 == 0
    assert rel(gp.rhs(z, u), O.rhs_forward(fp, z, u)) < (2e-6 if precision == "fp32" else floor)
    assert rel(gp.rhs(z, lam, u), O.rhs_adjoint(fp, z, lam, u)) < (2e-6 if mixed else floor)


# device blocks pass from one object of a context to the next, and objects may
# outlive their context
@pytest.mark.parametrize("nts", [(1024, 1024), (4096, 512), (512, 8192)])
def test_blocks_reused_between_problems(nts):
    ctx = Context(0)
    fps = [_problem(n, L=0.02) for n in nts]
    first = [GPUProblem(ctx, fp).forward()[0] for fp in fps]
    for fp, want in list(zip(fps, first))[::-1] * 2:
        gp = GPUProblem(ctx, fp)
        assert np.array_equal(gp.forward()[0], want)
    ctx.close()
    del gp
