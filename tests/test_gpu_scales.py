"""The error norm over the scales of its fields, and the stepper's own square
root, reciprocal and phasor over their arguments."""
import ctypes as C
import os

import numpy as np
import pytest

from fiberlab_gpu import _capi
from fiberlab_gpu import problem as P
from fiberlab_gpu._capi import GPUProblem

pytestmark = pytest.mark.gpu


# A linear fiber leaves every derivative exactly zero, whatever the weights of
# the error norm: bins without light have the absolute tolerance for a weight.
@pytest.mark.parametrize("abstol", [1e-160, 1e-300, 1e200])
@pytest.mark.parametrize("nt", [64, 1024, 8192])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_error_weights_over_tolerances(gpu_ctx, nt, precision, abstol):
    fp = P.single_mode_problem(nt=nt, time_window_ps=max(3.0, nt * 3e-3), L=0.05, power_w=0.08,
                               gamma=0.0, rep_rate_hz=80e6, raman_threshold_thz=-3.0,
                               validate_grid=False)
    fp.abstol = abstol
    u0 = fp.uw0.copy()
    u0[0, nt // 4:3 * nt // 4] = 0.0
    u, st = GPUProblem(gpu_ctx, fp, precision).forward(u0)
    assert st["status"] == 0 and st["nreject"] == 0
    want = u0 * np.exp(1j * np.asarray(fp.D) * fp.L)
    floor = 2 * np.finfo(float).eps * float(np.max(np.abs(fp.D))) * fp.L
    assert np.linalg.norm(u[-1] - want) < max(1e-12, floor) * np.linalg.norm(want)


def _math(which, a, b=None):
    if not os.path.exists(_capi.CHECKED_LIB_PATH):
        pytest.fail("the checked library is not built (run __graft_entry__.build())")
    lib = C.CDLL(_capi.CHECKED_LIB_PATH)
    lib.fl_check_math.argtypes = [C.c_int, C.c_int] + [C.c_void_p] * 3
    a = np.ascontiguousarray(a, dtype=np.float64)
    b = np.ascontiguousarray(np.zeros_like(a) if b is None else b, dtype=np.float64)
    out = np.empty(len(a) * (1 if which < 2 else 2))
    assert lib.fl_check_math(which, len(a), a.ctypes.data, b.ctypes.data, out.ctypes.data) == 0
    return out if which < 2 else out.view(np.complex128)


def _arguments():
    r = np.random.default_rng(3)
    n = 20000
    return np.concatenate([r.uniform(1.0, 4.0, n), np.exp2(r.uniform(-1020.0, 1020.0, n)),
                           np.exp2(np.arange(-1022.0, 1021.0))])


def test_square_root_and_reciprocal(gpu_ctx):
    # against long double (64 bits of mantissa)
    a = _arguments()
    for which, m, ref in ((0, np.append(a, 1.7976931348623157e308), np.sqrt), (1, a, np.reciprocal)):
        want = ref(m.astype(np.longdouble))
        ulp = np.spacing(want.astype(np.float64)).astype(np.longdouble)
        assert np.max(np.abs(_math(which, m) - want) / ulp) < 1.0
    assert np.array_equal(_math(0, [0.0, 5e-324, 2.2e-308]), [0.0, 0.0, 0.0])
    assert np.array_equal(_math(1, [5e307, 1e308, 1.7976931348623157e308]), [0.0, 0.0, 0.0])
    assert not np.any(np.isfinite(_math(0, [np.inf, np.nan, -1.0])))
    assert not np.any(np.isfinite(_math(1, [0.0, 1e-310, np.inf, np.nan])))


# FP64: the angle 2 pi r, |r| <= 1/8, in two roundings (1.2e-16), the series'
# first term left out (5e-17), the last roundings of its sums (2.5e-16): under
# 2 eps.  FP32: one more rounding (of r); under 3e-7.
@pytest.mark.parametrize("which,bound", [(2, 2 * np.finfo(np.float64).eps), (3, 3e-7)])
def test_phasor(gpu_ctx, which, bound):
    r = np.random.default_rng(4)
    n = 20000
    edges = np.arange(-64, 65) / 16.0  # quarter turns, and the octants between them
    d = np.concatenate([r.uniform(-2.0, 2.0, n), r.uniform(-1e6, 1e6, n), edges,
                        np.nextafter(edges, 9.0), np.nextafter(edges, -9.0),
                        np.ldexp(r.uniform(-1.0, 1.0, 500), r.integers(-1000, 48, 500)), [0.0, -0.0]])
    z = np.concatenate([r.uniform(0.0, 1.0, n), r.uniform(0.0, 3.0, n),
                        np.ones(len(d) - 2 * n)])
    t = d * z                       # rounded as the device does
    f = (t - np.rint(t)).astype(np.longdouble)
    ang = 2 * np.longdouble("3.14159265358979323846264338327950288") * f
    got = _math(which, d, z)
    assert np.max(np.abs(got.real - np.cos(ang))) < bound
    assert np.max(np.abs(got.imag - np.sin(ang))) < bound
    assert np.array_equal(got[-2:], [1.0, 1.0])
