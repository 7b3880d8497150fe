"""Double precision over any number of CTAs per solve, directly and served."""
import numpy as np
import pytest

from fiberlab_gpu import problem as P
from fiberlab_gpu._capi import GPUProblem
from fiberlab_gpu.serving import Server

pytestmark = pytest.mark.gpu


def _problem(nt, L=0.03):
    return P.single_mode_problem(nt=nt, time_window_ps=max(3.0, nt * 3e-3), L=L, power_w=0.08,
                                 rep_rate_hz=80e6, raman_threshold_thz=-3.0, validate_grid=False)


# 1 solve: four CTAs (2^12) or eight (2^13); 20: four; 40: two; 80: one each.
# The stage vectors are FP64 here, in kernels of their own.
@pytest.mark.parametrize("nt", [4096, 8192])
def test_same_bits_in_double_precision(gpu_ctx, nt):
    phis = 0.3 * np.random.default_rng(nt).standard_normal((80, nt))
    gp = GPUProblem(gpu_ctx, _problem(nt), "fp64")
    J, g, st = gp.phase_gradient_batch(phis)
    assert all(s["status"] == 0 for s in st)
    for n in (1, 20, 40):
        Jn, gn, _ = gp.phase_gradient_batch(phis[80 - n:])
        assert np.array_equal(Jn, J[80 - n:]) and np.array_equal(gn, g[80 - n:])


# a request's bits do not depend on what is served beside it
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_served_as_solved(gpu_ctx, precision):
    nts = [2048, 4096, 8192]
    gps = {nt: GPUProblem(gpu_ctx, _problem(nt), precision) for nt in nts}
    phis = {nt: 0.3 * np.random.default_rng(nt).standard_normal(nt) for nt in nts}
    want = {nt: gps[nt].phase_gradient_batch(phis[nt])[:2] for nt in nts}
    server = Server(gpu_ctx, checkpoints=32, segment_steps=64)
    for count in (1, 12, 40):
        live = [server.submit_band_gradient(gps[nts[i % 3]], phis[nts[i % 3]])
                for i in range(count)]
        for i, r in enumerate(live):
            done = server.wait(r)
            J, g = want[nts[i % 3]]
            assert done.J == J[0] and np.array_equal(done.out_grad, g[0])
    server.close()
