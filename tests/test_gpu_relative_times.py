"""Times of the stepper against one another on one device, for the grids,
modes and batch sizes that no timed case covers: kernel time per right-hand
side evaluation, the least of some calls."""
import numpy as np
import pytest

from fiberlab_gpu import problem as P
from fiberlab_gpu._capi import Context, GPUProblem

pytestmark = pytest.mark.gpu


def _evaluation_us(nt, precision="fp32", batch=1, L=0.1):
    fp = P.single_mode_problem(nt=nt, time_window_ps=max(3.0, nt * 3e-3), L=L, power_w=0.08,
                               rep_rate_hz=80e6, raman_threshold_thz=-3.0, validate_grid=False)
    ctx = Context(0, checkpoints=8, segment_steps=32)
    gp = GPUProblem(ctx, fp, precision)
    phis = 0.3 * np.random.default_rng(nt).standard_normal((batch, nt))
    best = np.inf
    for _ in range(6):
        _, _, st = gp.phase_gradient_batch(phis)
        evals = np.mean([s["nf"] + s["adj_nf"] for s in st])
        best = min(best, ctx.timing()[1] * 1e3 / evals)
    return best


# 64 points (two per lane of one warp) against 128 (four per lane)
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("batch", [1, 148])
def test_smallest_grid_against_the_next(gpu_ctx, precision, batch):
    assert _evaluation_us(64, precision, batch) < 1.15 * _evaluation_us(128, precision, batch)


# FP64 stage vectors (more registers) against FP32 ones under the cap of 128
@pytest.mark.parametrize("nt,batch", [(256, 592), (2048, 1), (2048, 148)])
def test_double_precision_against_single(gpu_ctx, nt, batch):
    assert _evaluation_us(nt, "fp64", batch) < 1.1 * _evaluation_us(nt, "fp32", batch)
