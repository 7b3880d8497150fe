"""Objects of one context after one another: tables, workspaces and staging
areas in blocks that earlier objects of other shapes have used."""
import numpy as np
import pytest

from fiberlab_gpu import problem as P
from fiberlab_gpu._capi import Context, GPUProblem

pytestmark = pytest.mark.gpu


def _single(nt):
    return P.single_mode_problem(nt=nt, time_window_ps=max(3.0, nt * 3e-3), L=0.02, power_w=0.08,
                                 rep_rate_hz=80e6, raman_threshold_thz=-3.0, validate_grid=False)


def _multi(order, nt):
    return P.multimode_problem(order, 32, nt, max(3.0, nt * 1.5e-3), 0.02, 2e-9, 200e-15, 1,
                               raman_threshold_thz=-3.0)


# single mode, 3 modes, 6 and 10 modes (images of the tensor-core operands)
@pytest.mark.parametrize("budget", [0, 64 << 20])
def test_gradients_in_used_blocks(budget):
    fps = [_single(1024), _multi(1, 512), _multi(2, 256), _single(4096), _multi(3, 128)]
    phis = [0.3 * np.random.default_rng(i).standard_normal((2, fp.nt)) for i, fp in enumerate(fps)]
    opts = dict(checkpoints=2, segment_steps=8)
    want = [GPUProblem(Context(0, **opts), fp).phase_gradient_batch(ph)[:2]
            for fp, ph in zip(fps, phis)]
    ctx = Context(0, hbm_budget_bytes=budget, **opts)
    for i in [0, 1, 2, 3, 4, 3, 1, 0, 2, 4, 0]:
        gp = GPUProblem(ctx, fps[i])
        J, g, st = gp.phase_gradient_batch(phis[i])
        assert all(s["status"] == 0 for s in st)
        assert np.array_equal(J, want[i][0]) and np.array_equal(g, want[i][1])
        gp.close()


def test_a_budget_bounds_what_a_context_keeps():
    torch = pytest.importorskip("torch")
    budget = 48 << 20
    fp = _single(8192)
    GPUProblem(Context(0), fp).forward()  # the kernels' own device memory
    ctx = Context(0, checkpoints=8, segment_steps=16, hbm_budget_bytes=budget)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info(0)[0]
    gps = [GPUProblem(ctx, fp) for _ in range(8)]
    for gp in gps:
        gp.forward()
    assert before - torch.cuda.mem_get_info(0)[0] > 2 * budget
    for gp in gps:
        gp.close()
    # cudaMalloc maps whole 2 MiB pages
    assert before - torch.cuda.mem_get_info(0)[0] <= budget + (4 << 20)
