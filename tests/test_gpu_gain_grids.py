"""Pump-gain propagation over its grids against the FP64 oracle."""
import numpy as np
import pytest

from fiberlab_gpu import gain as G
from fiberlab_gpu import problem as P
from fiberlab_gpu._capi import GPUProblem
from oracle import oracle as O
from test_gain_oracle import _synthetic_sections

pytestmark = pytest.mark.gpu


# one warp (2^6, 2^7), whole chunks of eight points (2^11) and two of them per
# thread (2^12, 2^13); a rejected step and a save position inside a step among
# them.  The bounds of the suite's other pump-gain checks.
@pytest.mark.parametrize("logn", [6, 7, 9, 11, 12, 13])
@pytest.mark.parametrize("model", ["constant", "ydfa"])
def test_gain_every_grid(gpu_ctx, logn, model):
    nt = 1 << logn
    fp = P.single_mode_problem(nt=nt, time_window_ps=max(3.0, nt * 3e-3), L=0.1, power_w=0.08,
                               rep_rate_hz=80e6, wavelength_m=1030e-9, validate_grid=False)
    gain = 0.8 if model == "constant" else G.ydfa_params(fp.sim, *_synthetic_sections())
    zs = [0.0, 0.013, 0.05, fp.L]
    out, pumps, st = GPUProblem(gpu_ctx, fp).forward_gain(gain, 0.05, saveat=zs)
    ref, pumps_ref, _ = O.forward_gain(fp, gain, 0.05, zsave=zs)
    assert st["status"] == 0 and st["nf"] == 3 + 6 * (st["naccept"] + st["nreject"])
    for i in range(len(zs)):
        assert np.linalg.norm(out[i] - ref[i]) < 1e-5 * np.linalg.norm(ref[i])
        assert pumps[i] == pytest.approx(pumps_ref[i], rel=1e-6)
