"""The monitored kernel and the one that carries the options come once per
form of the PCG, as the plain one does.  The monitor (its gate off) and the
TMA-staged sweeps leave the iteration's arithmetic as it is, so each gives the
plain kernel's bits, whatever the number of tiles per CTA."""
import numpy as np
import pytest

from coldplate_solver_b200 import cps, geometry

pytestmark = pytest.mark.gpu

TILES = 8 * 8  # of the 61 x 233 design, ragged in both directions


# up to 2 tiles per CTA, up to 7 (12 in mixed precision), p on chip, global memory
@pytest.mark.parametrize("per_cta", [1, 2, 7, 13, 64])
@pytest.mark.parametrize("precision", [cps.CPS_FP64, cps.CPS_MIXED])
def test_monitored_and_option_kernels_give_the_plain_bits(per_cta, precision, monkeypatch):
    d = geometry.channel_network(M=61, N=233, h=20e-6, wmin=4, wmax=8, seed=6).replace(maxPressureIter=40)
    out = {}
    for which in ("plain", "monitored", "options"):
        monkeypatch.setenv("CPS_STAGE_SWEEPS", "1" if which == "options" else "0")
        with cps.Solver(d, precision=precision, grid_ctas=-(-TILES // per_cta)) as s:
            if which == "monitored":
                s.set_dp_monitor(gate=False, window=1, percent=0.0, ramp_steps=0, x_core_in=0.0, x_core_out=d.N * d.hx)
                h = s.solve_monitored(6, eps=0.0)[0]
            else:
                h = s.solve(6, eps=0.0)
            out[which] = (h, s.download())
    h0, f0 = out["plain"]
    assert h0[:, 5].max() > 2
    for which in ("monitored", "options"):
        h, f = out[which]
        assert np.array_equal(h, h0), which
        assert all(np.array_equal(f[k], f0[k]) for k in f0), which
