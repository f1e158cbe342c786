"""The largest pressure-drop window a monitor takes, per tile shape and
precision: it runs, and one value more is refused."""
import numpy as np
import pytest

from coldplate_solver_b200 import cps, geometry

pytestmark = pytest.mark.gpu

LARGEST = {(16, cps.CPS_FP64): 12384, (16, cps.CPS_MIXED): 13248, (32, cps.CPS_FP64): 12664,
           (32, cps.CPS_MIXED): 13488, (64, cps.CPS_FP64): 13644, (64, cps.CPS_MIXED): 14328}


@pytest.mark.parametrize("tile_j,precision", sorted(LARGEST))
def test_largest_window(tile_j, precision):
    d = geometry.straight_channel(M=20, N=40, band=(5, 15))
    most = LARGEST[tile_j, precision]
    with cps.Solver(d, precision=precision, tile_j=tile_j) as s:
        kw = dict(percent=0.1, slope_gate=True, slope_max_delta=1.0, ramp_steps=0, x_core_in=0.0,
                  x_core_out=d.N * d.hx)
        s.set_dp_monitor(gate=True, window=most - 40, slope_window=40, **kw)
        h, dp, conv = s.solve_monitored(most + 2, eps=0.0)  # past the first full window
        assert np.isfinite(h).all() and np.isfinite(dp).all()
        with pytest.raises(cps.CpsError) as e:
            s.set_dp_monitor(gate=True, window=most - 40, slope_window=41, **kw)
        assert e.value.status == cps.CPS_ERR_ARG and str(most) in str(e.value)
