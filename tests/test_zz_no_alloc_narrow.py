"""cps_solve_noalloc's scratch is shared by calls of different shapes, and a
diverged call leaves NaN in it.  A narrow design of many tiles per CTA (the
PCG that streams its vectors) reads the conductances west of its first column
and south of its first row, which no phase writes: a call after a diverged one
of another shape gives what cps_solve gives, with the parity tests' per-step
tolerance."""
import numpy as np
import pytest

from coldplate_solver_b200 import cps, geometry
from test_zz_no_alloc import OUT_FIELDS, REL_STEP, CallerBuffers, call_noalloc, rel

pytestmark = pytest.mark.gpu


def random_state(d, seed):
    rng = np.random.default_rng(seed)
    return {"u": rng.normal(0, 0.05, (d.M + 1, d.N)), "v": rng.normal(0, 0.02, (d.M, d.N + 1)),
            "p": rng.normal(0, 5.0, (d.M + 1, d.N + 1))}


def test_narrow_design_after_a_diverged_one():
    lib = cps.load_library()
    wide = geometry.straight_channel(M=1023, N=127, band=(200, 800))
    bad = random_state(wide, 1)
    bad["u"][...] = np.nan
    with pytest.raises(AssertionError, match=str(cps.CPS_ERR_DIVERGED)):  # the call's status
        call_noalloc(lib, wide, CallerBuffers(wide, 128, bad), 1)
    d = geometry.straight_channel(M=32767, N=3, band=(8000, 24000))  # 4096 tiles; the same (M + 1) * pitch
    init = random_state(d, 2)
    buf = CallerBuffers(d, 4, init)
    h = call_noalloc(lib, d, buf, 3)
    f = buf.fields()
    with cps.Solver(d) as ref:
        ref.upload_fields(**init)
        h_ref = ref.solve(3, eps=0.0)
        f_ref = ref.download()
    assert h_ref[:, 5].max() > 1  # the PCG goes beyond its first iteration
    assert np.array_equal(h[:, 5:], h_ref[:, 5:]), (h[:, 5:], h_ref[:, 5:])
    for k in OUT_FIELDS:
        assert rel(f[k], f_ref[k]) <= REL_STEP, (k, rel(f[k], f_ref[k]))
