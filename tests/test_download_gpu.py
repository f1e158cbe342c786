"""cps_download_fields returns what cps_upload_fields stored, element for
element: from the smallest grid (one thread, one row per slot of the stage) to
grids whose fields several threads write, in both layouts."""
import ctypes

import numpy as np
import pytest

from coldplate_solver_b200 import cps, geometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N", [(3, 3), (3, 700), (15, 9), (61, 233), (251, 499), (331, 642)])
@pytest.mark.parametrize("layout", [cps.CPS_ROW_MAJOR, cps.CPS_COL_MAJOR])
def test_download_returns_the_uploaded_fields(M, N, layout):
    rng = np.random.default_rng(M)
    g = np.ones((M, N))
    d = geometry.Design(M=M, N=N, hx=1e-5, hy=1e-5, inletVelocity=0.1, gamma=g, alpha=0 * g)
    want = {"u": rng.normal(size=(M + 1, N)), "v": rng.normal(size=(M, N + 1)), "p": rng.normal(size=(M + 1, N + 1))}
    order = "C" if layout == cps.CPS_ROW_MAJOR else "F"
    ptr = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))  # noqa: E731
    with cps.Solver(d) as s:
        up = [np.asarray(want[k], order=order) for k in ("u", "v", "p")]
        assert s.lib.cps_upload_fields(s.ctx, *[ptr(a) for a in up], layout) == cps.CPS_OK
        out = {k: np.full(sh, np.nan, order=order) for k, sh in cps.field_shapes(M, N).items()}
        names = ("u", "v", "p", "pStar", "uStar", "vStar", "dE", "dN")
        assert s.lib.cps_download_fields(s.ctx, *[ptr(out[k]) for k in names], layout) == cps.CPS_OK
        some = np.full((M, N + 1), np.nan, order=order)
        assert s.lib.cps_download_fields(s.ctx, None, ptr(some), None, None, None, None, None, None, layout) == cps.CPS_OK
    for k in want:
        assert np.array_equal(out[k], want[k]), k
    assert np.array_equal(some, want["v"])
    assert all(np.array_equal(out[k], np.zeros_like(out[k])) for k in names[3:])  # not computed yet
