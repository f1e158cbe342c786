"""The PCG's forms (one cluster of CTAs, a CTA's tiles on chip, p of them on
chip, global memory), which the number of tiles and of tiles per CTA selects,
against the oracle: one outer
iteration from a random state, at the edges of each form's range and of the
ways an iteration can end (the cap, the tolerance after one or several
iterations, no iteration at all).

Tolerances as for one step from an identical state: FP64 fields 1e-10 relative
L2 with equal inner counts (only the grouping of the grid-wide sums differs);
mixed precision 1e-3 (its inner solves stop at their tolerances on FP32-stored
values)."""
import numpy as np
import pytest

from coldplate_solver_b200 import cps, geometry
from oracle import restatement as rs

pytestmark = pytest.mark.gpu

TILES = 8 * 8  # of the 61 x 233 design, ragged in both directions


def run_both(precision, grid_ctas, M=61, N=233, **settings):
    d = geometry.channel_network(M=M, N=N, h=20e-6, wmin=4, wmax=8, seed=6).replace(**settings)
    rng = np.random.default_rng(3)
    init = {"u": rng.normal(0, 0.05, (d.M + 1, d.N)), "v": rng.normal(0, 0.02, (d.M, d.N + 1)),
            "p": rng.normal(0, 5.0, (d.M + 1, d.N + 1))}
    with cps.Solver(d, precision=precision, grid_ctas=grid_ctas) as s:
        s.upload_fields(**init)
        h = s.solve(1, eps=0.0)
        f = s.download()
    fr = rs.new_fields(d)
    for k in init:
        fr[k][...] = init[k]
    hr = rs.solve(d, fr, 1, stop_on_conv=False)
    err = {k: np.linalg.norm(f[k] - fr[k]) / max(np.linalg.norm(fr[k]), 1e-300) for k in ("u", "v", "p")}
    return h, hr, err


# tiles per CTA: 1 and 2 in registers, 3 and 7 on chip, 8 and 30 with p on chip, 32 and 64 from global memory
@pytest.mark.parametrize("per_cta", [1, 2, 3, 7, 8, 30, 32, 64])
@pytest.mark.parametrize("settings", [dict(maxPressureIter=30), dict(maxPressureIter=200, pTol=2e-2),
                                      dict(maxPressureIter=1), dict(maxPressureIter=2), dict(maxPressureIter=0),
                                      dict(maxPressureIter=20, pTol=1e3)])
def test_pcg_forms_match_the_oracle(per_cta, settings):
    h, hr, err = run_both(cps.CPS_FP64, -(-TILES // per_cta), **settings)
    assert np.array_equal(h[:, 5:], hr[:, 5:]), (h[:, 5:], hr[:, 5:])
    assert max(err.values()) <= 1e-10, err


@pytest.mark.parametrize("per_cta", [1, 2, 3, 12, 13, 32, 64])
def test_mixed_pcg_forms_are_close_to_the_oracle(per_cta):
    _, _, err = run_both(cps.CPS_MIXED, -(-TILES // per_cta), maxPressureIter=30)
    assert err["u"] <= 1e-3 and err["v"] <= 1e-3, err


# one tile per CTA, on one cluster: 16 tiles (one per CTA of it) in three shapes, a tile column and row more,
# and as many as fit; 15 tiles are below its range
@pytest.mark.parametrize("M,N", [(33, 129), (9, 513), (129, 33), (34, 130), (41, 97), (113, 225), (100, 200)])
@pytest.mark.parametrize("settings", [dict(maxPressureIter=30), dict(maxPressureIter=200, pTol=2e-2),
                                      dict(maxPressureIter=3)])
def test_cluster_pcg_matches_the_oracle(M, N, settings):
    h, hr, err = run_both(cps.CPS_FP64, 0, M, N, **settings)
    assert np.array_equal(h[:, 5:], hr[:, 5:]), (h[:, 5:], hr[:, 5:])
    assert max(err.values()) <= 1e-10, err


@pytest.mark.parametrize("precision", [cps.CPS_FP64, cps.CPS_MIXED])
@pytest.mark.parametrize("M,N", [(33, 129), (61, 233), (100, 200)])
def test_cluster_pcg_has_the_bits_of_the_grid_form(precision, M, N):
    """The batch's waves solve a design on as many CTAs as tiles without a cluster."""
    d = geometry.channel_network(M=M, N=N, h=20e-6, wmin=4, wmax=8, seed=6).replace(maxPressureIter=60)
    out = []
    for wave in (False, True):
        with cps.Solver(d, precision=precision) as s:
            if wave:
                cps.batch_solve([s], 12, eps=0.0, tiles_per_cta=1)
                h = cps.get_history(s, 12)
            else:
                h = s.solve(12, eps=0.0)
            out.append((h, s.download()))
    assert np.array_equal(out[0][0], out[1][0])
    assert all(np.array_equal(out[0][1][k], out[1][1][k]) for k in out[0][1])
