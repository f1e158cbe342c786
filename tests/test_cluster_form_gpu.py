"""Which designs take the cluster form of the PCG (one tile per CTA, 16 tiles
to as many as the device holds at one CTA per SM in whole clusters of 16: 112
on B200), and that it is what ran where it is compared: with the oracle and
with the grid form, which the batch's waves run.

Tolerances as in test_pcg_forms_gpu.py."""
import numpy as np
import pytest

from coldplate_solver_b200 import cps, geometry
from oracle import restatement as rs

pytestmark = pytest.mark.gpu


def design(M, N, **settings):
    return geometry.channel_network(M=M, N=N, h=20e-6, wmin=2, wmax=4, seed=6).replace(**settings)


def state(d):
    rng = np.random.default_rng(3)
    return {"u": rng.normal(0, 0.05, (d.M + 1, d.N)), "v": rng.normal(0, 0.02, (d.M, d.N + 1)),
            "p": rng.normal(0, 5.0, (d.M + 1, d.N + 1))}


def run(d, n, precision=cps.CPS_FP64, grid_ctas=0):
    with cps.Solver(d, precision=precision, grid_ctas=grid_ctas) as s:
        s.upload_fields(**state(d))
        return s.solve(n, eps=0.0), s.download(), s.last_pcg_form


# 15 tiles, 16, 98, 112 in three shapes, 113 and 119
@pytest.mark.parametrize("precision", [cps.CPS_FP64, cps.CPS_MIXED])
@pytest.mark.parametrize("M,N,cluster", [(25, 160, False), (33, 129, True), (113, 225, True), (113, 257, True),
                                         (129, 225, True), (9, 3585, True), (9, 3617, False), (137, 225, False)])
def test_which_designs_take_the_cluster_form(M, N, cluster, precision):
    d = geometry.straight_channel(M=M, N=N, band=(M // 4, 3 * M // 4))
    with cps.Solver(d, precision=precision) as s:
        s.solve(1, eps=0.0)
        assert s.last_pcg_form == (cps.CPS_PCG_FORM_CLUSTER if cluster else cps.CPS_PCG_FORM_FEW)


@pytest.mark.parametrize("cap,cluster", [(2, False), (3, True), (100000, True), (100001, False)])
def test_caps_that_take_the_cluster_form(cap, cluster):
    d = geometry.straight_channel().replace(maxPressureIter=cap, pTol=1e3)
    with cps.Solver(d) as s:
        s.solve(1, eps=0.0)
        assert s.last_pcg_form == (cps.CPS_PCG_FORM_CLUSTER if cluster else cps.CPS_PCG_FORM_FEW)


@pytest.mark.parametrize("M,N", [(33, 129), (100, 200), (113, 257), (129, 225)])
def test_the_largest_clusters_match_the_oracle(M, N):
    d = design(M, N, maxPressureIter=30)
    h, f, form = run(d, 1)
    assert form == cps.CPS_PCG_FORM_CLUSTER
    fr = rs.new_fields(d)
    for k, a in state(d).items():
        fr[k][...] = a
    hr = rs.solve(d, fr, 1, stop_on_conv=False)
    assert np.array_equal(h[:, 5:], hr[:, 5:])
    for k in ("u", "v", "p"):
        assert np.linalg.norm(f[k] - fr[k]) <= 1e-10 * np.linalg.norm(fr[k]), k


@pytest.mark.parametrize("M,N", [(33, 129), (61, 233), (129, 225)])
def test_mixed_cluster_is_close_to_the_oracle(M, N):
    d = design(M, N, maxPressureIter=30)
    _, f, form = run(d, 1, cps.CPS_MIXED)
    assert form == cps.CPS_PCG_FORM_CLUSTER
    fr = rs.new_fields(d)
    for k, a in state(d).items():
        fr[k][...] = a
    rs.solve(d, fr, 1, stop_on_conv=False)
    for k in ("u", "v"):
        assert np.linalg.norm(f[k] - fr[k]) <= 1e-3 * np.linalg.norm(fr[k]), k


@pytest.mark.parametrize("precision", [cps.CPS_FP64, cps.CPS_MIXED])
@pytest.mark.parametrize("M,N", [(33, 129), (100, 200), (113, 257), (129, 225)])
def test_cluster_bits_against_waves(M, N, precision):
    """The batch's waves solve a design on as many CTAs as tiles without a cluster."""
    d = design(M, N, maxPressureIter=60)
    h, f, form = run(d, 8, precision)
    assert form == cps.CPS_PCG_FORM_CLUSTER
    with cps.Solver(d, precision=precision) as s:
        s.upload_fields(**state(d))
        cps.batch_solve([s], 8, eps=0.0, tiles_per_cta=1)
        hw, fw = cps.get_history(s, 8), s.download()
        assert s.last_pcg_form == cps.CPS_PCG_FORM_NONE
    assert np.array_equal(h, hw)
    assert all(np.array_equal(f[k], fw[k]) for k in f)
