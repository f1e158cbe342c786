"""A step whose residual is not finite ends the same way in every form of the
PCG: CPS_ERR_DIVERGED, every CTA having finished the step, and a context that
goes on working.  The NaN comes from the host, in an uploaded velocity; the
PCG then runs to its cap, which keeps the CTAs outside the cluster waiting for
several hundred microseconds with the diverged status already set.

With a NaN step length p' is NaN everywhere, so that no field depends on how
the sums were grouped: the cluster form (one tile per CTA) and a grid of one
CTA less, which cannot run as a cluster, leave the same fields."""
import numpy as np
import pytest

from coldplate_solver_b200 import cps, geometry

pytestmark = pytest.mark.gpu


def design(M, N):
    return geometry.channel_network(M=M, N=N, h=20e-6, wmin=4, wmax=8, seed=6).replace(maxPressureIter=200)


def state(d):
    rng = np.random.default_rng(5)
    return {"u": rng.normal(0, 0.05, (d.M + 1, d.N)), "v": rng.normal(0, 0.02, (d.M, d.N + 1)),
            "p": rng.normal(0, 5.0, (d.M + 1, d.N + 1))}


def diverge(s, d):
    bad = state(d)
    bad["u"][d.M // 2, d.N // 3] = np.nan
    s.upload_fields(**bad)
    with pytest.raises(cps.CpsError) as e:
        s.solve(4, eps=0.0)
    assert e.value.status == cps.CPS_ERR_DIVERGED
    return s.download()


# 16, 64 and 91 tiles, and 112, the most that fit
@pytest.mark.parametrize("precision", [cps.CPS_FP64, cps.CPS_MIXED])
@pytest.mark.parametrize("M,N,tiles", [(33, 129, 16), (61, 233, 64), (100, 200, 91), (129, 225, 112)])
def test_diverged_step_is_finished_by_every_cta(M, N, tiles, precision):
    d = design(M, N)
    fields = []
    for ctas in (0, tiles - 1):
        with cps.Solver(d, precision=precision, grid_ctas=ctas) as s:
            fields.append(diverge(s, d))
    for k in fields[0]:
        assert np.array_equal(fields[0][k], fields[1][k], equal_nan=True), k


def test_context_works_after_a_diverged_step():
    d = design(100, 200)
    with cps.Solver(d) as fresh:
        fresh.upload_fields(**state(d))
        h0, f0 = fresh.solve(3, eps=0.0), fresh.download()
    with cps.Solver(d) as s:
        diverge(s, d)
        s.reset_fields()
        s.upload_fields(**state(d))
        h, f = s.solve(3, eps=0.0), s.download()
    assert np.array_equal(h, h0)
    assert all(np.array_equal(f[k], f0[k]) for k in f0)


def test_batch_goes_on_after_a_diverged_design():
    """One group of CTAs takes the designs one after the other; the first one
    diverges and the others get what they get alone."""
    d = design(61, 233)
    with cps.Solver(d) as a, cps.Solver(d) as b, cps.Solver(d) as alone:
        bad = state(d)
        bad["u"][d.M // 2, d.N // 3] = np.nan
        a.upload_fields(**bad)
        for s in (b, alone):
            s.upload_fields(**state(d))
        cps.batch_solve([alone], 5, eps=0.0, group_ctas=148)
        res, _ = cps.batch_solve([a, b], 5, eps=0.0, group_ctas=148, max_clusters=1)
        assert res[0]["status"] == cps.CPS_ERR_DIVERGED and res[0]["n_done"] == 1
        assert res[1]["status"] == cps.CPS_OK and res[1]["n_done"] == 5
        f, f0 = b.download(), alone.download()
    assert all(np.array_equal(f[k], f0[k]) for k in f0)
