"""Contexts of small designs on several host threads share the GPU: a solve
that finds another one in flight takes the form that leaves room beside it,
with the bits of the form it takes alone."""
import threading

import numpy as np
import pytest

from coldplate_solver_b200 import cps, geometry

pytestmark = pytest.mark.gpu


def bits(s, n):
    s.reset_fields()
    return s.solve(n, eps=0.0), s.download()


@pytest.mark.parametrize("precision", [cps.CPS_FP64, cps.CPS_MIXED])
def test_a_solve_beside_another_leaves_it_room(precision):
    d = geometry.straight_channel()  # 91 tiles
    with cps.Solver(d, precision=precision) as long, cps.Solver(d, precision=precision) as short:
        assert short.last_pcg_form == cps.CPS_PCG_FORM_NONE
        h0, f0 = bits(short, 20)
        assert short.last_pcg_form == cps.CPS_PCG_FORM_CLUSTER
        t = threading.Thread(target=lambda: long.solve(8000, eps=0.0))  # about half a second
        forms = []
        t.start()
        while t.is_alive():
            h, f = bits(short, 20)
            forms.append(short.last_pcg_form)
            assert np.array_equal(h, h0) and all(np.array_equal(f[k], f0[k]) for k in f0)
        t.join()
        assert cps.CPS_PCG_FORM_FEW in forms
        bits(short, 20)
        assert short.last_pcg_form == cps.CPS_PCG_FORM_CLUSTER


def test_three_threads_get_what_they_get_alone():
    designs = [geometry.straight_channel(), geometry.channel_network(M=61, N=233, h=20e-6, wmin=4, wmax=8, seed=6),
               geometry.channel_network(M=129, N=225, h=20e-6, wmin=4, wmax=8, seed=7)]
    solvers = [cps.Solver(d) for d in designs]
    try:
        want = [bits(s, 30) for s in solvers]
        got = [[] for _ in solvers]

        def work(k):
            for _ in range(6):
                got[k].append(bits(solvers[k], 30))

        threads = [threading.Thread(target=work, args=(k,)) for k in range(3)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for k in range(3):
            assert len(got[k]) == 6
            for h, f in got[k]:
                assert np.array_equal(h, want[k][0])
                assert all(np.array_equal(f[q], want[k][1][q]) for q in f)
    finally:
        for s in solvers:
            s.close()
