"""The heat solve's multigrid over the shapes its levels can take: a single
column, lines, odd and power-of-two sides, one to 64 layers, one to three
sweeps, everything in one CTA or levels across the grid; the solution against
the oracle's direct one.  At rtol 1e-10 the iterate is within the system's
condition of it: 1e-5 relative, as in the other solution tests."""
import numpy as np
import pytest

from coldplate_solver_b200 import thermal as pt
from oracle import thermal as th

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nx,Ny,nzs,nzf,sweeps", [
    (1, 1, 2, 7, 2), (1, 9, 2, 7, 2), (7, 1, 2, 7, 2), (2, 2, 1, 1, 2), (16, 16, 2, 7, 2), (17, 13, 2, 7, 1),
    (33, 29, 2, 7, 3), (64, 32, 2, 7, 2), (47, 21, 1, 1, 2), (9, 5, 20, 44, 2), (31, 18, 20, 44, 2), (127, 65, 2, 7, 2)])
def test_solution_over_level_shapes(Nx, Ny, nzs, nzf, sweeps):
    rng = np.random.default_rng(Nx * 131 + Ny)
    gamma = (rng.random((Ny, Nx)) > 0.4).astype(float)
    gamma[rng.random((Ny, Nx)) > 0.85] = 0.37
    gamma[:, 0] = 1.0
    u = np.abs(rng.normal(0.2, 0.15, (Ny, Nx))) * gamma
    v = rng.normal(0.0, 0.05, (Ny, Nx)) * gamma
    c = pt.ThermalCase(gamma=gamma, u=u, v=v, dx=20e-6, dy=20e-6, q=8e5, H_t=4e-4, nz_solid=nzs, nz_fluid=nzf, rtol=1e-10)
    with pt.ThermalSolver(c, mg_sweeps=sweeps) as s:
        r = s.solve()
        T = s.temperature()
        r2 = s.solve()
        T2 = s.temperature()
    p = th.ThermalParams(Nx=Nx, Ny=Ny, dx=c.dx, dy=c.dy, nz_solid=nzs, nz_fluid=nzf, H_t=c.H_t, rtol=c.rtol)
    Td = th.solve_direct(p, c.gamma, c.u, c.v, c.heat_flux())
    assert r["converged"] and r == r2 and np.array_equal(T, T2), (r, r2)
    assert np.linalg.norm(T - Td) <= 1e-5 * np.linalg.norm(Td - c.T_inlet)


# the second level (a quarter of the cells) just below and above the 113 664 threads of a launch at three CTAs
# per SM of 148, where its right-hand side is formed by lanes and by threads, odd sides, and small cases
@pytest.mark.parametrize("Nx,Ny", [(221, 225), (223, 225), (226, 224), (127, 65), (30, 33)])
def test_first_iterations_equal_the_same_algorithm_on_the_cpu(Nx, Ny):
    """Three BiCGStab iterations (six V-cycles) from T_inlet: the same exact
    arithmetic, other rounding.  Each of some hundred operations per value
    rounds at 1e-16, and the coefficients of three iterations amplify that by
    far less than 1e5: 1e-9 relative."""
    rng = np.random.default_rng(Nx)
    gamma = (rng.random((Ny, Nx)) > 0.4).astype(float)
    gamma[:, 0] = 1.0
    u = np.abs(rng.normal(0.2, 0.15, (Ny, Nx))) * gamma
    v = rng.normal(0.0, 0.05, (Ny, Nx)) * gamma
    c = pt.ThermalCase(gamma=gamma, u=u, v=v, dx=20e-6, dy=20e-6, q=8e5, H_t=4e-4, rtol=1e-12, maxiter=3)
    with pt.ThermalSolver(c) as s:
        r = s.solve()
        T = s.temperature()
    p = th.ThermalParams(Nx=Nx, Ny=Ny, dx=c.dx, dy=c.dy, H_t=c.H_t, rtol=c.rtol, maxiter=3)
    Tc, its, _, _ = th.mg_bicgstab_cpu(p, c.gamma, c.u, c.v, c.heat_flux())
    assert r["iterations"] == its == 3
    assert np.linalg.norm(T - Tc) <= 1e-9 * np.linalg.norm(Tc - c.T_inlet)
