"""Grids whose multigrid plan fills the shared memory of a block to within a
kilobyte: solved by multigrid (at most 20 iterations, as on every other grid) and
to the Jacobi-preconditioned solution (both to 1e-12; 1e-9 of its largest value)."""
import numpy as np
import pytest

from conftest import rel_err
import mpm2d
import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nx, Ny", [(5, 1133), (11, 1922), (1133, 5), (3778, 17)])
def test_tight_plans_are_multigrid(Nx, Ny):
    h, rho = 1.0 / 64, 2450.0
    sc = scenes.column(Nx=Nx, Ny=Ny, h=h, width=min(Nx - 1, 200) * h, height=min(Ny - 2, 200) * h,
                       material="g_nonlocal_mu2", rho=rho, dt=1e-5, gravity=-9.8, mp={"grains_d": 5.3e-4, "A": 0.48})
    p = sc["particles"]
    p["syy"] = -rho * 9.8 * (np.max(p["y"]) + h / 4 - p["y"]) - 500.0
    p["sxx"] = 0.4 * p["syy"]
    gf = {}
    for precond in ("multigrid", "jacobi"):
        sim = mpm2d.Simulation(sc, solver_tol=1e-12, solver_maxit=50000, precond=precond)
        sim.step(1)
        rc, it, resid = sim.last_solve()
        assert rc == 0 and resid <= 1e-12
        assert precond == "jacobi" or it <= 20, it
        gf[precond] = sim.get("node_gf")
    assert np.max(np.abs(gf["jacobi"])) > 0
    assert rel_err(gf["multigrid"], gf["jacobi"]) <= 1e-9
