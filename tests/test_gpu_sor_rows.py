"""The wrapping lexicographic SOR (csrc/epic_sor.cu) against the oracle, bit for bit: the smallest lattice, sides
around a warp of rows, more rows than columns and the reverse, several warps per quarter of the SM, the largest
lattice that fits and the first that does not, caps before, at and between the residual checks."""
import numpy as np
import pytest

from oracle import oracle as O
from tests import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bc", ["periodic", "dirichlet_x"])
@pytest.mark.parametrize("nx,ny,cap", [(4, 4, 20000), (31, 9, 20000), (32, 33, 20000), (33, 32, 20000), (34, 34, 20000),
                                       (65, 20, 20000), (20, 65, 20000), (64, 64, 1), (64, 64, 26), (64, 64, 40),
                                       (150, 40, 30), (200, 120, 3), (160, 160, 2), (161, 161, 2)])
def test_wrapping_sor_is_iterate_exact(gpu_lib, tmp_path, bc, nx, ny, cap):
    ini = decks.write(decks.deck(nx=nx, ny=ny, ne=1000, ni=1000, solver="gs", tol="1e-6", maxit=cap,
                                 solver_extra="sor_omega = 1.8\npoisson_bc = %s\n" % bc), str(tmp_path))
    orc = O.OracleSim(ini, load=False, initial_field=False)
    rho = np.random.default_rng(nx * 1000 + ny).normal(size=(nx + 1, ny + 1))
    rho[:, -1] = rho[:, 0]
    if bc == "periodic":
        rho[-1] = rho[0]
    rho = rho.ravel()
    phi, err, it, conv = orc.R.gs_solve(rho, omega=1.8)
    sim = gpu_lib.Simulation.from_ini(ini)
    sim.set_grid("rho", rho)
    for _ in range(2):  # the second solve meets the first one's workspace
        it_g, _, conv_g = sim.potential_solver()
        assert (it_g, conv_g) == (it, bool(conv))
        assert np.array_equal(sim.grid("phi"), phi)


@pytest.mark.parametrize("nx,ny,cap", [(2, 2, 20000), (3, 5, 20000), (9, 8, 20000), (33, 9, 20000), (34, 34, 20000),
                                       (35, 34, 20000), (66, 30, 20000), (30, 66, 20000), (65, 64, 1), (65, 64, 2),
                                       (65, 64, 26), (65, 64, 40), (65, 64, 20000), (98, 97, 20000), (130, 60, 400),
                                       (60, 130, 400), (155, 100, 60), (170, 170, 30)])
def test_walled_sor_is_iterate_exact(gpu_lib, tmp_path, nx, ny, cap):
    """The sweeps streamed through a cluster: one to fifteen CTAs, one to four slots, rows at and beyond a warp, rows
    that set the period, caps around the residual checks, more checks than snapshots, and a lattice too large for it."""
    ini = decks.write(decks.deck(nx=nx, ny=ny, ne=1000, ni=1000, solver="gs", tol="1e-7", maxit=cap,
                                 solver_extra="sor_omega = 1.7\n"), str(tmp_path))
    orc = O.OracleSim(ini, load=False, initial_field=False)
    rho = np.random.default_rng(nx * 1000 + ny).normal(size=(nx + 1) * (ny + 1))
    phi, err, it, conv = orc.R.gs_solve(rho, omega=1.7)
    sim = gpu_lib.Simulation.from_ini(ini)
    sim.set_grid("rho", rho)
    for _ in range(3):
        it_g, _, conv_g = sim.potential_solver()
        assert (it_g, conv_g) == (it, bool(conv))
        assert np.array_equal(sim.grid("phi"), phi)


@pytest.mark.parametrize("nx,ny,cap", [(5, 4, 20000), (33, 34, 20000), (64, 64, 51), (64, 64, 20000), (97, 60, 20000)])
def test_boltzmann_sor_matches_the_oracle(gpu_lib, tmp_path, nx, ny, cap):
    """The same with the source (rho - exp phi) K: equal sweep counts, phi to 1e-12 (exp's last bit)."""
    ini = decks.write(decks.deck(nx=nx, ny=ny, ne=1000, ni=1000, solver="gshybrid", tol="1e-6", maxit=cap),
                      str(tmp_path))  # the oracle's gsfluidsolver has the reference's omega, 1.4
    orc = O.OracleSim(ini, load=False, initial_field=False)
    rho = np.random.default_rng(nx * 1000 + ny).normal(size=(nx + 1) * (ny + 1)) * 0.1
    phi, err, it, conv, _ = orc.R.gsfluid_solve(rho)
    sim = gpu_lib.Simulation.from_ini(ini)
    for _ in range(2):
        sim.set_grid("rho", rho)
        it_g, _, conv_g = sim.potential_solver()
        assert (it_g, conv_g) == (it, bool(conv))
        assert np.max(np.abs(sim.grid("phi") - phi)) <= 1e-12 * np.max(np.abs(phi))
