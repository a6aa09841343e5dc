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
