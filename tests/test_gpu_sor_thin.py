"""Wrapping lattices with many more rows than nodes a row (walls in x): a sweep starts every nyi steps while the last of
nxi rows ends a sweep about nxi steps after the first, so from some length on the first row is 25 sweeps ahead when a
checked sweep ends.  The last lattices where it is not, the first where it is, and beyond, against the oracle, bit for
bit, with caps around the residual checks."""
import numpy as np
import pytest

from oracle import oracle as O
from tests import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(96, 4), (97, 4), (109, 4), (128, 4), (201, 8), (257, 9), (257, 10), (257, 11)])
@pytest.mark.parametrize("cap", [1, 26, 40, 20000])
def test_thin_wrapping_sor_is_iterate_exact(gpu_lib, tmp_path, nx, ny, cap):
    ini = decks.write(decks.deck(nx=nx, ny=ny, ne=1000, ni=1000, solver="gs", tol="1e-3", maxit=cap,
                                 solver_extra="sor_omega = 1.8\npoisson_bc = dirichlet_x\n"), str(tmp_path))
    orc = O.OracleSim(ini, load=False, initial_field=False)
    rho = np.random.default_rng(nx * 1000 + ny).normal(size=(nx + 1, ny + 1))
    rho[:, -1] = rho[:, 0]
    rho = rho.ravel()
    phi, err, it, conv = orc.R.gs_solve(rho, omega=1.8)
    sim = gpu_lib.Simulation.from_ini(ini)
    sim.set_grid("rho", rho)
    for _ in range(2):  # the second solve meets the first one's workspace
        it_g, err_g, conv_g = sim.potential_solver()
        assert (it_g, conv_g) == (it, bool(conv))
        assert np.array_equal(sim.grid("phi"), phi)
        assert abs(err_g - err) <= 1e-12 * err
    sim.close()
