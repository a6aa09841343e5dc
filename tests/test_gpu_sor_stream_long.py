"""The streamed SOR's rings over many turns: thousands of sweeps without convergence, every message word and snapshot used
again hundreds of times, on lattices of one to four slots a CTA, with the shortest ring and with a padded one.  Bit for bit
the oracle's, solve after solve."""
import numpy as np
import pytest

from oracle import oracle as O
from tests import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(9, 8), (64, 64), (130, 60), (60, 130)])
def test_many_turns_of_the_rings(gpu_lib, tmp_path, nx, ny):
    cap = 3000
    ini = decks.write(decks.deck(nx=nx, ny=ny, ne=1000, ni=1000, solver="gs", tol="1e-300", maxit=cap,
                                 solver_extra="sor_omega = 1.7\n"), str(tmp_path))
    orc = O.OracleSim(ini, load=False, initial_field=False)
    rho = np.random.default_rng(nx).normal(size=(nx + 1) * (ny + 1))
    phi, _, it, conv = orc.R.gs_solve(rho, omega=1.7)
    sim = gpu_lib.Simulation.from_ini(ini)
    sim.set_grid("rho", rho)
    for _ in range(5):
        it_g, _, conv_g = sim.potential_solver()
        assert (it_g, conv_g) == (it, bool(conv))
        assert np.array_equal(sim.grid("phi"), phi)
    sim.close()
