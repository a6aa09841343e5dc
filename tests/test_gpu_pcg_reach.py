"""How far the PCG in the eigenbasis reaches: 4,096 components a block, 622,592 on 152.  Twenty iterations on a lattice just
inside (one launch: it writes the duplicated nodes itself) and on one just beyond (the global-memory kernel and the
nodes' fill), both against the oracle's iterates."""
import numpy as np
import pytest

from oracle import oracle as O
from tests import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,launches", [(1109, 1109, 1), (1120, 1120, 2)])
def test_the_largest_plan_and_beyond(gpu_lib, tmp_path, nx, ny, launches):
    import torch

    components = (nx - 1) * (ny // 2 + 1)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert (components <= 4096 * sms) == (launches == 1)
    ini = decks.write(decks.deck(nx=nx, ny=ny, ne=1000, ni=1000, solver="cg", tol="1e-300", maxit=20,
                                 solver_extra="poisson_bc = dirichlet_x\n"), str(tmp_path))
    orc = O.OracleSim(ini, load=False, initial_field=False)
    rho = np.random.default_rng(nx).normal(size=(nx + 1, ny + 1))
    rho[:, -1] = rho[:, 0]
    rho = rho.ravel()
    phi, _, it, conv = orc.R.pcg_solve(rho)
    assert it == 20 and not conv
    sim = gpu_lib.Simulation.from_ini(ini)
    sim.set_grid("rho", rho)
    before = sim.launches
    it_g, _, conv_g = sim.potential_solver()
    assert sim.launches - before == launches
    assert it_g == 20 and not conv_g
    assert np.max(np.abs(sim.grid("phi") - phi)) <= 1e-12 * np.max(np.abs(phi))
    sim.close()
