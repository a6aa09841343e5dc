"""What a call returns is the same from a state's first calls (copied straight to the caller) and from later ones (through
its pinned buffer, up to 64 KB), and device errors are reported by both and leave the state usable."""
import numpy as np
import pytest

from tests import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(16, 16), (90, 90), (90, 91), (120, 80)])
def test_results_and_errors_early_and_late(gpu_lib, tmp_path, nx, ny):
    E = gpu_lib
    n = 500
    ini = decks.write(decks.deck(nx=nx, ny=ny, ne=n, ni=n, solver="cg"), str(tmp_path))
    sim = E.Simulation.from_ini(ini)
    rng = np.random.default_rng(nx * ny)
    good = rng.random((n, 5)) * [nx, ny, 1, 1, 1]
    bad = good.copy()
    bad[7, 0] = -3.0
    seen = []
    for _ in range(6):
        sim.set_particles(0, bad)
        with pytest.raises(E.EpicError):
            sim.scatter_species(0)
        sim.set_particles(0, good)
        sim.set_particles(1, good)
        for s in range(2):
            sim.scatter_species(s)
        sim.compute_rho()
        it = sim.potential_solver()
        sim.calculate_efield()
        seen.append((sim.num_particles(0), it, sim.grid("rho"), sim.grid("phi"), sim.grid("efx"), sim.den(1),
                     sim.compute_ke(0), sim.compute_momentum(1), sim.compute_pe(), sim.delta_phi()))
    for later in seen[1:]:
        for a, b in zip(seen[0], later):
            assert np.array_equal(a, b)
    sim.close()
