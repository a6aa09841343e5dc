"""Unsorted mixed states deposit through bands of node words in shared memory (one launch more a push) up to eight bands,
counted as the launch forms them: on the last grids of eight bands, the first of nine, and elongated ones."""
import numpy as np
import pytest

from tests import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,bands", [(64, 64, True), (450, 450, True), (449, 450, True), (457, 457, False),
                                         (457, 456, False), (64, 3264, False), (64, 2900, True), (3264, 63, True),
                                         (480, 480, False)])
def test_at_most_eight_bands(gpu_lib, tmp_path, nx, ny, bands):
    ini = decks.write(decks.deck(nx=nx - 1, ny=ny - 1, ne=500, ni=500, solver="cg", tol="1e-3"), str(tmp_path))
    sim = gpu_lib.Simulation.from_ini(ini, precision=1, sort_every=0)
    p = np.random.default_rng(nx).random((500, 5)) * [nx - 1, ny - 1, 1, 1, 1]
    for s in range(2):
        sim.set_particles(s, p)
    before = sim.launches
    sim.push_species(0)
    assert sim.launches - before == (2 if bands else 1)
    sim.close()
