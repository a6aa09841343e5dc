"""Open walls: the erasing push over many ordered tiles keeps what the same push keeps of pieces that fit one tile, in
the same order and bit for bit: long stretches of tiles that lose nothing, everything, or every other particle, and
counts around a tile and around the 32 tiles a look-back reads at once."""
import numpy as np
import pytest

from tests import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [1023, 1025, 32 * 1024 + 1, 33 * 1024 + 5, 200007])
@pytest.mark.parametrize("pattern", ["stretches", "alternate", "random"])
def test_tiles_equal_pieces(gpu_lib, tmp_path, precision, n, pattern):
    E = gpu_lib
    ini = decks.write(decks.deck(nx=24, ny=20, ne=n, ni=n, bc="open", solver="cg"), str(tmp_path))
    sim = E.Simulation.from_ini(ini, precision=precision)
    rng = np.random.default_rng(n)
    p = rng.random((n, 5)) * [24, 20, 1, 1, 1]
    sim.set_particles(0, p)
    sim.set_particles(1, p)
    sim.initial_field()
    leave = {"stretches": (np.arange(n) // 9000) % 2 == 1, "alternate": np.arange(n) % 2 == 1,
             "random": rng.random(n) < 0.3}[pattern]
    p[leave, 2] = 1e6
    p[:, 4] = np.arange(n)
    sim.set_particles(0, p)
    sim.push_species(0)
    whole = sim.particles(0)
    pieces = []
    for a in range(0, n, 1000):
        sim.set_particles(0, p[a:a + 1000])
        sim.push_species(0)
        pieces.append(sim.particles(0))
    assert np.array_equal(whole, np.concatenate(pieces))
    assert not np.isin(whole[:, 4], np.flatnonzero(leave)).any() and len(whole) > 0
    sim.close()
