"""The mixed form's cell sort at particle counts around its vector loads, a tile and its scratch's smallest sizes: the
stable argsort of the cells, bit for bit, with one, two and three digit passes."""
import numpy as np
import pytest

from tests import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(16, 16), (64, 48), (520, 511)])
@pytest.mark.parametrize("n,cap", [(1, 1), (2, 3), (5, 5), (10, 10), (13, 13), (14, 16), (1023, 1023), (4095, 4096),
                                   (4097, 4097), (20006, 30001)])
def test_sort_mixed_counts(gpu_lib, tmp_path, nx, ny, n, cap):
    ini = decks.write(decks.deck(nx=nx, ny=ny, ne=n, ni=n), str(tmp_path))
    sim = gpu_lib.Simulation.from_ini(ini, precision=1, capacity=cap)
    rng = np.random.default_rng(n + nx)
    p = rng.random((n, 5))
    p[:, 0] *= nx
    p[:, 1] *= ny
    p[: n // 2, :2] = np.floor(p[: n // 2, :2] / 8) * 8 + 0.25  # many share a cell
    sim.set_particles(0, p)
    before = sim.particles(0)
    sim.sort_species(0)
    key = before[:, 0].astype(np.int64) * (ny + 1) + before[:, 1].astype(np.int64)
    assert np.array_equal(sim.particles(0), before[np.argsort(key, kind="stable")])
    sim.close()
