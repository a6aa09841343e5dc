"""The mixed form's deposit of unsorted particles through bands of node words in shared memory: densities, potential and
particles equal those of the same state sorted by cell first (whose deposit merges neighbours and adds to the grid), bit
for bit: the sums are integers.  Grids of one band, of several with a ragged last one, of the most bands and one beyond
(where the fused push deposits); particle counts at the edges of a thread's, a CTA's and a slice's share; particles
crowded into one cell, whose words carry past 32 bits."""
import numpy as np
import pytest

from tests import decks

pytestmark = pytest.mark.gpu


def _sim(E, ini, parts, sort_every):
    sim = E.Simulation.from_ini(ini, precision=1, sort_every=sort_every)
    for s in range(2):
        sim.set_particles(s, parts[s])
    sim.initial_field()
    return sim


@pytest.mark.parametrize("nx,ny,n,bc,crowd", [
    (5, 5, 1, "pbc", False), (16, 24, 8191, "reflective", False), (60, 33, 8193, "pbc", False),
    (64, 64, 200001, "pbc", True), (166, 168, 30000, "pbc", False), (168, 166, 30007, "open", False),
    (250, 301, 300005, "reflective", False), (456, 455, 60001, "pbc", False), (474, 473, 60001, "pbc", False),
    (480, 476, 60001, "pbc", False)])
def test_bands_equal_sorted_deposit(gpu_lib, tmp_path, nx, ny, n, bc, crowd):
    E = gpu_lib
    ini = decks.write(decks.deck(nx=nx, ny=ny, ne=n, ni=n, bc=bc, solver="cg", tol="1e-8", maxit=100000), str(tmp_path))
    rng = np.random.default_rng(nx + n)
    parts = []
    for s in range(2):
        p = np.empty((n, 5))
        p[:, 0] = rng.random(n) * nx
        p[:, 1] = rng.random(n) * ny
        if crowd:
            p[: n // 2, :2] = 7.0 + rng.random((n // 2, 2))
        p[:, 2:] = rng.standard_normal((n, 3)) * (1.0 if s == 0 else 0.02)
        parts.append(p)
    a, b = _sim(E, ini, parts, 0), _sim(E, ini, parts, 1)
    for steps in (1, 3):
        a.run(steps)
        b.run(steps)
        for s in range(2):
            assert a.num_particles(s) == b.num_particles(s)
            assert np.array_equal(a.den(s), b.den(s))
            pa, pb = a.particles(s), b.particles(s)
            assert np.array_equal(pa[np.lexsort(pa.T)], pb[np.lexsort(pb.T)])
        assert np.array_equal(a.grid("rho"), b.grid("rho")) and np.array_equal(a.grid("phi"), b.grid("phi"))
    a.close()
    b.close()
