"""The density's and the E-field's divisions, done as products where that gives the same double: bit for bit the quotients
IEEE division gives, for cells of one unit, of another power of two and of neither, and for divisors so extreme that the
division itself runs."""
import numpy as np
import pytest

from tests import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dx,density", [(1.0, None), (0.5, None), (0.3, None), (1.0, 1e-320), (1.0, 3.7e200)])
def test_quotients(gpu_lib, tmp_path, dx, density):
    E = gpu_lib
    n, nx, ny = 3001, 20, 17
    ini = decks.write(decks.deck(nx=nx, ny=ny, ne=n, ni=n, bc="reflective", solver="cg"), str(tmp_path))
    over = dict(precision=1, dx=dx, dy=dx)
    if density:
        over["density"] = density
    sim = E.Simulation.from_ini(ini, **over)
    rng = np.random.default_rng(5)
    S = 1 << 20
    i, j = rng.integers(0, nx, n), rng.integers(0, ny, n)
    a, b = rng.integers(0, S, n), rng.integers(0, S, n)
    p = np.zeros((n, 5))
    p[:, 0] = (i + a / S) * dx
    p[:, 1] = (j + b / S) * dx
    sim.set_particles(0, p)
    got = sim.particles(0)
    cell = np.floor(got[:, :2] / dx).astype(int)  # as stored (a product may round into the next cell)
    off = ((got[:, :2] / dx - cell).astype(np.float32) * np.float32(S)).astype(np.int64)
    acc = np.zeros((nx + 1, ny + 1), dtype=np.int64)
    for di in (0, 1):
        for dj in (0, 1):
            wx = off[:, 0] if di else S - off[:, 0]
            wy = off[:, 1] if dj else S - off[:, 1]
            np.add.at(acc, (cell[:, 0] + di, cell[:, 1] + dj), wx * wy)
    sim.scatter_species(0)
    c = sim.cfg
    with np.errstate(over="ignore", divide="ignore"):
        want = acc.astype(np.float64) * 2.0 ** -40 * sim.species[0].spwt / (c.dx * c.dy * (c.L * c.L) * c.density)
    want[[0, -1]] *= 0.5
    want[:, [0, -1]] *= 0.5
    if dx != 0.3:  # offsets are exact then
        assert np.array_equal(sim.den(0).reshape(nx + 1, ny + 1), want)
    phi = rng.standard_normal((nx + 1, ny + 1)) * 10.0 ** rng.integers(-3, 4, (nx + 1, ny + 1))
    sim.set_grid("phi", phi.ravel())
    sim.calculate_efield()
    ex = -(phi[2:] - phi[:-2]) / (2 * dx)
    ey = -(phi[:, 2:] - phi[:, :-2]) / (2 * dx)
    assert np.array_equal(sim.grid("efx").reshape(nx + 1, ny + 1)[1:-1], ex)
    assert np.array_equal(sim.grid("efy").reshape(nx + 1, ny + 1)[:, 1:-1], ey)
    sim.close()
