"""Kinetic energies of both precisions against exactly rounded sums of the stored velocities' squares: particle counts
around a vector load's and a thread's share, speeds of one size and over twenty decades, one huge among small ones,
subnormals, infinities and NaN.

Bound: all terms are positive, so every rounding counts at most 2^-53 of the sum.  A thread's share (up to two
particles at these sizes) 2 at most, the scaling 2, the trees of a warp, a CTA and of the CTAs' partials 5 + 8 + 38 + 5,
the normalisation and the expectation's own about 10: 70 roundings."""
import math

import numpy as np
import pytest

from tests import decks

pytestmark = pytest.mark.gpu


def _speeds(kind, n, rng):
    v = rng.standard_normal((n, 3))
    if kind == "decades":
        v *= 10.0 ** rng.uniform(-12, 8, (n, 3))
    elif kind == "outlier":
        v[n // 2] = [3e9, -7e11, 1.0]
    elif kind == "tiny":
        v *= 1e-42
        v[0, 0] = 1e-19
    return v


@pytest.mark.parametrize("precision,kind", [(0, "unit"), (0, "decades"), (0, "outlier"), (1, "unit"), (1, "decades"),
                                            (1, "outlier"), (1, "tiny")])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 1027, 311299, 500002])
def test_energies_match_exact_sums(gpu_lib, tmp_path, precision, kind, n):
    E = gpu_lib
    ini = decks.write(decks.deck(nx=16, ny=16, ne=n, ni=n, solver="cg"), str(tmp_path))
    sim = E.Simulation.from_ini(ini, precision=precision)
    rng = np.random.default_rng(n)
    p = np.empty((n, 5))
    p[:, :2] = rng.random((n, 2)) * 16
    p[:, 2:] = _speeds(kind, n, rng)
    unit = p.copy()
    unit[:, 2:] = 1.0
    sim.set_particles(0, unit)
    one = sim.compute_ke(0) / n  # the scale of a unit speed's square
    sim.set_particles(0, p)
    v = p[:, 2:].astype(np.float32).astype(np.float64) if precision else p[:, 2:]
    want = np.array([math.fsum(v[:, c] ** 2) for c in range(3)]) * one
    assert np.all(np.abs(sim.compute_ke(0) - want) <= 2 * 70 * 2.0 ** -53 * want)
    sim.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_energies_carry_infinities(gpu_lib, tmp_path, precision):
    E = gpu_lib
    n = 1001
    ini = decks.write(decks.deck(nx=16, ny=16, ne=n, ni=n, solver="cg"), str(tmp_path))
    sim = E.Simulation.from_ini(ini, precision=precision)
    p = np.ones((n, 5))
    p[17, 2] = np.inf
    p[400, 3] = np.nan
    p[401, 3] = 1e30
    sim.set_particles(0, p)
    ke = sim.compute_ke(0)
    assert ke[0] == np.inf and np.isnan(ke[1]) and np.isfinite(ke[2])
    sim.close()
