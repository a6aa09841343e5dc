"""The PCG solve's sums against exact ones.

Stopped after one iteration from a zero start, phi is -alpha b with alpha = (b, b)/(b, L b), so its projection on b gives
alpha to below the last bit.  The bound: alpha is rounded once (2^-53).  Each of the two sums crosses the blocks in at most
160 words rounded to a unit of 2^-58 of the total, evenly spread: sqrt(2 160/12) 2^-58 = 1.8e-17.  What a component of phi
carries beside it is r's rounding over alpha L, 4/L 2^-53/sqrt(12) of it, which leaves at most 2.2e-17 of the projection on
these lattices (summed over their eigenvalues).  With 5 sigma of both: 2.6e-16, whatever the number of components.  Sides
n with n + 1 = 2^odd (walls) and n = 4^k (periodic), where the transforms' scales are exact.

Stopped before the first iteration, phi is 0 and the reported error the root of the sum of b^2: large terms first and
then many that an FP64 sum beside them would lose."""
import math
from fractions import Fraction

import numpy as np
import pytest

from tests import decks

pytestmark = pytest.mark.gpu


def _sim(E, d, nx, ny, cap, extra=""):
    ini = decks.write(decks.deck(nx=nx - 1, ny=ny - 1, ne=1000, ni=1000, solver="cg", tol="1e-300", maxit=cap,
                                 solver_extra=extra), str(d))
    sim = E.Simulation.from_ini(ini)
    assert sim.cfg.dx == 1.0
    return sim, (sim.cfg.L * sim.cfg.L) / (sim.cfg.LDe * sim.cfg.LDe)


def _sum(x):
    s = math.fsum(x)
    return Fraction(s) + Fraction(math.fsum(np.append(x, -s)))


@pytest.mark.parametrize("nx,ny,wrap", [(31, 127, False), (129, 1025, True), (513, 1025, True)])
def test_first_step_length(gpu_lib, tmp_path, nx, ny, wrap):
    sim, K = _sim(gpu_lib, tmp_path, nx, ny, 1, "poisson_bc = dirichlet_x\n" if wrap else "")
    off = []
    for seed in range(6):
        g = np.random.default_rng(seed).integers(-1000, 1001, size=(nx, ny))
        g[0] = g[-1] = 0
        if wrap:
            g[:, -1] = g[:, 0]
            m = g[:, :-1]
            Lm = 4 * m - np.roll(m, 1, 1) - np.roll(m, -1, 1)
            Lm[1:] -= m[:-1]
            Lm[:-1] -= m[1:]
        else:
            g[:, 0] = g[:, -1] = 0
            m = g.reshape(ny, nx)  # the reference's lattice: the grid's nodes in rows of nx
            p = np.pad(m, 1)
            Lm = 4 * m - p[:-2, 1:-1] - p[2:, 1:-1] - p[1:-1, :-2] - p[1:-1, 2:]
        alpha = Fraction(int((m * m).sum()), int((m * Lm).sum()))
        sim.set_grid("rho", g.astype(float).ravel())
        it, _, conv = sim.potential_solver()
        assert it == 1 and not conv
        phi = sim.grid("phi").reshape(g.shape)
        phi = phi[:, :-1] if wrap else phi.reshape(m.shape)
        b = m * K
        got = _sum((phi * b).ravel()) / _sum((b * b).ravel())
        off.append(abs(float(abs(got) / alpha - 1)))
    sim.close()
    print("first step, %d x %d: off by %s" % (nx, ny, " ".join("%.2e" % o for o in off)))
    assert max(off) <= 2.6e-16


@pytest.mark.parametrize("nx,ny", [(60, 61), (1025, 1025)])
def test_reported_error_is_the_exact_sum(gpu_lib, tmp_path, nx, ny):
    sim, K = _sim(gpu_lib, tmp_path, nx, ny, 0)
    rho = np.full((ny, nx), 2.0 ** -27)
    rho.ravel()[: min(46000, nx * ny // 2)] = 1.0  # beyond every thread's first term
    rho = rho.ravel()
    edge = np.zeros((nx, ny), dtype=bool)
    edge[0] = edge[-1] = edge[:, 0] = edge[:, -1] = True
    sim.set_grid("rho", rho)
    it, err, conv = sim.potential_solver()
    assert it == 0 and not conv and not sim.grid("phi").any()
    b = np.where(edge.ravel(), 0.0, rho * K)
    assert err == math.sqrt(math.fsum(b * b)) / (nx * ny)
    sim.close()
