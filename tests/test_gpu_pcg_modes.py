"""The PCG solve in the eigenbasis of its operator (csrc/epic_pcg.cu) against the oracle, at the edges of its plan:
the smallest lattices, odd and even sides of every boundary (the folds of the transforms and of equal eigenvalues),
the largest one-cluster and the smallest whole-GPU lattice, one to sixteen components per thread, tables that leave
the small buffer, and the sides where the global-memory kernel takes over.

The solve is conjugate gradients on the same system in another orthonormal basis, so the iterates agree up to
rounding: the iteration counts are equal, and phi agrees within the 1e-12 that every FP64 solve is held to."""
import numpy as np
import pytest

from oracle import oracle as O
from tests import decks

pytestmark = pytest.mark.gpu

BOUNDARY = {0: "", 1: "poisson_bc = periodic", 2: "poisson_bc = dirichlet_x"}


@pytest.mark.parametrize("nx,ny,mode,blocks,tol", [
    (3, 3, 0, 0, "1e-10"), (2, 7, 0, 0, "1e-10"), (4, 4, 1, 0, "1e-10"), (4, 5, 2, 0, "1e-10"), (5, 4, 1, 0, "1e-10"),
    (16, 23, 0, 0, "1e-10"), (23, 16, 1, 0, "1e-10"), (15, 15, 1, 0, "1e-10"), (17, 16, 2, 0, "1e-10"),
    (21, 21, 0, 0, "1e-10"), (22, 22, 0, 0, "1e-10"),      # 253 and 276 components: one CTA, a cluster of three
    (89, 89, 0, 0, "1e-10"), (90, 90, 0, 0, "1e-10"),      # 4095 and 4186: one cluster, the whole GPU
    (180, 179, 1, 0, "1e-8"), (129, 130, 2, 0, "1e-8"),
    (300, 260, 2, 0, "1e-6"),                              # two components per thread
    (128, 128, 0, 16, "1e-8"), (128, 128, 0, 8, "1e-8"), (128, 128, 0, 3, "1e-8"),  # four, eight, sixteen
    (2046, 4, 0, 0, "1e-6"), (2049, 4, 0, 0, "1e-6"),      # the largest side of the tables, and beyond
])
def test_pcg_matches_the_oracle(gpu_lib, tmp_path, nx, ny, mode, blocks, tol):
    ini = decks.write(decks.deck(nx=nx, ny=ny, ne=1000, ni=1000, solver="cg", tol=tol, maxit=100000,
                                 solver_extra=BOUNDARY[mode]), str(tmp_path))
    orc = O.OracleSim(ini, load=False, initial_field=False)
    rho = np.random.default_rng(nx * 1000 + ny).normal(size=(nx + 1, ny + 1))
    rho[:, -1] = rho[:, 0]
    rho[-1] = rho[0]
    rho = rho.ravel()
    phi, err, it, conv = orc.R.pcg_solve(rho)
    assert conv
    sim = gpu_lib.Simulation.from_ini(ini, solver_blocks=blocks)
    sim.set_grid("rho", rho)
    for _ in range(2):  # the second solve meets the first one's workspace
        it_g, _, conv_g = sim.potential_solver()
        assert conv_g and it_g == it
        assert np.max(np.abs(sim.grid("phi") - phi)) <= 1e-12 * np.max(np.abs(phi))


def test_pcg_stops_at_the_cap_and_solves_a_zero_density(gpu_lib, tmp_path):
    ini = decks.write(decks.deck(nx=60, ny=60, ne=1000, ni=1000, solver="cg", tol="1e-10", maxit=7), str(tmp_path))
    orc = O.OracleSim(ini, load=False, initial_field=False)
    rho = np.random.default_rng(3).normal(size=61 * 61)
    phi, _, it, conv = orc.R.pcg_solve(rho)
    assert it == 7 and not conv
    sim = gpu_lib.Simulation.from_ini(ini)
    sim.set_grid("rho", rho)
    it_g, _, conv_g = sim.potential_solver()
    assert it_g == 7 and not conv_g
    assert np.max(np.abs(sim.grid("phi") - phi)) <= 1e-12 * np.max(np.abs(phi))
    sim.set_grid("rho", np.zeros_like(rho))
    it_g, _, conv_g = sim.potential_solver()
    assert it_g == 0 and conv_g and not sim.grid("phi").any()
