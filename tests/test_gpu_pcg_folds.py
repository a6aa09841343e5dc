"""The transforms of the FP64 PCG solve fold a line a second time where its length allows it (periodic sides of even
length, by the remainder of 4; walled sides of odd length, by the parity of half of it): every small length of each
kind against the oracle, with equal iteration counts and phi within the 1e-12 that every FP64 solve is held to."""
import numpy as np
import pytest

from tests import test_gpu_pcg_modes as modes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,mode", [(4, 6, 1), (5, 8, 1), (6, 9, 1), (7, 10, 1), (11, 12, 1), (28, 30, 1), (29, 31, 1),
                                        (4, 6, 2), (5, 7, 2), (6, 8, 2), (7, 9, 2), (8, 10, 2), (9, 12, 2), (10, 11, 2),
                                        (33, 34, 2), (4, 5, 0), (6, 7, 0), (8, 9, 0), (10, 12, 0), (31, 32, 0)])
def test_every_fold(gpu_lib, tmp_path, nx, ny, mode):
    modes.test_pcg_matches_the_oracle(gpu_lib, tmp_path, nx, ny, mode, 0, "1e-10")
