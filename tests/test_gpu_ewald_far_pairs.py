"""Smith-Ewald tensor through the reference's entry point, which takes pair vectors as
they are: vectors many boxes long, where the per-axis products of exponentials
would leave the FP64 range, against the oracle on the same vectors."""
import math

import numpy as np
import pytest

from conftest import rel_err
from test_gpu_tensors import _beads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(2, 4), (1, 2), (3, 4)])
@pytest.mark.parametrize("alpha,boxes", [(math.sqrt(math.pi), k) for k in (0, 1, 3, 111, 112, 113, 400)] +
                         [(16.0, k) for k in (0, 1, 2, 5)] + [(7.0, 6), (7.0, 8), (0.5, 1500)])
def test_pair_vectors_outside_the_box(oracle_lib, alpha, boxes, m, n):
    from pybrown_b200.diffusion import RPY_Smith_M_matrix
    L, N = 200.0, 9
    rng = np.random.default_rng(11)
    pos, radii = rng.uniform(-L / 2, L / 2, size=(N, 3)), rng.uniform(5.0, 9.0, size=N)
    rij = oracle_lib.pointers(pos, L)
    # every vector moved by whole boxes, another multiple along each axis
    shift = L * boxes * np.array([1.0, -1.0, 0.0])
    upper = np.triu(np.ones((N, N)), 1)[:, :, None]
    rij = rij + shift * upper - shift * upper.transpose(1, 0, 2)
    ref = oracle_lib.smith(radii, rij, L, alpha, m, n)
    assert np.all(np.isfinite(ref))
    got = RPY_Smith_M_matrix(_beads(pos, radii), rij, L, alpha, m, n)
    assert rel_err(got, ref) <= 1e-10
