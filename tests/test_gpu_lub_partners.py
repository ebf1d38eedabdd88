"""Lubrication correction at partner counts around the 32 that a bead's warp
evaluates together: none, one, 31, 32, 33, a scan chunk that overflows a started
list, several lists; against the oracle."""
import numpy as np
import pytest

from conftest import rel_err
from test_gpu_tensors import TOL, _beads, _random_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cutoff", [0.4, 2.0, 50.0])
@pytest.mark.parametrize("N", [2, 3, 32, 33, 34, 64, 65, 66, 100])
def test_lubrication_partner_counts(oracle_lib, N, cutoff):
    from pybrown_b200.diffusion import JO_R_lubrication_correction_matrix
    L = max(8.0, (N / 0.02) ** (1 / 3))
    pos, radii = _random_config(40 + N, N, L, 0.8, 1.2, gap=0.05)
    rij = oracle_lib.pointers(pos, L)
    ref = oracle_lib.lubrication(radii, rij, cutoff, True)
    got = JO_R_lubrication_correction_matrix(_beads(pos, radii), rij, cutoff, True)
    assert rel_err(got, ref) <= TOL
    assert np.array_equal(got != 0, ref != 0)
