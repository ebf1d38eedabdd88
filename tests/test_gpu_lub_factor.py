"""FP64 lubricated path: chol(D) read off the factor that D = kBT inv(R) comes
from, against numpy's of the same D, at orders on and beside the 64-wide tiles;
and the factorisation of D itself when a step takes chol(D) without a new D."""
import math

import numpy as np
import pytest

from conftest import rel_err
from test_gpu_box import _box, _config, _inp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme", ["ermak", "midpoint"])
@pytest.mark.parametrize("N", [1, 2, 21, 22, 43, 64])
def test_factor_of_D_lubricated(N, scheme):
    a = 20.0
    L = (N * 4 * math.pi * a ** 3 / 3 / 0.25) ** (1 / 3) if N > 2 else 150.0
    pos, radii = _config(7 + N, N, L, a, a, 0.05 * a)
    box = _box(pos, radii, _inp(box_length=L, hydrodynamics="rpy_smith_lub", propagation_scheme=scheme))
    for flags in ((True, True, True), (False, False, True), (True, True, True)):
        box.propagate(1e-4, *flags)
        D, B = box.D, box.B
        # cond(D) < 1e4 at these gaps: n eps cond < 1e-10
        assert rel_err(np.tril(B), np.linalg.cholesky(D)) <= 1e-10, flags
        assert not np.triu(B, 1).any(), flags
