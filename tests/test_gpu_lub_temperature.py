"""FP64 lubricated steps at temperatures without a diffusion matrix to factor: D = kBT
inv(R) is zero or negative definite and chol(D) is refused, as np.linalg.cholesky
does."""
import math

import numpy as np
import pytest

from test_gpu_box import _box, _config, _inp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme", ["ermak", "midpoint"])
@pytest.mark.parametrize("T", [0.0, -293.15])
def test_refused_without_a_positive_temperature(T, scheme):
    from pybrown_b200 import _lib
    N, a = 22, 20.0
    L = (N * 4 * math.pi * a ** 3 / 3 / 0.2) ** (1 / 3)
    pos, radii = _config(3, N, L, a, a, 0.05 * a)
    box = _box(pos, radii, _inp(box_length=L, T=T, hydrodynamics="rpy_smith_lub", propagation_scheme=scheme))
    # (the midpoint scheme goes on from the NaN that the refused factor leaves, and its
    # rebuild at the predicted positions is refused as well)
    with pytest.raises(_lib.PbgError, match="cholesky info 1, inverse info " + ("0/0" if scheme == "ermak" else "")):
        box.propagate(1e-4)
    D = box.D
    assert np.all(D == 0.0) if T == 0.0 else np.all(np.diag(D) < 0.0)
