"""A factorisation that is refused in one step does not follow the system into later
ones: after a refused chol(D) without a new D, a full step from good positions
succeeds and moves the beads as if nothing had happened."""
import math

import numpy as np
import pytest

from test_gpu_box import _box, _config, _inp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme", ["ermak", "midpoint"])
@pytest.mark.parametrize("precision,matrix", [("fp64", "D"), ("mixed", "R")])
def test_full_step_after_a_refused_factorisation(precision, matrix, scheme):
    from pybrown_b200 import _lib
    N, a = 22, 20.0
    L = (N * 4 * math.pi * a ** 3 / 3 / 0.2) ** (1 / 3)
    pos, radii = _config(3, N, L, a, a, 0.05 * a)
    inp = _inp(box_length=L, hydrodynamics="rpy_smith_lub", propagation_scheme=scheme, precision=precision)
    box, ref = _box(pos, radii, inp), _box(pos, radii, inp)
    for b in (box, ref):
        b.propagate(1e-4)
    bad = -np.eye(3 * N)
    _lib.call("pbg_set_matrix", box._h, _lib.MAT[matrix], bad.ctypes.data, box._stream)
    with pytest.raises(_lib.PbgError, match="not positive definite"):
        box.propagate(1e-4, False, False, True)
    ref.propagate(1e-4, False, False, True)  # takes the same noise
    for b in (box, ref):
        b._pos[...] = pos
        b.propagate(1e-4)
    assert np.array_equal(box.positions(), ref.positions())
