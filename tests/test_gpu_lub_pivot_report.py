"""A resistance matrix that is not positive definite is reported by its first
non-positive pivot in its own order (1-based), whatever order it is factored in."""
import re

import numpy as np
import pytest

from test_gpu_box import _box, _inp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme", ["ermak", "midpoint"])
@pytest.mark.parametrize("chol", [True, False])
@pytest.mark.parametrize("bad", [(0,), (5, 40), (17, 63), (65,)])
def test_first_pivot_of_R(bad, chol, scheme):
    from pybrown_b200 import _lib
    # 22 beads far apart: no lubricated pair, so R = Rff
    pos = np.array([[x, y, z] for x in (-300.0, 0.0, 300.0) for y in (-300.0, 0.0, 300.0)
                    for z in (-300.0, 0.0, 300.0)])[:22]
    radii = np.full(len(pos), 20.0)
    box = _box(pos, radii, _inp(box_length=1000.0, hydrodynamics="rpy_smith_lub", propagation_scheme=scheme))
    box.propagate(1e-4)
    R = np.eye(3 * len(pos))
    for k in bad:
        R[k, k] = -1.0
    _lib.call("pbg_set_matrix", box._h, _lib.MAT["Rff"], R.ctypes.data, box._stream)
    for _ in range(2):  # the second step builds nothing: it reports the same
        with pytest.raises(_lib.PbgError) as e:
            box.propagate(1e-4, False, _ == 0, chol and _ == 0)
        assert int(re.search(r"inverse info 0/(\d+)", str(e.value))[1]) == bad[0] + 1
    box._pos[...] = pos
    box.propagate(1e-4)
    assert np.all(np.isfinite(box.positions()))
