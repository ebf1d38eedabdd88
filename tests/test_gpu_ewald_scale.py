"""The mixed-precision Smith-Ewald tensor takes its scale in FP64: scales beyond the
FP32 range give finite elements where the scaled tensor is in range, and every
element is the FP64 product rounded once."""
import math

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


def _tensor(pos, radii, L, prec, scale):
    import torch
    from pybrown_b200 import _lib
    n3 = 3 * len(radii)
    dpos, drad = torch.tensor(pos.reshape(-1), device="cuda"), torch.tensor(radii, device="cuda")
    M = torch.empty((n3, n3), dtype=torch.float64 if prec == 0 else torch.float32, device="cuda")
    _lib.call("pbg_dev_smith_matrix", dpos.data_ptr(), drad.data_ptr(), len(radii), L, math.sqrt(math.pi), 2, 4, scale,
              prec, M.data_ptr(), n3, None)
    torch.cuda.synchronize()
    return M.double().cpu().numpy()


def _config():
    # radii of a thousand: elements of about 1e-5, overlapping pairs among them
    rng = np.random.default_rng(5)
    return rng.uniform(-1e4, 1e4, size=(40, 3)), rng.uniform(900.0, 1500.0, size=40)


@pytest.mark.parametrize("scale", [1e-41, 1.0, 3e38, 1e40, 3e42])
def test_scales_beyond_fp32(scale):
    pos, radii = _config()
    ref = _tensor(pos, radii, 2e4, 0, scale)
    got = _tensor(pos, radii, 2e4, 1, scale)
    assert np.all(np.isfinite(got))
    # 2e-6: the bar of the FP32 tensor; 2^-149: the spacing of subnormal floats
    assert np.max(np.abs(got - ref)) <= 2e-6 * np.max(np.abs(ref)) + 2.0 ** -149


def test_powers_of_two_scale_exactly():
    pos, radii = _config()
    one = _tensor(pos, radii, 2e4, 1, 1.0)
    assert np.array_equal(_tensor(pos, radii, 2e4, 1, 2.0 ** 130), one * 2.0 ** 130)


def test_scaled_once():
    """1 + 2^-24 rounds to 1 in FP32 (a tie), so a scale taken in FP32 leaves every
    element as it is; the FP64 product of a float of mantissa m in (1, 2) moves
    by m / 2 > 1/2 of its spacing, to the next float: all pair elements off their
    blocks' diagonals (two thirds) and about half of the others."""
    pos, radii = _config()
    one = _tensor(pos, radii, 2e4, 1, 1.0)
    two = _tensor(pos, radii, 2e4, 1, 1.0 + 2.0 ** -24)
    assert rel_err(two, one) <= 1.2e-7 and np.count_nonzero(two != one) > 0.6 * one.size
