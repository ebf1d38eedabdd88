"""Mixed-precision factor of matrices with elements up to the largest float: the
tiles that the solves split into TF32 halves hold such elements (L does not:
below 2^64), so 4^63 A must factor to 2^63 times the factor of A, bit for bit."""
import numpy as np
import pytest

from test_gpu_factor_scaling import _factor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [1, 2])
@pytest.mark.parametrize("n", [64, 192, 193, 257, 330])
def test_elements_up_to_the_largest_float(n, prec):
    rng = np.random.default_rng(n)
    v = rng.uniform(1.38, 1.42, size=n)  # elements of all 24 bits: their TF32 halves do not vanish
    A = np.outer(v, v) + np.diag(rng.uniform(1.5, 1.9, size=n))
    A = A.astype(np.float32).astype(np.float64)
    L = _factor(A, prec)
    assert np.max(np.abs(L @ L.T - A)) <= 1e-5
    big = np.ldexp(A, 126)
    assert np.max(big) < np.finfo(np.float32).max
    assert np.array_equal(_factor(big, prec), np.ldexp(L, 63))
