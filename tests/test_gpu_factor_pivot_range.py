"""Pivots at the ends of the range: those that the factorisation cannot take are
reported as non-positive instead of leaving infinities or NaN behind info = 0."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _factor(A, prec):
    import torch
    from pybrown_b200 import _lib
    n, ld = len(A), (len(A) + 63) // 64 * 64
    dtype = torch.float64 if prec == 0 else torch.float32
    buf = torch.zeros((ld, ld), dtype=dtype, device="cuda")
    buf[:n, :n] = torch.tensor(A).to(dtype)
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.call("pbg_dev_cholesky", buf.data_ptr(), n, ld, prec, info.data_ptr(), None)
    torch.cuda.synchronize()
    return np.tril(buf[:n, :n].double().cpu().numpy()), int(info.item())


@pytest.mark.parametrize("n", [1, 8, 64, 70])
@pytest.mark.parametrize("pivot", [5e-324, 2.0 ** -1030, np.nextafter(2.0 ** -1022, 0), 1.5 * 2.0 ** 1022, 2.0 ** 1023,
                                   np.inf, np.nan, 0.0, -1.0])
def test_refused_last_pivot_fp64(n, pivot):
    A = np.eye(n)
    A[-1, -1] = pivot
    assert _factor(A, 0)[1] == n


@pytest.mark.parametrize("n", [1, 8, 64, 70])
@pytest.mark.parametrize("pivot", [2.0 ** -1022, 2.0 ** -1000, 2.0 ** 1000, 2.0 ** 1022])
def test_accepted_last_pivot_fp64(n, pivot):
    A = np.eye(n)
    A[-1, -1] = pivot
    L, info = _factor(A, 0)
    assert info == 0 and np.array_equal(L, np.sqrt(A))


@pytest.mark.parametrize("n", [1, 64, 70])
def test_subnormal_floats(n):
    A = np.eye(n)
    A[-1, -1] = 2.0 ** -140
    assert _factor(A, 1)[1] == n
    L, info = _factor(A, 2)
    assert info == 0 and np.array_equal(L, np.sqrt(A))
