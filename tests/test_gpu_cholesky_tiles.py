"""The single-matrix factorisation at the sizes where its task list changes
shape (one to six tile rows, ragged last tiles), in the three precisions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ORDERS = [1, 7, 8, 63, 64, 65, 128, 129, 192, 193, 256, 257, 321, 383]


def _factor(A, prec):
    import torch
    from pybrown_b200 import _lib
    n = len(A)
    ld = (n + 63) // 64 * 64
    buf = torch.zeros((ld, ld), dtype=torch.float64 if prec == 0 else torch.float32, device="cuda")
    buf[:n, :n] = torch.tensor(A).to(buf.dtype)
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.call("pbg_dev_cholesky", buf.data_ptr(), n, ld, prec, info.data_ptr(), None)
    torch.cuda.synchronize()
    return np.tril(buf[:n, :n].double().cpu().numpy()), int(info.item())


def _spd(n):
    rng = np.random.default_rng(n)
    g = rng.normal(size=(n, 32))
    return 2.0 * np.eye(n) + g @ g.T / 16.0


@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("n", ORDERS)
def test_backward_error(n, prec):
    """|A - L L^T| stays below the rounding bound of a Cholesky factorisation,
    (n + 1) u |L| |L^T| (Higham, Accuracy and Stability of Numerical
    Algorithms, theorem 10.3), u the unit roundoff of FP64 or of a 3xTF32
    product (2^-22), with a factor of 4 for the blocks' own inverses."""
    A = _spd(n)
    if prec:
        A = A.astype(np.float32).astype(np.float64)
    L, info = _factor(A, prec)
    assert info == 0
    u = 2.0 ** -53 if prec == 0 else 2.0 ** -22
    bound = 4 * (n + 1) * u * (np.abs(L) @ np.abs(L).T)
    assert np.all(np.abs(A - L @ L.T) <= bound)


@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("n,bad", [(8, 0), (64, 63), (65, 64), (130, 7), (200, 128), (321, 320)])
def test_first_bad_pivot(n, bad, prec):
    """A negative diagonal entry that no earlier column touches is the first
    non-positive pivot, whatever follows it."""
    A = _spd(n)
    A[bad, :] = A[:, bad] = 0.0
    A[bad, bad] = -1.0
    assert _factor(A, prec)[1] == bad + 1
