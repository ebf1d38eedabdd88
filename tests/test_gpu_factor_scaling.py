"""Factorisation and inverse of matrices far from 1: every operation of them commutes
with a power of two as long as no intermediate leaves the range of its type, so the
factor of 4^k A is 2^k times that of A, and the inverse 4^-k times, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spd(n):
    rng = np.random.default_rng(n)
    g = rng.normal(size=(n, 32))
    A = np.eye(n) + g @ g.T / 64.0
    return A / (1.01 * np.max(A))  # elements below 1


def _device(A, ld, torch_dtype):
    import torch
    buf = torch.zeros((ld, ld), dtype=torch_dtype, device="cuda")
    buf[:len(A), :len(A)] = torch.tensor(A).to(torch_dtype)
    return buf, torch.zeros(1, dtype=torch.int32, device="cuda")


def _factor(A, prec):
    import torch
    from pybrown_b200 import _lib
    n, ld = len(A), (len(A) + 63) // 64 * 64
    buf, info = _device(A, ld, torch.float64 if prec == 0 else torch.float32)
    _lib.call("pbg_dev_cholesky", buf.data_ptr(), n, ld, prec, info.data_ptr(), None)
    torch.cuda.synchronize()
    assert int(info.item()) == 0
    return np.tril(buf[:n, :n].double().cpu().numpy())


def _inverse(A):
    import torch
    from pybrown_b200 import _lib
    n, ld = len(A), (len(A) + 63) // 64 * 64
    buf, info = _device(A, ld, torch.float64)
    _lib.call("pbg_dev_spd_inverse", buf.data_ptr(), n, ld, info.data_ptr(), None)
    torch.cuda.synchronize()
    assert int(info.item()) == 0
    return buf[:n, :n].cpu().numpy()


@pytest.mark.parametrize("n", [2, 8, 61, 64, 130, 257])
def test_fp64_factor_scales(n):
    A = _spd(n)
    L = _factor(A, 0)
    for k in (-470, -400, -280, -200, 200, 280, 400, 500):
        assert np.array_equal(_factor(np.ldexp(A, 2 * k), 0), np.ldexp(L, k)), k


@pytest.mark.parametrize("n", [8, 130])
def test_fp64_inverse_scales(n):
    A = _spd(n)
    X = _inverse(A)
    for k in (-400, -280, 280, 400):
        assert np.array_equal(_inverse(np.ldexp(A, 2 * k)), np.ldexp(X, -2 * k)), k


@pytest.mark.parametrize("prec", [1, 2])
@pytest.mark.parametrize("n", [8, 64, 130, 257])
def test_fp32_factor_scales(n, prec):
    A = _spd(n).astype(np.float32).astype(np.float64)
    L = _factor(A, prec)
    for k in (-30, 30, 60):
        assert np.array_equal(_factor(np.ldexp(A, 2 * k), prec), np.ldexp(L, k)), k
