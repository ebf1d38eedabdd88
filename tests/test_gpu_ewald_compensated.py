"""FP32 Smith-Ewald tensor with many real-space images: their sum is compensated, so
its error does not grow with their number."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tensor(pos, radii, L, alpha, m, n_max, prec):
    import torch
    from pybrown_b200 import _lib
    n3 = 3 * len(radii)
    dpos, drad = torch.tensor(pos.reshape(-1), device="cuda"), torch.tensor(radii, device="cuda")
    M = torch.empty((n3, n3), dtype=torch.float64 if prec == 0 else torch.float32, device="cuda")
    _lib.call("pbg_dev_smith_matrix", dpos.data_ptr(), drad.data_ptr(), len(radii), L, alpha, m, n_max, 1.0, prec,
              M.data_ptr(), n3, None)
    torch.cuda.synchronize()
    return M.double().cpu().numpy()


@pytest.mark.parametrize("m", [2, 3, 8, 16])
def test_image_sum_error_does_not_grow(m):
    """alpha = 0.05 makes up to 6017 images count, all of one sign in the diagonal
    elements of a pair block.  A term is off by erfc's 1.5e-7 (absolute; erfc > 0.4
    on the average over these images) and about six roundings, a compensated sum by
    two: 1.5e-7 / 0.4 + 8 * 2^-24 < 9e-7 of the element, whatever m.  (The plain sum
    in this order is off by 3e-6 at m = 8 and 6e-6 at m = 16.)"""
    N, L = 60, 100.0
    rng = np.random.default_rng(7)
    pos, radii = rng.uniform(-L / 2, L / 2, size=(N, 3)), np.full(N, 1.0)
    ref = _tensor(pos, radii, L, 0.05, m, 1, 0)
    got = _tensor(pos, radii, L, 0.05, m, 1, 1)
    i = np.arange(3 * N)
    pair_diagonals = (i[:, None] // 3 != i[None, :] // 3) & (i[:, None] % 3 == i[None, :] % 3)
    assert np.max(np.abs(got - ref)[pair_diagonals] / np.abs(ref[pair_diagonals])) <= 9e-7
