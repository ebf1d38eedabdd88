"""The Smith-Ewald tensor over the lattice sizes of both forms of its sums
(unrolled for ewald_real <= 2 and ewald_imag <= 4, rolled above), tile edges,
and row strides and bases that rule out 16-byte stores, against the oracle."""
import math

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


def _config(n, L, seed):
    """Uniform positions: overlapping and engulfed pairs occur among them."""
    rng = np.random.default_rng(seed)
    return rng.uniform(-L / 2, L / 2, size=(n, 3)), rng.uniform(10.0, 40.0, size=n)


def _device(pos, radii, L, alpha, m, n_max, prec, ld, offset=0):
    import torch
    from pybrown_b200 import _lib
    dtype = torch.float64 if prec == 0 else torch.float32
    n3 = 3 * len(radii)
    dpos = torch.tensor(pos.reshape(-1), device="cuda")
    drad = torch.tensor(radii, device="cuda")
    buf = torch.full((offset + n3 * ld,), -7.0, dtype=dtype, device="cuda")
    M = buf[offset:]
    _lib.call("pbg_dev_smith_matrix", dpos.data_ptr(), drad.data_ptr(), len(radii), L, alpha, m, n_max, 1.0, prec,
              M.data_ptr(), ld, None)
    torch.cuda.synchronize()
    out = M.view(n3, ld).double().cpu().numpy()
    assert np.all(buf[:offset].cpu().numpy() == -7.0) and np.all(out[:, n3:] == -7.0)
    return out[:, :n3]


def _oracle(lib, pos, radii, L, alpha, m, n_max):
    return lib.smith(radii, lib.pointers(pos, L), L, alpha, m, n_max)


@pytest.mark.parametrize("m,n_max", [(0, 0), (1, 0), (0, 1), (1, 2), (2, 3), (2, 4), (3, 4), (2, 5), (4, 6), (5, 7)])
def test_lattice_sizes(oracle_lib, m, n_max):
    L, alpha = 400.0, math.sqrt(math.pi)
    pos, radii = _config(35, L, 1)
    ref = _oracle(oracle_lib, pos, radii, L, alpha, m, n_max)
    assert rel_err(_device(pos, radii, L, alpha, m, n_max, 0, 105), ref) <= 1e-10
    assert rel_err(_device(pos, radii, L, alpha, m, n_max, 1, 105), ref) <= 2e-6


@pytest.mark.parametrize("alpha", [1.0, 2.5])
def test_other_alpha(oracle_lib, alpha):
    L = 600.0
    pos, radii = _config(20, L, 2)
    for m, n_max in ((2, 4), (3, 5)):
        ref = _oracle(oracle_lib, pos, radii, L, alpha, m, n_max)
        assert rel_err(_device(pos, radii, L, alpha, m, n_max, 0, 60), ref) <= 1e-10
        assert rel_err(_device(pos, radii, L, alpha, m, n_max, 1, 60), ref) <= 2e-6


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 33])
@pytest.mark.parametrize("extra,offset", [(0, 0), (1, 0), (4, 0), (4, 1)])
def test_tile_edges(oracle_lib, n, extra, offset):
    """Rows of 3n + extra elements (odd strides, 16-byte multiples) from a base
    `offset` elements past an aligned one; nothing outside 3n x 3n is written."""
    L, alpha = 500.0, math.sqrt(math.pi)
    pos, radii = _config(n, L, 3 + n)
    ref = _oracle(oracle_lib, pos, radii, L, alpha, 2, 4)
    assert rel_err(_device(pos, radii, L, alpha, 2, 4, 0, 3 * n + extra, offset), ref) <= 1e-10
    assert rel_err(_device(pos, radii, L, alpha, 2, 4, 1, 3 * n + extra, offset), ref) <= 2e-6


def test_refused_lattices():
    """Lattices beyond the tables' limits stay refused, whatever form the sums take."""
    from pybrown_b200 import _lib
    import torch
    z = torch.ones(64, dtype=torch.float64, device="cuda")
    for prec, n_max, ok in ((0, 7, True), (0, 8, False), (1, 9, True), (1, 10, False)):
        rc = _lib.lib.pbg_dev_smith_matrix(z.data_ptr(), z.data_ptr(), 1, 100.0, 1.7, 2, n_max, 1.0, prec,
                                           z.data_ptr(), 3, None)
        assert (rc == 0) == ok, (prec, n_max, rc)
    torch.cuda.synchronize()
