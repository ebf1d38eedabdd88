"""Mixed batched factorisation (left-looking, K-steps of 64 through two operand
buffers and two accumulators of four K-steps each): B against numpy's factor of
the same D at tile counts around the buffers' and accumulators' turns, odd and
even (a last task with one row of tiles), and ragged orders; replicas alone and
together bit for bit."""
import numpy as np
import pytest

from conftest import rel_err
from test_gpu_box import _config

pytestmark = pytest.mark.gpu

# tile counts 1, 2, 3, 4, 5, 6, 9, 10, 11, 14 with ragged and full last tiles
SIZES = (1, 22, 60, 64, 97, 128, 185, 213, 220, 298)


def _batch(sizes):
    from pybrown_b200.batch import ReplicaBatch
    batch = ReplicaBatch(precision="mixed")
    slots = []
    for N in sizes:
        L = (N * 4 * np.pi * 20.0 ** 3 / 3 / 0.1) ** (1 / 3) if N > 1 else 100.0
        pos, radii = _config(300 + N, N, L, 20.0, 20.0, 0.5)
        slots.append(batch.add(pos, radii, L, seed=N))
    batch.propagate(1e-3)
    return batch, slots


def test_mixed_batch_factor_tile_counts():
    batch, slots = _batch(SIZES)
    B = [np.tril(batch.matrix(s, "B")) for s in slots]
    for N, s, b in zip(SIZES, slots, B):
        # FP32 storage and 3xTF32 products (2^-22) over n <= 900 terms of a matrix
        # with condition below 100: below 1e-5, the bar of the other mixed tests
        assert rel_err(b, np.linalg.cholesky(batch.matrix(s, "D"))) <= 1e-5, N
    batch.close()
    for k in (2, 5, 9):
        alone, (s,) = _batch(SIZES[k:k + 1])
        assert np.array_equal(np.tril(alone.matrix(s, "B")), B[k]), SIZES[k]
        alone.close()
