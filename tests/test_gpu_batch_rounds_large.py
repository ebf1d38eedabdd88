"""Attempt rounds of replicas beyond 512 columns: the product of eight noise vectors
stages them 256 columns at a time through two shared-memory buffers, so a buffer is
first used again at the third block.  Odd and even orders just above two and three
blocks, against one attempt after the other, bit for bit."""
import numpy as np
import pytest

from test_gpu_batch_rounds import _batch

pytestmark = pytest.mark.gpu

SIZES = [171, 172, 257, 341, 342, 400]  # orders 513, 516, 771, 1023, 1026, 1200


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_rounds_of_large_replicas(precision):
    a, sa = _batch(precision, SIZES)
    b, sb = _batch(precision, SIZES)
    most = [0] * len(SIZES)
    for _ in range(8):
        a.propagate(0.1, device_loop=True)
        b.propagate(0.1, device_loop=False)
        for k, (x, y) in enumerate(zip(sa, sb)):
            assert a.last_move_attempts(x) == b.last_move_attempts(y)
            assert a.draws(x) == b.draws(y)
            assert np.array_equal(a.positions(x), b.positions(y))
            most[k] = max(most[k], a.last_move_attempts(x))
    # every replica was rejected at least once, so a round of eight attempts ran for each
    assert min(most) >= 2, most
