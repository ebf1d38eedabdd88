"""Attempt rounds of a batched step with many rejections: several attempts of a
replica in one round must leave exactly what one attempt after the other does
-- positions, attempts, draws -- for bead counts around the row and bead blocks
of the kernels and for attempt limits that end inside a round."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _crowd(seed, n):
    """n beads in a box at a volume fraction of 0.15, radii 5 .. 8 (the step used
    below moves a bead by a few tenths: most moves of larger crowds overlap)."""
    rng = np.random.default_rng(seed)
    radii = rng.uniform(5.0, 8.0, size=n)
    L = max(40.0, float((np.sum(4.0 / 3.0 * np.pi * radii ** 3) / 0.15) ** (1.0 / 3.0)))
    pos = np.empty((n, 3))
    for k in range(n):
        while True:
            p = rng.uniform(-L / 2, L / 2, size=3)
            d = pos[:k] - p
            d -= L * np.round(d / L)
            if np.all((d * d).sum(1) > (radii[:k] + radii[k] + 0.02) ** 2):
                break
        pos[k] = p
    return pos, radii, L


def _batch(precision, sizes, limit=10 ** 6, check=True):
    from pybrown_b200.batch import ReplicaBatch
    batch = ReplicaBatch(precision=precision)
    slots = []
    for k, n in enumerate(sizes):
        pos, radii, L = _crowd(50 + n, n)
        slots.append(batch.add(pos, radii, L, seed=1000 + k, noise="device", max_move_attempts=limit,
                               check_overlaps=check))
    return batch, slots


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_rounds_equal_attempts_in_a_row(precision):
    sizes = [1, 2, 7, 8, 9, 16, 21, 43, 64, 90]
    a, sa = _batch(precision, sizes)
    b, sb = _batch(precision, sizes)
    taken = 0
    for _ in range(4):
        a.propagate(0.4, device_loop=True)
        b.propagate(0.4, device_loop=False)
        for x, y in zip(sa, sb):
            assert a.last_move_attempts(x) == b.last_move_attempts(y)
            assert a.draws(x) == b.draws(y)
            assert np.array_equal(a.positions(x), b.positions(y))
            taken = max(taken, a.last_move_attempts(x))
    assert taken > 9  # a first attempt, a whole round after it and some more


@pytest.mark.parametrize("limit", [1, 2, 8, 9, 12])
def test_attempt_limit_inside_a_round(limit):
    """Replicas that use up their attempts keep the positions that the same
    rejected attempts, made one by one, leave."""
    sizes = [90, 64, 5]
    a, sa = _batch("fp64", sizes, limit)
    b, sb = _batch("fp64", sizes, limit)
    over = []
    for batch, loop in ((a, True), (b, False)):
        try:
            batch.propagate(6.0, device_loop=loop)  # far too long a step for the crowds
            over.append(False)
        except AssertionError:
            over.append(True)
    assert over == [True, True]
    for x, y in zip(sa, sb):
        assert a.last_move_attempts(x) == b.last_move_attempts(y) <= limit
        assert a.draws(x) == b.draws(y)
        assert np.array_equal(a.positions(x), b.positions(y))


def test_without_overlap_check():
    a, sa = _batch("mixed", [3, 30], check=False)
    a.propagate(0.4)
    assert [a.last_move_attempts(s) for s in sa] == [1, 1]
