"""The merged task list of a batch as the library builds it (host only, no GPU):
every replica's segments exactly once and in their own order, in all merge orders,
so that each replica's part replays with every wait satisfied (test_task_lists)."""
import ctypes

import numpy as np
import pytest

from test_task_lists import (PREC_FP64, PREC_MIXED, _lib, replay_left_looking, replay_right_looking, task_list)

ORDERS = 7
TILE_COUNTS = [[1], [5, 5, 5, 5], [1, 24], [24, 1, 2, 3, 1, 7], [3, 8, 2, 8, 5, 1, 13, 11, 2]]


def merge(precision, order, nts, cap=None):
    lib = _lib()
    cap = cap if cap is not None else 4 * sum(nts) + 8 * len(nts)
    out, n = (ctypes.c_int * (2 * max(cap, 1)))(), ctypes.c_int()
    rc = lib.pbg_cholesky_merge_list(precision, order, (ctypes.c_int * max(len(nts), 1))(*nts), len(nts), out, cap,
                                     ctypes.byref(n))
    return rc, n.value, [(out[2 * e], out[2 * e + 1]) for e in range(min(n.value, cap))]


@pytest.mark.parametrize("precision", [PREC_MIXED, PREC_FP64])
@pytest.mark.parametrize("order", range(ORDERS))
@pytest.mark.parametrize("nts", TILE_COUNTS + [[96, 1, 40]])
def test_every_segment_once_and_in_order(precision, order, nts):
    if precision == PREC_FP64 and max(nts) > 24:
        nts = [min(nt, 30) for nt in nts]
    rc, n, merged = merge(precision, order, nts)
    assert rc == 0
    lists = [task_list(nt, precision) for nt in nts]
    assert n == sum(len(seg) - 1 for _, seg in lists)
    replay = replay_left_looking if precision == PREC_MIXED else replay_right_looking
    for q, (tasks, seg) in enumerate(lists):
        own = [s for r, s in merged if r == q]
        assert own == list(range(len(seg) - 1))
        mine = np.concatenate([tasks[seg[s]:seg[s + 1]] for s in own])
        done = replay(nts[q], mine)
        assert sorted(done) == sorted((r, c) for c in range(nts[q]) for r in range(c, nts[q]))


@pytest.mark.parametrize("order", [0, 1, 2])
def test_spread_over_the_longest(order):
    """Segment s of n stands where segment s longest / n of the longest stands."""
    nts = [3, 8, 2, 8, 5, 1, 13, 11, 2]
    _, _, merged = merge(PREC_MIXED, order, nts)
    longest = 2 * max(nts)
    place = [s * longest // (2 * nts[q]) for q, s in merged]
    assert place == sorted(place)


def test_refused_arguments():
    assert merge(PREC_MIXED, 0, [])[0] == -2
    assert merge(PREC_MIXED, ORDERS, [3])[0] == -2 and merge(PREC_MIXED, -1, [3])[0] == -2
    assert merge(PREC_MIXED, 0, [3, 0])[0] == -2
    rc, n, _ = merge(PREC_MIXED, 0, [3, 2], cap=9)
    assert rc == -2 and n == 10
