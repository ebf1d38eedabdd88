"""The wait-expiry self-test at the smallest poll limits: the waits that depend on
other CTAs give up at once, those inside one tile's factorisation do not (they
would read panels that are not there and report a pivot), so the aborted launch
always reports info = -1 and the barrier bit, and the next factorisation
succeeds."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu
PBG_DEV_ERR_BARRIER = 2


@pytest.mark.parametrize("limit", [1, 2, 3, 16, 200])
def test_small_limits_report_the_expired_wait(limit):
    from pybrown_b200 import _lib
    info, err = ctypes.c_int(0), ctypes.c_uint(0)
    for _ in range(5):
        assert _lib.lib.pbg_selftest_wait_expiry(limit, ctypes.byref(info), ctypes.byref(err)) == 0, _lib.last_error()
        assert info.value == -1 and err.value & PBG_DEV_ERR_BARRIER
