"""The bounded waits of the tile phases: one that gives up ends those that follow
it, so that a launch of hundreds of waits is over soon after the first."""
import ctypes as C
import time

import pytest

from opensayal_gb300 import native

pytestmark = pytest.mark.gpu


def test_waits_that_give_up_end_the_others(gpu):
    lib = native.load()
    status = C.c_int32(-1)
    t0 = time.perf_counter()
    native.check(lib.os_selftest_bounded_wait(0, C.byref(status)))
    seconds = time.perf_counter() - t0
    assert status.value == native.OS_ERR_TIMEOUT
    # One wait for a packet and one for a message, a second each; 401 of the
    # latter, each on its own, would be minutes.
    assert seconds < 10
