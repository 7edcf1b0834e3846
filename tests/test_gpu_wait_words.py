"""The bounded waits of both contraction kernels and the words that they report
a timeout in.

sht_selftest_device_timeout runs the split kernel's own wait and then the FP64
kernels' own wait, each on a barrier that nothing arrives at;
sht_selftest_device_timeout_dev runs the FP64 one on the plan's stream and
returns, as a device call does.  In each block a second warp waits with the
full limit of two seconds and has to leave on the first one's abort flag, so a
run that takes much longer than its limit shows a flag that does not work."""
import time

import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu

TIMEOUT = 7


def test_both_kernels_waits_run_out_and_report():
    P = pkg()
    lib = P.load_library()
    s = P.SpmlUtil(64, 32, 1, 21)
    try:
        assert lib.sht_selftest_device_timeout(s._h, 1) == TIMEOUT  # builds the digit tables
        limit = 0.2
        t0 = time.perf_counter()
        assert lib.sht_selftest_device_timeout(s._h, int(1e3 * limit)) == TIMEOUT, lib.sht_last_error()
        dt = time.perf_counter() - t0
        assert 2 * limit <= dt < 2 * limit + 1.0, dt
        assert lib.sht_synchronize(s._h) == 0
    finally:
        s.final()


def test_fp64_wait_on_the_plans_stream():
    P = pkg()
    lib = P.load_library()
    s = P.SpmlUtil(64, 32, 1, 21)
    try:
        x = np.random.default_rng(1).standard_normal((3, 32, 64))
        want = s.wa_xya(x)
        assert lib.sht_selftest_device_timeout_dev(s._h, 0) == 1
        assert lib.sht_selftest_device_timeout_dev(s._h, 1001) == 1
        t0 = time.perf_counter()
        assert lib.sht_selftest_device_timeout_dev(s._h, 300) == 0
        assert time.perf_counter() - t0 < 0.2  # enqueued only
        assert lib.sht_synchronize(s._h) == TIMEOUT
        assert 0.3 <= time.perf_counter() - t0 < 1.3
        assert b"legendre" in lib.sht_last_error()
        assert lib.sht_synchronize(s._h) == 0
        assert np.array_equal(s.wa_xya(x), want)
    finally:
        s.final()


def test_timeouts_in_both_words_are_reported_once():
    P = pkg()
    lib = P.load_library()
    s = P.SpmlUtil(64, 32, 1, 21)
    try:
        x = np.random.default_rng(2).standard_normal((2, 32, 64))
        want = s.wa_xya(x)
        assert lib.sht_selftest_device_timeout(s._h, 1) == TIMEOUT  # builds the digit tables
        t0 = time.perf_counter()
        assert lib.sht_selftest_device_timeout_dev(s._h, 100) == 0
        assert lib.sht_synchronize(s._h) == TIMEOUT
        assert time.perf_counter() - t0 >= 0.2  # both waits ran
        assert lib.sht_synchronize(s._h) == 0
        assert np.array_equal(s.wa_xya(x), want)
    finally:
        s.final()
