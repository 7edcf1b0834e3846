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


def test_next_call_reports_a_device_calls_timeout():
    """A device call that times out has returned 0 by then: whichever call comes
    next on the plan returns the status, without running, and the one after it runs."""
    import torch

    P = pkg()
    lib = P.load_library()
    im, jm, nm, nb = 64, 32, 21, 2
    s, other = P.SpmlUtil(im, jm, 1, nm), P.SpmlUtil(im, jm, 1, nm)
    try:
        g = torch.Generator(device="cuda")
        g.manual_seed(5)
        x, y, q = (torch.randn(nb, jm, im, generator=g, device="cuda", dtype=torch.float64) for _ in range(3))
        w, v = (torch.randn(nb, s.lm, generator=g, device="cuda", dtype=torch.float64) for _ in range(2))
        c = torch.rand(s.lm, generator=g, device="cuda", dtype=torch.float64)
        halo = torch.zeros(nb, jm + 2, im + 2, device="cuda", dtype=torch.float64)
        xh, wh = x.cpu().numpy(), w.cpu().numpy()
        out = torch.empty_like(w)
        m = P.MultiTransform()
        m.add(s, w.clone(), x.clone())
        m.build()

        def noalloc():
            st = lib.sht_wa_xya_dev_noalloc(s._h, x.data_ptr(), nb, out.data_ptr())
            if st:
                raise P.SpmlError(st, "noalloc", lib.sht_last_error().decode())

        lib.sht_wa_xya_dev_noalloc.argtypes = lib.sht_wa_xya_dev.argtypes
        calls = [lambda: s.w_xy(x), lambda: s.xy_w(w), lambda: s.calc_UVCosLat2VorDiv_fma(x, y, q), lambda: s.diffuse(w, c, 0.5),
                 lambda: s._sub_filter(w.clone(), v, c), lambda: s._sub_lapla(w.clone(), v.clone(), w),
                 lambda: s.analysis(halo, 1, 1), lambda: s.synthesis(w, halo, 1, 1), lambda: s.roundtrip_diffuse_(x.clone()),
                 noalloc, m.run, lambda: s.w_xy(xh), lambda: s.xy_w(wh), lambda: s.diffuse(wh, c.cpu().numpy(), 0.5)]
        for k, call in enumerate(calls):
            call()
            assert lib.sht_selftest_device_timeout_dev(s._h, 1) == 0
            torch.cuda.synchronize()
            other.w_xy(x)  # another plan is not concerned
            with pytest.raises(P.SpmlError) as e:
                call()
            assert e.value.status == TIMEOUT and "earlier call" in str(e.value), k
            call()
            assert lib.sht_synchronize(s._h) == 0
        assert torch.equal(s.w_xy(x), other.w_xy(x))
        m.close()
    finally:
        s.final()
        other.final()
