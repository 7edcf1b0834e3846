"""The one-pass spectral tails of the batched tendencies, equal bit for bit to
the separate passes (same products and differences, rounded one by one), at
level counts around a block of 8 and with non-finite entries; and the tendency
functions with arguments that the one-pass form does not take."""
import importlib

import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [1, 7, 8, 9, 40])
def test_tails_equal_separate_passes(nb):
    import torch

    P = pkg()
    sp = P.SpmlUtil(64, 32, 1, 21)
    try:
        g = torch.Generator(device="cuda")
        g.manual_seed(nb)
        rnd = lambda *s: torch.randn(s, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
        a, b, c, f = rnd(nb, sp.lm), rnd(nb, sp.lm), rnd(nb, sp.lm), rnd(sp.lm)
        a[0, 3], c[0, 5], b[-1, 0] = float("nan"), float("inf"), -0.0
        same = lambda x, y: torch.equal(x.view(torch.int64), y.view(torch.int64))  # noqa: E731
        ref = (a - b) * f[None, :]
        out = sp._sub_filter(a.clone(), b, f)
        assert same(torch.nan_to_num(out, nan=7.0), torch.nan_to_num(ref, nan=7.0))
        p, q = sp._sub_lapla(a.clone(), b.clone(), c)
        assert same(torch.nan_to_num(p, nan=7.0), torch.nan_to_num(a - sp.w_Lapla_w(c), nan=7.0))
        assert same(q, -b)
    finally:
        sp.final()


def test_other_arguments_take_the_separate_passes():
    import torch

    P, C = pkg(), importlib.import_module("dennou-ogcm_b200.callers")
    sp = P.SpmlUtil(64, 32, 1, 21)
    try:
        g = [torch.randn(3, 32, 64, dtype=torch.float64, device="cuda") for _ in range(5)]
        f = torch.rand(sp.lm, dtype=torch.float64, device="cuda")
        ref = C.htrc_rhs(sp, *g[:4], f, g[4])
        # a strided filter, and numpy arrays throughout
        strided = torch.stack([f, f], 1)[:, 0]
        assert not strided.is_contiguous()
        assert torch.equal(C.htrc_rhs(sp, *g[:4], strided, g[4]), ref)
        host = [x.cpu().numpy() for x in g]
        out = C.htrc_rhs(sp, *host[:4], f.cpu().numpy(), host[4])
        assert abs(out - ref.cpu().numpy()).max() <= 1e-13 * float(ref.abs().max())
        u, v = C.momrhs_vordiv(sp, *g[:3])
        uh, vh = C.momrhs_vordiv(sp, *host[:3])
        scale = max(float(u.abs().max()), float(v.abs().max()))
        assert abs(uh - u.cpu().numpy()).max() <= 1e-13 * scale and abs(vh - v.cpu().numpy()).max() <= 1e-13 * scale
    finally:
        sp.final()
