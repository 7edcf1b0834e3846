"""The narrow-batch kernels (contraction and layout conversion in one) against
the oracle for every analysis and synthesis operator: level counts around a
block's two and four, latitude and degree counts around its 8-row tiles, both
sides of the size at which wider batches leave them, the axisymmetric plan,
and the same bits one level at a time as in a batch that takes the wide
path.  Bound: 1e-11 per field."""
import numpy as np
import pytest

import oracle as O
from conftest import pkg, relerr, workloads

pytestmark = pytest.mark.gpu

TOL = 1e-11

# (im, jm, nm, levels)
GRIDS = [(16, 6, 1, (1, 5)), (32, 18, 13, (1, 4, 5)), (48, 30, 14, (2, 3)), (64, 34, 30, (1, 8, 9)),
         (128, 64, 42, (1, 60)), (256, 128, 85, (1, 3, 30, 31, 60, 61)), (320, 160, 106, (2,)), (512, 256, 170, (1, 9))]


@pytest.mark.parametrize("I,J,N,levels", GRIDS)
def test_narrow_operators(I, J, N, levels):
    P, W = pkg(), workloads()
    a = 6.371e6
    sp = P.SpmlUtil(I, J, 1, N, None, a)
    try:
        ora = O.OraclePlan(I, J, N, a)
        for nb in levels:
            rng = np.random.default_rng(N + nb)
            w, w2 = W.seeded_spectra(N, nb, 1.0, rng=rng), W.seeded_spectra(N, nb, 1.0, rng=rng)
            x, y = rng.standard_normal((nb, J, I)), rng.standard_normal((nb, J, I))
            pairs = {"w_xy": (sp.wa_xya(x), ora.wa_xya(x)), "xy_w": (sp.xya_wa(w), ora.xya_wa(w)),
                     "divlam": (sp.wa_DivLambda_xya(x), ora.wa_divlambda_xya(x)),
                     "divmu": (sp.wa_DivMu_xya(x), ora.wa_divmu_xya(x)),
                     "alpha_w": (sp.wa_AlphaOptr_xya(x, y), ora.wa_alphaoptr_xya(x, y)),
                     "alpha_x": (sp.xya_AlphaOptr_wa(w, w2), ora.xya_alphaoptr_wa(w, w2)),
                     "gradlam": (sp.xya_GradLambda_wa(w), ora.xya_gradlambda_wa(w)),
                     "gradmu": (sp.xya_GradMu_wa(w), ora.xya_gradmu_wa(w))}
            lon, lat = sp.xy_HGrad_w(w)
            pairs["hgrad_lon"], pairs["hgrad_lat"] = (lon, ora.xya_gradlon_wa(w)), (lat, ora.xya_gradlat_wa(w))
            for k, g, o in zip("UV", sp.calc_VorDiv2UV(w, w2), ora.vordiv2uv(w, w2)):
                pairs[k] = (g, o)
            for k, g, o in zip(("vor", "div"), sp.calc_UVCosLat2VorDiv(x, y), ora.uvcoslat2vordiv(x, y)):
                pairs[k] = (g, o)
            bad = {k: relerr(g, o) for k, (g, o) in pairs.items() if not relerr(g, o) < TOL}
            assert not bad, (nb, bad)
    finally:
        sp.final()


def test_one_level_equals_the_batch():
    import torch

    P, W = pkg(), workloads()
    for I, J, N, nb in ((256, 128, 85, 200), (1, 64, 42, 700)):
        sp = P.SpmlUtil(I, J, 1, N)
        try:
            g = torch.Generator(device="cuda")
            g.manual_seed(3)
            w = torch.randn((nb, sp.lm), generator=g, device="cuda", dtype=torch.float64)
            x = sp.xy_w(w)
            c = sp.w_DivMu_xy(x)
            for k in (0, 7, nb - 1):
                assert torch.equal(sp.xy_w(w[k:k + 1]), x[k:k + 1])
                assert torch.equal(sp.w_DivMu_xy(x[k:k + 1]), c[k:k + 1])
        finally:
            sp.final()


def test_non_finite_values_stay_in_their_level():
    P, W = pkg(), workloads()
    I, J, N, nb = 64, 36, 21, 3
    sp = P.SpmlUtil(I, J, 1, N)
    try:
        w = W.seeded_spectra(N, nb, 1.0)
        g = sp.xya_wa(w)
        back = sp.wa_xya(g)
        wb, gb = w.copy(), g.copy()
        wb[1, 5], gb[1, 3, 7] = np.inf, np.nan
        g2, b2 = sp.xya_wa(wb), sp.wa_xya(gb)
        for k in (0, 2):
            assert np.array_equal(g2[k], g[k]) and np.array_equal(b2[k], back[k])
        assert not np.isfinite(g2[1]).all() and not np.isfinite(b2[1]).all()
    finally:
        sp.final()
