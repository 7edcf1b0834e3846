"""The band Legendre kernels (the automatic FP64 choice) against the oracle
where a tile, a stage or a column block can go wrong: latitude halves and
degree counts around multiples of 8 and 16, the smallest bands, column counts
around 8, 16 and 32 (the warps split the rows of narrow batches), outputs tall
enough for several items per band, the axisymmetric plan, and non-finite
coefficients, which must stay in their own field-level.  Bound: 1e-11 per
field, the repository's bar."""
import numpy as np
import pytest

import oracle as O
from conftest import pkg, relerr, workloads

pytestmark = pytest.mark.gpu

TOL = 1e-11

# (im, jm, nm, nb): JH = jm/2 and (nm + 2)/2 rows around the tile edges
GRIDS = [(16, 6, 0, 1), (16, 10, 4, 7), (32, 14, 10, 8), (32, 18, 12, 9), (48, 30, 13, 15), (48, 34, 14, 17),
         (64, 46, 30, 31), (64, 50, 31, 33), (96, 62, 46, 24), (128, 126, 60, 41), (128, 130, 62, 5),
         (256, 136, 127, 3), (512, 250, 200, 2), (512, 514, 255, 1)]


@pytest.mark.parametrize("I,J,N,nb", GRIDS)
def test_band_kernels(I, J, N, nb):
    P, W = pkg(), workloads()
    sp = P.SpmlUtil(I, J, 1, N, None, 6.371e6)
    try:
        ora = O.OraclePlan(I, J, N, 6.371e6)
        rng = np.random.default_rng(I + J + N)
        w, w2 = W.seeded_spectra(N, nb, 1.0, rng=rng), W.seeded_spectra(N, nb, 1.0, rng=rng)
        x, y = rng.standard_normal((nb, J, I)), rng.standard_normal((nb, J, I))
        u, v = sp.calc_VorDiv2UV(w, w2)
        uo, vo = ora.vordiv2uv(w, w2)
        res = {"xy_w": relerr(sp.xya_wa(w), ora.xya_wa(w)), "w_xy": relerr(sp.wa_xya(x), ora.wa_xya(x)),
               "gradmu": relerr(sp.xya_GradMu_wa(w), ora.xya_gradmu_wa(w)),
               "alpha": relerr(sp.wa_AlphaOptr_xya(x, y), ora.wa_alphaoptr_xya(x, y))}
        if N > 0:
            res["u"], res["v"] = relerr(u, uo), relerr(v, vo)
        bad = {k: e for k, e in res.items() if not e < TOL}
        assert not bad, bad
    finally:
        sp.final()


@pytest.mark.parametrize("nb", [1, 8, 9, 33])
def test_non_finite_values_stay_in_their_level(nb):
    P, W = pkg(), workloads()
    I, J, N = 64, 36, 21
    sp = P.SpmlUtil(I, J, 1, N)
    try:
        w = W.seeded_spectra(N, nb, 1.0)
        g = sp.xya_wa(w)
        back = sp.wa_xya(g)
        bad = nb // 2
        wb, gb = w.copy(), g.copy()
        wb[bad, 5], gb[bad, 3, 7] = np.inf, np.nan
        g2, b2 = sp.xya_wa(wb), sp.wa_xya(gb)
        keep = np.arange(nb) != bad
        assert np.array_equal(g2[keep], g[keep]) and np.array_equal(b2[keep], back[keep])
        assert not np.isfinite(g2[bad]).all() and not np.isfinite(b2[bad]).all()
    finally:
        sp.final()
