"""The mixed-radix longitude transforms (im with factors 3 and 5) against the
oracle, whose transform of such counts is a direct sum: every radix of both
classes (up to 16, and 18 to 32), odd half counts, row pairs that do not fill
a tile, the largest and smallest truncations, and the product and
multiply-add load modes.  A count with another prime factor (112 = 16 * 7)
keeps the direct sum.  Bound: 1e-11 per field, the repository's bar.
"""
import numpy as np
import pytest

import oracle as O
from conftest import pkg, relerr, workloads

pytestmark = pytest.mark.gpu

TOL = 1e-11

# (im, jm, nm, nb)
GRIDS = [(18, 10, 5, 3), (20, 10, 9, 3), (24, 12, 7, 2), (30, 16, 14, 5), (36, 18, 11, 3), (50, 26, 16, 2),
         (54, 26, 17, 2), (90, 46, 29, 3), (96, 48, 31, 40), (100, 50, 33, 3), (112, 56, 37, 2), (160, 78, 53, 5),
         (180, 90, 59, 2), (240, 120, 79, 9), (320, 160, 106, 4), (360, 100, 90, 2), (384, 130, 127, 2),
         (480, 162, 159, 2), (540, 100, 90, 2), (640, 100, 99, 3), (720, 82, 80, 2), (750, 60, 50, 2),
         (810, 60, 50, 2), (960, 66, 64, 2), (1250, 40, 30, 2), (1280, 66, 64, 1), (1536, 40, 39, 2),
         (1620, 40, 30, 1), (1800, 40, 30, 1), (1920, 66, 65, 2), (1944, 30, 20, 1)]


@pytest.mark.parametrize("I,J,N,nb", GRIDS)
def test_mixed_radix_transforms(I, J, N, nb):
    P, W = pkg(), workloads()
    sp = P.SpmlUtil(I, J, 1, N, None, 6.371e6)
    try:
        ora = O.OraclePlan(I, J, N, 6.371e6)
        rng = np.random.default_rng(20261205 + I)
        w = W.seeded_spectra(N, nb, 1.0, rng=rng)
        x, y, q = (rng.standard_normal((nb, J, I)) for _ in range(3))
        z1, z2 = rng.standard_normal((nb, J, I)), rng.standard_normal((nb, J, I))
        cs = np.cos(sp.y_Lat)[None, :, None]
        res = {"xy_w": relerr(sp.xya_wa(w), ora.xya_wa(w)), "w_xy": relerr(sp.wa_xya(x), ora.wa_xya(x)),
               "prod": relerr(sp.w_AlphaOptrProd_xy(x, y, q), ora.wa_alphaoptr_xya(x * q, y * q))}
        v, d = sp.calc_UVCosLat2VorDiv_fma(x, y, q, z1, z2)
        vo, do = ora.uvcoslat2vordiv(cs * (x * q + z1), cs * (y * q + z2))
        res["vor"], res["div"] = relerr(v, vo), relerr(d, do)
        bad = {k: e for k, e in res.items() if not e < TOL}
        assert not bad, bad
    finally:
        sp.final()


def test_longitude_points_beyond_the_truncation():
    # the longest truncation a count allows (im = 2 nm + 2): both Z_k and
    # Z_{NC-k} of every pair carry an order
    P, W = pkg(), workloads()
    I, J, N = 96, 52, 47
    sp = P.SpmlUtil(I, J, 1, N, None, 1.0)
    try:
        ora = O.OraclePlan(I, J, N, 1.0)
        w = W.seeded_spectra(N, 3, 0.5)
        g = ora.xya_wa(w)
        assert relerr(sp.xya_wa(w), g) < TOL
        assert relerr(sp.wa_xya(g), ora.wa_xya(g)) < TOL
    finally:
        sp.final()
