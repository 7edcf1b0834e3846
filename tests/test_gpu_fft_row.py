"""The longitude transforms of im = 64 to 1024 (whole rows and mirrored pairs
as one complex row) against the oracle: row pairs that do not fill a tile, the
smallest and the largest truncation a count allows (im = 2 nm + 2), and the
product and multiply-add load modes.  Bound: 1e-11 per field."""
import numpy as np
import pytest

import oracle as O
from conftest import pkg, relerr, workloads

pytestmark = pytest.mark.gpu

TOL = 1e-11

# (im, jm, nm, nb)
GRIDS = [(64, 2, 0, 3), (64, 34, 31, 9), (64, 66, 21, 20), (128, 18, 1, 2), (128, 66, 63, 5), (128, 80, 42, 7),
         (256, 30, 3, 3), (256, 130, 127, 2), (256, 140, 85, 4), (512, 26, 2, 2), (512, 258, 255, 1),
         (512, 180, 170, 2), (1024, 14, 5, 2), (1024, 514, 511, 1), (1024, 350, 341, 1)]


@pytest.mark.parametrize("I,J,N,nb", GRIDS)
def test_row_transforms(I, J, N, nb):
    P, W = pkg(), workloads()
    sp = P.SpmlUtil(I, J, 1, N, None, 6.371e6)
    try:
        ora = O.OraclePlan(I, J, N, 6.371e6)
        rng = np.random.default_rng(I + 7 * J + N)
        w = W.seeded_spectra(N, nb, 1.0, rng=rng)
        x, y, q, z1, z2 = (rng.standard_normal((nb, J, I)) for _ in range(5))
        cs = np.cos(sp.y_Lat)[None, :, None]
        res = {"xy_w": relerr(sp.xya_wa(w), ora.xya_wa(w)), "w_xy": relerr(sp.wa_xya(x), ora.wa_xya(x))}
        if N > 0:
            res["prod"] = relerr(sp.w_AlphaOptrProd_xy(x, y, q), ora.wa_alphaoptr_xya(x * q, y * q))
            v, d = sp.calc_UVCosLat2VorDiv_fma(x, y, q, z1, z2)
            vo, do = ora.uvcoslat2vordiv(cs * (x * q + z1), cs * (y * q + z2))
            res["vor"], res["div"] = relerr(v, vo), relerr(d, do)
        bad = {k: e for k, e in res.items() if not e < TOL}
        assert not bad, bad
    finally:
        sp.final()
