"""Split-precision analyses of fewer latitudes than a contraction chunk (64),
which have an instance of their own: latitude counts around the 16 of a
converting thread, odd ones (8-byte loads) among them, and columns around the
64 of a tile, against the oracle; non-finite values stay in their column; an
instance for longer contractions on the other side of the line."""
import numpy as np
import pytest

import oracle as O
from conftest import pkg, relerr

pytestmark = pytest.mark.gpu

TOL = 1e-11  # the split mode's documented bound per field

# (im, jm / 2, nm)
GRIDS = [(16, 3, 3), (16, 8, 5), (16, 15, 5), (32, 16, 10), (32, 17, 10), (64, 31, 21), (64, 32, 30), (48, 33, 15),
         (96, 47, 31), (96, 48, 31), (96, 49, 31), (128, 63, 42), (128, 64, 42), (1, 17, 20), (1, 63, 42)]


@pytest.mark.parametrize("im,JH,nm", GRIDS)
def test_short_analyses(im, JH, nm):
    P = pkg()
    jm = 2 * JH
    sp = P.SpmlUtil(im, jm, 1, nm)
    try:
        sp.set_precision(P.SHT_PREC_SPLIT)
        rng = np.random.default_rng(100 * im + JH)
        if im > 1:
            ora = O.OraclePlan(im, jm, nm)
            ref = lambda x: ora.wa_xya(x)  # noqa: E731
        else:  # the axisymmetric plan against FP64 arithmetic of the same library
            fp = P.SpmlUtil(im, jm, 1, nm)
            ref = lambda x: fp.wa_xya(x)  # noqa: E731
        for nb in (1, 63, 65):
            x = rng.standard_normal((nb, jm, im)) * 10.0 ** rng.integers(-6, 7, (nb, 1, 1))
            w = sp.wa_xya(x)
            assert relerr(w, ref(x)) < TOL, nb
            if nb > 1:
                y = x.copy()
                y[1, jm // 3, im // 2] = np.nan
                v = sp.wa_xya(y)
                assert all(np.array_equal(v[k], w[k]) for k in range(nb) if k != 1)
    finally:
        sp.final()
