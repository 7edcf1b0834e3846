"""The stage fills of the split-precision contraction: sub-items with several
K chunks and several pairs of output segments, whose stages are kept from one
pair to the next or come back from the digit cache.  Against the FP64
contraction of the same plan (itself tested against the oracle), to the
documented 1e-11 of the split mode, and bit for bit against the same columns in
another batch (the level sums are exact integers, so neither the order of the
chunks nor the place in a tile may show)."""
import numpy as np
import pytest

from conftest import pkg, relerr, workloads

TOL = 1e-11

pytestmark = pytest.mark.gpu

# analysis: K = jm/2 latitudes, up to (nm+3)/2 rows; synthesis: the reverse
GRIDS = [
    (512, 646, 170),  # 323 terms (odd, six chunks, the last of 3) x 86 rows; 86 terms (two chunks) x 323 rows
    (800, 402, 266),  # 201 terms (odd, four chunks) x 134 rows; 134 terms (three chunks) x 201 rows
    (640, 480, 213),  # 240 terms (32-byte loads) x 108 rows; 108 terms x 240 rows
    (256, 130, 85),   # 65 terms (two chunks, the last of 1) x 44 rows; 44 terms x 65 rows (three segments)
]


@pytest.mark.parametrize("grid", GRIDS)
def test_stage_fills_vs_fp64(grid):
    P, W = pkg(), workloads()
    I, J, N = grid
    gpu = P.SpmlUtil(I, J, 1, N, None, 1.0)
    try:
        nb = 65  # one column past a tile
        rng = np.random.default_rng(N)
        w = W.seeded_spectra(N, nb, 2.0, rng=rng)
        x = rng.standard_normal((nb, J, I))
        g64, w64 = gpu.xya_wa(w), gpu.wa_xya(x)
        gpu.set_precision(P.SHT_PREC_SPLIT)
        g, c = gpu.xya_wa(w), gpu.wa_xya(x)
        gpu.synchronize()  # reads the error word of the bounded waits
        assert relerr(g, g64) < TOL
        assert relerr(c, w64) < TOL
        assert np.array_equal(gpu.xya_wa(w[-3:]), g[-3:])
        assert np.array_equal(gpu.wa_xya(x[-3:]), c[-3:])
    finally:
        gpu.final()
