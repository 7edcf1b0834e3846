"""Device memory of a plan: one Legendre table, not two.  A plan may hold its
table (padded to whole 8 x 8 blocks), and a tenth more for everything else; the
first split-precision call allocates digit tables beside it, sized by the same
table (seven digit bytes per value and direction) and a cache per SM."""
import ctypes

import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu

SLACK = 8 << 20  # allocation granularity and the driver's own


def table_bytes(N, JH, orders):
    tiles = sum(((r + 1) // 2 + 7) // 8 + (r // 2 + 7) // 8 for r in (N + 2 - m for m in range(orders)))
    return 512 * tiles * ((JH + 7) // 8)


@pytest.mark.parametrize("im,jm,nm", [(1024, 512, 341), (640, 320, 213), (1, 512, 341)])
def test_one_legendre_table(im, jm, nm):
    import torch

    P = pkg()
    lib = P.load_library()
    warm = P.SpmlUtil(64, 32, 1, 21)  # the library's own first allocations
    try:
        torch.cuda.synchronize()
        free0 = torch.cuda.mem_get_info()[0]
        h = ctypes.c_void_p()
        assert lib.sht_init(im, jm, 1, nm, 1.0, ctypes.byref(h)) == 0
        torch.cuda.synchronize()
        used = free0 - torch.cuda.mem_get_info()[0]
        assert lib.sht_final(h) == 0
        most = 1.1 * table_bytes(nm, jm // 2, 1 if im == 1 else nm + 1) + SLACK
        assert used <= most, (used, most)
    finally:
        warm.final()
