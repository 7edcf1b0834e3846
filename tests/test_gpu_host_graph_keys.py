"""Staged host calls keep one graph per piece of work: option values that run the
same kernels (the tile option, Legendre kernels 0 to 3) share it, the
single-kernel transform (4, or 0 where it is the automatic choice) has its own."""
import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,small_is_automatic", [((64, 32, 21), False), ((32, 16, 10), True)])
def test_options_that_change_nothing_share_a_graph(grid, small_is_automatic):
    P = pkg()
    sp = P.SpmlUtil(grid[0], grid[1], 1, grid[2])
    try:
        x = np.random.default_rng(8).standard_normal((grid[1], grid[0]))

        def calls():
            out = [sp.w_xy(x) for _ in range(3)]
            assert all(np.array_equal(o, out[0]) for o in out)
            return out[0]

        band, small = {}, {}
        for tile in (0, 8, 32):
            sp.set_option(P.SHT_OPT_LEGENDRE_TILE, tile)
            for kern in (1, 2, 3, 0, 4):
                sp.set_option(P.SHT_OPT_LEGENDRE_KERNEL, kern)
                one_kernel = kern == 4 or (kern == 0 and small_is_automatic)
                (small if one_kernel else band)[tile, kern] = calls()
                assert sp.get_option(P.SHT_OPT_LEGENDRE_TILE) == tile
        assert sp.get_option(P.SHT_OPT_HOST_GRAPH_COUNT) == 2
        for group in (band, small):
            first = next(iter(group.values()))
            assert all(np.array_equal(v, first) for v in group.values())
    finally:
        sp.final()
