"""Host-pointer calls on pageable arrays: grids up to 16 KB are copied, larger
ones are read and written in place in the staging buffer.  Results equal the
device-pointer calls bit for bit, for one and two inputs and outputs, odd
spectral lengths, first (direct) and repeated (graph) calls, with stage timing
on (copies), and from page-locked arrays."""
import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu

# 16 x 8 and 64 x 32: up to 16 KB per level; 64 x 34: just above; mixed radix, zonal, direct sums
GRIDS = [(16, 8, 5), (64, 32, 20), (64, 34, 21), (96, 48, 31), (256, 128, 84), (1, 32, 20), (44, 22, 14), (1024, 64, 20)]


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("nb", [1, 3])
def test_host_calls_equal_device_calls(grid, nb):
    import torch

    P = pkg()
    im, jm, nm = grid
    sp = P.SpmlUtil(im, jm, 1, nm, None, 6.4e6)
    try:
        rng = np.random.default_rng(im + nb)
        w, w2 = rng.standard_normal((2, nb, sp.lm))
        x, y = rng.standard_normal((2, nb, jm, im))
        calls = [(sp.xy_w, (w,)), (sp.w_xy, (x,)), (sp.w_AlphaOptr_xy, (x, y)), (sp.calc_UVCosLat2VorDiv, (x, y)),
                 (sp.calc_VorDiv2UV, (w, w2)), (sp.xy_AlphaOptr_w, (w, w2)), (sp.w_AlphaOptrProd_xy, (x, y, x)),
                 (sp.xy_HGrad_xy, (x,)), (sp.xy_FluxDiv_xy, (x, y)), (sp.AvrLonLat_xy, (x,))]
        for fn, args in calls:
            dev = fn(*[torch.from_numpy(a).cuda() for a in args])
            dev = [d.cpu().numpy() for d in (dev if isinstance(dev, tuple) else (dev,))]
            keep = [a.copy() for a in args]

            def same(out):
                return all(np.array_equal(o, d) for o, d in zip(out if isinstance(out, tuple) else (out,), dev))

            for _ in range(4):
                assert same(fn(*args)), fn.__name__
            assert same(fn(*[torch.from_numpy(a).pin_memory().numpy() for a in args])), fn.__name__
            sp.set_timing(True)
            assert same(fn(*args)), fn.__name__
            sp.set_timing(False)
            assert same(fn(*args)), fn.__name__
            assert all(np.array_equal(a, k) for a, k in zip(args, keep))
    finally:
        sp.final()
