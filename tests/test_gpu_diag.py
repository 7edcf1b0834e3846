"""The diagonal spectral operators on device tensors: entry counts around a
block of 256, level counts around a block of 8, the inverse Laplacian's zero
mode, and diffusion out of place (the input untouched) and in place, with and
without a filter, equal bit for bit to the same arithmetic in torch."""
import ctypes

import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("im,jm,nm", [(32, 16, 3), (32, 18, 14), (64, 32, 15), (48, 24, 15), (1, 32, 20)])
@pytest.mark.parametrize("nb", [1, 7, 8, 9, 40])
def test_diagonal_operators(im, jm, nm, nb):
    import torch

    P = pkg()
    lib = P.load_library()
    sp = P.SpmlUtil(im, jm, 1, nm)
    try:
        g = torch.Generator(device="cuda")
        g.manual_seed(im + nm + nb)
        rnd = lambda *s: torch.randn(s, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
        w, coef, filt = rnd(nb, sp.lm), -rnd(sp.lm).abs(), rnd(sp.lm)
        keep = w.clone()
        rn = torch.from_numpy(sp.rn).cuda()
        assert torch.equal(sp.w_Lapla_w(w), w * rn)
        assert torch.equal(sp.w_LaplaInv_w(w), torch.where(rn == 0, 0.0, w / torch.where(rn == 0, 1.0, rn)))
        assert torch.equal(sp.diffuse(w, coef, 0.5), w / (1.0 - 0.5 * coef))
        assert torch.equal(sp.diffuse(w, coef, 0.5, filt), filt * w / (1.0 - 0.5 * coef))
        assert torch.equal(w, keep)
        st = lib.sht_wa_diffuse_dev(sp._h, w.data_ptr(), nb, coef.data_ptr(), ctypes.c_double(0.5), None)
        sp.synchronize()
        assert st == 0 and torch.equal(w, keep / (1.0 - 0.5 * coef))
        assert lib.sht_wa_diffuse_to_dev(sp._h, w.data_ptr(), nb, coef.data_ptr(), ctypes.c_double(0.5), None, None) == 1
    finally:
        sp.final()
