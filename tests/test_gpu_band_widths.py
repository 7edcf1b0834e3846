"""The FP64 contraction gives a field-level the same bits whatever batch it is
in: the narrow-batch kernels (m8n8k4 products), the band kernels with the warps
splitting the rows (small batches) or the columns (large ones), in m16n8k8
products for pairs of row tiles and m8n8k4 for an odd one or a tail of up to
four terms, one block of three teams or three of one, and any share of the SMs.
That holds because an m16n8k8 product accumulates its two halves in the order
of two m8n8k4 products; nothing in the code rounds differently.  And T341 in
FP64 against the oracle (1e-11 per field, the repository's bar)."""
import numpy as np
import pytest

import oracle as O
from conftest import pkg, relerr, workloads

pytestmark = pytest.mark.gpu

# row tiles per parity (analysis) and latitude tiles (synthesis), odd and even,
# up to 8 in one item and several items; degree counts that leave tails of 1..16
GRIDS = [(16, 8, 5, 100), (64, 34, 21, 300), (96, 48, 31, 300), (128, 72, 62, 300), (192, 104, 63, 200), (256, 128, 85, 200),
         (256, 128, 86, 200), (384, 200, 127, 90), (400, 210, 128, 90), (512, 256, 170, 70)]


@pytest.mark.parametrize("I,J,N,nb", GRIDS)
def test_same_bits_in_any_batch(I, J, N, nb):
    import torch

    P = pkg()
    sp = P.SpmlUtil(I, J, 1, N)
    try:
        g = torch.Generator(device="cuda")
        g.manual_seed(N)
        w = torch.randn((nb, sp.lm), generator=g, device="cuda", dtype=torch.float64)
        v = torch.randn((nb, sp.lm), generator=g, device="cuda", dtype=torch.float64)
        x = sp.xy_w(w)
        c, u = sp.w_xy(x), sp.calc_VorDiv2UV(w, v)
        for n in (1, 2, 5, 8, 9, 17, 33, 64):
            for k in (0, (nb - n) // 2, nb - n):
                s = slice(k, k + n)
                assert torch.equal(sp.xy_w(w[s]), x[s]), (n, k)
                assert torch.equal(sp.w_xy(x[s]), c[s]), (n, k)
                assert all(torch.equal(a, b[s]) for a, b in zip(sp.calc_VorDiv2UV(w[s], v[s]), u)), (n, k)
    finally:
        sp.final()


def test_same_bits_on_a_share_of_the_sms():
    import torch

    P = pkg()
    grids = [(128, 64, 42, 70), (256, 128, 85, 40), (512, 256, 170, 20)]
    plans = [P.SpmlUtil(*d[:2], 1, d[2]) for d in grids]
    m = P.MultiTransform()
    try:
        g = torch.Generator(device="cuda")
        g.manual_seed(11)
        ws = [torch.randn((d[3], sp.lm), generator=g, device="cuda", dtype=torch.float64) for d, sp in zip(grids, plans)]
        arrays = [(w.clone(), torch.empty((d[3], d[1], d[0]), device="cuda", dtype=torch.float64)) for d, w in zip(grids, ws)]
        for sp, (w, x) in zip(plans, arrays):
            m.add(sp, w, x)
        m.build(autotune=False, side_by_side=True)
        assert all(0 < s["sms"] < 148 for s in m.groups())
        for w, (a, _) in zip(ws, arrays):
            a.copy_(w)
        torch.cuda.synchronize()
        m.run()
        m.synchronize()
        for sp, w, (a, x) in zip(plans, ws, arrays):
            ref = sp.xy_w(w)
            assert torch.equal(x, ref) and torch.equal(a, sp.w_xy(ref))
    finally:
        m.close()
        for sp in plans:
            sp.final()


@pytest.mark.parametrize("nb", [1, 19])
def test_t341_fp64_against_the_oracle(nb):
    P, W = pkg(), workloads()
    I, J, N = 1024, 512, 341
    sp = P.SpmlUtil(I, J, 1, N)
    try:
        ora = O.OraclePlan(I, J, N)
        rng = np.random.default_rng(nb)
        w, w2 = W.seeded_spectra(N, nb, 1.0, rng=rng), W.seeded_spectra(N, nb, 1.0, rng=rng)
        x = rng.standard_normal((nb, J, I))
        assert relerr(sp.xya_wa(w), ora.xya_wa(w)) < 1e-11
        assert relerr(sp.wa_xya(x), ora.wa_xya(x)) < 1e-11
        assert relerr(sp.xya_GradMu_wa(w2), ora.xya_gradmu_wa(w2)) < 1e-11
    finally:
        sp.final()
