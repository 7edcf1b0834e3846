"""Layout conversions of axisymmetric plans in wide batches (their own kernels,
a thread per degree and level): the same bits as one level at a time, which takes
the narrow-batch kernels and their own conversion, for every operator, at degree
counts around a block's 8 and level counts around its 32; non-finite values stay
in their level; and batches registered by column tables."""
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu

# (jm, nm, levels): more levels than the narrow-batch kernels take
GRIDS = [(16, 5, 6017), (16, 6, 5313), (16, 7, 4705), (64, 41, 640), (64, 42, 671), (130, 85, 225)]


@pytest.mark.parametrize("jm,nm,nb", GRIDS)
def test_batch_equals_single_levels(jm, nm, nb):
    import torch

    P = pkg()
    sp = P.SpmlUtil(1, jm, 1, nm, None, 6.371e6)
    try:
        assert (nb + 3) // 4 * (nm + 2) * (jm // 2) > 84000
        g = torch.Generator(device="cuda")
        g.manual_seed(nb)
        rnd = lambda *s: torch.randn(s, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
        x, y, q, w, v = rnd(nb, jm, 1), rnd(nb, jm, 1), rnd(nb, jm, 1), rnd(nb, sp.lm), rnd(nb, sp.lm)
        x[1, jm // 2], w[1, 0] = float("nan"), float("inf")
        calls = {"w_xy": (sp.w_xy, x), "divlam": (sp.w_DivLambda_xy, x), "divmu": (sp.w_DivMu_xy, x),
                 "alpha": (sp.w_AlphaOptr_xy, x, y), "prod": (sp.w_AlphaOptrProd_xy, x, y, q),
                 "vordiv": (sp.calc_UVCosLat2VorDiv, x, y), "xy_w": (sp.xy_w, w), "gradlam": (sp.xy_GradLambda_w, w),
                 "gradmu": (sp.xy_GradMu_w, w), "hgrad": (sp.xy_HGrad_w, w), "alpha_w": (sp.xy_AlphaOptr_w, w, v),
                 "uv": (sp.calc_VorDiv2UV, w, v)}
        tup = lambda o: o if isinstance(o, tuple) else (o,)  # noqa: E731
        bits = lambda t: torch.nan_to_num(t, nan=3.0, posinf=5.0, neginf=7.0)  # noqa: E731
        for name, (fn, *args) in calls.items():
            batch = tup(fn(*args))
            for k in (0, 1, 2, 31, 32, nb // 2, nb - 1):
                one = tup(fn(*[a[k:k + 1] for a in args]))
                for a, b in zip(batch, one):
                    assert torch.equal(bits(a[k]), bits(b[0])), (name, k)
            for a in batch:
                bad = (~torch.isfinite(a.reshape(nb, -1))).any(1).nonzero().flatten().tolist()
                assert bad in ([], [1]), (name, bad)
    finally:
        sp.final()


def test_column_tables():
    import torch

    P = pkg()
    sp = P.SpmlUtil(1, 64, 1, 42)
    m = P.MultiTransform()
    try:
        g = torch.Generator(device="cuda")
        g.manual_seed(9)
        ws = [torch.randn(nb, sp.lm, generator=g, device="cuda", dtype=torch.float64) for nb in (1, 5, 40)]
        pairs = [(w.clone(), torch.zeros(w.shape[0], 64, 1, device="cuda", dtype=torch.float64)) for w in ws]
        for w, x in pairs:
            m.add(sp, w, x)
        m.build(autotune=False)
        for w, (wm, xm) in zip(ws, pairs):
            wm.copy_(w)
            xm.zero_()
        torch.cuda.synchronize()
        m.run()
        m.synchronize()
        for w, (wm, xm) in zip(ws, pairs):
            x = sp.xy_w(w)
            assert torch.equal(xm, x) and torch.equal(wm, sp.w_xy(x))
    finally:
        m.close()
        sp.final()
