"""Tendencies on a SpmlUtil subclass that keeps what its transforms return: the
spectra that it kept are as they were, and the result is the plain plan's, bit
for bit."""
import importlib

import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["htrc_rhs", "momrhs_vordiv", "momrhs_vordiv_fma"])
def test_kept_spectra_are_not_overwritten(name):
    import torch

    P, C = pkg(), importlib.import_module("dennou-ogcm_b200.callers")

    class Keeps(P.SpmlUtil):
        """Remembers every spectrum it hands out (a model that stores its tendencies)."""

        def _run(self, *a, **kw):
            out = super()._run(*a, **kw)
            for o in out if isinstance(out, tuple) else (out,):
                self.kept.append((o, o.clone()))
            return out

    plain, sp = P.SpmlUtil(64, 32, 1, 21), Keeps(64, 32, 1, 21)
    sp.kept = []
    try:
        g = torch.Generator(device="cuda")
        g.manual_seed(6)
        x = [torch.randn(3, 32, 64, generator=g, device="cuda", dtype=torch.float64) for _ in range(5)]
        f = torch.rand(sp.lm, generator=g, device="cuda", dtype=torch.float64)
        args = {"htrc_rhs": (*x[:4], f, x[4]), "momrhs_vordiv": x[:3], "momrhs_vordiv_fma": (*x, x[0])}[name]
        fn = getattr(C, name)
        out, ref = fn(sp, *args), fn(plain, *args)
        for a, b in zip(out if isinstance(out, tuple) else (out,), ref if isinstance(ref, tuple) else (ref,)):
            assert torch.equal(a, b)
        assert sp.kept and all(torch.equal(o, c) for o, c in sp.kept)
    finally:
        plain.final()
        sp.final()
