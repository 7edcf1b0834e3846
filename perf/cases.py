"""Performance cases of the spherical-harmonic transform.

A case is one pass of what a host model does with the package through its
public entry points (SpmlUtil, callers, MultiTransform), on a grid of im
longitudes by jm Gauss latitudes, truncation nm, nb field-levels:

    roundtrip  xy_w of nb spectra, then w_xy of the grids
    uv         calc_VorDiv2UV, then calc_UVCosLat2VorDiv of U, V cos(phi)
    hgrad      xy_HGrad_xy: both horizontal gradients of nb tracer grids
    tracer     callers.htrc_rhs: the tracer tendency of a leapfrog stage
    momentum   callers.momrhs_vordiv_fma: the velocity tendency
    diffusion  xy_w, w_xy and the backward-Euler lateral diffusion
    mixed      MultiTransform round trip over instances of T21/T42/T85/T170

`precision` is the plan's mode (0 FP64, 1 split, 2 per direction); `host`
calls take numpy arrays (pageable memory), the others CUDA tensors.
"""
from __future__ import annotations

import importlib
import math

import numpy as np
import torch

P = importlib.import_module("dennou-ogcm_b200")
callers = importlib.import_module("dennou-ogcm_b200.callers")

RADIUS = 6.371e6
GRIDS = {"T21": (64, 32, 21), "T42": (128, 64, 42), "T85": (256, 128, 85), "T170": (512, 256, 170)}
MIX = ["T21"] * 8 + ["T42"] * 4 + ["T85"] * 2 + ["T170"]


def _case(op, im, jm, nm, nb, precision=0, host=False, name=None):
    c = {"op": op, "im": im, "jm": jm, "nm": nm, "nb": nb, "precision": precision, "host": host}
    return {"name": name, **c} if name else c


def listed():
    return [
        # one 2-D field on the coarsest model grid: the barotropic sub-cycle's calls
        _case("roundtrip", 64, 32, 21, 1, name="t21_level"),
        # the velocity <-> vorticity/divergence pair of the barotropic sub-cycle at T85
        _case("uv", 256, 128, 85, 1, name="t85_level_uv"),
        # the Fortran host's unmodified per-level loop: one level through host arrays
        _case("roundtrip", 256, 128, 85, 1, host=True, name="t85_host_level"),
        # Redi/GM tracer gradients of one tracer on the T42 grid
        _case("hgrad", 128, 64, 42, 60, name="t42_hgrad"),
        # a factor-3 longitude count and an odd level count
        _case("uv", 192, 96, 63, 37, name="t63_uv"),
        # tracer tendency of one tracer, all levels in one call
        _case("tracer", 256, 128, 85, 60, name="t85_tracer"),
        # velocity tendency, all levels in one call
        _case("momentum", 256, 128, 85, 60, name="t85_momentum"),
        # every level of eight fields: the headline batch
        _case("roundtrip", 256, 128, 85, 480, name="t85_roundtrip"),
        # the T106 grid (factor 5), three fields of 60 levels
        _case("roundtrip", 320, 160, 106, 180, name="t106_roundtrip"),
        # twelve fields of 60 levels at T170, plain FP64
        _case("roundtrip", 512, 256, 170, 720, name="t170_roundtrip"),
        # sixteen fields of 60 levels at T341 with diffusion, precision picked per direction
        _case("diffusion", 1024, 512, 341, 960, precision=2, name="t341_diffusion"),
        # 64 instances of mixed truncation, levels 10-60, 3-8 fields, one step
        {"name": "mixed_batch", "op": "mixed", "count": 64},
    ]


def draw(rng):
    kind = rng.random()
    if kind < 0.06:
        return {"op": "mixed", "count": rng.randrange(4, 25)}
    im = rng.choice([32, 64, 128, 256, 512, 1024] if kind < 0.66 else [48, 80, 96, 160, 192, 240, 320, 384, 480, 640])
    jm = im // 2 + (2 * rng.randrange(-2, 3) if rng.random() < 0.3 else 0)
    nm = (im - 1) // 3 - (rng.randrange(0, im // 12 + 1) if rng.random() < 0.5 else 0)
    op = rng.choice(["roundtrip", "roundtrip", "roundtrip", "uv", "hgrad", "tracer", "momentum", "diffusion"])
    most = max(1, min(2000, 96_000_000 // (im * jm)))
    nb = max(1, min(most, round(math.exp(rng.uniform(0.0, math.log(most + 0.99))))))
    precision, host = 0, False
    how = rng.random()
    if how < 0.1 and im * jm * nb < 8_000_000:
        op, host = "roundtrip", True
    elif how < 0.4 and im >= 128 and im & (im - 1) == 0 and jm == im // 2:
        precision = rng.choice([1, 2])
    return _case(op, im, jm, nm, nb, precision, host)


# ------------------------------------------------------------------ inputs

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _spectra(N, nb, power, gen):
    """a_n^m ~ N(0,1) (n+1)^-power in the SPML real layout l = n(n+1) + m."""
    n = torch.repeat_interleave(torch.arange(N + 1, device="cuda"), 2 * torch.arange(N + 1, device="cuda") + 1)
    m = torch.arange((N + 1) ** 2, device="cuda") - n * (n + 1)
    s = (n + 1.0).double() ** -power * torch.where(m == 0, 1.0, math.sqrt(2.0)).double()
    return torch.randn((nb, s.numel()), generator=gen, device="cuda", dtype=torch.float64) * s


def _grids(im, jm, nb, gen, size=1.0):
    """Large-scale waves of random phase with a little grid-scale structure."""
    k = 6
    lon = torch.arange(im, device="cuda", dtype=torch.float64) * (2 * math.pi / im)
    lat = (torch.arange(jm, device="cuda", dtype=torch.float64) + 0.5) * (math.pi / jm)
    wave = torch.cat([torch.cos(torch.arange(k, device="cuda")[:, None] * lon), torch.sin(torch.arange(k, device="cuda")[:, None] * lon)])
    prof = torch.stack([torch.sin(lat) ** (q // 2 + 1) * (torch.cos(lat) if q % 2 else 1.0) for q in range(2 * k)])
    amp = torch.randn((nb, 1, 2 * k), generator=gen, device="cuda", dtype=torch.float64)
    out = torch.matmul(prof.T[None] * amp, wave)
    out += 0.05 * torch.randn((nb, jm, im), generator=gen, device="cuda", dtype=torch.float64) * torch.sin(lat)[None, :, None]
    return out.mul_(size)


def _mixed_instances(count):
    rng = np.random.default_rng(20261203)
    out = []
    for k in range(count):
        levels, fields = int(rng.integers(10, 61)), int(rng.integers(3, 9))
        out.append((MIX[k % len(MIX)], levels * fields))
    return out


def _inputs(case, seed):
    g = _generator(seed)
    op = case["op"]
    if op == "mixed":
        return [_spectra(GRIDS[t][2], nb, 1.5, g) for t, nb in _mixed_instances(case["count"])]
    im, jm, N, nb = case["im"], case["jm"], case["nm"], case["nb"]
    if op == "roundtrip":
        return [_spectra(N, nb, 1.5, g)]
    if op == "diffusion":
        return [_spectra(N, nb, 2.0, g), _diffusion_coef(N)]
    if op == "uv":
        return [_spectra(N, nb, 2.0, g) * 1e-5, _spectra(N, nb, 2.0, g) * 1e-6]
    if op == "hgrad":
        return [_grids(im, jm, nb, g, 10.0)]
    if op == "tracer":
        u, v, t, z, h = (_grids(im, jm, nb, g, s) for s in (1.0, 0.5, 300.0, 1e-5, 1e-5))
        return [u, v, t, z, torch.exp(-0.01 * torch.rand((N + 1) ** 2, generator=g, device="cuda", dtype=torch.float64)), h]
    if op == "momentum":
        return [_grids(im, jm, nb, g, s) for s in (1.0, 0.5, 1e-5, 1e-5, 1e-5, 10.0)]
    raise ValueError(op)


def _diffusion_coef(N):
    n = torch.sqrt(torch.arange((N + 1) ** 2, device="cuda", dtype=torch.float64)).floor()
    return -1e-3 * (n * (n + 1.0) / (N * (N + 1.0))) ** 4


def prepare(case, seed):
    x = _inputs(case, seed)
    if case["op"] == "mixed":
        # all instances' arrays side by side, as a host that owns one pool lays them out
        plans = {t: P.SpmlUtil(g[0], g[1], 1, g[2], None, RADIUS) for t, g in GRIDS.items()}
        inst = _mixed_instances(case["count"])
        spec = torch.zeros(sum(w.numel() for w in x), dtype=torch.float64, device="cuda")
        grid = torch.empty(sum(nb * GRIDS[t][0] * GRIDS[t][1] for t, nb in inst), dtype=torch.float64, device="cuda")
        multi, at, ag = P.MultiTransform(), 0, 0
        for t, nb in inst:
            im, jm, N = GRIDS[t]
            nw, ng = nb * (N + 1) ** 2, nb * im * jm
            multi.add(plans[t], spec[at:at + nw].view(nb, -1), grid[ag:ag + ng].view(nb, jm, im))
            at, ag = at + nw, ag + ng
        torch.cuda.synchronize()
        multi.build(autotune=True)
        multi.set_stream(torch.cuda.current_stream())
        spec.copy_(torch.cat([w.reshape(-1) for w in x]))
        return {"op": "mixed", "multi": multi, "plans": plans, "spec": spec, "grid": grid}
    sp = P.SpmlUtil(case["im"], case["jm"], 1, case["nm"], None, RADIUS)
    sp.set_precision(case["precision"])
    if case["host"]:
        x = [a.cpu().numpy() for a in x]
    cos = torch.cos(torch.as_tensor(sp.y_Lat, dtype=torch.float64, device="cuda"))[None, :, None]
    return {"op": case["op"], "sp": sp, "x": x, "cos": cos}


def run(state):
    op = state["op"]
    if op == "mixed":
        state["multi"].run(P.SHT_MULTI_ROUND_TRIP)
        return state["grid"], state["spec"]
    sp, x = state["sp"], state["x"]
    if op == "roundtrip":
        g = sp.xy_w(x[0])
        return g, sp.w_xy(g)
    if op == "diffusion":
        g = sp.xy_w(x[0])
        return g, sp.diffuse(sp.w_xy(g), x[1], 1.0)
    if op == "uv":
        u, v = sp.calc_VorDiv2UV(x[0], x[1])
        vor, div = sp.calc_UVCosLat2VorDiv(u * state["cos"], v * state["cos"])
        return u, v, vor, div
    if op == "hgrad":
        return sp.xy_HGrad_xy(x[0])
    if op == "tracer":
        return callers.htrc_rhs(sp, *x)
    return callers.momrhs_vordiv_fma(sp, *x)


# -------------------------------------------------------------------- work

def _transform_flops(im, jm, N, cols):
    """One direction, cols field-levels: the contraction of each latitude half with
    one parity of the degrees, and a real FFT per row."""
    return cols * (jm * (N + 1.0) * (N + 2.0) + jm * 2.5 * im * math.log2(im))


def work(case):
    """Arrays of each call read and written once; both directions' arithmetic."""
    if case["op"] == "mixed":
        parts = [work(_case("roundtrip", *GRIDS[t], nb)) for t, nb in _mixed_instances(case["count"])]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    im, jm, N, nb = case["im"], case["jm"], case["nm"], case["nb"]
    g, w = 8.0 * nb * im * jm, 8.0 * nb * (N + 1) ** 2
    #            grids, spectra read or written by the calls; columns transformed
    ng, nw, cols = {"roundtrip": (2, 2, 2), "diffusion": (2, 2, 2), "uv": (4, 4, 4), "hgrad": (3, 0, 3),
                    "tracer": (6, 0, 4), "momentum": (8, 0, 5)}[case["op"]]
    return {"bytes": ng * g + nw * w, "flops": _transform_flops(im, jm, N, cols * nb)}


# ------------------------------------------------------- the sums in 64 bits

def _gauss(jm):
    """Gauss-Legendre nodes and weights (sum 2), refined by Newton steps in extended precision."""
    x = np.polynomial.legendre.leggauss(jm)[0].astype(np.longdouble)
    for _ in range(3):
        p0, p1 = np.ones_like(x), x
        for n in range(2, jm + 1):
            p0, p1 = p1, ((2 * n - 1) * x * p1 - (n - 1) * p0) / n
        dp = jm * (x * p1 - p0) / (x * x - 1)
        x, w = x - p1 / dp, 2 / ((1 - x * x) * dp * dp)
    return x.astype(np.float64), w.astype(np.float64)


class _Direct:
    """The transform as written, in torch FP64: cuFFT rows, one matrix product per order."""

    def __init__(self, im, jm, N):
        self.im, self.jm, self.N = im, jm, N
        mu, w = _gauss(jm)
        dev = lambda a: torch.as_tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
        self.mu, self.w = dev(mu), dev(w / 2.0)
        self.c2 = 1.0 - self.mu ** 2
        m = torch.arange(N + 1, device="cuda", dtype=torch.float64)[:, None]

        def eps(n):
            return torch.sqrt(torch.clamp(n * n - m * m, min=0.0) / (4.0 * n * n - 1.0)) if n > 0 else torch.zeros_like(m)
        k = torch.arange(1, N + 1, dtype=torch.float64)
        lead = torch.cat([torch.zeros(1), torch.cumsum(torch.log(torch.sqrt((2 * k + 1) / (2 * k))), 0)]).cuda()[:, None]
        top = torch.exp(lead + 0.5 * m * torch.log(self.c2)[None, :])  # Pbar_m^m
        # T[n, m, j] = Pbar_n^m(mu_j), n = 0..N+1
        T = torch.zeros((N + 2, N + 1, jm), dtype=torch.float64, device="cuda")
        for n in range(N + 2):
            if n >= 1:
                prev2 = T[n - 2] if n >= 2 else torch.zeros_like(T[0])
                e = eps(n)
                T[n] = torch.where(m < n, (self.mu * T[n - 1] - eps(n - 1) * prev2) / torch.where(e > 0, e, 1.0), 0.0)
            if n <= N:
                T[n, n] = top[n]
        self.T = T
        # (1 - mu^2) dPbar/dmu = (n+1) eps_n Pbar_{n-1} - n eps_{n+1} Pbar_{n+1}
        self.H = torch.stack([(n + 1) * eps(n) * (T[n - 1] if n else 0.0) - n * eps(n + 1) * T[n + 1] for n in range(N + 1)])
        self.n = torch.repeat_interleave(torch.arange(N + 1, device="cuda"), 2 * torch.arange(N + 1, device="cuda") + 1)

    def _lm(self, m):
        n = torch.arange(m, self.N + 1, device="cuda")
        return n * (n + 1) + m, n * (n + 1) - m

    def synth(self, parts, scale=None):
        """sum over (table, coefficient, times i m) of table . coefficient -> grid."""
        nb = parts[0][1].shape[0]
        G = torch.zeros((nb, self.jm, self.im // 2 + 1), dtype=torch.complex128, device="cuda")
        for m in range(self.N + 1):
            lc, ls = self._lm(m)
            for table, w, im in parts:
                t = table[m:self.N + 1, m]
                re, q = torch.matmul(w[:, lc], t), (torch.matmul(w[:, ls], t) if m else None)
                s = 1.0 if m == 0 else math.sqrt(0.5)
                z = torch.complex(re * s, q * s) if m else torch.complex(re, torch.zeros_like(re))
                G[:, :, m] += 1j * m * z if im else z
        g = torch.fft.irfft(G, n=self.im, dim=2, norm="forward")
        return g if scale is None else g.mul_(scale[None, :, None])

    def fourier(self, g, scale=None):
        G = torch.fft.rfft(g, dim=2, norm="forward")[:, :, :self.N + 1]
        s = self.w if scale is None else self.w * scale
        return G * s[None, :, None]

    def analyse(self, parts):
        """sum over (table, Fourier array, times i m, factor) -> spectra."""
        nb = parts[0][1].shape[0]
        out = torch.zeros((nb, (self.N + 1) ** 2), dtype=torch.float64, device="cuda")
        for m in range(self.N + 1):
            lc, ls = self._lm(m)
            z = 0
            for table, G, im, f in parts:
                t = table[m:self.N + 1, m].T * f
                x = G[:, :, m]
                c = torch.complex(torch.matmul(x.real.contiguous(), t), torch.matmul(x.imag.contiguous(), t))
                z = z + (1j * m * c if im else c)
            if m == 0:
                out[:, lc] = z.real
            else:
                out[:, lc], out[:, ls] = z.real * math.sqrt(2.0), z.imag * math.sqrt(2.0)
        return out

    def xy_w(self, w):
        return self.synth([(self.T, w, False)])

    def w_xy(self, g):
        return self.analyse([(self.T, self.fourier(g), False, 1.0)])

    def alpha(self, a, b):
        """(1/a) ((1/(1-mu^2)) dA/dlambda + dB/dmu), the second by parts."""
        A, B = self.fourier(a, 1.0 / self.c2), self.fourier(b, 1.0 / self.c2)
        return self.analyse([(self.T, A, True, 1.0 / RADIUS), (self.H, B, False, -1.0 / RADIUS)])

    def vordiv(self, uc, vc):
        U, V = self.fourier(uc, 1.0 / self.c2), self.fourier(vc, 1.0 / self.c2)
        return (self.analyse([(self.T, V, True, 1.0 / RADIUS), (self.H, U, False, 1.0 / RADIUS)]),
                self.analyse([(self.T, U, True, 1.0 / RADIUS), (self.H, V, False, -1.0 / RADIUS)]))

    def uv(self, vor, div):
        nn = (self.n * (self.n + 1)).double()
        inv = torch.where(nn > 0, -RADIUS ** 2 / torch.where(nn > 0, nn, 1.0), 0.0)
        psi, chi = vor * inv, div * inv
        s = 1.0 / (RADIUS * torch.sqrt(self.c2))
        return (self.synth([(self.T, chi, True), (self.H, -psi, False)], s),
                self.synth([(self.T, psi, True), (self.H, chi, False)], s))


def exact(case, seed):
    x = _inputs(case, seed)
    if case["op"] == "mixed":
        d = {t: _Direct(*GRIDS[t]) for t in {t for t, _ in _mixed_instances(case["count"])}}
        grid, spec = [], []
        for (t, _), w in zip(_mixed_instances(case["count"]), x):
            g = d[t].xy_w(w)
            grid.append(g.reshape(-1))
            spec.append(d[t].w_xy(g).reshape(-1))
        return torch.cat(grid), torch.cat(spec)
    d, op = _Direct(case["im"], case["jm"], case["nm"]), case["op"]
    cos = torch.sqrt(d.c2)[None, :, None]
    if op == "roundtrip":
        g = d.xy_w(x[0])
        return g, d.w_xy(g)
    if op == "diffusion":
        g = d.xy_w(x[0])
        return g, d.w_xy(g) / (1.0 - x[1])
    if op == "uv":
        u, v = d.uv(x[0], x[1])
        return (u, v, *d.vordiv(u * cos, v * cos))
    if op == "hgrad":
        w = d.w_xy(x[0])
        s = 1.0 / torch.sqrt(d.c2)
        return d.synth([(d.T, w, True)], s), d.synth([(d.H, w, False)], s)
    if op == "tracer":
        u, v, t, z, filt, h = x
        return d.xy_w((d.w_xy(z) - d.alpha(u * t, v * t)) * filt) + h
    u, v, vor, za, zb, c = x
    wv, wd = d.vordiv(cos * (vor * u + za), cos * (vor * v + zb))
    lap = -(d.n * (d.n + 1)).double()
    return d.uv(-wd, wv - lap * d.w_xy(c))
