// sht_spectral.cu -- spectral-side kernels: conversion between the SPML
// real layout wa[b][l] and the internal complex layout S[row][col], fused
// with the derivative recurrences of the operators, plus the diagonal
// spectral operators and the Gauss-weighted grid integrals.
//
//   analysis side ("pack", internal c -> wa):
//     plain      w_xy                              c_n
//     divlambda  w_DivLambda_xy                    i m c_n
//     divmu      w_DivMu_xy                        D(c)_n = -((n+1) eps_n c_{n-1} - n eps_{n+1} c_{n+1})
//     alpha      w_AlphaOptr_xy(A,B)               (i m cA_n + D(cB)_n) / a
//     vordiv     calc_UVCosLat2VorDiv(Ucos,Vcos)   vor = (i m cV - D(cU))/a, div = (i m cU + D(cV))/a
//   synthesis side ("unpack", wa -> internal a, n = m..N+1):
//     plain      xy_w                              a_n
//     gradlambda xy_GradLambda_w / GradLon         i m a_n
//     hgrad      GradLon and GradLat together      i m a_n and R(a)_n (two column sets)
//     gradmu     xy_GradMu_w / GradLat             R(a)_n = (n+2) eps_{n+1} a_{n+1} - (n-1) eps_n a_{n-1}
//     alpha      xy_AlphaOptr_w(A,B)               i m aA_n + R(aB)_n
//     vordiv2uv  calc_VorDiv2UV(vor,div)           psi,chi = -a^2 x/(n(n+1));
//                                                  U = i m chi - R(psi), V = i m psi + R(chi)
// The eps recurrence is space_discretization.tex:250-257; the U, V form is
// :369-379; D is the by-parts form of :262-267; the 1/a factors are
// SpmlUtil_mod.f90:410,426 and the a^2 LaplaInv at SpmlUtil_mod.f90:335-336.
//
// Both conversions tile by (total degree n, a chunk of 32 orders m, 32
// field-levels) so that global reads and writes are 256-512 byte runs.
#include "sht_spectral.cuh"

namespace sht {

namespace {

using namespace spec;

constexpr int kMC = 32;  // orders per tile
constexpr int kBC = 32;  // field-levels per tile
template <int OP>
__global__ void __launch_bounds__(256) k_pack(SpecArgs a)
{
  __shared__ double out[2][2][kMC][kBC + 1];  // [array][cos/sin][m][b]
  const int2 t = a.tiles[blockIdx.x];
  const int n = t.x, m0 = t.y;
  const int b0 = blockIdx.y * kBC;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b = b0 + lane;
  constexpr int NOUT = (OP == PACK_VORDIV) ? 2 : 1;
  constexpr int NI = kMC / 8;  // orders per warp
  // every load of the thread is issued before any is used: out-of-range
  // entries read element 0 and are replaced by zero
  double2 c[NI][3][2];
  double ev[NI][2];  // eps_n^m and eps_{n+1}^m, loaded with the coefficients
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    const int m = m0 + warp + 8 * i;
    const bool ok = m <= n && m < a.M && b < a.nb;
    if (OP != PACK_PLAIN && OP != PACK_DIVLAMBDA) {
      ev[i][0] = ok ? eps_at(a, m, n) : 0.0;
      ev[i][1] = ok ? eps_at(a, m, n + 1) : 0.0;
    }
    const long long base = ok ? (long long)spec_row(a.N, m, n) * a.ncolS + b : 0;
#pragma unroll
    for (int dn = -1; dn <= 1; ++dn)
#pragma unroll
      for (int set = 0; set < 2; ++set) {
        c[i][dn + 1][set] = make_double2(0.0, 0.0);
        if (!pack_needs<OP>(dn, set)) continue;
        const bool okk = ok && n + dn >= m && n + dn <= a.N + 1;
        const double2 x = a.S[okk ? base + (long long)dn * a.ncolS + set * a.nb : 0];
        if (okk) c[i][dn + 1][set] = x;
      }
  }
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    const int mi = warp + 8 * i, m = m0 + mi;
    double2 v0 = make_double2(0.0, 0.0), v1 = make_double2(0.0, 0.0);
    if (m <= n && m < a.M && b < a.nb) pack_combine<OP>(c[i], n, m, ev[i][0], ev[i][1], a.radius, v0, v1);
    const double s = (m == 0) ? 1.0 : kSqrt2;
    out[0][0][mi][lane] = v0.x * s;
    out[0][1][mi][lane] = v0.y * s;
    if (NOUT == 2) {
      out[1][0][mi][lane] = v1.x * s;
      out[1][1][mi][lane] = v1.y * s;
    }
  }
  __syncthreads();
  // write runs w[b][n(n+1) + m] and w[b][n(n+1) - m]
  const int mi = lane, m = m0 + mi;
  if (m > n || m >= a.M) return;
  const long long lc = spml_l(a, n, m, 0), ls = spml_l(a, n, m, 1);
#pragma unroll
  for (int q = 0; q < kBC / 8; ++q) {
    const int bi = warp + 8 * q, bb = b0 + bi;
    if (bb >= a.nb) break;
#pragma unroll
    for (int o = 0; o < NOUT; ++o) {
      double *w = (o == 0 && a.ocol) ? a.ocol[bb] : ((o == 0) ? a.o0 : a.o1) + (long long)bb * a.L;
      w[lc] = out[o][0][mi][bi];
      if (m > 0) w[ls] = out[o][1][mi][bi];
    }
  }
}


// A warp takes field-levels b0 + 8 i' + w with its lanes along the orders
// (256-byte runs of the SPML rows), applies the operator there, and stages
// only the results, transposed, for stores with the lanes along the
// field-levels.  Staging the entries instead (up to twelve runs, 101 KB for
// U, V from vorticity and divergence) and dividing by n(n+1) in every
// thread's inner loop took 63 us for that operator at T85 with 480 levels, 41
// now (116 MB).
template <int OP>
__global__ void __launch_bounds__(256) k_unpack(SpecArgs a)
{
  constexpr int NIN = (OP == UNPACK_ALPHA || OP == UNPACK_VORDIV2UV) ? 2 : 1;
  constexpr int NOUT = unpack_outputs<OP>();
  constexpr bool kEps = OP != UNPACK_PLAIN && OP != UNPACK_GRADLAMBDA;
  __shared__ double ws[2 * NOUT][kMC][kBC + 1];  // [output, re/im][m][b]
  const int2 t = a.tiles[blockIdx.x];
  const int n = t.x, m0 = t.y;
  const int b0 = blockIdx.y * kBC;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int NQ = kBC / 8;
  const int m = m0 + lane;
  // the SPML offset of each run (dn = -1..1, cos/sin part; -1 where the entry
  // does not exist) and the recurrence's coefficients, formed once
  int off[6];
#pragma unroll
  for (int r = 0; r < 6; ++r) {
    const int nn = n + r / 2 - 1, sn = r & 1;
    const bool ok = nn >= 0 && nn <= a.N && m <= nn && m < a.M && !(sn && m == 0);
    off[r] = ok ? (int)spml_l(a, nn, m, sn) : -1;
  }
  const double *wr[NIN][NQ];
#pragma unroll
  for (int in = 0; in < NIN; ++in)
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int bb = b0 + 8 * q + warp;
      wr[in][q] = bb >= a.nb ? nullptr
                : (in == 0 && a.icol) ? a.icol[bb] : ((in == 0) ? a.w0 : a.w1) + (long long)bb * a.L;
    }
  double x[NQ][NIN][3][2];
#pragma unroll
  for (int in = 0; in < NIN; ++in)
#pragma unroll
    for (int r = 0; r < 6; ++r)
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        x[q][in][r / 2][r & 1] = 0.0;
        if (!unpack_needs<OP>(in, r / 2 - 1)) continue;
        const double *w = wr[in][q];
        const int o = off[r];
        if (w && o >= 0) x[q][in][r / 2][r & 1] = __ldg(w + o);
      }
  const bool mok = m <= n && m <= a.N && m < a.M;
  double ep = 0.0, em = 0.0;
  if (kEps && mok) {
    ep = (n + 2) * eps_at(a, m, n + 1);
    em = (n - 1) * eps_at(a, m, n);
  }
  double lap[3];
  lap_factors<OP>(n, a.radius, lap);
  const double s = (m == 0) ? 1.0 : kRSqrt2;
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    double2 v0, v1 = make_double2(0.0, 0.0);
    unpack_combine<OP>(x[q], m, ep, em, lap, s, v0, v1);
    ws[0][lane][8 * q + warp] = v0.x;
    ws[1][lane][8 * q + warp] = v0.y;
    if constexpr (NOUT == 2) {
      ws[2][lane][8 * q + warp] = v1.x;
      ws[3][lane][8 * q + warp] = v1.y;
    }
  }
  __syncthreads();
  const int b = b0 + lane;
  if (b >= a.nb) return;
  int rows[kMC / 8];  // internal rows of this warp's orders
#pragma unroll
  for (int i = 0; i < kMC / 8; ++i) {
    const int mw = m0 + warp + 8 * i;
    rows[i] = (mw <= n && mw <= a.N && mw < a.M) ? spec_row(a.N, mw, n) : -1;
  }
#pragma unroll
  for (int i = 0; i < kMC / 8; ++i) {
    const int mi = warp + 8 * i;
    if (rows[i] < 0) continue;
    double2 *So = a.So + (long long)rows[i] * a.ncolS + b;
    So[0] = make_double2(ws[0][mi][lane], ws[1][mi][lane]);
    if constexpr (NOUT == 2) So[a.nb] = make_double2(ws[2][mi][lane], ws[3][mi][lane]);
  }
}

// ------------------------------------------------------ axisymmetric plans
// One order: the tiles above would leave 31 of 32 lanes (or 7 of 8 warps)
// idle.  A thread takes one degree of one field-level; the lanes run over the
// levels (whole runs of the internal rows), a block's eight warps over the
// degrees, so that the sectors of a level's row are used while they are in L1.
// Whole calls with the tiles before / as they are now in the other plans /
// here, us: 1 x 64 points, 960 levels, flux-form analysis of a product 18.1 / 20.5 /
// 14.4; 1 x 128, 4000 levels, xy_GradMu_w 43 / 48 / 21, calc_VorDiv2UV 117 / 113 /
// 28.  Below about 200 levels the narrow-batch kernels run instead.
template <int OP>
__global__ void __launch_bounds__(256) k_pack_zonal(SpecArgs a)
{
  const int b = blockIdx.x * 32 + (threadIdx.x & 31), n = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (b >= a.nb || n > a.N) return;
  double2 c[3][2];
#pragma unroll
  for (int dn = -1; dn <= 1; ++dn)
#pragma unroll
    for (int set = 0; set < 2; ++set) {
      c[dn + 1][set] = make_double2(0.0, 0.0);
      if (pack_needs<OP>(dn, set) && n + dn >= 0) c[dn + 1][set] = a.S[(long long)(n + dn) * a.ncolS + set * a.nb + b];
    }
  double e0 = 0.0, e1 = 0.0;
  if (OP != PACK_PLAIN && OP != PACK_DIVLAMBDA) {
    e0 = eps_at(a, 0, n);
    e1 = eps_at(a, 0, n + 1);
  }
  double2 v0, v1 = make_double2(0.0, 0.0);
  pack_combine<OP>(c, n, 0, e0, e1, a.radius, v0, v1);
  (a.ocol ? a.ocol[b] : a.o0 + (long long)b * a.L)[n] = v0.x;
  if constexpr (OP == PACK_VORDIV) a.o1[(long long)b * a.L + n] = v1.x;
}

template <int OP>
__global__ void __launch_bounds__(256) k_unpack_zonal(SpecArgs a)
{
  constexpr int NIN = (OP == UNPACK_ALPHA || OP == UNPACK_VORDIV2UV) ? 2 : 1;
  const int b = blockIdx.x * 32 + (threadIdx.x & 31), n = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (b >= a.nb || n > a.N + 1) return;
  double x[NIN][3][2];
#pragma unroll
  for (int in = 0; in < NIN; ++in) {
    const double *w = (in == 0 && a.icol) ? a.icol[b] : (in == 0 ? a.w0 : a.w1) + (long long)b * a.L;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int nn = n + d - 1;
      x[in][d][0] = unpack_needs<OP>(in, d - 1) && nn >= 0 && nn <= a.N ? __ldg(w + nn) : 0.0;
      x[in][d][1] = 0.0;
    }
  }
  double ep = 0.0, em = 0.0, lap[3];
  if (OP != UNPACK_PLAIN && OP != UNPACK_GRADLAMBDA) {
    ep = (n + 2) * eps_at(a, 0, n + 1);
    em = (n - 1) * eps_at(a, 0, n);
  }
  lap_factors<OP>(n, a.radius, lap);
  double2 v0, v1 = make_double2(0.0, 0.0);
  unpack_combine<OP>(x, 0, ep, em, lap, 1.0, v0, v1);
  double2 *So = a.So + (long long)n * a.ncolS + b;
  So[0] = v0;
  if constexpr (unpack_outputs<OP>() == 2) So[a.nb] = v1;
}

// --------------------------------------------------------- diagonal ops
// Both diagonal operators: one thread per spectral entry and kDiagLevels
// field-levels, so that the entry's factor is read once and no index is
// divided (a 64-bit remainder per element bound the earlier form: 960 levels
// at T341, diffusion 434 us in place after a 284 us copy -> 263 us out of
// place, 1.8 GB).
constexpr int kDiagLevels = 8;

__global__ void __launch_bounds__(256) k_lapla(const double *__restrict__ w, const double *__restrict__ rn, int nb, int L,
                                               double *__restrict__ out, int inverse)
{
  const int l = blockIdx.x * 256 + threadIdx.x, b0 = blockIdx.y * kDiagLevels;
  if (l >= L) return;
  const double e = __ldg(rn + l);
  const long long at = (long long)b0 * L + l;
  double x[kDiagLevels];
#pragma unroll
  for (int k = 0; k < kDiagLevels; ++k) x[k] = b0 + k < nb ? w[at + (long long)k * L] : 0.0;
#pragma unroll
  for (int k = 0; k < kDiagLevels; ++k)
    if (b0 + k < nb) out[at + (long long)k * L] = inverse ? ((e == 0.0) ? 0.0 : x[k] / e) : x[k] * e;
}

// in == out is allowed
__global__ void __launch_bounds__(256) k_diffuse(const double *in, int nb, int L, const double *__restrict__ coef,
                                                 double dt, const double *__restrict__ filter, double *out)
{
  const int l = blockIdx.x * 256 + threadIdx.x, b0 = blockIdx.y * kDiagLevels;
  if (l >= L) return;
  const double f = filter ? __ldg(filter + l) : 1.0, d = 1.0 - dt * __ldg(coef + l);
  const long long at = (long long)b0 * L + l;
  double x[kDiagLevels];
#pragma unroll
  for (int k = 0; k < kDiagLevels; ++k) x[k] = b0 + k < nb ? in[at + (long long)k * L] : 0.0;
#pragma unroll
  for (int k = 0; k < kDiagLevels; ++k)
    if (b0 + k < nb) out[at + (long long)k * L] = f * x[k] / d;
}

// The spectral tails of the tracer and momentum tendencies, in place, where the
// operators and the differences are otherwise a pass each (60 levels at T85:
// subtract and scale 7.2 -> 3.4 us, negate, Laplacian and subtract 7.5 -> 3.8).
// Products and differences round one by one, as in separate passes.
__global__ void __launch_bounds__(256) k_sub_filter(double *a, const double *__restrict__ b, int nb, int L,
                                                    const double *__restrict__ filter)
{
  const int l = blockIdx.x * 256 + threadIdx.x, b0 = blockIdx.y * kDiagLevels;
  if (l >= L) return;
  const double f = __ldg(filter + l);
  const long long at = (long long)b0 * L + l;
  double x[kDiagLevels], y[kDiagLevels];
#pragma unroll
  for (int k = 0; k < kDiagLevels; ++k) {
    x[k] = b0 + k < nb ? a[at + (long long)k * L] : 0.0;
    y[k] = b0 + k < nb ? __ldg(b + at + (long long)k * L) : 0.0;
  }
#pragma unroll
  for (int k = 0; k < kDiagLevels; ++k)
    if (b0 + k < nb) a[at + (long long)k * L] = __dmul_rn(__dsub_rn(x[k], y[k]), f);
}

// p <- p - lap(c), q <- -q
__global__ void __launch_bounds__(256) k_sub_lapla(double *p, double *q, const double *__restrict__ c,
                                                   const double *__restrict__ rn, int nb, int L)
{
  const int l = blockIdx.x * 256 + threadIdx.x, b0 = blockIdx.y * kDiagLevels;
  if (l >= L) return;
  const double e = __ldg(rn + l);
  const long long at = (long long)b0 * L + l;
  double x[kDiagLevels], y[kDiagLevels], z[kDiagLevels];
#pragma unroll
  for (int k = 0; k < kDiagLevels; ++k) {
    const bool in = b0 + k < nb;
    x[k] = in ? p[at + (long long)k * L] : 0.0;
    y[k] = in ? q[at + (long long)k * L] : 0.0;
    z[k] = in ? __ldg(c + at + (long long)k * L) : 0.0;
  }
#pragma unroll
  for (int k = 0; k < kDiagLevels; ++k)
    if (b0 + k < nb) {
      p[at + (long long)k * L] = __dsub_rn(x[k], __dmul_rn(z[k], e));
      q[at + (long long)k * L] = -y[k];
    }
}

// kind 0: IntLonLat, 1: AvrLonLat, 2: ya_IntLon, 3: ya_AvrLon
__global__ void __launch_bounds__(256) k_lonlat(const double *__restrict__ g, int I, int J,
                                                const double *__restrict__ wgt, double *__restrict__ out, int kind)
{
  __shared__ double part[8];
  const int b = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double *gb = g + (long long)b * I * J;
  const double dl = 2.0 * M_PI / I;
  double acc = 0.0;
  for (int j = warp; j < J; j += 8) {
    double s = 0.0;
    for (int i = lane; i < I; i += 32) s += __ldg(gb + (long long)j * I + i);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (kind >= 2) {
      if (lane == 0) out[(long long)b * J + j] = (kind == 3) ? s / I : s * dl;
    } else {
      acc += s * dl * 2.0 * __ldg(wgt + j);
    }
  }
  if (kind < 2) {
    if (lane == 0) part[warp] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int w = 0; w < 8; ++w) t += part[w];
      out[b] = (kind == 1) ? t / (4.0 * M_PI) : t;
    }
  }
}

}  // namespace

int launch_pack(const sht_plan *p, int op, const double2 *S, int ncolS, int nb, double *w0,
                double *w1, cudaStream_t s, double *const *wcol)
{
  if (nb <= 0) return SHT_OK;
  SpecArgs a{};
  a.ocol = wcol;
  a.S = S; a.ncolS = ncolS; a.o0 = w0; a.o1 = w1 ? w1 : w0;
  a.nb = nb; a.N = p->N; a.L = p->L; a.radius = p->radius;
  a.eps = p->d_eps; a.tiles = p->d_spec_tiles;
  a.M = p->M; a.zonal = p->zonal ? 1 : 0;
  const unsigned groups = (unsigned)((nb + kBC - 1) / kBC);
  auto launch = [&](auto tiles, auto zonal) {
    if (p->zonal) zonal<<<dim3(groups, (unsigned)(p->N + 1 + 7) / 8), 256, 0, s>>>(a);
    else tiles<<<dim3((unsigned)p->n_pack_tiles, groups), 256, 0, s>>>(a);
  };
  switch (op) {
  case PACK_PLAIN: launch(k_pack<PACK_PLAIN>, k_pack_zonal<PACK_PLAIN>); break;
  case PACK_DIVLAMBDA: launch(k_pack<PACK_DIVLAMBDA>, k_pack_zonal<PACK_DIVLAMBDA>); break;
  case PACK_DIVMU: launch(k_pack<PACK_DIVMU>, k_pack_zonal<PACK_DIVMU>); break;
  case PACK_ALPHA: launch(k_pack<PACK_ALPHA>, k_pack_zonal<PACK_ALPHA>); break;
  case PACK_VORDIV: launch(k_pack<PACK_VORDIV>, k_pack_zonal<PACK_VORDIV>); break;
  default: set_error("pack: unknown operator"); return SHT_ERR_INVALID_ARG;
  }
  count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? SHT_OK : cuda_fail(e, "k_pack");
}

int launch_unpack(const sht_plan *p, int op, const double *w0, const double *w1, int nb,
                  double2 *S, int ncolS, cudaStream_t s, const double *const *wcol)
{
  if (nb <= 0) return SHT_OK;
  SpecArgs a{};
  a.icol = wcol;
  a.So = S; a.ncolS = ncolS; a.w0 = w0; a.w1 = w1 ? w1 : w0;
  a.nb = nb; a.N = p->N; a.L = p->L; a.radius = p->radius;
  a.eps = p->d_eps; a.tiles = p->d_spec_tiles;
  a.M = p->M; a.zonal = p->zonal ? 1 : 0;
  const unsigned groups = (unsigned)((nb + kBC - 1) / kBC);
  auto launch = [&](auto tiles, auto zonal) {
    if (p->zonal) zonal<<<dim3(groups, (unsigned)(p->N + 2 + 7) / 8), 256, 0, s>>>(a);
    else tiles<<<dim3((unsigned)p->n_spec_tiles, groups), 256, 0, s>>>(a);
  };
  switch (op) {
  case UNPACK_PLAIN: launch(k_unpack<UNPACK_PLAIN>, k_unpack_zonal<UNPACK_PLAIN>); break;
  case UNPACK_GRADLAMBDA: launch(k_unpack<UNPACK_GRADLAMBDA>, k_unpack_zonal<UNPACK_GRADLAMBDA>); break;
  case UNPACK_GRADMU: launch(k_unpack<UNPACK_GRADMU>, k_unpack_zonal<UNPACK_GRADMU>); break;
  case UNPACK_ALPHA: launch(k_unpack<UNPACK_ALPHA>, k_unpack_zonal<UNPACK_ALPHA>); break;
  case UNPACK_VORDIV2UV: launch(k_unpack<UNPACK_VORDIV2UV>, k_unpack_zonal<UNPACK_VORDIV2UV>); break;
  case UNPACK_HGRAD: launch(k_unpack<UNPACK_HGRAD>, k_unpack_zonal<UNPACK_HGRAD>); break;
  default: set_error("unpack: unknown operator"); return SHT_ERR_INVALID_ARG;
  }
  count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? SHT_OK : cuda_fail(e, "k_unpack");
}

static dim3 diag_grid(const sht_plan *p, int nb)
{
  return dim3((unsigned)((p->L + 255) / 256), (unsigned)((nb + kDiagLevels - 1) / kDiagLevels));
}

// blocks of levels are a grid's y extent: at most 65535 of them per launch
static constexpr int kDiagMost = 65535 * kDiagLevels;

int launch_lapla(const sht_plan *p, const double *w, int nb, double *out, bool inverse, cudaStream_t s)
{
  for (int b = 0; b < nb; b += kDiagMost) {
    const int n = nb - b < kDiagMost ? nb - b : kDiagMost;
    const long long at = (long long)b * p->L;
    k_lapla<<<diag_grid(p, n), 256, 0, s>>>(w + at, p->d_rn, n, p->L, out + at, inverse ? 1 : 0);
    count_launch();
  }
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? SHT_OK : cuda_fail(e, "k_lapla");
}

int launch_diffuse(const sht_plan *p, const double *w, int nb, const double *coef, double dt,
                   const double *filter, double *out, cudaStream_t s)
{
  for (int b = 0; b < nb; b += kDiagMost) {
    const int n = nb - b < kDiagMost ? nb - b : kDiagMost;
    const long long at = (long long)b * p->L;
    k_diffuse<<<diag_grid(p, n), 256, 0, s>>>(w + at, n, p->L, coef, dt, filter, out + at);
    count_launch();
  }
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? SHT_OK : cuda_fail(e, "k_diffuse");
}

int launch_sub_filter(const sht_plan *p, double *a, const double *w, int nb, const double *filter, cudaStream_t s)
{
  for (int b = 0; b < nb; b += kDiagMost) {
    const int n = nb - b < kDiagMost ? nb - b : kDiagMost;
    const long long at = (long long)b * p->L;
    k_sub_filter<<<diag_grid(p, n), 256, 0, s>>>(a + at, w + at, n, p->L, filter);
    count_launch();
  }
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? SHT_OK : cuda_fail(e, "k_sub_filter");
}

int launch_sub_lapla(const sht_plan *p, double *a, double *neg, const double *c, int nb, cudaStream_t s)
{
  for (int b = 0; b < nb; b += kDiagMost) {
    const int n = nb - b < kDiagMost ? nb - b : kDiagMost;
    const long long at = (long long)b * p->L;
    k_sub_lapla<<<diag_grid(p, n), 256, 0, s>>>(a + at, neg + at, c + at, p->d_rn, n, p->L);
    count_launch();
  }
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? SHT_OK : cuda_fail(e, "k_sub_lapla");
}

int launch_lonlat_reduce(const sht_plan *p, const double *g, int nb, double *out, int kind, cudaStream_t s)
{
  if (nb <= 0) return SHT_OK;
  k_lonlat<<<nb, 256, 0, s>>>(g, p->I, p->J, p->d_wgt, out, kind);
  count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? SHT_OK : cuda_fail(e, "k_lonlat");
}

}  // namespace sht
