// sht_spectral.cuh -- the spectral-side operators, element by element: what an
// entry of the SPML layout becomes in the internal one and the reverse, shared
// by the layout conversions of sht_spectral.cu and the narrow-batch kernels of
// sht_narrow.cu.  The formulas are listed at the top of sht_spectral.cu.
#pragma once

#include "sht_internal.h"

namespace sht {
namespace spec {

constexpr double kSqrt2 = 1.41421356237309504880;
constexpr double kRSqrt2 = 0.70710678118654752440;

struct SpecArgs {
  const double2 *S;   // pack input
  double2 *So;        // unpack output
  int ncolS;
  const double *w0, *w1;  // unpack inputs
  double *o0, *o1;        // pack outputs
  int nb, N, L;
  double radius;
  const double *eps;      // [m][n], n = 0..N+2
  const int2 *tiles;      // (n, m0) per tile
  double *const *ocol;        // optional per-field-level pack destinations
  const double *const *icol;  // optional per-field-level unpack sources
  int M;                      // orders present: N + 1, or 1 for a zonal plan
  int zonal;                  // SPML index l = n (wa_zonal_module) instead of n(n+1) +- m
};

// 0-based SPML index of (n, m), cos (sn = 0) or sin (sn = 1) part
__device__ __forceinline__ long long spml_l(const SpecArgs &a, int n, int m, int sn)
{
  return a.zonal ? (long long)n : (long long)n * (n + 1) + (sn ? -m : m);
}

__device__ __forceinline__ double eps_at(const SpecArgs &a, int m, int n)
{
  return (n < 0 || n > a.N + 2) ? 0.0 : __ldg(a.eps + (long long)m * (a.N + 3) + n);
}

// Internal row of (m, n): rowoff(m) + n - m, with rowoff(m) = sum over m' < m
// of the N + 2 - m' rows of band m' (the plan's row table in closed form, so
// that no dependent load precedes the coefficient loads)
__device__ __forceinline__ int spec_row(int N, int m, int n) { return m * (N + 2) - m * (m - 1) / 2 + (n - m); }
__device__ __forceinline__ double2 cadd(double2 x, double2 y) { return make_double2(x.x + y.x, x.y + y.y); }
__device__ __forceinline__ double2 csub(double2 x, double2 y) { return make_double2(x.x - y.x, x.y - y.y); }
__device__ __forceinline__ double2 cscale(double2 x, double s) { return make_double2(x.x * s, x.y * s); }
__device__ __forceinline__ double2 times_im(double2 x, int m) { return make_double2(-m * x.y, m * x.x); }

// Which internal rows a pack operator reads: degree offset dn in -1..1 of
// column set `set` (0: the first input's columns, 1: the second's).
template <int OP>
__host__ __device__ constexpr bool pack_needs(int dn, int set)
{
  return OP == PACK_PLAIN || OP == PACK_DIVLAMBDA ? (dn == 0 && set == 0)
       : OP == PACK_DIVMU                         ? (dn != 0 && set == 0)
       : OP == PACK_ALPHA                         ? (set == 0 ? dn == 0 : dn != 0)
                                                  : true;  // VORDIV
}

// The outputs of a pack operator at (n, m): c[dn + 1][set], e0 = eps_n^m, e1 =
// eps_{n+1}^m; without the SPML factor sqrt(2) of m > 0.
template <int OP>
__device__ __forceinline__ void pack_combine(const double2 (&c)[3][2], int n, int m, double e0, double e1, double radius,
                                             double2 &v0, double2 &v1)
{
  auto D = [&](int set) -> double2 {  // -( (n+1) eps_n c_{n-1} - n eps_{n+1} c_{n+1} )
    const double f0 = (n + 1) * e0, f1 = n * e1;
    const double2 cm = c[0][set], cp = c[2][set];
    return make_double2(f1 * cp.x - f0 * cm.x, f1 * cp.y - f0 * cm.y);
  };
  if (OP == PACK_PLAIN) {
    v0 = c[1][0];
  } else if (OP == PACK_DIVLAMBDA) {
    v0 = times_im(c[1][0], m);
  } else if (OP == PACK_DIVMU) {
    v0 = D(0);
  } else if (OP == PACK_ALPHA) {
    v0 = cscale(cadd(times_im(c[1][0], m), D(1)), 1.0 / radius);
  } else {  // PACK_VORDIV: set 0 = U cos, set 1 = V cos
    v0 = cscale(csub(times_im(c[1][1], m), D(0)), 1.0 / radius);
    v1 = cscale(cadd(times_im(c[1][0], m), D(1)), 1.0 / radius);
  }
}

// Which SPML entries an unpack operator reads: input `in`, degree offset dn.
template <int OP>
__host__ __device__ constexpr bool unpack_needs(int in, int dn)
{
  return OP == UNPACK_PLAIN || OP == UNPACK_GRADLAMBDA ? (in == 0 && dn == 0)
       : OP == UNPACK_GRADMU                          ? (in == 0 && dn != 0)
       : OP == UNPACK_HGRAD                           ? (in == 0)
       : OP == UNPACK_ALPHA                           ? (in == 0 ? dn == 0 : dn != 0)
                                                      : true;  // VORDIV2UV
}
template <int OP>
__host__ __device__ constexpr int unpack_outputs() { return OP == UNPACK_VORDIV2UV || OP == UNPACK_HGRAD ? 2 : 1; }

// -a^2/(k(k+1)) for the degrees k = n - 1, n, n + 1 (zero for k < 1)
template <int OP>
__device__ __forceinline__ void lap_factors(int n, double radius, double (&lap)[3])
{
  lap[0] = lap[1] = lap[2] = 0.0;
  if constexpr (OP == UNPACK_VORDIV2UV) {
    const double a2 = radius * radius;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double k = n + d - 1.0;
      lap[d] = k >= 1.0 ? -a2 / (k * (k + 1.0)) : 0.0;
    }
  }
}

// The outputs of an unpack operator at (n, m) from the SPML entries
// x[input][dn + 1][cos/sin]; ep = (n+2) eps_{n+1}, em = (n-1) eps_n of
// R(x)_n = ep x_{n+1} - em x_{n-1}; s the SPML factor (1/sqrt(2) for m > 0).
template <int OP, int NIN>
__device__ __forceinline__ void unpack_combine(const double (&x)[NIN][3][2], int m, double ep, double em,
                                               const double (&lap)[3], double s, double2 &v0, double2 &v1)
{
  auto coef = [&](int in, int dn) { return make_double2(x[in][dn + 1][0] * s, x[in][dn + 1][1] * s); };
  auto R = [&](int in, bool inv_lap) {
    double2 xp = coef(in, 1), xm = coef(in, -1);
    if (inv_lap) {
      xp = cscale(xp, lap[2]);
      xm = cscale(xm, lap[0]);
    }
    return make_double2(ep * xp.x - em * xm.x, ep * xp.y - em * xm.y);
  };
  if (OP == UNPACK_PLAIN) {
    v0 = coef(0, 0);
  } else if (OP == UNPACK_GRADLAMBDA) {
    v0 = times_im(coef(0, 0), m);
  } else if (OP == UNPACK_GRADMU) {
    v0 = R(0, false);
  } else if (OP == UNPACK_HGRAD) {
    v0 = times_im(coef(0, 0), m);
    v1 = R(0, false);
  } else if (OP == UNPACK_ALPHA) {
    v0 = cadd(times_im(coef(0, 0), m), R(NIN - 1, false));
  } else {  // UNPACK_VORDIV2UV: input 0 = vor, 1 = div
    const double2 psi = cscale(coef(0, 0), lap[1]), chi = cscale(coef(NIN - 1, 0), lap[1]);
    v0 = csub(times_im(chi, m), R(0, true));
    v1 = cadd(times_im(psi, m), R(NIN - 1, true));
  }
}

}  // namespace spec
}  // namespace sht
