// sht_narrow.cu -- Legendre contraction and spectral layout conversion in one
// kernel, for batches of a few field-levels.
//
// A model's 2-D fields and its per-level loops call the transform with one
// level at a time.  Such a call is bound by its launches (three kernels of 2 to
// 6 us, 3 us of host time each), so here the contraction and the conversion
// share one: an order's coefficients of all degrees fit in one block, and the
// operators couple degrees of one order only.  A block takes one order m and
// four complex columns (the two inputs or outputs of two levels, or four
// levels), and its warps take (parity, 8-row tile) units of FP64 products
// (mma.sync.m8n8k4.f64, the four columns' real and imaginary parts as the
// eight-wide side).
//   analysis:  Fourier columns -> shared memory | products, table blocks read
//              from L2 | operator (pack_combine) and SPML entries
//   synthesis: SPML entries, operator (unpack_combine) -> coefficients in
//              shared memory | products | Fourier runs
// Sums: space_discretization.tex:197-200 and :212-216, tables and layouts as in
// sht_legendre_band.cu.  The SPML entries are 8-byte accesses at stride 2n,
// which a wide batch would pay for; the rule for taking these kernels is at
// use_narrow.
#include "sht_spectral.cuh"
#include "sht_dmma.cuh"
#include "sht_l2.cuh"

namespace sht {

namespace {

using namespace spec;
using dmma::mma884;

constexpr int kNT = 256, kNW = kNT / 32;

struct NarrowArgs {
  SpecArgs s;           // spectra, operator data (S and tiles unused)
  const double *P;      // blocked Legendre table
  const long long *boff;
  const double2 *F;     // analysis input
  double2 *Fo;          // synthesis output
  int J, JH, ncol;
};

// Coefficient rows of a block: [parity][k] of six double2 (four columns; the
// stride spreads a fragment load over all banks)
constexpr int kCS = 6;
__host__ __device__ __forceinline__ int row_cap(int N, int m) { return ((N + 3 - m) / 2 + 7) & ~7; }  // rows of one parity, padded

template <int OP>
__global__ void __launch_bounds__(kNT) k_narrow_inv(NarrowArgs a)
{
  constexpr int NIN = (OP == UNPACK_ALPHA || OP == UNPACK_VORDIV2UV) ? 2 : 1;
  constexpr int NOUT = unpack_outputs<OP>(), G = 4 / NOUT;
  extern __shared__ __align__(16) double2 sm_narrow[];
  const int m = blockIdx.x, b0 = blockIdx.y * G;
  const int N = a.s.N, R = N + 2 - m, Kp = row_cap(N, m);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

  const double s = (m == 0) ? 1.0 : kRSqrt2;
  for (int idx = threadIdx.x; idx < 2 * Kp * G; idx += kNT) {
    const int r = idx / G, g = idx % G, n = m + r, b = b0 + g;
    double2 v0 = make_double2(0.0, 0.0), v1 = v0;
    if (r < R && b < a.s.nb) {
      double x[NIN][3][2];
#pragma unroll
      for (int in = 0; in < NIN; ++in) {
        const double *w = (in == 0 ? a.s.w0 : a.s.w1) + (long long)b * a.s.L;
#pragma unroll
        for (int d = 0; d < 3; ++d)
#pragma unroll
          for (int sn = 0; sn < 2; ++sn) {
            const int nn = n + d - 1;
            const bool ok = unpack_needs<OP>(in, d - 1) && nn >= m && nn <= N && !(sn && m == 0);
            x[in][d][sn] = ok ? __ldg(w + spml_l(a.s, nn, m, sn)) : 0.0;
          }
      }
      double ep = 0.0, em = 0.0, lap[3];
      if (OP != UNPACK_PLAIN && OP != UNPACK_GRADLAMBDA) {
        ep = (n + 2) * eps_at(a.s, m, n + 1);
        em = (n - 1) * eps_at(a.s, m, n);
      }
      lap_factors<OP>(n, a.s.radius, lap);
      unpack_combine<OP>(x, m, ep, em, lap, s, v0, v1);
    }
    double2 *row = sm_narrow + ((r & 1) * Kp + (r >> 1)) * kCS;
    row[g] = v0;
    if constexpr (NOUT == 2) row[G + g] = v1;
  }
  __syncthreads();

  const int nlt = (a.JH + 7) >> 3, nn = lane >> 2, q = lane & 3;
  const double *sd = reinterpret_cast<const double *>(sm_narrow);
  for (int unit = warp; unit < 2 * nlt; unit += kNW) {
    const int par = unit >= nlt, lt = unit - par * nlt;
    const int cnt = par ? R / 2 : (R + 1) / 2, nrt = (cnt + 7) >> 3;
    const double *P = a.P + (a.boff[2 * m + par] + (long long)lt * nrt) * 64 + 8 * q + (nn ^ (4 * (q >> 1)));
    const double *B = sd + (par * Kp + q) * 2 * kCS + nn;
    double acc[2] = {0.0, 0.0};  // one chain, in the order of the band kernels: the same bits in any batch
#pragma unroll 4
    for (int rt = 0; rt < nrt; ++rt) {
      const double p0 = __ldg(P + rt * 64), p1 = __ldg(P + rt * 64 + 32);
      mma884(acc, p0, B[rt * 16 * kCS]);
      mma884(acc, p1, B[rt * 16 * kCS + 8 * kCS]);
    }
    const int jh = 8 * lt + nn, b = b0 + q % G;
    if (jh < a.JH && b < a.s.nb)
      a.Fo[((long long)m * a.ncol + (q / G) * a.s.nb + b) * a.J + par * a.JH + jh] =
          make_double2(acc[0], acc[1]);
  }
}

template <int OP>
__global__ void __launch_bounds__(kNT) k_narrow_fwd(NarrowArgs a)
{
  constexpr int NSET = (OP == PACK_ALPHA || OP == PACK_VORDIV) ? 2 : 1, G = 4 / NSET;
  constexpr int NOUT = (OP == PACK_VORDIV) ? 2 : 1;
  extern __shared__ __align__(16) double2 sm_narrow[];
  const int m = blockIdx.x, b0 = blockIdx.y * G;
  const int N = a.s.N, R = N + 2 - m, nlt = (a.JH + 7) >> 3, JHp = 8 * nlt;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double2 *const Fs = sm_narrow, *const C = sm_narrow + 4 * (2 * JHp + 1);  // columns 2 JHp + 1 apart: conflict-free fragments

  for (int idx = threadIdx.x; idx < 8 * JHp; idx += kNT) {
    const int c = idx / (2 * JHp), e = idx - c * 2 * JHp, par = e >= JHp, jh = e - par * JHp, b = b0 + c % G;
    double2 v = make_double2(0.0, 0.0);
    if (jh < a.JH && b < a.s.nb) v = a.F[((long long)m * a.ncol + (c / G) * a.s.nb + b) * a.J + par * a.JH + jh];
    Fs[c * (2 * JHp + 1) + e] = v;
  }
  __syncthreads();

  const int nn = lane >> 2, q = lane & 3;
  const int cntE = (R + 1) / 2, cntO = R / 2, tE = (cntE + 7) >> 3, tO = (cntO + 7) >> 3;
  const double *fd = reinterpret_cast<const double *>(Fs) + 2 * ((nn >> 1) * (2 * JHp + 1) + 2 * q) + (nn & 1);
  for (int unit = warp; unit < tE + tO; unit += kNW) {
    const int par = unit >= tE, rt = unit - par * tE, cnt = par ? cntO : cntE, nrt = par ? tO : tE;
    const double *P = a.P + (a.boff[2 * m + par] + rt) * 64 + 8 * nn + 2 * (q ^ (nn & 2));
    const double *B = fd + 2 * par * JHp;
    double acc[2] = {0.0, 0.0};  // one chain, in the order of the band kernels: the same bits in any batch
#pragma unroll 4
    for (int lt = 0; lt < nlt; ++lt) {
      // the two steps take latitudes 2q and 2q + 1 of the tile's eight
      const double2 p = __ldg(reinterpret_cast<const double2 *>(P + (long long)lt * nrt * 64));
      mma884(acc, p.x, B[16 * lt]);
      mma884(acc, p.y, B[16 * lt + 2]);
    }
    const int k = 8 * rt + nn;
    if (k < cnt) C[(2 * k + par) * 4 + q] = make_double2(acc[0], acc[1]);
  }
  __syncthreads();

  const double s = (m == 0) ? 1.0 : kSqrt2;
  for (int idx = threadIdx.x; idx < (N + 1 - m) * G; idx += kNT) {
    const int r = idx / G, g = idx % G, n = m + r, b = b0 + g;
    if (b >= a.s.nb) continue;
    double2 c[3][2];
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
      for (int set = 0; set < 2; ++set) {
        const int rr = r + d - 1;
        c[d][set] = make_double2(0.0, 0.0);
        if (pack_needs<OP>(d - 1, set) && rr >= 0 && rr < R) c[d][set] = C[rr * 4 + set * G + g];
      }
    double e0 = 0.0, e1 = 0.0;
    if (OP != PACK_PLAIN && OP != PACK_DIVLAMBDA) {
      e0 = eps_at(a.s, m, n);
      e1 = eps_at(a.s, m, n + 1);
    }
    double2 v0 = make_double2(0.0, 0.0), v1 = v0;
    pack_combine<OP>(c, n, m, e0, e1, a.s.radius, v0, v1);
    const long long lc = spml_l(a.s, n, m, 0), ls = spml_l(a.s, n, m, 1);
    double *w = a.s.o0 + (long long)b * a.s.L;
    w[lc] = v0.x * s;
    if (m > 0) w[ls] = v0.y * s;
    if constexpr (NOUT == 2) {
      w = a.s.o1 + (long long)b * a.s.L;
      w[lc] = v1.x * s;
      if (m > 0) w[ls] = v1.y * s;
    }
  }
}

NarrowArgs narrow_args(const sht_plan *p, int nb, int ncol)
{
  NarrowArgs a{};
  a.s.nb = nb; a.s.N = p->N; a.s.L = p->L; a.s.radius = p->radius;
  a.s.eps = p->d_eps; a.s.M = p->M; a.s.zonal = p->zonal ? 1 : 0;
  a.P = p->d_band_P; a.boff = p->d_band_off;
  a.J = p->J; a.JH = p->JH; a.ncol = ncol;
  return a;
}

size_t smem_inv(const sht_plan *p) { return sizeof(double2) * 2 * row_cap(p->N, 0) * kCS; }
size_t smem_fwd(const sht_plan *p)
{
  const size_t JHp = (p->JH + 7) & ~7;
  return sizeof(double2) * (4 * (2 * JHp + 1) + 4 * (size_t)(p->N + 2));
}

int launch(void (*kern)(NarrowArgs), size_t smem, int groups, const NarrowArgs &a, cudaStream_t s, const char *name)
{
  cudaError_t e = kernel_setup((const void *)kern, smem, kNT);
  if (e != cudaSuccess) return cuda_fail(e, name);
  kern<<<dim3((unsigned)a.s.M, (unsigned)groups), kNT, smem, s>>>(a);
  count_launch();
  e = cudaGetLastError();
  return e == cudaSuccess ? SHT_OK : cuda_fail(e, name);
}

}  // namespace

// Narrow enough for these kernels: groups of four columns times the size of the
// contraction.  Both kernels of the wide path against the one here, us,
// synthesis / analysis (a saved launch is worth about one more): one level T21
// 4.7 / 4.7 -> 2.4 / 2.8, T85 5.8 / 6.2 -> 4.2 / 4.6, T170 8.5 / 10.7 -> 8.3 /
// 8.2; at the line T42, 160 columns 7.3 / 7.4 -> 6.1 / 6.9, T85, 60 9.4 / 10.6
// -> 9.7 / 10.5, T106, 32 9.2 / 10.1 -> 9.7 / 11.4; above it T85, 96 11.4 / 12.4
// -> 13.3 / 14.6, T170, 16 11.5 / 12.6 -> 14.6 / 15.9.
bool use_narrow(const sht_plan *p, int nb, int sets)
{
  const size_t lim = 227 * 1024;
  const long long groups = (nb + 4 / sets - 1) / (4 / sets);
  return groups * (p->N + 2) * p->JH <= 84000 && smem_inv(p) <= lim && smem_fwd(p) <= lim;
}

int launch_narrow_fwd(const sht_plan *p, int op, const double2 *F, int ncol, int nb, double *w0, double *w1, cudaStream_t s)
{
  if (nb <= 0) return SHT_OK;
  NarrowArgs a = narrow_args(p, nb, ncol);
  a.F = F; a.s.o0 = w0; a.s.o1 = w1 ? w1 : w0;
  const size_t smem = smem_fwd(p);
  const int g4 = (nb + 3) / 4, g2 = (nb + 1) / 2;
  switch (op) {
  case PACK_PLAIN: return launch(k_narrow_fwd<PACK_PLAIN>, smem, g4, a, s, "k_narrow_fwd");
  case PACK_DIVLAMBDA: return launch(k_narrow_fwd<PACK_DIVLAMBDA>, smem, g4, a, s, "k_narrow_fwd");
  case PACK_DIVMU: return launch(k_narrow_fwd<PACK_DIVMU>, smem, g4, a, s, "k_narrow_fwd");
  case PACK_ALPHA: return launch(k_narrow_fwd<PACK_ALPHA>, smem, g2, a, s, "k_narrow_fwd");
  case PACK_VORDIV: return launch(k_narrow_fwd<PACK_VORDIV>, smem, g2, a, s, "k_narrow_fwd");
  default: set_error("pack: unknown operator"); return SHT_ERR_INVALID_ARG;
  }
}

int launch_narrow_inv(const sht_plan *p, int op, const double *w0, const double *w1, int nb, double2 *F, int ncol,
                      cudaStream_t s)
{
  if (nb <= 0) return SHT_OK;
  NarrowArgs a = narrow_args(p, nb, ncol);
  a.Fo = F; a.s.w0 = w0; a.s.w1 = w1 ? w1 : w0;
  const size_t smem = smem_inv(p);
  const int g4 = (nb + 3) / 4, g2 = (nb + 1) / 2;
  switch (op) {
  case UNPACK_PLAIN: return launch(k_narrow_inv<UNPACK_PLAIN>, smem, g4, a, s, "k_narrow_inv");
  case UNPACK_GRADLAMBDA: return launch(k_narrow_inv<UNPACK_GRADLAMBDA>, smem, g4, a, s, "k_narrow_inv");
  case UNPACK_GRADMU: return launch(k_narrow_inv<UNPACK_GRADMU>, smem, g4, a, s, "k_narrow_inv");
  case UNPACK_ALPHA: return launch(k_narrow_inv<UNPACK_ALPHA>, smem, g4, a, s, "k_narrow_inv");
  case UNPACK_VORDIV2UV: return launch(k_narrow_inv<UNPACK_VORDIV2UV>, smem, g2, a, s, "k_narrow_inv");
  case UNPACK_HGRAD: return launch(k_narrow_inv<UNPACK_HGRAD>, smem, g2, a, s, "k_narrow_inv");
  default: set_error("unpack: unknown operator"); return SHT_ERR_INVALID_ARG;
  }
}

}  // namespace sht
