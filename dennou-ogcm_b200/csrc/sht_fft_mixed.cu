// sht_fft_mixed.cu -- batched real FFT in longitude for counts with factors 3
// and 5 (96, 160, 192, 240, 320, 384, 480, 640, ... points; the counts that
// ISPACK's FFT takes, util/grid/DOGCM_GaussSpmVFvmGrid_mod.f90:209-211).
//
// Same sums, row scales, Gs/Ga and E/O layouts as the power-of-two kernels of
// sht_fft.cu.  A row of I = 2 NC real points is NC complex points, transformed
// in two passes, NC = R1 R2, with both radices at most 16 (or 32) and run-time
// values: each pass switches once per tile to the code of its radix.  A tile
// is JT/2 mirrored row pairs of one field-level in one shared-memory buffer,
// row r at r RS; element (k1, u) of a row sits at k1 S + u with S odd, so that
// both the first pass (lanes along u) and the second (lanes along k1, stride
// S) touch eight distinct 16-byte bank groups per phase, and RS is odd, so that
// lanes along the rows do too.  Every pass works in place on its own elements:
//
//   forward:  load rows, R1-point DFTs, twiddle, store (k1, u) | R2-point DFTs
//             in place | real unpack of Z_m and Z_{NC-m}, sums over the mirrored
//             rows, runs of JT/2 rows to the Fourier array
//   inverse:  Fourier runs -> north/south rows -> real pack of Z_k and Z_{NC-k}
//             | R1-point DFTs, twiddle | R2-point DFTs, scale, store rows
//
// A tile's loads overlap other resident blocks' arithmetic (three to five
// blocks per SM).  What it replaces, the direct sum over longitudes, is O(I N)
// per row and bound by its FP64 products.  The T106 grid (320 x 160, 180
// field-levels, 123 MB per direction): forward / inverse 0.730 / 1.289 ms ->
// 0.034 / 0.038 ms with cold caches, 3.6 / 3.2 TB/s (0.031 / 0.037 back to back);
// 192 x 96, 74 columns: 61 / 112 -> 9.5 / 11.3 us (6.9 / 7.1 back to back).
#include "sht_fft_tile.cuh"
#include "sht_fft_mixed.cuh"

#include <algorithm>
#include <type_traits>

namespace sht {

namespace {

// cos(2 pi t / R) and sin(2 pi t / R) for the twiddles inside the 9-, 25- and
// 27-point transforms (32 significant digits, rounded once)
__host__ __device__ constexpr double tcos(int R, int t)
{
  if (R == 9) {
    constexpr double c[5] = {1.0, 0.76604444311897803520239265055542, 0.17364817766693034885171662676931, -0.5,
      -0.93969262078590838405410927732473};
    return c[t];
  }
  if (R == 25) {
    constexpr double c[17] = {1.0, 0.96858316112863111949016837546474, 0.87630668004386358730811590392206,
      0.72896862742141152314673031905526, 0.53582679497899661827130876786764,
      0.30901699437494742410229341718282, 0.062790519529313376076178224565631,
      -0.18738131458572463054255073444729, -0.42577929156507264886250244574425,
      -0.63742398974868971017671281167602, -0.80901699437494742410229341718282,
      -0.92977648588825140366094255622199, -0.99211470131447783104979304278578,
      -0.99211470131447783104979304278578, -0.92977648588825140366094255622199,
      -0.80901699437494742410229341718282, -0.63742398974868971017671281167602};
    return c[t];
  }
  constexpr double c[17] = {1.0, 0.9730448705798238388328851727847, 0.89363264032341224819257418686666,
      0.76604444311897803520239265055542, 0.59715859170278616485185216058396,
      0.39607976603915682369604339160974, 0.17364817766693034885171662676931,
      -0.058144828910475828538748016847072, -0.28680323271109025310328017316716, -0.5,
      -0.68624163786873358572960499961754, -0.83548781141293641965382617001958,
      -0.93969262078590838405410927732473, -0.9932383577419429885478955521937,
      -0.9932383577419429885478955521937, -0.93969262078590838405410927732473,
      -0.83548781141293641965382617001958};
  return c[t];
}
__host__ __device__ constexpr double tsin(int R, int t)
{
  if (R == 9) {
    constexpr double c[5] = {0.0, 0.64278760968653932632264340990726, 0.98480775301220805936674302458952,
      0.86602540378443864676372317075294, 0.34202014332566873304409961468226};
    return c[t];
  }
  if (R == 25) {
    constexpr double c[17] = {0.0, 0.24868988716485478824228374600645, 0.48175367410171527498719150287213,
      0.68454710592868867373228335762121, 0.84432792550201507854855806396668,
      0.95105651629515357211643933337938, 0.99802672842827156195233680686345,
      0.98228725072868868108564174286527, 0.9048270524660195277136686479327,
      0.77051324277578923080300963639618, 0.58778525229247312916870595463907,
      0.36812455268467795915694714749296, 0.12533323356430424537311875981651,
      -0.12533323356430424537311875981651, -0.36812455268467795915694714749296,
      -0.58778525229247312916870595463907, -0.77051324277578923080300963639618};
    return c[t];
  }
  constexpr double c[17] = {0.0, 0.23061587074244017845019834929294, 0.44879918020046217278504033473314,
      0.64278760968653932632264340990726, 0.80212319275504378508329489193393,
      0.91821610688027401475896141531464, 0.98480775301220805936674302458952,
      0.99830815827126820804782070878328, 0.95798951231548887443737476695675,
      0.86602540378443864676372317075294, 0.72737364157304869598717641766382,
      0.54950897807080603526278037405013, 0.34202014332566873304409961468226,
      0.11609291412523022967566652338071, -0.11609291412523022967566652338071,
      -0.34202014332566873304409961468226, -0.54950897807080603526278037405013};
  return c[t];
}

__host__ __device__ constexpr int cgcd(int a, int b) { return b == 0 ? a : cgcd(b, a % b); }
// a^-1 mod m (m small)
__host__ __device__ constexpr int cinv(int a, int m)
{
  for (int x = 0; x < m; ++x)
    if ((a * x) % m == 1 % m) return x;
  return 0;
}
// first factor of a composite radix: the power of two of it, else its 3
__host__ __device__ constexpr int first_factor(int R)
{
  int p = 1;
  while (R % (2 * p) == 0) p *= 2;
  return p > 1 ? p : 3 * (R % 3 == 0) + 5 * (R % 3 != 0);
}
__host__ __device__ constexpr int log2i(int R) { return R <= 1 ? 0 : 1 + log2i(R / 2); }

// In-register DFT of R points, natural order in and out, sign -1 or +1 (INV).
// Powers of two by the radix-2 code of sht_fft_tile.cuh; 3 and 5 by their
// symmetric forms (sums and differences of the conjugate pairs); coprime
// products by the prime-factor index maps (Good 1958), which need no
// twiddles; 9 = 3 x 3, 25 = 5 x 5 and 27 = 3 x 9 by Cooley-Tukey.
template <int R, bool INV>
__device__ __forceinline__ void dft_nat(double2 (&v)[R])
{
  if constexpr (R == 1) {
    return;
  } else if constexpr ((R & (R - 1)) == 0) {
    constexpr int LOG = log2i(R);
    dft_reg<LOG, INV>(v);
    double2 t[R];
#pragma unroll
    for (int k = 0; k < R; ++k) t[k] = v[brev<LOG>(k)];
#pragma unroll
    for (int k = 0; k < R; ++k) v[k] = t[k];
  } else if constexpr (R == 3) {
    constexpr double s3 = INV ? -0.86602540378443864676372317075294 : 0.86602540378443864676372317075294;
    const double2 s = make_double2(v[1].x + v[2].x, v[1].y + v[2].y);
    const double dx = s3 * (v[1].x - v[2].x), dy = s3 * (v[1].y - v[2].y);
    const double2 t = make_double2(v[0].x - 0.5 * s.x, v[0].y - 0.5 * s.y);
    v[0] = make_double2(v[0].x + s.x, v[0].y + s.y);
    v[1] = make_double2(t.x + dy, t.y - dx);
    v[2] = make_double2(t.x - dy, t.y + dx);
  } else if constexpr (R == 5) {
    constexpr double c1 = 0.30901699437494742410229341718282, c2 = -0.80901699437494742410229341718282;
    constexpr double s1 = INV ? -0.95105651629515357211643933337938 : 0.95105651629515357211643933337938;
    constexpr double s2 = INV ? -0.58778525229247312916870595463907 : 0.58778525229247312916870595463907;
    const double2 p = make_double2(v[1].x + v[4].x, v[1].y + v[4].y), q = make_double2(v[2].x + v[3].x, v[2].y + v[3].y);
    const double2 d = make_double2(v[1].x - v[4].x, v[1].y - v[4].y), e = make_double2(v[2].x - v[3].x, v[2].y - v[3].y);
    const double2 m1 = make_double2(fma(c2, q.x, fma(c1, p.x, v[0].x)), fma(c2, q.y, fma(c1, p.y, v[0].y)));
    const double2 m2 = make_double2(fma(c1, q.x, fma(c2, p.x, v[0].x)), fma(c1, q.y, fma(c2, p.y, v[0].y)));
    const double2 n1 = make_double2(fma(s2, e.x, s1 * d.x), fma(s2, e.y, s1 * d.y));
    const double2 n2 = make_double2(fma(-s1, e.x, s2 * d.x), fma(-s1, e.y, s2 * d.y));
    v[0] = make_double2(v[0].x + p.x + q.x, v[0].y + p.y + q.y);
    v[1] = make_double2(m1.x + n1.y, m1.y - n1.x);
    v[4] = make_double2(m1.x - n1.y, m1.y + n1.x);
    v[2] = make_double2(m2.x + n2.y, m2.y - n2.x);
    v[3] = make_double2(m2.x - n2.y, m2.y + n2.x);
  } else {
    constexpr int P = first_factor(R), Q = R / P;
    double2 a[Q][P], out[R];
    if constexpr (cgcd(P, Q) == 1) {
      constexpr int eP = Q * cinv(Q % P, P), eQ = P * cinv(P % Q, Q);  // 1 mod P and 0 mod Q, and the reverse
#pragma unroll
      for (int n2 = 0; n2 < Q; ++n2) {
#pragma unroll
        for (int n1 = 0; n1 < P; ++n1) a[n2][n1] = v[(Q * n1 + P * n2) % R];
        dft_nat<P, INV>(a[n2]);
      }
#pragma unroll
      for (int k1 = 0; k1 < P; ++k1) {
        double2 b[Q];
#pragma unroll
        for (int n2 = 0; n2 < Q; ++n2) b[n2] = a[n2][k1];
        dft_nat<Q, INV>(b);
#pragma unroll
        for (int k2 = 0; k2 < Q; ++k2) out[(k1 * eP + k2 * eQ) % R] = b[k2];
      }
    } else {
#pragma unroll
      for (int n2 = 0; n2 < Q; ++n2) {
#pragma unroll
        for (int n1 = 0; n1 < P; ++n1) a[n2][n1] = v[Q * n1 + n2];
        dft_nat<P, INV>(a[n2]);
      }
#pragma unroll
      for (int k1 = 0; k1 < P; ++k1) {
        double2 b[Q];
#pragma unroll
        for (int n2 = 0; n2 < Q; ++n2) {
          const int t = n2 * k1;
          const double c = tcos(R, t), s = INV ? -tsin(R, t) : tsin(R, t);  // e^{-+ 2 pi i t / R}
          const double2 x = a[n2][k1];
          b[n2] = t == 0 ? x : make_double2(x.x * c + x.y * s, x.y * c - x.x * s);
        }
        dft_nat<Q, INV>(b);
#pragma unroll
        for (int k2 = 0; k2 < Q; ++k2) out[k1 + P * k2] = b[k2];
      }
    }
#pragma unroll
    for (int k = 0; k < R; ++k) v[k] = out[k];
  }
}

struct MixArgs {
  FftArgs f;
  int R1, R2, S, RS;  // radices and the buffer's strides (double2)
  int lgh;            // log2 of the row pairs per tile
};

// Runs F<radix>(...) for a run-time radix of the class.
template <int MAXR, class F>
__device__ __forceinline__ void with_radix(int r, F &&f)
{
  using std::integral_constant;
  switch (r) {
  case 2: f(integral_constant<int, 2>()); break;
  case 3: f(integral_constant<int, 3>()); break;
  case 4: f(integral_constant<int, 4>()); break;
  case 5: f(integral_constant<int, 5>()); break;
  case 6: f(integral_constant<int, 6>()); break;
  case 8: f(integral_constant<int, 8>()); break;
  case 9: f(integral_constant<int, 9>()); break;
  case 10: f(integral_constant<int, 10>()); break;
  case 12: f(integral_constant<int, 12>()); break;
  case 15: f(integral_constant<int, 15>()); break;
  case 16: f(integral_constant<int, 16>()); break;
  default:
    if constexpr (MAXR > 16) {
      if (r == 18) f(integral_constant<int, 18>());
      if (r == 20) f(integral_constant<int, 20>());
    }
    if constexpr (MAXR > 20) {
      switch (r) {
      case 24: f(integral_constant<int, 24>()); break;
      case 25: f(integral_constant<int, 25>()); break;
      case 27: f(integral_constant<int, 27>()); break;
      case 30: f(integral_constant<int, 30>()); break;
      case 32: f(integral_constant<int, 32>()); break;
      default: break;
      }
    }
  }
}

struct MixShared {
  double2 *buf, *stw, *stwI;
  unsigned short *pos;
};

__device__ __forceinline__ MixShared mix_shared(const MixArgs &a, int NC)
{
  extern __shared__ __align__(16) double2 smem_mix[];
  MixShared s;
  s.stw = smem_mix;               // stw[k1 R2 + u] = e^{-2 pi i u k1 / NC}
  s.stwI = smem_mix + NC;         // e^{-2 pi i m / I}
  s.buf = smem_mix + 2 * NC;
  s.pos = reinterpret_cast<unsigned short *>(s.buf + (2 << a.lgh) * a.RS);
  for (int q = threadIdx.x; q < NC; q += blockDim.x) {
    s.stw[q] = __ldg(a.f.tw + (q % a.R2) * (q / a.R2));
    s.stwI[q] = __ldg(a.f.twI + q);
  }
  return s;
}

template <int MAXR, int MUL>
__global__ void __launch_bounds__(256, MAXR <= 16 ? 2 : 1) k_mix_fwd(MixArgs a)
{
  const FftArgs &f = a.f;
  const int NC = f.I / 2, R1 = a.R1, R2 = a.R2, S = a.S, RS = a.RS;
  const int JTh = 1 << a.lgh, NT = blockDim.x, tid = threadIdx.x;
  const MixShared sh = mix_shared(a, NC);
  double2 *const buf = sh.buf;
  for (int m = tid; m < NC; m += NT) sh.pos[m] = (unsigned short)((m % R1) * S + m / R1);
  __syncthreads();

  const unsigned ntile = (unsigned)((f.JH + JTh - 1) >> a.lgh);
  const unsigned ntot = (unsigned)f.ncol * ntile;
  const long long IJ = (long long)f.I * f.J;
  const long long mstride = (long long)f.ncolF * f.J;
  const uint64_t keep = l2::keep_policy();
  for (unsigned t0 = blockIdx.x; t0 < ntot; t0 += gridDim.x) {
    // last column first, as in the power-of-two kernels: a synthesis that just
    // wrote the grid left its last columns in L2
    const unsigned t = ntot - 1 - t0, c2 = t / ntile;
    const int h0 = (int)(t - c2 * ntile) << a.lgh;
    const int col = f.mul_pair ? (int)(c2 >> 1) + (int)(c2 & 1) * f.nsplit : (int)c2;
    const double *gb = f.gcol ? f.gcol[col]
                     : (col < f.nsplit) ? f.g0 + (long long)col * IJ : f.g1 + (long long)(col - f.nsplit) * IJ;
    const double *fb = MUL ? f.mul + (long long)(col % f.nmul) * IJ : nullptr;
    const double *zb = (MUL && f.add0) ? (col < f.nsplit ? f.add0 + (long long)col * IJ
                                                         : f.add1 + (long long)(col - f.nsplit) * IJ) : nullptr;
    with_radix<MAXR>(R1, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int idx = tid; idx < 2 * JTh * R2; idx += NT) {
        const int row = idx / R2, u = idx - row * R2;
        const int jh = h0 + (row & (JTh - 1)), j = row < JTh ? f.JH + jh : f.JH - 1 - jh;
        const bool valid = jh < f.JH;
        const long long off = (long long)(valid ? j : 0) * NC + u;
        const double2 *src = reinterpret_cast<const double2 *>(gb) + off;
        double2 v[R];
#pragma unroll
        for (int n = 0; n < R; ++n) v[n] = valid ? __ldcs(src + R2 * n) : make_double2(0.0, 0.0);
        if (MUL) {
          const double2 *fr = reinterpret_cast<const double2 *>(fb) + off;
#pragma unroll
          for (int n = 0; n < R; ++n) {
            const double2 q = valid ? __ldg(fr + R2 * n) : make_double2(0.0, 0.0);
            v[n] = make_double2(v[n].x * q.x, v[n].y * q.y);
          }
          if (zb) {
            const double2 *zr = reinterpret_cast<const double2 *>(zb) + off;
#pragma unroll
            for (int n = 0; n < R; ++n) {
              const double2 z = valid ? __ldg(zr + R2 * n) : make_double2(0.0, 0.0);
              v[n] = make_double2(v[n].x + z.x, v[n].y + z.y);
            }
          }
        }
        dft_nat<R, false>(v);
        double2 *o = buf + row * RS + u;
        o[0] = v[0];
#pragma unroll
        for (int k = 1; k < R; ++k) o[k * S] = cmul(v[k], sh.stw[k * R2 + u]);
      }
    });
    __syncthreads();
    with_radix<MAXR>(R2, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int idx = tid; idx < 2 * JTh * R1; idx += NT) {
        const int row = idx / R1, k1 = idx - row * R1;
        double2 *o = buf + row * RS + k1 * S;
        double2 v[R];
#pragma unroll
        for (int n = 0; n < R; ++n) v[n] = o[n];
        dft_nat<R, false>(v);
#pragma unroll
        for (int n = 0; n < R; ++n) o[n] = v[n];
      }
    });
    __syncthreads();
    // real unpack X_m = E - i W^m D, E/D = (Z_m +- conj Z_{NC-m})/2, of the north
    // row i and the south row JTh + i; their sum and difference go out
    double2 *Fb = f.F + (long long)(f.colF0 + col) * f.J + h0;
    for (int idx = tid; idx < (f.N + 1) << a.lgh; idx += NT) {
      const int m = idx >> a.lgh, i = idx & (JTh - 1);
      if (h0 + i >= f.JH) continue;
      const int pm = sh.pos[m], pc = sh.pos[m == 0 ? 0 : NC - m];
      const double2 w = sh.stwI[m];
      auto row_x = [&](const double2 *z, double sc) {
        const double2 zm = z[pm], zc = z[pc];
        const double er = 0.5 * (zm.x + zc.x), ei = 0.5 * (zm.y - zc.y);
        const double dr = 0.5 * (zm.x - zc.x), di = 0.5 * (zm.y + zc.y);
        const double tr = w.x * dr - w.y * di, ti = w.x * di + w.y * dr;
        return make_double2((er + ti) * sc, (m == 0) ? 0.0 : (ei - tr) * sc);
      };
      const double2 gn = row_x(buf + i * RS, __ldg(f.rowscale + f.JH + h0 + i));
      const double2 gs = row_x(buf + (JTh + i) * RS, __ldg(f.rowscale + f.JH - 1 - h0 - i));
      l2::st_keep(Fb + m * mstride + i, make_double2(gn.x + gs.x, gn.y + gs.y), keep);
      l2::st_keep(Fb + m * mstride + f.JH + i, make_double2(gn.x - gs.x, gn.y - gs.y), keep);
    }
    __syncthreads();  // the next tile reuses the buffer
  }
}

template <int MAXR>
__global__ void __launch_bounds__(256, MAXR <= 16 ? 2 : 1) k_mix_inv(MixArgs a)
{
  const FftArgs &f = a.f;
  const int NC = f.I / 2, R1 = a.R1, R2 = a.R2, S = a.S, RS = a.RS;
  const int JTh = 1 << a.lgh, NT = blockDim.x, tid = threadIdx.x;
  const MixShared sh = mix_shared(a, NC);
  double2 *const buf = sh.buf;
  for (int k = tid; k < NC; k += NT) sh.pos[k] = (unsigned short)((k / R2) * S + k % R2);
  __syncthreads();

  const unsigned ntile = (unsigned)((f.JH + JTh - 1) >> a.lgh);
  const unsigned ntot = (unsigned)f.ncol * ntile;
  const long long IJ = (long long)f.I * f.J;
  const long long mstride = (long long)f.ncolF * f.J;
  const bool drop = JTh * 16 % 128 == 0 && f.JH % JTh == 0;  // the runs are whole 128-byte lines
  for (unsigned t = blockIdx.x; t < ntot; t += gridDim.x) {
    const int col = (int)(t / ntile), h0 = (int)(t - (unsigned)col * ntile) << a.lgh;
    const double2 *Fb = f.Fc + (long long)(f.colF0 + col) * f.J + h0;
    // Z_k = (X_k + conj X_{NC-k}) + i w^k (X_k - conj X_{NC-k}), w = e^{+2 pi i / I},
    // for k and NC - k together (w^{NC-k} = -conj w^k); X north = E + O, south = E - O
#pragma unroll 2
    for (int idx = tid; idx < (NC / 2 + 1) << a.lgh; idx += NT) {
      const int k = idx >> a.lgh, i = idx & (JTh - 1), kk = NC - k;
      const bool in = h0 + i < f.JH;
      double2 e = make_double2(0.0, 0.0), o = e, e2 = e, o2 = e;
      if (in && k <= f.N) {
        e = Fb[k * mstride + i];
        o = Fb[k * mstride + f.JH + i];
        if (k == 0) e.y = o.y = 0.0;
      }
      if (in && k > 0 && kk <= f.N) {
        e2 = Fb[kk * mstride + i];
        o2 = Fb[kk * mstride + f.JH + i];
      }
      const double2 w = make_double2(sh.stwI[k].x, -sh.stwI[k].y);  // w^k
      const int p1 = sh.pos[k], p2 = k > 0 ? sh.pos[kk] : 0;
      auto put = [&](double2 *z, double2 X, double2 Y) {
        // Y = X_{NC-k}
        const double dr = X.x - Y.x, di = X.y + Y.y, sr = X.x + Y.x, si = X.y - Y.y;
        const double tr = w.x * dr - w.y * di, ti = w.x * di + w.y * dr;  // w^k (X - conj Y)
        z[p1] = make_double2(sr - ti, si + tr);
        // Z_{NC-k} = conj(sum) + i conj(w^k) conj(X - conj Y) = conj(sum) + i conj(t)
        if (k > 0 && kk != k) z[p2] = make_double2(sr + ti, tr - si);
      };
      put(buf + i * RS, make_double2(e.x + o.x, e.y + o.y), make_double2(e2.x + o2.x, e2.y + o2.y));
      put(buf + (JTh + i) * RS, make_double2(e.x - o.x, e.y - o.y), make_double2(e2.x - o2.x, e2.y - o2.y));
    }
    __syncthreads();
    if (drop) {
      // no later kernel reads these lines: drop them from L2 without a write-back
      const int lpr = JTh * 16 / 128;
      for (int q = tid; q < (f.N + 1) * 2 * lpr; q += NT) {
        const int m = q / (2 * lpr), rest = q - m * 2 * lpr;
        l2::discard_line(reinterpret_cast<const char *>(Fb + m * mstride + (rest < lpr ? 0 : f.JH)) + 128 * (rest % lpr));
      }
    }
    with_radix<MAXR>(R1, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int idx = tid; idx < 2 * JTh * R2; idx += NT) {
        const int row = idx / R2, u = idx - row * R2;
        double2 *o = buf + row * RS + u;
        double2 v[R];
#pragma unroll
        for (int n = 0; n < R; ++n) v[n] = o[n * S];
        dft_nat<R, true>(v);
        o[0] = v[0];
#pragma unroll
        for (int k = 1; k < R; ++k) o[k * S] = cmulc(v[k], sh.stw[k * R2 + u]);
      }
    });
    __syncthreads();
    double *dst = f.ocol ? f.ocol[col]
                : (col < f.nsplit) ? f.o0 + (long long)col * IJ : f.o1 + (long long)(col - f.nsplit) * IJ;
    with_radix<MAXR>(R2, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int idx = tid; idx < 2 * JTh * R1; idx += NT) {
        const int row = idx / R1, k1 = idx - row * R1;
        const int jh = h0 + (row & (JTh - 1)), j = row < JTh ? f.JH + jh : f.JH - 1 - jh;
        const double2 *o = buf + row * RS + k1 * S;
        double2 v[R];
#pragma unroll
        for (int n = 0; n < R; ++n) v[n] = o[n];
        dft_nat<R, true>(v);
        if (jh < f.JH) {
          const double sc = __ldg(f.rowscale + j);
          double2 *rowp = reinterpret_cast<double2 *>(dst + (long long)j * f.I) + k1;
#pragma unroll
          for (int n = 0; n < R; ++n) rowp[R1 * n] = make_double2(v[n].x * sc, v[n].y * sc);
        }
      }
    });
    __syncthreads();  // the next tile refills the buffer
  }
}

// ------------------------------------------- mirrored pairs as one complex row
// For I = R1 R2 itself (im up to 960 or so) the north and south row of a
// mirrored pair are the real and imaginary part of one complex row of I points,
// as in sht_fft_row.cu: both unpack from Z_m and Z_{I-m} without a twiddle, and
// only the outputs m <= N and m >= I - N pass through shared memory.  The
// inverse's Fourier runs of the next tile stream into their own buffer
// (cp.async) while this one is transformed.
struct PairShared {
  double2 *stw, *buf, *runs;
  unsigned short *pos;
};

// stw[k1 R2 + u] = W_I^{u k1}; pos[m]: the slot of order m (I - m below m = 0)
template <bool INV>
__device__ __forceinline__ PairShared pair_shared(const MixArgs &a)
{
  extern __shared__ __align__(16) double2 smem_mix[];
  const int I = a.f.I, R1 = a.R1, R2 = a.R2;
  PairShared s;
  s.stw = smem_mix;
  s.buf = smem_mix + I;
  s.runs = s.buf + (a.RS << a.lgh);
  s.pos = reinterpret_cast<unsigned short *>(s.runs + (INV ? (a.f.N + 1) * (2 << a.lgh) : 0));
  for (int q = threadIdx.x; q < I; q += blockDim.x) {
    const int t = (q % R2) * (q / R2);
    const double2 w = __ldg(a.f.twI + (t < I / 2 ? t : t - I / 2));
    s.stw[q] = t < I / 2 ? w : make_double2(-w.x, -w.y);
    s.pos[q] = (unsigned short)(INV ? (q / R2) * a.S + q % R2 : (q % R1) * a.S + q / R1);
  }
  return s;
}

template <int MAXR, int MUL>
__global__ void __launch_bounds__(256, MAXR <= 20 ? 2 : 1) k_mixpair_fwd(MixArgs a)
{
  const FftArgs &f = a.f;
  const int I = f.I, R1 = a.R1, R2 = a.R2, S = a.S, RS = a.RS;
  const int JTh = 1 << a.lgh, NT = blockDim.x, tid = threadIdx.x;
  const PairShared sh = pair_shared<false>(a);
  double2 *const buf = sh.buf;
  __syncthreads();
  const unsigned ntile = (unsigned)((f.JH + JTh - 1) >> a.lgh);
  const unsigned ntot = (unsigned)f.ncol * ntile;
  const long long IJ = (long long)I * f.J, mstride = (long long)f.ncolF * f.J;
  const uint64_t keep = l2::keep_policy();
  for (unsigned t0 = blockIdx.x; t0 < ntot; t0 += gridDim.x) {
    // last column first, as in the power-of-two kernels
    const unsigned t = ntot - 1 - t0, c2 = t / ntile;
    const int h0 = (int)(t - c2 * ntile) << a.lgh;
    const int col = f.mul_pair ? (int)(c2 >> 1) + (int)(c2 & 1) * f.nsplit : (int)c2;
    const double *gb = f.gcol ? f.gcol[col]
                     : (col < f.nsplit) ? f.g0 + (long long)col * IJ : f.g1 + (long long)(col - f.nsplit) * IJ;
    const double *fb = MUL ? f.mul + (long long)(col % f.nmul) * IJ : nullptr;
    const double *zb = (MUL && f.add0) ? (col < f.nsplit ? f.add0 + (long long)col * IJ
                                                         : f.add1 + (long long)(col - f.nsplit) * IJ) : nullptr;
    with_radix<MAXR>(R1, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int idx = tid; idx < R2 << a.lgh; idx += NT) {
        const int row = idx / R2, u = idx - row * R2;
        const bool valid = h0 + row < f.JH;
        const int jn = f.JH + (valid ? h0 + row : 0), js = f.J - 1 - jn;
        const int on = jn * I + u, os = js * I + u;
        double2 v[R];
#pragma unroll
        for (int n = 0; n < R; ++n)
          v[n] = valid ? make_double2(__ldcs(gb + on + R2 * n), __ldcs(gb + os + R2 * n)) : make_double2(0.0, 0.0);
        if (MUL && valid) {
#pragma unroll
          for (int n = 0; n < R; ++n) {
            v[n].x *= __ldg(fb + on + R2 * n);
            v[n].y *= __ldg(fb + os + R2 * n);
          }
          if (zb) {
#pragma unroll
            for (int n = 0; n < R; ++n) {
              v[n].x += __ldg(zb + on + R2 * n);
              v[n].y += __ldg(zb + os + R2 * n);
            }
          }
        }
        dft_nat<R, false>(v);
        double2 *o = buf + row * RS + u;
        o[0] = v[0];
#pragma unroll
        for (int k = 1; k < R; ++k) o[k * S] = cmul(v[k], sh.stw[k * R2 + u]);
      }
    });
    __syncthreads();
    with_radix<MAXR>(R2, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int idx = tid; idx < R1 << a.lgh; idx += NT) {
        const int row = idx / R1, k1 = idx - row * R1;
        double2 *o = buf + row * RS + k1 * S;
        double2 v[R];
#pragma unroll
        for (int n = 0; n < R; ++n) v[n] = o[n];
        dft_nat<R, false>(v);
#pragma unroll
        for (int n = 0; n < R; ++n) {
          const int m = k1 + R1 * n;
          if (m <= f.N || m >= I - f.N) o[n] = v[n];
        }
      }
    });
    __syncthreads();
    // Gs = X + Y and Ga = X - Y from U = Z_m + conj Z_{I-m}, V = Z_m - conj Z_{I-m}
    double2 *Fb = f.F + (long long)(f.colF0 + col) * f.J + h0;
    for (int idx = tid; idx < (f.N + 1) << a.lgh; idx += NT) {
      const int m = idx >> a.lgh, i = idx & (JTh - 1);
      if (h0 + i >= f.JH) continue;
      const double sc = 0.5 * __ldg(f.rowscale + f.JH + h0 + i);  // the scales are symmetric in latitude
      const double2 x = buf[i * RS + sh.pos[m]], y = buf[i * RS + sh.pos[m == 0 ? 0 : I - m]];
      const double ux = x.x + y.x, uy = x.y - y.y, vx = x.x - y.x, vy = x.y + y.y;
      l2::st_keep(Fb + m * mstride + i, make_double2((ux + vy) * sc, m == 0 ? 0.0 : (uy - vx) * sc), keep);
      l2::st_keep(Fb + m * mstride + f.JH + i, make_double2((ux - vy) * sc, m == 0 ? 0.0 : (uy + vx) * sc), keep);
    }
    __syncthreads();  // the next tile reuses the buffer
  }
}

template <int MAXR>
__global__ void __launch_bounds__(256, MAXR <= 20 ? 2 : 1) k_mixpair_inv(MixArgs a)
{
  const FftArgs &f = a.f;
  const int I = f.I, R1 = a.R1, R2 = a.R2, S = a.S, RS = a.RS;
  const int JTh = 1 << a.lgh, MS = 2 * JTh, NT = blockDim.x, tid = threadIdx.x;
  const PairShared sh = pair_shared<true>(a);
  double2 *const buf = sh.buf, *const runs = sh.runs;
  const unsigned ntile = (unsigned)((f.JH + JTh - 1) >> a.lgh);
  const unsigned ntot = (unsigned)f.ncol * ntile;
  const long long IJ = (long long)I * f.J, mstride = (long long)f.ncolF * f.J;
  const bool drop = JTh * 16 % 128 == 0 && f.JH % JTh == 0;  // the runs are whole 128-byte lines
  // runs[m MS + i] takes E, runs[m MS + JTh + i] O, of row pair h0 + i
  auto issue = [&](unsigned t) {
    const int col = (int)(t / ntile), h0 = (int)(t - (unsigned)col * ntile) << a.lgh;
    const double2 *Fb = f.Fc + (long long)(f.colF0 + col) * f.J + h0;
    for (int idx = tid; idx < (f.N + 1) << (a.lgh + 1); idx += NT) {
      const int m = idx >> (a.lgh + 1), rr = idx & (MS - 1), i = rr & (JTh - 1);
      const bool in = h0 + i < f.JH;
      cp_async16(runs + idx, in ? Fb + m * mstride + (rr < JTh ? 0 : f.JH) + i : Fb, in);
    }
  };
  unsigned t = blockIdx.x;
  if (t < ntot) issue(t);
  cp_async_commit();
  for (; t < ntot; t += gridDim.x) {
    const int col = (int)(t / ntile), h0 = (int)(t - (unsigned)col * ntile) << a.lgh;
    const double2 *Fb = f.Fc + (long long)(f.colF0 + col) * f.J + h0;
    cp_async_wait<0>();
    __syncthreads();  // the runs (and the tables) are in; the row buffer is free
    // Z_m = X + i Y and Z_{I-m} = conj X + i conj Y, X = E + O (north), Y = E - O
    for (int idx = tid; idx < (f.N + 1) << a.lgh; idx += NT) {
      const int m = idx >> a.lgh, i = idx & (JTh - 1);
      const double2 e = runs[m * MS + i], o = runs[m * MS + JTh + i];
      const double xr = e.x + o.x, yr = e.x - o.x;
      const double xi = m == 0 ? 0.0 : e.y + o.y, yi = m == 0 ? 0.0 : e.y - o.y;
      double2 *const z = buf + i * RS;
      z[sh.pos[m]] = make_double2(xr - yi, xi + yr);
      if (m > 0) z[sh.pos[I - m]] = make_double2(xr + yi, yr - xi);
    }
    __syncthreads();  // the runs are consumed, the rows complete
    if (drop) {
      // no later kernel reads these lines: drop them from L2 without a write-back
      const int lpr = JTh * 16 / 128;
      for (int q = tid; q < (f.N + 1) * 2 * lpr; q += NT) {
        const int m = q / (2 * lpr), rest = q - m * 2 * lpr;
        l2::discard_line(reinterpret_cast<const char *>(Fb + m * mstride + (rest < lpr ? 0 : f.JH)) + 128 * (rest % lpr));
      }
    }
    if (t + gridDim.x < ntot) issue(t + gridDim.x);
    cp_async_commit();
    with_radix<MAXR>(R1, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int idx = tid; idx < R2 << a.lgh; idx += NT) {
        const int row = idx / R2, u = idx - row * R2;
        double2 *o = buf + row * RS + u;
        double2 v[R];
#pragma unroll
        for (int n = 0; n < R; ++n) {
          const int m = R2 * n + u;
          v[n] = make_double2(0.0, 0.0);
          if (m <= f.N || m >= I - f.N) v[n] = o[n * S];
        }
        dft_nat<R, true>(v);
        o[0] = v[0];
#pragma unroll
        for (int k = 1; k < R; ++k) o[k * S] = cmulc(v[k], sh.stw[k * R2 + u]);
      }
    });
    __syncthreads();
    double *dst = f.ocol ? f.ocol[col]
                : (col < f.nsplit) ? f.o0 + (long long)col * IJ : f.o1 + (long long)(col - f.nsplit) * IJ;
    with_radix<MAXR>(R2, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int idx = tid; idx < R1 << a.lgh; idx += NT) {
        const int row = idx / R1, k1 = idx - row * R1;
        const double2 *o = buf + row * RS + k1 * S;
        double2 v[R];
#pragma unroll
        for (int n = 0; n < R; ++n) v[n] = o[n];
        dft_nat<R, true>(v);
        if (h0 + row < f.JH) {
          const int jn = f.JH + h0 + row, js = f.J - 1 - jn;
          const double sc = __ldg(f.rowscale + jn);  // the scales are symmetric in latitude
          double *const rn = dst + jn * I + k1, *const rs = dst + js * I + k1;
#pragma unroll
          for (int n = 0; n < R; ++n) {
            rn[R1 * n] = v[n].x * sc;
            rs[R1 * n] = v[n].y * sc;
          }
        }
      }
    });
  }
  cp_async_wait<0>();
}

constexpr int kRadices[] = {2, 3, 4, 5, 6, 8, 9, 10, 12, 15, 16, 18, 20, 24, 25, 27, 30, 32};

// NC = R1 R2 over the radices above with the smallest larger one, which comes
// first; false where no such product exists (another prime factor, or e.g.
// 972 = 4 3^5)
bool radices(int NC, int *R1, int *R2)
{
  int best = 0;
  for (int r : kRadices)
    for (int q : kRadices)
      if (r >= q && r * q == NC && (best == 0 || r < best)) {
        best = r;
        *R1 = r;
        *R2 = q;
      }
  return best != 0;
}

struct MixShape {
  MixArgs a;
  bool pair;  // mirrored pairs as one complex row of I points; otherwise rows of I/2
  int threads;
  size_t smem;
};

// Pairs in the inverse up to radix 20; otherwise rows of I/2 while their
// radices stay at 16, then pairs.  Stage times (each with a launch gap of a few
// us), rows / pairs, us: inverse im = 96,
// 2000 field-levels 52 / 39, 240, 300 56 / 37, 320, 180 48 / 41, 480, 80 50 /
// 62, 640, 60 125 / 72; forward 96 40 / 39, 192, 500 36 / 39, 320 38 / 42, 480
// 39 / 67, 640 86 / 76.
bool mix_shape(int I, int N, bool inverse, MixShape *s)
{
  const int NC = I / 2;
  MixArgs &a = s->a;
  int p1 = 0, p2 = 0, h1 = 0, h2 = 0;
  const bool pair_ok = radices(I, &p1, &p2), half_ok = radices(NC, &h1, &h2);
  if (!pair_ok && !half_ok) return false;
  s->pair = pair_ok && (!half_ok || h1 > 16 || (inverse && p1 <= 20));
  a.R1 = s->pair ? p1 : h1;
  a.R2 = s->pair ? p2 : h2;
  a.S = a.R2 | 1;
  a.RS = (a.R1 * a.S) | 1;
  auto bytes = [&](int lgh) {
    if (s->pair)
      return sizeof(double2) * (((size_t)a.RS << lgh) + I + (inverse ? (size_t)(N + 1) * (2 << lgh) : 0)) + sizeof(short) * ((size_t)I + 8);
    return sizeof(double2) * ((size_t)(2 << lgh) * a.RS + 2 * (size_t)NC) + sizeof(short) * ((size_t)NC + 8);
  };
  // eight row pairs per tile (128-byte Fourier runs) where at least three such
  // tiles share an SM, else four
  a.lgh = bytes(3) <= 75 * 1024 ? 3 : 2;
  s->smem = bytes(a.lgh);
  // threads: the most resident transforms per unit of pass time (rows R2
  // transforms of R1 points, then rows R1 of R2 points; 128 or 255 registers a
  // thread)
  const int rows = s->pair ? 1 << a.lgh : 2 << a.lgh;
  const int by_smem = (int)(227 * 1024 / (s->smem + 1024));
  double best = 0.0;
  for (int nt = 96; nt <= 256; nt += 32) {
    const int i1 = rows * a.R2, i2 = rows * a.R1;
    const int blocks = std::min(by_smem, (a.R1 <= 20 ? 512 : 256) / nt);
    const double rate = blocks / (double)((i1 + nt - 1) / nt * a.R1 + (i2 + nt - 1) / nt * a.R2);
    if (rate > best) {
      best = rate;
      s->threads = nt;
    }
  }
  return s->smem <= 227 * 1024 && best > 0.0;
}

}  // namespace

bool fft_mixed_supported(int I, int N)
{
  MixShape s{};
  return I % 2 == 0 && mix_shape(I, N, false, &s) && mix_shape(I, N, true, &s);
}

int run_fft_mixed(bool inverse, const sht_plan *p, const FftArgs &args, cudaStream_t s)
{
  MixShape sh{};
  if (!mix_shape(p->I, p->N, inverse, &sh)) { set_error("fft: longitude count without a two-pass factorisation"); return SHT_ERR_UNSUPPORTED_SIZE; }
  sh.a.f = args;
  const int JTh = 1 << sh.a.lgh;
  const long long ntiles = (long long)args.ncol * ((p->JH + JTh - 1) / JTh);
  if (ntiles <= 0) return SHT_OK;
  if (ntiles > 0x7fffffffLL) { set_error("fft: too many field-levels for one call"); return SHT_ERR_TOO_LARGE; }
  void (*kern)(MixArgs) = nullptr;
  const int R = sh.a.R1;
  if (sh.pair) {
    auto pick = [&](auto mr) {
      constexpr int MR = decltype(mr)::value;
      kern = inverse ? k_mixpair_inv<MR> : args.mul ? k_mixpair_fwd<MR, 1> : k_mixpair_fwd<MR, 0>;
    };
    if (R <= 16) pick(std::integral_constant<int, 16>());
    else if (R <= 20) pick(std::integral_constant<int, 20>());
    else pick(std::integral_constant<int, 32>());
  } else {
    const bool wide = R > 16;
    kern = inverse ? (wide ? k_mix_inv<32> : k_mix_inv<16>)
         : args.mul ? (wide ? k_mix_fwd<32, 1> : k_mix_fwd<16, 1>)
                    : (wide ? k_mix_fwd<32, 0> : k_mix_fwd<16, 0>);
  }
  int occ = 0;
  cudaError_t e = kernel_setup((const void *)kern, sh.smem, sh.threads, &occ);
  if (e != cudaSuccess) return cuda_fail(e, "fft smem attribute");
  const long long g = (long long)(occ < 1 ? 1 : occ) * grid_sms(p);
  kern<<<(int)(ntiles < g ? ntiles : g), sh.threads, sh.smem, s>>>(sh.a);
  count_launch();
  e = cudaGetLastError();
  return e == cudaSuccess ? SHT_OK : cuda_fail(e, inverse ? "k_mix_inv" : "k_mix_fwd");
}

}  // namespace sht
