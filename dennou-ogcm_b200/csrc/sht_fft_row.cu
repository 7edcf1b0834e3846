// sht_fft_row.cu -- batched real FFT in longitude for im = 64 to 1024 (powers
// of two), FP64.  Sums, row scales, Gs/Ga and E/O layouts as in sht_fft.cu.
//
// A row of NC = I/2 complex points is NC = R1 R2 with R2 = H R1, H = 1 or 2:
// T = R2 threads per row, R1 points per thread.
//   pass A: thread u takes points R2 n1 + u, an R1-point DFT over n1 and the
//           twiddle W_NC^{u k1}; element (k1, u) goes to k1 S + u.
//   pass B: for every k1 an R2-point DFT over u.  H = 1: one thread.  H = 2:
//           two neighbouring lanes take the even and the odd u, R1 points
//           each, trade half of their results by shuffles and finish with one
//           radix-2 step, so that every thread keeps R1 points and no lane
//           idles.  Output k1 + R1 k2, k2 = q + R1 p (p < H).
// R1 = 8 needs 80 registers and R1 = 16 128 to 168, for 12 to 24 warps per SM;
// the kernels it replaced held up to 32 points per thread (255 registers, 8
// warps at NC = 512).  What bounds it is the shared-memory pipe (62 % of its
// cycles at T85, with the FP64 pipe at 37 % and DRAM at 37 %): the
// exchange, the unpack and their barriers.  Pairs as one complex row (below)
// take a quarter fewer shared-memory wavefronts.
//
// Forward: the second pass leaves Z in its own slots; after a barrier each
// thread unpacks one order of a mirrored row pair from four elements (Z_m and
// Z_{NC-m} of the north and south rows) and writes their sum and difference as
// runs of JTh rows, no staging.  The next tile's rows are loaded into the free
// registers before the unpack.
// Inverse: the Fourier runs of the next tile stream into their own buffer
// (cp.async) while this one is transformed; each thread packs Z_k and
// Z_{NC-k} of a row pair from it.
//
// Shared-memory conflicts: S = 1 (H = 1) or 2 (H = 2) mod 8 makes the lanes
// (k1, u mod H) of pass B fall on distinct 16-byte bank groups; row strides
// are chosen below for the phases whose lanes run over the rows.
#include "sht_fft_row.cuh"

#include <type_traits>

namespace sht {

namespace {

template <int R1, int H, int JTh>
struct RowShape {
  static constexpr int R2 = R1 * H, NC = R1 * R2, T = R2, JT = 2 * JTh, NT = JT * T;
  static constexpr int S = H == 1 ? (R2 | 1) : R2 + 2;
  static_assert(T >= 8 && (H == 1 || S % 8 == 2), "bank layout");
  // forward: lanes over rows read one element each: odd; inverse with JTh = 4:
  // lanes over four rows and two neighbouring elements: 2 (mod 8)
  static constexpr int RSF = (R1 * S) | 1;
  static constexpr int rs_inv()
  {
    int s = R1 * S;
    while (JTh == 4 ? s % 8 != 2 : s % 2 != 1) ++s;
    return s;
  }
  static constexpr int RSI = rs_inv();
  static constexpr int MS = JTh == 4 ? 12 : 2 * JTh;  // staged Fourier runs: stride per order
  static size_t smem(bool inverse, int N)
  {
    return sizeof(double2) * (inverse ? JT * RSI + 2 * NC + (size_t)(N + 1) * MS : (size_t)JT * RSF + 2 * NC);
  }
};

// Slot of output Z_m in its row after pass B: thread (k1, h) keeps its R1
// results at its own pass-B addresses k1 S + h + H slot.
template <int R1, int H>
__device__ __forceinline__ int row_pos(int m, int S)
{
  const int k1 = m % R1, k2 = m / R1;  // powers of two: shifts
  if constexpr (H == 1) return k1 * S + k2;
  const int q = k2 % R1, p = k2 / R1;
  return k1 * S + q / (R1 / 2) + 2 * (q % (R1 / 2) + (R1 / 2) * p);
}

__device__ __forceinline__ double2 shfl_xor1(double2 v)
{
  return make_double2(__shfl_xor_sync(0xffffffffu, v.x, 1), __shfl_xor_sync(0xffffffffu, v.y, 1));
}

constexpr int ilog2(int x) { return x <= 1 ? 0 : 1 + ilog2(x / 2); }

// Pass B of one thread: reads its R1 elements (u = H j + h), returns
// z[slot] with slot = qq + (R1/H) p for q = h (R1/H) + qq.
template <int R1, int H, bool INV>
__device__ __forceinline__ void pass_b(const double2 *base, int h, double2 (&z)[R1])
{
  constexpr int LOG = ilog2(R1);
  double2 v[R1];
#pragma unroll
  for (int j = 0; j < R1; ++j) v[j] = base[H * j];
  dft_reg<LOG, INV>(v);
  if constexpr (H == 1) {
#pragma unroll
    for (int k = 0; k < R1; ++k) z[k] = v[brev<LOG>(k)];
  } else {
    // lane h keeps q in [h R1/2, (h+1) R1/2) and gets the partner's values there
    constexpr int HQ = R1 / 2;
#pragma unroll
    for (int qq = 0; qq < HQ; ++qq) {
      const double2 lo = v[brev<LOG>(qq)], hi = v[brev<LOG>(HQ + qq)];
      const double2 mine = h ? hi : lo, other = shfl_xor1(h ? lo : hi);
      const double2 a = h ? other : mine;  // even u
      double2 b = h ? mine : other;        // odd u, times W_{R2}^q = W_{2 R1}^{qq} (-+i)^h
      const int t = qq * (16 / R1);        // W_{2 R1}^{qq} = e^{-2 pi i t / 32}
      if constexpr (INV) {
        const double2 c = rot32(make_double2(b.x, -b.y), t);  // conj(b w) = conj(b) conj(w)
        b = h ? make_double2(c.y, c.x) : make_double2(c.x, -c.y);
      } else {
        const double2 c = rot32(b, t);
        b = h ? make_double2(c.y, -c.x) : c;
      }
      z[qq] = make_double2(a.x + b.x, a.y + b.y);
      z[qq + HQ] = make_double2(a.x - b.x, a.y - b.y);
    }
  }
}

template <int R1, int T, bool INV>
__device__ __forceinline__ void pass_a_store(double2 (&v)[R1], double2 *o, int S, const double2 *stw, int u)
{
  constexpr int LOG = ilog2(R1);
  dft_reg<LOG, INV>(v);
  PassTwiddles<R1, T> tw;
  tw.load(stw, u);
#pragma unroll
  for (int k = 0; k < R1; ++k) {
    double2 y = v[brev<LOG>(k)];
    if (k != 0) y = INV ? cmulc(y, tw(k)) : cmul(y, tw(k));
    o[k * S] = y;
  }
}

template <int R1, int H, int JTh, int MUL, int MINB, int PF>
__global__ void __launch_bounds__(RowShape<R1, H, JTh>::NT, MINB) k_row_fwd(FftArgs a)
{
  using P = RowShape<R1, H, JTh>;
  constexpr int R2 = P::R2, NC = P::NC, T = P::T, NT = P::NT, S = P::S, RS = P::RSF;
  extern __shared__ __align__(16) double2 smem_row[];
  double2 *const stw = smem_row, *const stwI = smem_row + NC, *const buf = smem_row + 2 * NC;
  load_twiddles<T, NC, NT>(a, stw, stwI);
  const int tid = threadIdx.x, r = tid / T, u = tid % T;
  const unsigned ntile = (unsigned)((a.JH + JTh - 1) / JTh);
  const unsigned ntot = (unsigned)a.ncol * ntile;  // the launcher checks that it fits
  const long long IJ = (long long)a.I * a.J, mstride = (long long)a.ncolF * a.J;
  auto where = [&](unsigned t, int &col, int &h0) {
    // last column first: a synthesis that has just written the grid left its
    // last columns in L2
    t = ntot - 1 - t;
    const unsigned c2 = t / ntile;
    h0 = (int)(t - c2 * ntile) * JTh;
    col = a.mul_pair ? (int)(c2 >> 1) + (int)(c2 & 1) * a.nsplit : (int)c2;
  };
  double2 v[R1];
  auto load = [&](unsigned t, auto lo, auto hi) {
    constexpr int LO = decltype(lo)::value, HI = decltype(hi)::value;
    int col, h0;
    where(t, col, h0);
    const int jh = h0 + r % JTh, j = r < JTh ? a.JH + jh : a.JH - 1 - jh;
    const bool valid = jh < a.JH;
    const double *gb = a.gcol ? a.gcol[col]
                     : (col < a.nsplit) ? a.g0 + (long long)col * IJ : a.g1 + (long long)(col - a.nsplit) * IJ;
    const long long off = (long long)(valid ? j : 0) * NC + u;
    const double2 *src = reinterpret_cast<const double2 *>(gb) + off;
#pragma unroll
    for (int n = LO; n < HI; ++n) v[n] = valid ? __ldcs(src + R2 * n) : make_double2(0.0, 0.0);
  };
  // the factors when the tile's turn comes, so that its prefetched rows are not
  // waited for before the unpack (products of two fields, T85 pairs, 480:
  // 103 -> 99 us; T341 rows, 48: 214 -> 191; no size slower)
  auto multiply = [&](unsigned t) {
    int col, h0;
    where(t, col, h0);
    const int jh = h0 + r % JTh, j = r < JTh ? a.JH + jh : a.JH - 1 - jh;
    const bool valid = jh < a.JH;
    const long long off = (long long)(valid ? j : 0) * NC + u;
    const double2 *fr = reinterpret_cast<const double2 *>(a.mul + (long long)(col % a.nmul) * IJ) + off;
#pragma unroll
    for (int n = 0; n < R1; ++n) {
      const double2 q = valid ? __ldg(fr + R2 * n) : make_double2(0.0, 0.0);
      v[n] = make_double2(v[n].x * q.x, v[n].y * q.y);
    }
    if (a.add0) {
      const double *zb = col < a.nsplit ? a.add0 + (long long)col * IJ : a.add1 + (long long)(col - a.nsplit) * IJ;
      const double2 *zr = reinterpret_cast<const double2 *>(zb) + off;
#pragma unroll
      for (int n = 0; n < R1; ++n) {
        const double2 z = valid ? __ldg(zr + R2 * n) : make_double2(0.0, 0.0);
        v[n] = make_double2(v[n].x + z.x, v[n].y + z.y);
      }
    }
  };
  const uint64_t keep = l2::keep_policy();
  unsigned t = blockIdx.x;
  constexpr std::integral_constant<int, 0> zero{};
  constexpr std::integral_constant<int, PF> pf{};
  constexpr std::integral_constant<int, R1> all{};
  if (t < ntot) load(t, zero, pf);
  __syncthreads();  // the twiddle tables are in
  for (; t < ntot; t += gridDim.x) {
    int col, h0;
    where(t, col, h0);
    if constexpr (PF < R1) load(t, pf, all);
    if (MUL) multiply(t);
    pass_a_store<R1, T, false>(v, buf + r * RS + u, S, stw, u);
    __syncthreads();
    {
      double2 *const own = buf + r * RS + (u / H) * S + u % H;
      double2 z[R1];
      pass_b<R1, H, false>(own, u % H, z);
#pragma unroll
      for (int k = 0; k < R1; ++k) own[H * k] = z[k];
    }
    if (t + gridDim.x < ntot) load(t + gridDim.x, zero, pf);
    __syncthreads();
    // X_m = E - i W^m D, E/D = (Z_m +- conj Z_{NC-m})/2, of the pair's two rows
    const int i = tid % JTh;
    if (h0 + i < a.JH) {
      double2 *const Fb = a.F + (long long)(a.colF0 + col) * a.J + h0 + i;
      const double scn = 0.5 * __ldg(a.rowscale + a.JH + h0 + i), scs = 0.5 * __ldg(a.rowscale + a.JH - 1 - h0 - i);
      const double2 *const zn = buf + i * RS, *const zs = zn + JTh * RS;
      for (int mm = tid / JTh; mm <= (JTh == 4 ? a.N | 7 : a.N); mm += NT / JTh) {
        // JTh = 4: a phase's two orders are 4 / H apart, 4 (mod 8) elements
        constexpr int B = H == 2 ? 1 : 2;
        const int m = JTh == 4 ? (mm & ~(1 | 1 << B)) | ((mm & 1) << B) | ((mm >> B) & 1) : mm;
        if (m > a.N) continue;
        const int pm = row_pos<R1, H>(m, S), pc = row_pos<R1, H>((NC - m) & (NC - 1), S);
        const double2 w = stwI[m];
        auto order = [&](const double2 *z, double sc) {
          const double2 x = z[pm], y = z[pc];
          const double er = x.x + y.x, ei = x.y - y.y, dr = x.x - y.x, di = x.y + y.y;
          return make_double2((er + (w.x * di + w.y * dr)) * sc, (ei - (w.x * dr - w.y * di)) * sc);
        };
        double2 gn = order(zn, scn), gs = order(zs, scs);
        if (m == 0) gn.y = gs.y = 0.0;
        l2::st_keep(Fb + m * mstride, make_double2(gn.x + gs.x, gn.y + gs.y), keep);
        l2::st_keep(Fb + m * mstride + a.JH, make_double2(gn.x - gs.x, gn.y - gs.y), keep);
      }
    }
    __syncthreads();  // the next tile reuses the buffer
  }
}

template <int R1, int H, int JTh, int MINB>
__global__ void __launch_bounds__(RowShape<R1, H, JTh>::NT, MINB) k_row_inv(FftArgs a)
{
  using P = RowShape<R1, H, JTh>;
  constexpr int R2 = P::R2, NC = P::NC, T = P::T, JT = P::JT, NT = P::NT, S = P::S, RS = P::RSI, MS = P::MS;
  extern __shared__ __align__(16) double2 smem_row[];
  double2 *const stw = smem_row, *const stwI = smem_row + NC, *const buf = smem_row + 2 * NC, *const runs = buf + JT * RS;
  load_twiddles<T, NC, NT>(a, stw, stwI);
  const int tid = threadIdx.x, r = tid / T, u = tid % T;
  const unsigned ntile = (unsigned)((a.JH + JTh - 1) / JTh);
  const unsigned ntot = (unsigned)a.ncol * ntile;
  const long long IJ = (long long)a.I * a.J, mstride = (long long)a.ncolF * a.J;
  // runs[m MS + i] takes E, runs[m MS + JTh + i] O, of row pair h0 + i
  auto issue = [&](unsigned t) {
    const int col = (int)(t / ntile), h0 = (int)(t - (unsigned)col * ntile) * JTh;
    const double2 *Fb = a.Fc + (long long)(a.colF0 + col) * a.J + h0;
    constexpr int STEP = NT / JT;
    const int rr = tid % JT, i = rr % JTh;
    const bool in = h0 + i < a.JH;
    const double2 *src = Fb + (rr < JTh ? 0 : a.JH) + i + (long long)(tid / JT) * mstride;
    for (int m = tid / JT; m <= a.N; m += STEP, src += STEP * mstride) cp_async16(runs + m * MS + rr, in ? src : Fb, in);
  };
  unsigned t = blockIdx.x;
  if (t < ntot) issue(t);
  cp_async_commit();
  for (; t < ntot; t += gridDim.x) {
    const int col = (int)(t / ntile), h0 = (int)(t - (unsigned)col * ntile) * JTh;
    cp_async_wait<0>();
    __syncthreads();  // the runs (and the twiddle tables) are in; the row buffer is free
    // Z_k = (X_k + conj X_{NC-k}) + i w^k (X_k - conj X_{NC-k}), w = e^{+2 pi i/I},
    // for k and NC - k together; X north = E + O, south = E - O
    {
      const int i = tid % JTh;
      for (int k = tid / JTh; k <= NC / 2; k += NT / JTh) {
        const int kk = NC - k;
        double2 e = make_double2(0.0, 0.0), o = e, e2 = e, o2 = e;
        if (k <= a.N) {
          e = runs[k * MS + i];
          o = runs[k * MS + JTh + i];
          if (k == 0) e.y = o.y = 0.0;
        }
        if (k > 0 && kk <= a.N) {
          e2 = runs[kk * MS + i];
          o2 = runs[kk * MS + JTh + i];
        }
        const double2 w = make_double2(stwI[k].x, -stwI[k].y);
        const int p1 = (k / R2) * S + k % R2, p2 = (kk / R2) * S + kk % R2;
        auto put = [&](double2 *z, double2 X, double2 Y) {
          const double dr = X.x - Y.x, di = X.y + Y.y, sr = X.x + Y.x, si = X.y - Y.y;
          const double tr = w.x * dr - w.y * di, ti = w.x * di + w.y * dr;
          z[p1] = make_double2(sr - ti, si + tr);
          if (k > 0 && kk != k) z[p2] = make_double2(sr + ti, tr - si);
        };
        put(buf + i * RS, make_double2(e.x + o.x, e.y + o.y), make_double2(e2.x + o2.x, e2.y + o2.y));
        put(buf + (JTh + i) * RS, make_double2(e.x - o.x, e.y - o.y), make_double2(e2.x - o2.x, e2.y - o2.y));
      }
    }
    __syncthreads();  // the runs are consumed, the rows complete
    if constexpr (JTh * 16 % 128 == 0) {
      // whole 128-byte lines that no later kernel reads: drop them from L2
      // without a write-back
      if (a.JH % JTh == 0) {
        constexpr int LPR = JTh * 16 / 128;
        const double2 *Fb = a.Fc + (long long)(a.colF0 + col) * a.J + h0;
        for (int q = tid; q < (a.N + 1) * 2 * LPR; q += NT) {
          const int m = q / (2 * LPR), rest = q - m * 2 * LPR;
          l2::discard_line(reinterpret_cast<const char *>(Fb + m * mstride + (rest < LPR ? 0 : a.JH)) + 128 * (rest % LPR));
        }
      }
    }
    if (t + gridDim.x < ntot) issue(t + gridDim.x);
    cp_async_commit();
    {
      double2 *const own = buf + r * RS + u;
      double2 v[R1];
#pragma unroll
      for (int n = 0; n < R1; ++n) v[n] = own[n * S];
      pass_a_store<R1, T, true>(v, own, S, stw, u);
    }
    __syncthreads();
    double2 z[R1];
    const int k1 = u / H, h = u % H;
    pass_b<R1, H, true>(buf + r * RS + k1 * S + h, h, z);
    const int jh = h0 + r % JTh, j = r < JTh ? a.JH + jh : a.JH - 1 - jh;
    if (jh < a.JH) {
      double *dst = a.ocol ? a.ocol[col]
                  : (col < a.nsplit) ? a.o0 + (long long)col * IJ : a.o1 + (long long)(col - a.nsplit) * IJ;
      double2 *rowp = reinterpret_cast<double2 *>(dst + (long long)j * a.I) + k1 + R1 * h * (R1 / H);
      const double sc = __ldg(a.rowscale + j);
#pragma unroll
      for (int k = 0; k < R1; ++k) {
        // slot k = qq + (R1/H) p holds point k1 + R1 (h (R1/H) + qq + R1 p)
        const int qq = k % (R1 / H), p = k / (R1 / H);
        rowp[R1 * (qq + R1 * p)] = make_double2(z[k].x * sc, z[k].y * sc);  // default policy: may stay in L2 for an analysis
      }
    }
  }
  cp_async_wait<0>();
}

// ------------------------------------------------- mirrored pairs as one row
// The north row x and the south row y of a mirrored pair are the real and
// imaginary part of one complex row z = x + i y of I = R1 R2 points.  With
// Z its transform, X_m = (Z_m + conj Z_{I-m})/2 and Y_m = -i (Z_m - conj Z_{I-m})/2,
// so both rows unpack from two elements without a twiddle, and only the
// outputs m <= N and m >= I - N are kept.
template <int R1, int H, int JTh>
struct PairShape {
  static constexpr int R2 = R1 * H, I = R1 * R2, T = R2, NT = JTh * T;
  static constexpr int S = H == 1 ? (R2 | 1) : R2 + 2;
  static constexpr int RS = (R1 * S) | 1;
  static constexpr int MS = 2 * JTh;
  static size_t smem(bool inverse, int N)
  {
    return sizeof(double2) * ((size_t)JTh * RS + I + (inverse ? (size_t)(N + 1) * MS : 0));
  }
};

// stw[k1 T + u] = W_I^{u k1} from the half table e^{-2 pi i t / I}, t < I/2
template <int T, int I, int NT>
__device__ __forceinline__ void load_pair_twiddles(const FftArgs &a, double2 *stw)
{
  for (int q = threadIdx.x; q < I; q += NT) {
    const int t = (q % T) * (q / T);
    const double2 w = __ldg(a.twI + (t < I / 2 ? t : t - I / 2));
    stw[q] = t < I / 2 ? w : make_double2(-w.x, -w.y);
  }
}

template <int R1, int H, int JTh, int MUL, int MINB>
__global__ void __launch_bounds__(PairShape<R1, H, JTh>::NT, MINB) k_pair_fwd(FftArgs a)
{
  using P = PairShape<R1, H, JTh>;
  constexpr int R2 = P::R2, I = P::I, T = P::T, NT = P::NT, S = P::S, RS = P::RS;
  extern __shared__ __align__(16) double2 smem_row[];
  double2 *const stw = smem_row, *const buf = smem_row + I;
  load_pair_twiddles<T, I, NT>(a, stw);
  const int tid = threadIdx.x, r = tid / T, u = tid % T;
  const unsigned ntile = (unsigned)((a.JH + JTh - 1) / JTh);
  const unsigned ntot = (unsigned)a.ncol * ntile;  // the launcher checks that it fits
  const long long IJ = (long long)I * a.J, mstride = (long long)a.ncolF * a.J;
  auto where = [&](unsigned t, int &col, int &h0) {
    // last column first: a synthesis that has just written the grid left its
    // last columns in L2
    t = ntot - 1 - t;
    const unsigned c2 = t / ntile;
    h0 = (int)(t - c2 * ntile) * JTh;
    col = a.mul_pair ? (int)(c2 >> 1) + (int)(c2 & 1) * a.nsplit : (int)c2;
  };
  double2 v[R1];
  auto load = [&](unsigned t) {
    int col, h0;
    where(t, col, h0);
    const bool valid = h0 + r < a.JH;
    const int jn = a.JH + (valid ? h0 + r : 0), js = 2 * a.JH - 1 - jn;
    const double *gb = a.gcol ? a.gcol[col]
                     : (col < a.nsplit) ? a.g0 + (long long)col * IJ : a.g1 + (long long)(col - a.nsplit) * IJ;
    const int on = jn * I + u, os = js * I + u;
#pragma unroll
    for (int n = 0; n < R1; ++n)
      v[n] = valid ? make_double2(__ldcs(gb + on + R2 * n), __ldcs(gb + os + R2 * n)) : make_double2(0.0, 0.0);
  };
  // the factors when the tile's turn comes (see k_row_fwd)
  auto multiply = [&](unsigned t) {
    int col, h0;
    where(t, col, h0);
    const bool valid = h0 + r < a.JH;
    const int jn = a.JH + (valid ? h0 + r : 0), js = 2 * a.JH - 1 - jn;
    const int on = jn * I + u, os = js * I + u;
    const double *f = a.mul + (long long)(col % a.nmul) * IJ;
#pragma unroll
    for (int n = 0; n < R1; ++n) {
      v[n].x *= __ldg(f + on + R2 * n);
      v[n].y *= __ldg(f + os + R2 * n);
    }
    if (a.add0) {
      const double *z = col < a.nsplit ? a.add0 + (long long)col * IJ : a.add1 + (long long)(col - a.nsplit) * IJ;
#pragma unroll
      for (int n = 0; n < R1; ++n) {
        v[n].x += __ldg(z + on + R2 * n);
        v[n].y += __ldg(z + os + R2 * n);
      }
    }
    if (!valid)
#pragma unroll
      for (int n = 0; n < R1; ++n) v[n] = make_double2(0.0, 0.0);
  };
  const uint64_t keep = l2::keep_policy();
  unsigned t = blockIdx.x;
  if (t < ntot) load(t);
  __syncthreads();  // the twiddle table is in
  for (; t < ntot; t += gridDim.x) {
    int col, h0;
    where(t, col, h0);
    if (MUL) multiply(t);
    pass_a_store<R1, T, false>(v, buf + r * RS + u, S, stw, u);
    __syncthreads();
    {
      const int k1 = u / H, h = u % H;
      double2 *const own = buf + r * RS + k1 * S + h;
      double2 z[R1];
      pass_b<R1, H, false>(own, h, z);
#pragma unroll
      for (int k = 0; k < R1; ++k) {
        const int m = k1 + R1 * (h * (R1 / H) + k % (R1 / H) + R1 * (k / (R1 / H)));
        if (m <= a.N || m >= I - a.N) own[H * k] = z[k];
      }
    }
    if (t + gridDim.x < ntot) load(t + gridDim.x);
    __syncthreads();
    // Gs = X + Y and Ga = X - Y from U = Z_m + conj Z_{I-m}, V = Z_m - conj Z_{I-m}
    const int i = tid % JTh;
    if (h0 + i < a.JH) {
      double2 *const Fb = a.F + (long long)(a.colF0 + col) * a.J + h0 + i;
      const double sc = 0.5 * __ldg(a.rowscale + a.JH + h0 + i);  // the scales are symmetric in latitude
      const double2 *const z = buf + i * RS;
      for (int m = tid / JTh; m <= a.N; m += NT / JTh) {
        const double2 x = z[row_pos<R1, H>(m, S)], y = z[row_pos<R1, H>((I - m) & (I - 1), S)];
        const double ux = x.x + y.x, uy = x.y - y.y, vx = x.x - y.x, vy = x.y + y.y;
        l2::st_keep(Fb + m * mstride, make_double2((ux + vy) * sc, m == 0 ? 0.0 : (uy - vx) * sc), keep);
        l2::st_keep(Fb + m * mstride + a.JH, make_double2((ux - vy) * sc, m == 0 ? 0.0 : (uy + vx) * sc), keep);
      }
    }
    __syncthreads();  // the next tile reuses the buffer
  }
}

template <int R1, int H, int JTh, int MINB>
__global__ void __launch_bounds__(PairShape<R1, H, JTh>::NT, MINB) k_pair_inv(FftArgs a)
{
  using P = PairShape<R1, H, JTh>;
  constexpr int R2 = P::R2, I = P::I, T = P::T, NT = P::NT, S = P::S, RS = P::RS, MS = P::MS;
  extern __shared__ __align__(16) double2 smem_row[];
  double2 *const stw = smem_row, *const buf = smem_row + I, *const runs = buf + JTh * RS;
  load_pair_twiddles<T, I, NT>(a, stw);
  const int tid = threadIdx.x, r = tid / T, u = tid % T;
  const unsigned ntile = (unsigned)((a.JH + JTh - 1) / JTh);
  const unsigned ntot = (unsigned)a.ncol * ntile;
  const long long IJ = (long long)I * a.J, mstride = (long long)a.ncolF * a.J;
  // runs[m MS + i] takes E, runs[m MS + JTh + i] O, of row pair h0 + i
  auto issue = [&](unsigned t) {
    const int col = (int)(t / ntile), h0 = (int)(t - (unsigned)col * ntile) * JTh;
    const double2 *Fb = a.Fc + (long long)(a.colF0 + col) * a.J + h0;
    constexpr int STEP = NT / MS;
    const int rr = tid % MS, i = rr % JTh;
    const bool in = h0 + i < a.JH;
    const double2 *src = Fb + (rr < JTh ? 0 : a.JH) + i + (long long)(tid / MS) * mstride;
    for (int m = tid / MS; m <= a.N; m += STEP, src += STEP * mstride) cp_async16(runs + m * MS + rr, in ? src : Fb, in);
  };
  unsigned t = blockIdx.x;
  if (t < ntot) issue(t);
  cp_async_commit();
  for (; t < ntot; t += gridDim.x) {
    const int col = (int)(t / ntile), h0 = (int)(t - (unsigned)col * ntile) * JTh;
    cp_async_wait<0>();
    __syncthreads();  // the runs (and the twiddle table) are in; the row buffer is free
    // Z_m = X + i Y and Z_{I-m} = conj X + i conj Y, X = E + O (north), Y = E - O
    {
      const int i = tid % JTh;
      double2 *const z = buf + i * RS;
      for (int m = tid / JTh; m <= a.N; m += NT / JTh) {
        const double2 e = runs[m * MS + i], o = runs[m * MS + JTh + i];
        const double xr = e.x + o.x, yr = e.x - o.x;
        const double xi = m == 0 ? 0.0 : e.y + o.y, yi = m == 0 ? 0.0 : e.y - o.y;
        z[(m / R2) * S + m % R2] = make_double2(xr - yi, xi + yr);
        if (m > 0) z[((I - m) / R2) * S + (I - m) % R2] = make_double2(xr + yi, yr - xi);
      }
    }
    __syncthreads();  // the runs are consumed, the rows complete
    if constexpr (JTh * 16 % 128 == 0) {
      // whole 128-byte lines that no later kernel reads: drop them from L2
      // without a write-back
      if (a.JH % JTh == 0) {
        constexpr int LPR = JTh * 16 / 128;
        const double2 *Fb = a.Fc + (long long)(a.colF0 + col) * a.J + h0;
        for (int q = tid; q < (a.N + 1) * 2 * LPR; q += NT) {
          const int m = q / (2 * LPR), rest = q - m * 2 * LPR;
          l2::discard_line(reinterpret_cast<const char *>(Fb + m * mstride + (rest < LPR ? 0 : a.JH)) + 128 * (rest % LPR));
        }
      }
    }
    if (t + gridDim.x < ntot) issue(t + gridDim.x);
    cp_async_commit();
    {
      double2 *const own = buf + r * RS + u;
      double2 v[R1];
#pragma unroll
      for (int n = 0; n < R1; ++n) {
        const int m = R2 * n + u;
        v[n] = make_double2(0.0, 0.0);
        if (m <= a.N || m >= I - a.N) v[n] = own[n * S];
      }
      pass_a_store<R1, T, true>(v, own, S, stw, u);
    }
    __syncthreads();
    double2 z[R1];
    const int k1 = u / H, h = u % H;
    pass_b<R1, H, true>(buf + r * RS + k1 * S + h, h, z);
    if (h0 + r < a.JH) {
      double *dst = a.ocol ? a.ocol[col]
                  : (col < a.nsplit) ? a.o0 + (long long)col * IJ : a.o1 + (long long)(col - a.nsplit) * IJ;
      const int jn = a.JH + h0 + r, js = 2 * a.JH - 1 - jn, at = k1 + R1 * h * (R1 / H);
      double *const rn = dst + jn * I + at, *const rs = dst + js * I + at;
      const double sc = __ldg(a.rowscale + jn);  // the scales are symmetric in latitude
#pragma unroll
      for (int k = 0; k < R1; ++k) {
        // slot k = qq + (R1/H) p holds point k1 + R1 (h (R1/H) + qq + R1 p)
        const int o = R1 * (k % (R1 / H) + R1 * (k / (R1 / H)));
        rn[o] = z[k].x * sc;  // default policy: may stay in L2 for an analysis
        rs[o] = z[k].y * sc;
      }
    }
  }
  cp_async_wait<0>();
}

// Persistent grid: the resident blocks, never more than there are tiles.
int launch_rows(void (*kern)(FftArgs), int threads, size_t smem, int pairs, const sht_plan *p, const FftArgs &a,
                cudaStream_t s, const char *name)
{
  const long long ntiles = (long long)a.ncol * ((p->JH + pairs - 1) / pairs);
  if (ntiles <= 0) return SHT_OK;
  if (ntiles > 0x7fffffffLL) { set_error("fft: too many field-levels for one call"); return SHT_ERR_TOO_LARGE; }
  if (smem > 227 * 1024) { set_error("fft: shared-memory tile too large for this truncation"); return SHT_ERR_UNSUPPORTED_SIZE; }
  int occ = 0;
  cudaError_t e = kernel_setup((const void *)kern, smem, threads, &occ);
  if (e != cudaSuccess) return cuda_fail(e, "fft smem attribute");
  const long long g = (long long)(occ < 1 ? 1 : occ) * grid_sms(p);
  kern<<<(int)(ntiles < g ? ntiles : g), threads, smem, s>>>(a);
  count_launch();
  e = cudaGetLastError();
  return e == cudaSuccess ? SHT_OK : cuda_fail(e, name);
}

template <int R1, int H, int JTh, int MINB, int PF>
int row_fwd(const sht_plan *p, const FftArgs &a, cudaStream_t s)
{
  using P = RowShape<R1, H, JTh>;
  return launch_rows(a.mul ? k_row_fwd<R1, H, JTh, 1, MINB, PF> : k_row_fwd<R1, H, JTh, 0, MINB, PF>, P::NT,
                     P::smem(false, p->N), JTh, p, a, s, "k_row_fwd");
}
template <int R1, int H, int JTh, int MINB>
int row_inv(const sht_plan *p, const FftArgs &a, cudaStream_t s)
{
  using P = RowShape<R1, H, JTh>;
  return launch_rows(k_row_inv<R1, H, JTh, MINB>, P::NT, P::smem(true, p->N), JTh, p, a, s, "k_row_inv");
}
template <int R1, int H, int JTh, int MBF, int MBI>
int pairs(bool inverse, const sht_plan *p, const FftArgs &a, cudaStream_t s)
{
  using P = PairShape<R1, H, JTh>;
  return launch_rows(inverse ? k_pair_inv<R1, H, JTh, MBI>
                     : a.mul ? k_pair_fwd<R1, H, JTh, 1, MBF> : k_pair_fwd<R1, H, JTh, 0, MBF>,
                     P::NT, P::smem(inverse, p->N), JTh, p, a, s, inverse ? "k_pair_inv" : "k_pair_fwd");
}

}  // namespace

// Which counts and directions these kernels take.  im = 1024's inverse stays
// with k_fft_inv, whose one staging buffer leaves room for two blocks per SM
// (240 field-levels: 397 us against 431).
bool fft_row_supported(int NC, bool inverse) { return (NC >= 32 && NC <= 256) || (NC == 512 && !inverse); }

// The form per count, measured (forward / inverse, us, against the kernels
// they replaced): pairs where a pair's I points split as R1 x R1, single rows
// where the pair form would need the shuffles of H = 2 (T42 pairs: 63 / 68,
// T170 pairs: 291 / 302).
//   im = 64   pairs, 7110 field-levels   44 / 45 -> 37 / 39
//   im = 128  rows, 3095                 70 / 73 -> 62 / 64
//   im = 256  pairs, 480                 47 / 52 -> 43 / 45
//   im = 512  rows, 720                  258 / 275 -> 258 / 237
//   im = 1024 rows, 240                  510 -> 397 (half of the next tile's
//             rows prefetched; all of them spill: 432.  Two row pairs per block,
//             three blocks: 384, but its 32-byte pieces per order lose where
//             orders lie megabytes apart, 960: 1566 -> 1989)
int run_fft_row(bool inverse, const sht_plan *p, const FftArgs &a, cudaStream_t s)
{
  switch (p->NC) {
  case 32: return pairs<8, 1, 16, 5, 6>(inverse, p, a, s);
  case 64: return inverse ? row_inv<8, 1, 8, 6>(p, a, s) : row_fwd<8, 1, 8, 6, 8>(p, a, s);
  case 128: return pairs<16, 1, 8, 3, 3>(inverse, p, a, s);
  case 256: return inverse ? row_inv<16, 1, 4, 3>(p, a, s) : row_fwd<16, 1, 4, 3, 16>(p, a, s);
  case 512: if (!inverse) return row_fwd<16, 2, 4, 2, 8>(p, a, s);  // fall through
  default: set_error("fft: unsupported longitude count"); return SHT_ERR_UNSUPPORTED_SIZE;
  }
}

}  // namespace sht
