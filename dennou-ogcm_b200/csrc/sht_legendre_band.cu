// sht_legendre_band.cu -- FP64 Legendre contraction, one band and parity per
// thread block, any grid.
//
//   analysis  (space_discretization.tex:197-200):
//     S[row(m, r)][col] = sum_jh Pbar_{m+r}^m(mu_jh) F[m][col][par JH + jh],
//     par = r mod 2; the longitude transform delivers Gs (par 0) and Ga (par 1).
//   synthesis (:212-216):
//     F[m][col][par JH + jh] = sum over the r of parity par of Pbar S[row][col].
//
// Each is a dense product per (m, par) on the FP64 tensor path (mma.sync f64:
// m16n8k8 for pairs of 8-row tiles, m8n8k4 for an odd tile and for tails of up to
// four terms; 37 TF/s is also the FMA pipe's rate, the two share it).  A block takes one work item -- up to TM 8-row tiles of the output
// (degrees of one parity in the analysis, latitudes in the synthesis) -- and
// 8 CW field-level columns.  Warp w owns 8 columns (real and imaginary parts
// are two 8-wide tiles) and every RW-th row tile, CW RW = W, so a warp's
// fragment of the data serves all its row tiles and no product is repeated.
// With enough columns RW = 1 and all warps of a block carry equal work; batches
// of fewer than 8 W columns split the rows instead.
//
// Operands stream through NS shared-memory stages of 16 contraction terms.  One
// producer warp fills them with TMA: tensor copies of the data (out-of-range
// latitudes and columns read as zero, so ragged counts need no care) and bulk
// copies of the table; full/empty mbarriers connect it to the W consumer warps,
// which do nothing per stage but wait, load fragments and multiply.  The
// sequence of stages runs on across work units, so the next unit's first
// stages are in flight while a unit finishes.
//   * The Legendre table is stored in 8 x 8 blocks (degree x latitude, 512
//     bytes) in the order [m][par][latitude tile][row tile].  Within a block
//     the latitude index is XORed with 4 for degrees 2, 3, 6, 7: the analysis
//     (16-byte loads of two latitudes) and the synthesis (8-byte loads, degrees
//     as the contraction index) both read it without bank conflicts.
//   * Data tiles are 128-byte rows with the 128-byte TMA swizzle: rows of 8
//     latitudes of one column (analysis), or of 8 columns of one degree
//     (synthesis; lane n takes column n/2 + 4 (n mod 2) of the eight, which
//     spreads each 8-lane phase over all banks).
// Units are listed largest first and dealt out to the SMs forwards and backwards
// in turn, which balances the triangular bands; where units are long, the three
// teams of an SM share its units.  Three independent blocks with equal shares
// lose up to a quarter of the time there: the warp schedulers serve the oldest
// first, and the youngest is left to finish alone (T170: the blocks of an SM
// ended after 300, 325 and 420 thousand cycles).
//
// Bound: the FP64 tensor pipe from T170 up (82-86 % of its rate with the padding
// to 8-row tiles counted; the inner loop alone reaches 97 %), the Fourier
// array's traffic and the units' latency below.  Measured against the kernels it
// replaced (analysis / synthesis, us): T42, 3095 field-levels 52 / 48 -> 37 /
// 35; T85, 480: 39.6 / 42.0 -> 31.5 / 30.7; 320 x 160 (T106), 180: 70 / 82 -> 25
// / 26; T170, 720: 434 / 396 -> 208 / 195; T341, 240: 909 / 987 -> 483 / 473
// (30.5 TF/s of the 37 executed).  Filling the stages with cp.async from the
// consumer warps instead took 268 / 264 us at T170: their copy instructions
// (up to ten per product) held the pipe at 61 %.
#include "sht_internal.h"
#include "sht_dmma.cuh"
#include "sht_l2.cuh"
#include "sht_tc.cuh"

#include <algorithm>
#include <cstdlib>
#include <mutex>

namespace sht {

namespace {

using dmma::mma1688;
using dmma::mma884;

constexpr int kKC = 16;  // contraction terms per stage (two 8-term steps)


struct BandArgs {
  const double2 *F;   // analysis input F[m][col][j]
  double2 *S;         // analysis output S[row][col]
  const double2 *Sc;  // synthesis input
  double2 *Fo;        // synthesis output
  const double *P;    // blocked table
  const BandItem *items;
  int nunits, ncb;    // work units (item, column block) and column blocks
  int lgcw;           // log2 CW
  int J, JH, ncol;
  int drop;           // the Fourier lines are read by one item only: drop them from L2
  int *err;           // the plan's error word (page-locked host memory)
};

// k-th unit of block b: the largest-first list is dealt out to the G blocks
// forwards and backwards in turn, so that their shares differ by less than one
// unit's work
__device__ __forceinline__ int unit_of(int k)
{
  const int G = gridDim.x, b = blockIdx.x;
  return k * G + ((k & 1) ? G - 1 - b : b);
}

// Stage layout (bytes, each part 1024-byte aligned): 8 CW columns x 16 terms of
// data, then TM x 2 table blocks.
template <int W, int TM>
struct BandStage {
  static constexpr int BB = W * 8 * kKC * 16, AB = TM * 1024, BYTES = BB + AB;
};

// What a unit's first stage tells the consumers; col0 < 0: no more units.
struct alignas(16) BandUnit {
  BandItem item;
  int col0, pad[3];
};

// Barriers and unit slots of one team; the block's unit counter and abort flag
struct BandCtl {
  uint64_t *full, *empty;
  BandUnit *unit;
  int *taken, *abort_flag, *err;
};

constexpr uint64_t kBandWaitLimit = 2000000000ull;  // 2 s per bounded wait

// Waits for a phase, for at most limit_ns of wall time: then the error word is
// set and every role of the block leaves its loop.
__device__ __forceinline__ bool band_wait(const BandCtl &c, uint64_t *bar, uint32_t parity,
                                          uint64_t limit_ns = kBandWaitLimit)
{
  const uint32_t addr = tc::smem_addr(bar);
  bool ok = true;
  uint64_t t0 = 0;
  for (int i = 1; !tc::mbar_try(addr, parity); ++i) {
    if (i & 31) continue;
    if (*(volatile int *)c.abort_flag) { ok = false; break; }
    const uint64_t now = tc::globaltimer_ns();
    if (t0 == 0) t0 = now;
    if (now - t0 > limit_ns) {
      *(volatile int *)c.abort_flag = 1;
      *(volatile int *)c.err = SHT_ERR_DEVICE_TIMEOUT;
      __threadfence_system();
      ok = false;
      break;
    }
  }
  return __all_sync(0xffffffffu, ok);
}

__device__ __forceinline__ void tma_4d(void *dst, const CUtensorMap *map, int x, int y, int z, int w, uint64_t *bar)
{
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];\n" ::"r"(
          tc::smem_addr(dst)),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(tc::smem_addr(bar))
      : "memory");
}
__device__ __forceinline__ void tma_3d(void *dst, const CUtensorMap *map, int x, int y, int z, uint64_t *bar)
{
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(
          tc::smem_addr(dst)),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(tc::smem_addr(bar))
      : "memory");
}

// A team's producer warp: every stage of the team's units in order, then a stage
// that says there are no more.  The units come off the block's counter, so that
// whichever team is ahead takes the next one; one is fetched ahead, since the
// smallest units have a stage or two.
template <int W, int TM, int NS, int TEAMS, bool INV>
__device__ void band_produce(const BandArgs &a, const CUtensorMap *map, char *sm, const BandCtl &c)
{
  using St = BandStage<W, TM>;
  const int lane = threadIdx.x & 31, CW = 1 << a.lgcw;
  int taken = 0;
  auto take = [&] {
    int k = taken++;
    if constexpr (TEAMS > 1) {
      if (lane == 0) k = atomicAdd(c.taken, 1);
      k = __shfl_sync(0xffffffffu, k, 0);
    }
    return unit_of(k);
  };
  int g = 0;  // stages issued so far
  bool ok = true;
  int un = take();
  BandItem nxt = a.items[un < a.nunits ? un / a.ncb : 0];
  while (ok && un < a.nunits) {
    const int u = un, col0 = (u % a.ncb) * (8 << a.lgcw);
    const BandItem it = nxt;
    un = take();
    if (un < a.nunits) nxt = a.items[un / a.ncb];
    const int nrt = (it.cnt + 7) >> 3, nlt = (a.JH + 7) >> 3;
    const int nst = INV ? (nrt + 1) >> 1 : (nlt + 1) >> 1;
    const double *P = a.P + (INV ? it.blk + (long long)it.t0 * nrt : it.blk + it.t0) * 64;
    for (int st = 0; st < nst; ++st, ++g) {
      const int slot = g % NS;
      if (g >= NS && !(ok = band_wait(c, c.empty + slot, ((g / NS) - 1) & 1))) break;
      char *B = sm + slot * St::BYTES, *A = B + St::BB;
      uint64_t *bar = c.full + slot;
      const int two = 2 * st + 1 < (INV ? nrt : nlt) ? 2 : 1;  // contraction tiles in this stage
      if (lane == 0) {
        if (st == 0) {
          c.unit[slot].item = it;
          c.unit[slot].col0 = col0;
        }
        tc::mbar_arrive_expect_tx(bar, (INV ? CW * 8 * kKC * 16 : two * CW * 1024) + two * it.tt * 512);
      }
      __syncwarp();
      if constexpr (INV) {
        if (lane < CW) tma_3d(B + lane * 2048, map, 2 * (col0 + 8 * lane), it.row & 1, (it.row >> 1) + kKC * st, bar);
        if (lane < it.tt) tc::bulk_g2s(A + lane * 1024, P + ((long long)lane * nrt + 2 * st) * 64, two * 512, bar);
      } else {
        if (lane < two) {
          tma_4d(B + lane * CW * 1024, map, 16 * (2 * st + lane), it.par, col0, it.m, bar);
          tc::bulk_g2s(A + lane * it.tt * 512, P + (long long)(2 * st + lane) * nrt * 64, it.tt * 512, bar);
        }
      }
    }
  }
  if (ok && (g < NS || band_wait(c, c.empty + g % NS, ((g / NS) - 1) & 1))) {
    if (lane == 0) {
      c.unit[g % NS].col0 = -1;
      tc::mbar_arrive(c.full + g % NS);
    }
    return;
  }
  // aborted: leave only when the copies have landed in the block's shared memory
  for (int s = 0; s < NS && s < g; ++s) {
    const int last = g - 1 - (g - 1 - s) % NS;  // last stage issued to slot s
    const uint64_t t0 = tc::globaltimer_ns();
    while (!tc::mbar_try(tc::smem_addr(c.full + s), (last / NS) & 1))
      if (tc::globaltimer_ns() - t0 > kBandWaitLimit) break;
  }
}

// ------------------------------------------------------------------ analysis
// SPLIT: the warps split the row tiles (RW > 1); otherwise T is the item's
// tile count and every table offset is a constant.  Returns false on abort.
template <int W, int TM, int T, int NS, bool SPLIT>
__device__ __forceinline__ bool band_fwd(const BandArgs &a, const char *sm, const BandCtl &ctl, int &g, const BandItem &it,
                                         int col0)
{
  using St = BandStage<W, TM>;
  const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) % W;
  const int lgcw = SPLIT ? a.lgcw : __ffs(W) - 1;
  const int cg = warp & ((1 << lgcw) - 1), rw = SPLIT ? warp >> lgcw : 0;
  const int lgrw = SPLIT ? __ffs(W) - 1 - lgcw : 0, TT = SPLIT ? it.tt : T;
  const int nlt = (a.JH + 7) >> 3;

  double acc[T][2][2];
#pragma unroll
  for (int t = 0; t < T; ++t) acc[t][0][0] = acc[t][0][1] = acc[t][1][0] = acc[t][1][1] = 0.0;
  const int n = lane >> 2, q = lane & 3;
  // K order: a pair of steps takes latitudes 2q and 2q + 1 of the tile's eight
  const int b0 = (8 * cg + n) * 16 + 2 * ((2 * q) ^ n), b1 = (8 * cg + n) * 16 + 2 * ((2 * q + 1) ^ n);
  const int ao = 8 * n + 2 * (q ^ (n & 2));
  auto tile = [&](const double *B, const double *A) {
    const double2 be = *reinterpret_cast<const double2 *>(B + b0);
    const double2 bd = *reinterpret_cast<const double2 *>(B + b1);
    double2 av[T];
#pragma unroll
    for (int t = 0; t < T; ++t)
      av[t] = *reinterpret_cast<const double2 *>(A + ao + (SPLIT ? min(rw + (t << lgrw), TT - 1) : t) * 64);
#pragma unroll
    for (int t = 0; t + 1 < T; t += 2) {
      mma1688(acc[t][0], acc[t + 1][0], av[t].x, av[t + 1].x, av[t].y, av[t + 1].y, be.x, bd.x);
      mma1688(acc[t][1], acc[t + 1][1], av[t].x, av[t + 1].x, av[t].y, av[t + 1].y, be.y, bd.y);
    }
    if constexpr (T % 2 != 0) {
      mma884(acc[T - 1][0], av[T - 1].x, be.x);
      mma884(acc[T - 1][1], av[T - 1].x, be.y);
      mma884(acc[T - 1][0], av[T - 1].y, bd.x);
      mma884(acc[T - 1][1], av[T - 1].y, bd.y);
    }
  };
  for (int lt = 0; lt < nlt; lt += 2, ++g) {
    const int slot = g % NS;
    if (!band_wait(ctl, ctl.full + slot, (g / NS) & 1)) return false;
    const double *B = reinterpret_cast<const double *>(sm + slot * St::BYTES), *A = B + St::BB / 8;
    tile(B, A);
    if (lt + 1 < nlt) tile(B + (128 << lgcw), A + TT * 64);
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(ctl.empty + slot);
  }
  const int c0 = col0 + 8 * cg + 2 * q;
  double2 *S = a.S + ((long long)it.row + 16 * (it.t0 + rw) + 2 * n) * a.ncol + c0;
#pragma unroll
  for (int t = 0; t < T; ++t, S += (16ll << lgrw) * a.ncol) {
    const int tl = rw + (t << lgrw);
    if (tl >= TT || 8 * (it.t0 + tl) + n >= it.cnt) continue;
    if (c0 < a.ncol) S[0] = make_double2(acc[t][0][0], acc[t][1][0]);
    if (c0 + 1 < a.ncol) S[1] = make_double2(acc[t][0][1], acc[t][1][1]);
  }
  if (a.drop) {
    // no later kernel reads these Fourier lines: drop them without a write-back
    // (this warp's columns, or its share of them: their copies have landed)
    const int lpc = a.JH / 8;  // 128-byte lines per column
    const char *F = reinterpret_cast<const char *>(a.F + ((long long)it.m * a.ncol + col0 + 8 * cg) * a.J + it.par * a.JH);
    const int ncv = min(8, a.ncol - col0 - 8 * cg);
    for (int x = lane + 32 * rw; x < ncv * lpc; x += 32 << lgrw) {
      const int c = x / lpc;
      l2::discard_line(F + (long long)c * a.J * 16 + 128 * (x - c * lpc));
    }
  }
  return true;
}

// ----------------------------------------------------------------- synthesis
template <int W, int TM, int T, int NS, bool SPLIT>
__device__ __forceinline__ bool band_inv(const BandArgs &a, const char *sm, const BandCtl &ctl, int &g, const BandItem &it,
                                         int col0)
{
  using St = BandStage<W, TM>;
  const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) % W;
  const int lgcw = SPLIT ? a.lgcw : __ffs(W) - 1;
  const int cg = warp & ((1 << lgcw) - 1), rw = SPLIT ? warp >> lgcw : 0;
  const int lgrw = SPLIT ? __ffs(W) - 1 - lgcw : 0, TT = SPLIT ? it.tt : T;

  double acc[T][2][2];
#pragma unroll
  for (int t = 0; t < T; ++t) acc[t][0][0] = acc[t][0][1] = acc[t][1][0] = acc[t][1][1] = 0.0;
  const int n = lane >> 2, q = lane & 3;
  const int cn = (n >> 1) | ((n & 1) << 2);  // column of the group that lane n multiplies
  // row q of a step at 16 q, its 16-byte chunk XORed with row mod 8 = q or 4 + q
  const int b0 = cg * 256 + 16 * q + 2 * (cn ^ q), b1 = cg * 256 + 16 * (q + 4) + 2 * (cn ^ (q + 4));
  const int ao = 8 * q + (n ^ (4 * (q >> 1)));
  auto table = [&](const double *A, int t, int ks) {
    return A[ao + (SPLIT ? min(rw + (t << lgrw), TT - 1) : t) * 128 + 32 * ks];
  };
  auto two_steps = [&](const double *B, const double *A, int ks, double2 b, double2 d) {
    double av[T], aw[T];
#pragma unroll
    for (int t = 0; t < T; ++t) {
      av[t] = table(A, t, ks);
      aw[t] = table(A, t, ks + 1);
    }
#pragma unroll
    for (int t = 0; t + 1 < T; t += 2) {
      mma1688(acc[t][0], acc[t + 1][0], av[t], av[t + 1], aw[t], aw[t + 1], b.x, d.x);
      mma1688(acc[t][1], acc[t + 1][1], av[t], av[t + 1], aw[t], aw[t + 1], b.y, d.y);
    }
    if constexpr (T % 2 != 0) {
      mma884(acc[T - 1][0], av[T - 1], b.x);
      mma884(acc[T - 1][1], av[T - 1], b.y);
      mma884(acc[T - 1][0], aw[T - 1], d.x);
      mma884(acc[T - 1][1], aw[T - 1], d.y);
    }
  };
  auto data = [&](const double *B, int off, bool ok) {
    const double2 b = *reinterpret_cast<const double2 *>(B + off);
    return ok ? b : make_double2(0.0, 0.0);
  };
  for (int left = it.cnt; left > 0; left -= kKC, ++g) {  // degrees
    const int slot = g % NS;
    if (!band_wait(ctl, ctl.full + slot, (g / NS) & 1)) return false;
    const double *B = reinterpret_cast<const double *>(sm + slot * St::BYTES), *A = B + St::BB / 8;
    if (left >= kKC) {
      two_steps(B, A, 0, data(B, b0, true), data(B, b1, true));
      two_steps(B, A, 2, data(B, 128 + b0, true), data(B, 128 + b1, true));
    } else {
      // the tile rows past the last degree hold the next band's coefficients:
      // taken as zero, like the table's
      for (int s = 0; s < left; s += 8) {
        const int h = s >> 3;
        const double2 b = data(B, 128 * h + b0, s + q < left), d = data(B, 128 * h + b1, s + 4 + q < left);
        if (s + 4 < left) {
          two_steps(B, A, 2 * h, b, d);
        } else {
#pragma unroll
          for (int t = 0; t < T; ++t) {
            const double av = table(A, t, 2 * h);
            mma884(acc[t][0], av, b.x);
            mma884(acc[t][1], av, b.y);
          }
        }
      }
    }
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(ctl.empty + slot);
  }
  const uint64_t keep = l2::keep_policy();  // the Fourier runs stay in L2 for the longitude transform
  // accumulator columns 2q and 2q + 1 are columns q and q + 4 of the group
  const int c0 = col0 + 8 * cg + q, jh0 = 8 * (it.t0 + rw) + n;
  double2 *F = a.Fo + ((long long)it.m * a.ncol + c0) * a.J + it.par * a.JH + jh0;
  const bool k0 = c0 < a.ncol, k1 = c0 + 4 < a.ncol;
#pragma unroll
  for (int t = 0; t < T; ++t) {
    if (rw + (t << lgrw) >= TT || jh0 + (8 * t << lgrw) >= a.JH) continue;
    if (k0) l2::st_keep(F + (8 * t << lgrw), make_double2(acc[t][0][0], acc[t][1][0]), keep);
    if (k1) l2::st_keep(F + 4ll * a.J + (8 * t << lgrw), make_double2(acc[t][0][1], acc[t][1][1]), keep);
  }
  return true;
}

// TEAMS teams of W consumer warps and a producer warp, each with its own ring of
// stages and its own unit.  The row tiles per warp (tt / RW rounded
// up) select the unrolled code.
template <int W, int TM, int NS, int TEAMS, int MINB, bool INV, bool SPLIT>
__global__ void __launch_bounds__(32 * (W + 1) * TEAMS, MINB) k_leg_band(const __grid_constant__ CUtensorMap map, BandArgs a)
{
  extern __shared__ __align__(1024) char sm_band[];
  constexpr int SLOTS = TEAMS * NS, STB = BandStage<W, TM>::BYTES;
  BandUnit *units = reinterpret_cast<BandUnit *>(sm_band + SLOTS * STB);
  uint64_t *bars = reinterpret_cast<uint64_t *>(units + SLOTS);
  int *words = reinterpret_cast<int *>(bars + 2 * SLOTS);
  if (threadIdx.x == 0) {
    for (int s = 0; s < SLOTS; ++s) {
      tc::mbar_init(bars + s, 1);
      tc::mbar_init(bars + SLOTS + s, W);
    }
    words[0] = words[1] = 0;
    tc::mbar_fence_init();
  }
  __syncthreads();
  // warps: the teams' consumers, then their producers
  const int w = threadIdx.x >> 5, team = w < W * TEAMS ? w / W : w - W * TEAMS;
  const BandCtl ctl{bars + team * NS, bars + SLOTS + team * NS, units + team * NS, words, words + 1, a.err};
  char *const sm = sm_band + team * NS * STB;
  if (w >= W * TEAMS) {
    band_produce<W, TM, NS, TEAMS, INV>(a, &map, sm, ctl);
    return;
  }
  const int lgrw = SPLIT ? __ffs(W) - 1 - a.lgcw : 0;
  int g = 0;  // stages consumed
  while (true) {
    if (!band_wait(ctl, ctl.full + g % NS, (g / NS) & 1)) return;
    const BandItem it = ctl.unit[g % NS].item;
    const int col0 = ctl.unit[g % NS].col0;
    if (col0 < 0) return;
    bool ok = true;
    auto go = [&](auto tc) {
      constexpr int T = decltype(tc)::value;
      if constexpr (T <= TM) {
        if constexpr (INV) ok = band_inv<W, TM, T, NS, SPLIT>(a, sm, ctl, g, it, col0);
        else ok = band_fwd<W, TM, T, NS, SPLIT>(a, sm, ctl, g, it, col0);
      }
    };
    using std::integral_constant;
    switch ((it.tt + (1 << lgrw) - 1) >> lgrw) {
    case 1: go(integral_constant<int, 1>()); break;
    case 2: go(integral_constant<int, 2>()); break;
    case 3: go(integral_constant<int, 3>()); break;
    case 4: go(integral_constant<int, 4>()); break;
    case 5: go(integral_constant<int, 5>()); break;
    case 6: go(integral_constant<int, 6>()); break;
    case 7: go(integral_constant<int, 7>()); break;
    case 8: go(integral_constant<int, 8>()); break;
      default: break;
    }
    if (!ok) return;
  }
}

// The failure path of the waits above, run on purpose: the first warp waits on a
// barrier that nothing arrives at, gives up after limit_ns, raises the abort flag
// and records the timeout; the second, waiting on the same barrier with the full
// limit, leaves on the flag.  No copies are in flight.
__global__ void __launch_bounds__(64) k_band_wait_selftest(int *err, uint64_t limit_ns)
{
  __shared__ __align__(8) uint64_t bar;
  __shared__ int words[2];
  if (threadIdx.x == 0) {
    tc::mbar_init(&bar, 1);
    words[0] = words[1] = 0;
    tc::mbar_fence_init();
  }
  __syncthreads();
  const BandCtl c{&bar, &bar, nullptr, words, words + 1, err};
  band_wait(c, &bar, 0, threadIdx.x < 32 ? limit_ns : kBandWaitLimit);
}

int max_row_tiles(int N) { return ((N + 3) / 2 + 7) / 8; }

// row tiles per item: the tiles of the largest band split evenly into items
// of at most `cap`
int even_split(int tiles, int cap)
{
  const int nblk = (tiles + cap - 1) / cap;
  return (tiles + nblk - 1) / nblk;
}

// 8 tiles of accumulators are what 128 registers hold; items of up to 11 (160
// registers, two teams) re-read the data less often but took 506 / 508 us at
// T341 where these take 483 / 473.
constexpr int kItemCap = 8;

}  // namespace

// The plans' error words.  A page of them is ordinary memory of this process,
// never freed and registered with the plans' device, so that the host may read a
// word whatever became of the context it was registered in; a page whose
// registration went with a device reset is registered again for the next plan.
// A word belongs to one live plan, is zero when it is handed out, and comes back
// with sht_final.
namespace {

struct ErrorPage {
  int device;
  int *words;
  std::vector<int> unused;
};
constexpr int kPageWords = 1024;
std::mutex g_error_mutex;
std::vector<ErrorPage> &error_pages()
{
  static auto *pages = new std::vector<ErrorPage>;  // outlives plans that are finalised at exit
  return *pages;
}

// the page's address on its device (current), registering it where it is not
cudaError_t page_address(const ErrorPage &g, int **dev)
{
  cudaPointerAttributes at;
  cudaError_t e = cudaPointerGetAttributes(&at, g.words);
  if (e != cudaSuccess || at.type == cudaMemoryTypeUnregistered) {
    cudaGetLastError();
    if ((e = cudaHostRegister(g.words, sizeof(int) * kPageWords, cudaHostRegisterMapped)) != cudaSuccess) return e;
  }
  void *d = nullptr;
  e = cudaHostGetDevicePointer(&d, g.words, 0);
  *dev = static_cast<int *>(d);
  return e;
}

int take_error_word(sht_plan *p)
{
  std::lock_guard<std::mutex> lk(g_error_mutex);
  auto &pages = error_pages();
  ErrorPage *g = nullptr;
  for (ErrorPage &c : pages)
    if (!g && c.device == p->device && !c.unused.empty()) g = &c;
  if (!g) {
    int *w = static_cast<int *>(std::aligned_alloc(4096, sizeof(int) * kPageWords));
    if (!w) { set_error("error words: host allocation failed"); return SHT_ERR_ALLOC; }
    pages.push_back({p->device, w, {}});
    g = &pages.back();
    for (int k = kPageWords; k-- > 0;) g->unused.push_back(k);
  }
  int *dev = nullptr;
  const cudaError_t e = page_address(*g, &dev);
  if (e != cudaSuccess) return cuda_fail(e, "error words");
  const int k = g->unused.back();
  g->unused.pop_back();
  p->err_word = g->words + k;
  p->err_dev = dev + k;
  *(volatile int *)p->err_word = 0;
  return SHT_OK;
}

}  // namespace

void return_error_word(sht_plan *p)
{
  if (!p->err_word) return;
  std::lock_guard<std::mutex> lk(g_error_mutex);
  for (ErrorPage &g : error_pages())
    if (p->err_word >= g.words && p->err_word < g.words + kPageWords) g.unused.push_back((int)(p->err_word - g.words));
  p->err_word = p->err_dev = nullptr;
}

int launch_band_wait_selftest(const sht_plan *p, unsigned long long limit_ns, cudaStream_t s)
{
  k_band_wait_selftest<<<1, 64, 0, s>>>(p->err_dev, limit_ns);
  count_launch();
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? SHT_OK : cuda_fail(e, "k_band_wait_selftest");
}

int band_error_status(sht_plan *p)
{
  if (!p->err_word || *(volatile int *)p->err_word == 0) return SHT_OK;
  *(volatile int *)p->err_word = 0;
  set_error("legendre: a bounded shared-memory wait timed out");
  return SHT_ERR_DEVICE_TIMEOUT;
}

// The block offsets of every (m, parity) in the blocked table (the last entry
// is the block count) and the item lists of both directions, largest first.
int plan_band_items(sht_plan *p, std::vector<long long> &boff, std::vector<BandItem> &items)
{
  const int rc = take_error_word(p);
  if (rc) return rc;
  const int N = p->N, M = p->M, nlt = (p->JH + 7) / 8;
  auto count = [&](int m, int par) { const int R = N + 2 - m; return par ? R / 2 : (R + 1) / 2; };
  boff.resize(2 * M + 1);
  long long nb = 0;
  for (int m = 0; m < M; ++m)
    for (int par = 0; par < 2; ++par) {
      boff[2 * m + par] = nb;
      nb += (long long)nlt * ((count(m, par) + 7) / 8);
    }
  boff[2 * M] = nb;
  p->band_tf = even_split(max_row_tiles(N), kItemCap);
  p->band_ti = even_split(nlt, kItemCap);
  std::vector<BandItem> inv;
  for (int m = 0; m < M; ++m)
    for (int par = 0; par < 2; ++par) {
      const int cnt = count(m, par), nrt = (cnt + 7) / 8;
      auto item = [&](int t0, int tt) { return BandItem{m, par, t0, tt, boff[2 * m + par], p->h_rowoff[m] + par, cnt}; };
      for (int t = 0; t < nrt; t += p->band_tf) items.push_back(item(t, std::min(p->band_tf, nrt - t)));
      for (int t = 0; t < nlt && nrt > 0; t += p->band_ti) inv.push_back(item(t, std::min(p->band_ti, nlt - t)));
    }
  std::stable_sort(items.begin(), items.end(), [](const BandItem &x, const BandItem &y) { return x.tt > y.tt; });
  p->n_band_f = (int)items.size();
  p->n_band_i = (int)inv.size();
  items.insert(items.end(), inv.begin(), inv.end());
  return SHT_OK;
}

namespace {

// cuTensorMapEncodeTiled of the driver in use (no link-time dependency)
using EncodeTiled = decltype(&cuTensorMapEncodeTiled);
EncodeTiled encode_tiled()
{
  static const EncodeTiled fn = [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult st;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &st) != cudaSuccess ||
        st != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<EncodeTiled>(f);
  }();
  return fn;
}

// The data operand as a tensor.  Analysis: (re/im of a latitude, parity half,
// column, order); synthesis: (re/im of a column, row parity, row pair).  The
// strides are multiples of 16 bytes whatever the counts.
int data_map(const sht_plan *p, const BandArgs &a, bool inv, const CUtensorMap **out)
{
  auto &slot = p->band_map[inv];
  const void *ptr = inv ? a.Sc : a.F;
  *out = &slot.map;
  // a map is a function of the address and the counts alone
  if (slot.ptr == ptr && slot.ncol == a.ncol && slot.lgcw == a.lgcw) return SHT_OK;
  slot.ptr = nullptr;
  CUtensorMap *map = &slot.map;
  const EncodeTiled enc = encode_tiled();
  if (!enc) { set_error("legendre: the driver has no cuTensorMapEncodeTiled"); return SHT_ERR_CUDA; }
  const cuuint64_t nc = (cuuint64_t)a.ncol, col = 16ull * p->J;
  const cuuint32_t one[4] = {1, 1, 1, 1};
  CUresult r;
  if (inv) {
    const long long rows = p->zonal ? p->N + 2 : p->R;
    const cuuint64_t dims[3] = {2 * nc, 2, (cuuint64_t)(rows + 1) / 2}, str[2] = {16 * nc, 32 * nc};
    const cuuint32_t box[3] = {16, 1, kKC};
    r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<double2 *>(a.Sc), dims, str, box, one,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  } else {
    const cuuint64_t dims[4] = {2ull * p->JH, 2, nc, (cuuint64_t)p->M}, str[3] = {16ull * p->JH, col, nc * col};
    const cuuint32_t box[4] = {16, 1, 8u << a.lgcw, 1};
    r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, const_cast<double2 *>(a.F), dims, str, box, one,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  }
  if (r != CUDA_SUCCESS) { set_error("legendre: tensor map encoding failed"); return SHT_ERR_CUDA; }
  slot.ptr = ptr;
  slot.ncol = a.ncol;
  slot.lgcw = a.lgcw;
  return SHT_OK;
}

template <int W, int TM, int NS, int TEAMS, int MINB, bool INV>
int run_band(const sht_plan *p, BandArgs a, cudaStream_t s)
{
  constexpr size_t smem = (size_t)TEAMS * NS * (BandStage<W, TM>::BYTES + sizeof(BandUnit) + 16) + 16;
  static_assert(MINB * (smem + 1024) <= 228 * 1024, "stages");
  // Columns per block: 8 W where the batch has that many.  A batch whose units
  // would leave block slots empty takes fewer (the warps then split the rows):
  // in the synthesis until the slots are filled (T85, 60 field-levels: 7.3 ->
  // 6.6 us), in the analysis while all units still run at once (T42, 60: 4.4 us
  // with the synthesis's rule, 3.8 with this).
  const int items = INV ? p->n_band_i : p->n_band_f;
  int lg = 0;
  while ((1 << lg) < W && (8 << lg) < a.ncol) ++lg;
  auto units_at = [&](int l) { return (long long)items * ((a.ncol + (8 << l) - 1) / (8 << l)); };
  const long long slots = (long long)TEAMS * MINB * grid_sms(p);
  while (lg > 0 && (INV ? units_at(lg) < slots : units_at(lg - 1) <= slots)) --lg;
  a.lgcw = lg;
  a.ncb = (a.ncol + (8 << lg) - 1) / (8 << lg);
  const long long units = units_at(lg);
  if (units > 0x3fffffffLL) { set_error("legendre: too many field-levels for one call"); return SHT_ERR_TOO_LARGE; }
  a.nunits = (int)units;
  const CUtensorMap *map = nullptr;
  const int rc = data_map(p, a, INV, &map);
  if (rc) return rc;
  auto kern = (1 << lg) == W ? k_leg_band<W, TM, NS, TEAMS, MINB, INV, false>
                             : k_leg_band<W, TM, NS, TEAMS, MINB, INV, true>;
  constexpr int threads = 32 * (W + 1) * TEAMS;
  cudaError_t e = kernel_setup((const void *)kern, smem, threads);
  if (e != cudaSuccess) return cuda_fail(e, "legendre band smem attribute");
  kern<<<(unsigned)std::min<long long>(units, (long long)MINB * grid_sms(p)), threads, smem, s>>>(*map, a);
  count_launch();
  e = cudaGetLastError();
  return e == cudaSuccess ? SHT_OK : cuda_fail(e, "k_leg_band");
}

template <bool INV>
int launch_band(const sht_plan *p, BandArgs a, cudaStream_t s)
{
  a.P = p->d_band_P;
  a.items = p->d_band_items + (INV ? p->n_band_f : 0);
  a.J = p->J; a.JH = p->JH;
  a.err = p->err_dev;
  const int tm = INV ? p->band_ti : p->band_tf;
  // One block of three teams, or three blocks of one.  The teams share the SM's
  // units, which pays where a unit is long (analysis / synthesis, T170, 720:
  // 221 / 215 -> 208 / 195 us, T341, 240: 506 / 508 -> 483 / 473); below, blocks
  // that start and end apart are level or ahead (T85, 480: 31.5 / 30.7 either way,
  // T42, 3095: 39.8 / 36.9 shared, 37 / 35 apart).
  if (p->N > 127) return run_band<4, 8, 4, 3, 1, INV>(p, a, s);
  if (tm <= 6) return run_band<4, 6, 4, 1, 3, INV>(p, a, s);
  return run_band<4, 8, 4, 1, 3, INV>(p, a, s);
}

}  // namespace

int launch_leg_fwd_fp64(const sht_plan *p, const double2 *F, int ncol, double2 *S, cudaStream_t s)
{
  if (ncol <= 0) return SHT_OK;
  BandArgs a{};
  a.F = F; a.S = S; a.ncol = ncol;
  a.drop = p->JH % 8 == 0 && max_row_tiles(p->N) <= p->band_tf;
  return launch_band<false>(p, a, s);
}

int launch_leg_inv_fp64(const sht_plan *p, const double2 *S, int ncol, double2 *F, cudaStream_t s)
{
  if (ncol <= 0) return SHT_OK;
  BandArgs a{};
  a.Sc = S; a.Fo = F; a.ncol = ncol;
  return launch_band<true>(p, a, s);
}

}  // namespace sht
