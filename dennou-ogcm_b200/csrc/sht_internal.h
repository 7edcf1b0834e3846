// sht_internal.h -- plan state, device layouts and kernel launchers of the
// B200 spherical-harmonic transform.
//
// Device data layouts (all FP64):
//   grid      xya[b][j][i]        b < nb field-levels, j < J (mu ascending), i < I
//   spectral  wa[b][l]            SPML order l = n(n+1)+m, m in [-n, n]
//   Fourier   F[m][col][j]        complex G^m(mu_j) for m <= N, col < ncol
//                                 (ncol = nb, or 2 nb for two-input operators)
//   internal  S[row][col]         complex coefficient of Pbar_n^m, row = rowoff(m) + n - m,
//                                 n = m..N+1 (one extra degree so that the
//                                 (1-mu^2) d/dmu recurrences close), rowoff(m) =
//                                 sum_{m'<m} (N+2-m').
//   Legendre  P[poff(m) + (n-m) JH + jh]  Pbar_n^m at the northern Gauss rows
//                                 j = JH + jh (JH = J/2), n = m..N+1.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdint>
#include <cstddef>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/dogcm_sht.h"

namespace sht {

// Row-scale tables used by the longitude transforms (per Gauss row j).
enum RowScale : int {
  RS_FWD_PLAIN = 0,     // analysis: w_j / I
  RS_FWD_INV1MMU2 = 1,  // analysis: w_j / (I (1 - mu_j^2))
  RS_INV_PLAIN = 2,     // synthesis: 1
  RS_INV_INVCOS = 3,    // synthesis: 1 / cos(phi_j)
  RS_INV_INVA1MMU2 = 4, // synthesis: 1 / (a (1 - mu_j^2))
  RS_INV_INVACOS = 5,   // synthesis: 1 / (a cos(phi_j))
  RS_FWD_INVCOS = 6,    // analysis: w_j / (I cos(phi_j)) = w_j cos(phi_j) / (I (1 - mu_j^2))
  RS_COUNT = 7
};

// Spectral-side operators applied between the SPML layout and the internal one.
enum PackOp : int {
  PACK_PLAIN = 0,      // w = c
  PACK_DIVLAMBDA = 1,  // w = i m c
  PACK_DIVMU = 2,      // w = D(c) = -((n+1) eps_n c_{n-1} - n eps_{n+1} c_{n+1})
  PACK_ALPHA = 3,      // w = (i m cA + D(cB)) / a, D = the divmu form    (two column sets)
  PACK_VORDIV = 4,     // vor = (i m cV - D(cU))/a, div = (i m cU + D(cV))/a
};
enum UnpackOp : int {
  UNPACK_PLAIN = 0,      // a
  UNPACK_GRADLAMBDA = 1, // i m a
  UNPACK_GRADMU = 2,     // (k+2) eps_{k+1} a_{k+1} - (k-1) eps_k a_{k-1}
  UNPACK_ALPHA = 3,      // i m aA + GRADMU(aB)                   (two inputs)
  UNPACK_VORDIV2UV = 4,  // psi, chi = -a^2 a/(n(n+1)); U = i m chi - GRADMU(psi), V = i m psi + GRADMU(chi)
  UNPACK_HGRAD = 5,      // i m a and GRADMU(a) from one input    (two column sets)
};

struct Timing {
  bool on = false;
  cudaEvent_t ev[8] = {};
  float ms_fft = 0.f, ms_leg = 0.f, ms_spec = 0.f;
};

// A host-pointer call staged through the plan's page-locked buffer, kept as
// an instantiated CUDA graph (copy in, the operator's kernels, copy out).
// Every pointer in it is a plan buffer, so it replays for any caller arrays
// of the same operator and size until a buffer is reallocated (buf_gen).
struct HostGraph {
  int op = -1, nb = 0, precision = 0;
  bool small = false;              // captured with the single-kernel small-grid transform chosen
  unsigned long long gen = 0;
  cudaGraphExec_t exec = nullptr;  // null after the first call, or when not capturable
  bool failed = false;             // capture was refused: run this call uncaptured
  int launches = 0;                // kernels in the graph
};

// A work item of the band kernels: row tiles [t0, t0 + tt) of the output of
// band m and parity par, whose table starts at block blk, whose coefficients
// are the cnt internal rows row, row + 2, ...
struct alignas(16) BandItem {
  int m, par, t0, tt;
  long long blk;
  int row, cnt;
};

// The blocked Legendre table (sht_legendre_band.cu): element (k, jh) of a band
// and parity whose blocks begin at block blk and lie in rows of nrt row tiles --
// k-th degree of the parity, latitude jh.
__host__ __device__ inline long long band_at(long long blk, int nrt, int k, int jh)
{
  const int d = k & 7;
  return (blk + (long long)(jh >> 3) * nrt + (k >> 3)) * 64 + 8 * d + ((jh & 7) ^ (4 * ((d >> 1) & 1)));
}

}  // namespace sht

struct sht_plan_s {
  uint32_t magic = 0;
  int I = 0, J = 0, N = 0, K = 0, JH = 0, NC = 0, L = 0;
  long long R = 0;              // internal rows (N+1)(N+4)/2
  double radius = 1.0;
  int device = 0;
  cudaStream_t stream = nullptr;      // stream used by all work of the plan
  cudaStream_t own_stream = nullptr;  // stream created by sht_init (destroyed by sht_final)
  // host-pointer calls: copy streams and per-chunk events of the pipelined
  // host -> device -> host path (created on first use)
  cudaStream_t copy_in = nullptr, copy_out = nullptr;
  cudaEvent_t chunk_ev[16] = {};
  bool zonal = false;  // im = 1: the axisymmetric (m = 0) transform of wa_zonal_module, lm = nm + 1
  bool direct_dft = false;  // im not a power of two: mixed-radix FFT (factors 2, 3, 5) or, for other prime factors, direct summation
  int M = 0;           // orders transformed: N + 1, or 1 for a zonal plan
  int precision = SHT_PREC_FP64;
  int leg_kernel = 0;  // SHT_OPT_LEGENDRE_KERNEL: 4 single-kernel small-grid transform (plain analysis and synthesis,
                       // im <= 128); the other values all take the band kernels
  int leg_tile = 0;    // SHT_OPT_LEGENDRE_TILE: kept for the callers that set and read it, selects nothing

  // device tables, all in one allocation
  void *d_tables = nullptr;
  double *d_mu = nullptr, *d_wgt = nullptr, *d_rowscale = nullptr;
  double *d_P = nullptr;    // row-major Legendre table, where the small-grid kernel takes the plan
  int *d_rowoff = nullptr;
  double *d_eps = nullptr;  // [m][n], n = 0..N+2
  double2 *d_tw = nullptr;  // exp(-2 pi i k / NC), k < NC
  double2 *d_twI = nullptr; // exp(-2 pi i k / I),  k < NC
  double *d_rn = nullptr;   // -n(n+1) per l
  int2 *d_spec_tiles = nullptr;  // (n, m0) tiles of the spectral conversions
  int n_spec_tiles = 0;          // n = 0..N+1
  int n_pack_tiles = 0;          // n = 0..N (a prefix of the list)
  int2 *d_pairs = nullptr;       // band pairs (m, N-m), (N/2, -1) for even N
  int n_pairs = 0;
  int num_sms = 0;
  int sm_cap = 0;       // at most this many SMs' worth of persistent blocks (0: all); set by a batch that runs plans side by side

  // blocked Legendre table and work items of the band kernels (sht_legendre_band.cu)
  double *d_band_P = nullptr;
  long long *d_band_off = nullptr;
  sht::BandItem *d_band_items = nullptr;  // analysis items, then synthesis items
  int *err_word = nullptr, *err_dev = nullptr;  // host word their bounded waits report a timeout in, its device address
  int n_band_f = 0, n_band_i = 0;
  int band_tf = 0, band_ti = 0;  // most 8-row tiles of an item
  // the last data tensor map of each direction: encoding one costs a launch
  // about a microsecond of host time (used under the plan's mutex)
  struct BandMap {
    const void *ptr = nullptr;
    int ncol = 0, lgcw = 0;
    CUtensorMap map;
  };
  mutable BandMap band_map[2];

  // host copies
  std::vector<double> h_mu, h_wgt;
  std::vector<int> h_rowoff;

  // device workspace (Fourier + internal spectral), grown on demand
  void *d_ws = nullptr;
  size_t ws_bytes = 0;
  // device staging for the host-pointer API, grown on demand
  void *d_io = nullptr;
  size_t io_bytes = 0;
  // page-locked host staging for small host-pointer calls on pageable arrays
  void *h_stage = nullptr;
  size_t h_stage_bytes = 0;

  // split-precision tables (built lazily)
  void *tc_tables = nullptr;
  // device address of the allocation-free entry point's fixed scratch array
  // on this plan's device (looked up on that entry point's first call)
  void *noalloc_scratch = nullptr;

  // graphs of staged host-pointer calls (SHT_OPT_HOST_GRAPHS), the stream
  // they are captured on, and the generation of the buffers they name
  // (bumped whenever d_ws, d_io or h_stage is reallocated)
  bool host_graphs = true;
  std::vector<sht::HostGraph> graphs;
  cudaStream_t cap_stream = nullptr;
  unsigned long long buf_gen = 0;

  std::mutex mtx;
  sht::Timing timing;
};

namespace sht {

constexpr uint32_t kPlanMagic = 0x53485442u;  // "SHTB"

void set_error(const std::string &msg);
int cuda_fail(cudaError_t e, const char *what);
void count_launch(int n = 1);

// Dynamic shared-memory opt-in of a kernel and its resident blocks per SM at
// (smem, threads), on the current device.  The runtime calls behind them
// cost microseconds each, which a per-level call would pay on every launch,
// so the results are cached per device and kernel; the opt-in only grows.
cudaError_t kernel_setup(const void *kern, size_t smem, int threads, int *per_sm = nullptr);

// --- setup kernels (sht_setup.cu)
int build_tables(sht_plan *p);

// --- longitude transforms (sht_fft.cu)
// grid (up to two source arrays: columns [0, nsplit) from g0, the rest from g1;
// or, when gcol is given, column c at gcol[c]) -> F[m][colF0 + col][j],
// scaled per row by rowscale table `rs`.
int launch_fft_fwd(const sht_plan *p, const double *g0, const double *g1, int nsplit, int ncol,
                   double2 *F, int ncolF, int colF0, int rs, cudaStream_t s,
                   const double *const *gcol = nullptr, const double *mul = nullptr, int nmul = 0,
                   const double *add0 = nullptr, const double *add1 = nullptr);
// F -> grid (two destinations split at nsplit, or column c at ocol[c]),
// scaled per row by `rs`.
int launch_fft_inv(const sht_plan *p, const double2 *F, int ncolF, int colF0, int ncol,
                   double *g0, double *g1, int nsplit, int rs, cudaStream_t s,
                   double *const *ocol = nullptr);

// --- Legendre contraction, FP64: one band and parity per block, any grid
// (sht_legendre_band.cu)
int plan_band_items(sht_plan *p, std::vector<long long> &boff, std::vector<BandItem> &items);
int band_error_status(sht_plan *p);  // reads and clears the plan's error word (after a synchronisation)
void return_error_word(sht_plan *p);  // once none of the plan's kernels can run any more
int launch_leg_fwd_fp64(const sht_plan *p, const double2 *F, int ncol, double2 *S, cudaStream_t s);
int launch_leg_inv_fp64(const sht_plan *p, const double2 *S, int ncol, double2 *F, cudaStream_t s);

bool split_supported(const sht_plan *p);
// Whether a contraction runs in split precision: always under SHT_PREC_SPLIT;
// under SHT_PREC_AUTO when it is at least 128 terms long (jm/2 latitudes in
// the analysis, (nm+3)/2 degrees of one parity in the synthesis).  That is the
// mode's documented meaning.  The line was drawn where the int8 digit kernel beat
// the per-grid FP64 kernels of the time; the band kernels are now the faster on
// both sides of it (synthesis / analysis, T170, 720: 195 / 208 us against 403 /
// 327; T341, 960: 1746 / 1832 against 2439 / 2384), so SHT_PREC_FP64 is the mode
// for speed.
inline bool use_split(const sht_plan *p, bool analysis)
{
  if (p->precision == SHT_PREC_SPLIT) return true;
  if (p->precision != SHT_PREC_AUTO || !split_supported(p)) return false;
  return (analysis ? p->JH : (p->N + 3) / 2) >= 128;
}

// --- whole plain transforms of small grids in one kernel (sht_small.cu)
bool small_supported(const sht_plan *p);
int launch_small_fwd(const sht_plan *p, const double *g, const double *const *gcol, int ncol, double *w,
                     double *const *wcol, cudaStream_t s);
int launch_small_inv(const sht_plan *p, const double *w, const double *const *wcol, int ncol, double *g,
                     double *const *gcol, cudaStream_t s);
// plain analysis / synthesis by the single-kernel small-grid transform:
// chosen with SHT_OPT_LEGENDRE_KERNEL = 4, and by the automatic choice for
// im = 32 (16 complex points per row), the only size where it measured
// faster than the batched kernels (T10, 480 field-levels: round trip 23
// against 25 us); in FP64 only (split precision keeps the batched path)
inline bool wants_small(const sht_plan *p) { return p->leg_kernel == 4 || (p->leg_kernel == 0 && p->NC == 16); }
inline bool use_small(const sht_plan *p, bool analysis)
{
  return wants_small(p) && !use_split(p, analysis) && small_supported(p);
}

// SMs a plan's persistent kernels size their grids for
inline int grid_sms(const sht_plan *p)
{
  const int n = p->num_sms > 0 ? p->num_sms : 1;
  return (p->sm_cap > 0 && p->sm_cap < n) ? p->sm_cap : n;
}

// --- Legendre contraction, split precision on tcgen05 (sht_legendre_i8.cu)
int launch_leg_fwd_split(sht_plan *p, const double2 *F, int ncol, double2 *S, cudaStream_t s);
int launch_leg_inv_split(sht_plan *p, const double2 *S, int ncol, double2 *F, cudaStream_t s);
void free_split_tables(sht_plan *p);
int split_error_status(sht_plan *p);  // reads and clears the device error word (synchronous)
// one block each whose bounded wait runs out on purpose and sets the error word
int launch_band_wait_selftest(const sht_plan *p, unsigned long long limit_ns, cudaStream_t s);
int launch_split_wait_selftest(sht_plan *p, unsigned long long limit_ns, cudaStream_t s);
// Reads and clears every device error word of the plan (synchronous).
int device_error_status(sht_plan *p);
// What the host-readable one says of calls that have finished (no waiting).
int earlier_timeout_status(sht_plan *p);

// --- column-table pipelines (sht_capi.cu), used by the multi-instance batches
// F holds (N+1) J ncol complex values, S holds R ncol; the plan mutex is held
// by the caller.
int run_analysis_cols(sht_plan *p, const double *const *gcol, int ncol, double *const *wcol, double2 *F,
                      double2 *S, cudaStream_t s);
int run_synthesis_cols(sht_plan *p, const double *const *wcol, int ncol, double *const *gcol, double2 *F,
                       double2 *S, cudaStream_t s);

// --- contraction and layout conversion in one kernel, narrow batches
// (sht_narrow.cu): sets is the operator's inputs (analysis) or outputs
// (synthesis), ncol = sets nb the columns of F
bool use_narrow(const sht_plan *p, int nb, int sets);
int launch_narrow_fwd(const sht_plan *p, int op, const double2 *F, int ncol, int nb, double *w0, double *w1, cudaStream_t s);
int launch_narrow_inv(const sht_plan *p, int op, const double *w0, const double *w1, int nb, double2 *F, int ncol,
                      cudaStream_t s);

// --- spectral-side kernels (sht_spectral.cu)
// internal S (ncolS columns; set A at col 0, set B at col nb) -> SPML wa outputs
// (field-level b at w0 + b L, or at wcol[b] when a column table is given;
// tables serve the single-output operators)
int launch_pack(const sht_plan *p, int op, const double2 *S, int ncolS, int nb, double *w0,
                double *w1, cudaStream_t s, double *const *wcol = nullptr);
// SPML inputs -> internal S (ncolS columns); wcol as for launch_pack
int launch_unpack(const sht_plan *p, int op, const double *w0, const double *w1, int nb,
                  double2 *S, int ncolS, cudaStream_t s, const double *const *wcol = nullptr);
int launch_lapla(const sht_plan *p, const double *w, int nb, double *out, bool inverse,
                 cudaStream_t s);
int launch_sub_filter(const sht_plan *p, double *a, const double *w, int nb, const double *filter, cudaStream_t s);
int launch_sub_lapla(const sht_plan *p, double *a, double *neg, const double *c, int nb, cudaStream_t s);
int launch_diffuse(const sht_plan *p, const double *w, int nb, const double *coef, double dt,
                   const double *filter, double *out, cudaStream_t s);
int launch_lonlat_reduce(const sht_plan *p, const double *g, int nb, double *out, int kind,
                         cudaStream_t s);

}  // namespace sht
