// sht_setup.cu -- plan tables: Gauss-Legendre nodes/weights and the
// associated-Legendre table, both generated on the device in FP64, plus the
// small host-built tables (twiddles, recurrence coefficients, row scales).
//
// Follows doc/description/ogcm/space_discretization.tex:33-38 (Gauss grid,
// mu ascending), :205-209 (weights normalised to sum 1), :169 (Pbar
// normalised to 2) and :250-257 (normalised three-term recurrence), which is
// what wa_Initial sets up inside SPMODEL (SpmlUtil_mod.f90:218-223).
#include "sht_internal.h"

#include <cmath>
#include <cstring>
#include <type_traits>

namespace sht {

// One thread per positive root of P_J: Newton iteration on the three-term
// recurrence, started from the Tricomi-type estimate cos(pi (k+3/4)/(J+1/2)).
__global__ void k_gauss_nodes(int J, double *mu, double *wgt)
{
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (J + 1) / 2) return;
  double x = cos(M_PI * (k + 0.75) / (J + 0.5));
  double dp = 1.0;
  for (int it = 0; it < 100; ++it) {
    double p0 = 1.0, p1 = x;
    for (int n = 2; n <= J; ++n) {
      const double p2 = ((2.0 * n - 1.0) * x * p1 - (n - 1.0) * p0) / n;
      p0 = p1;
      p1 = p2;
    }
    dp = J * (x * p1 - p0) / (x * x - 1.0);
    const double dx = p1 / dp;
    x -= dx;
    if (fabs(dx) < 1e-16 * (1.0 + fabs(x)) && it > 2) break;
  }
  // derivative at the converged root
  {
    double p0 = 1.0, p1 = x;
    for (int n = 2; n <= J; ++n) {
      const double p2 = ((2.0 * n - 1.0) * x * p1 - (n - 1.0) * p0) / n;
      p0 = p1;
      p1 = p2;
    }
    dp = J * (x * p1 - p0) / (x * x - 1.0);
  }
  const double w = 1.0 / ((1.0 - x * x) * dp * dp);  // sums to 1 over all J roots
  mu[J - 1 - k] = x;
  mu[k] = -x;
  wgt[J - 1 - k] = w;
  wgt[k] = w;
  if ((J & 1) && k == J / 2) mu[k] = 0.0;
}

// Pbar_n^m(mu_j) for the northern rows, one thread per (m, jh):
//   Pbar_m^m = prod_{k<=m} sqrt((2k+1)/(2k)) (1-mu^2)^{m/2}
//   Pbar_{n+1}^m = (mu Pbar_n^m - eps_n^m Pbar_{n-1}^m) / eps_{n+1}^m,
// into the blocked table (zeros in the blocks' degrees and latitudes past the
// last) and, where a plan's small-grid kernel reads it, the row-major one: rows
// of JH latitudes in internal-row order.  Writing the blocks from a row-major
// table kept both on every plan: T341 248 MB and 5.6 ms of set-up, 128 MB and
// 5.2 ms with this (4.3 and 4.2 ms with one row-major table and this, elsewhere).
__global__ void k_legendre_table(int N, int J, int JH, const double *__restrict__ mu, const double *__restrict__ eps,
                                 const long long *__restrict__ boff, double *__restrict__ blocked,
                                 double *__restrict__ rows)
{
  const int jh = blockIdx.x * blockDim.x + threadIdx.x;
  const int m = blockIdx.y;
  if (jh >= ((JH + 7) & ~7)) return;
  const int R = N + 2 - m;
  const bool real = jh < JH;
  const double x = mu[J - JH + (real ? jh : 0)];
  const double s = sqrt((1.0 - x) * (1.0 + x));
  double pmm = 1.0;
  for (int k = 1; k <= m; ++k) pmm *= sqrt((2.0 * k + 1.0) / (2.0 * k)) * s;
  double *const row = rows && real ? rows + (long long)(m * (N + 2) - m * (m - 1) / 2) * JH + jh : nullptr;
  const double *e = eps + (long long)m * (N + 3);
  auto put = [&](int r, double v) {
    const int cnt = (r & 1) ? R / 2 : (R + 1) / 2;
    blocked[band_at(boff[2 * m + (r & 1)], (cnt + 7) >> 3, r >> 1, jh)] = real ? v : 0.0;
    if (row && r < R) row[(long long)r * JH] = v;
  };
  double pm2 = 0.0, pm1 = pmm;
  put(0, pmm);
  for (int n = m + 1; n <= N + 1; ++n) {
    const double pn = (x * pm1 - e[n - 1] * pm2) / e[n];
    put(n - m, pn);
    pm2 = pm1;
    pm1 = pn;
  }
  for (int par = 0; par < 2; ++par) {
    const int cnt = par ? R / 2 : (R + 1) / 2;
    for (int k = cnt; k < ((cnt + 7) & ~7); ++k) put(2 * k + par, 0.0);
  }
}

namespace {

// The plan's tables share one device allocation: parts are reserved first,
// then the host-built ones are written into one image that goes up in a
// single copy (a plan had a dozen allocations and uploads, which cost more
// than its kernels).
struct TableArena {
  size_t bytes = 0, host_bytes = 0;
  template <typename T>
  size_t reserve(size_t count)
  {
    const size_t at = bytes;
    bytes += (sizeof(T) * (count ? count : 1) + 255) & ~(size_t)255;
    return at;
  }
};

}  // namespace

int build_tables(sht_plan *p)
{
  const int I = p->I, J = p->J, N = p->N, JH = p->JH, NC = p->NC;
  p->R = (long long)(N + 1) * (N + 4) / 2;
  p->M = p->zonal ? 1 : N + 1;
  p->L = p->zonal ? N + 1 : (N + 1) * (N + 1);
  cudaError_t e;
  // --- host-built tables
  // recurrence coefficients eps_n^m, n = 0..N+2 (closed form)
  std::vector<double> eps((size_t)(N + 1) * (N + 3));
  for (int m = 0; m <= N; ++m)
    for (int n = 0; n <= N + 2; ++n)
      eps[(size_t)m * (N + 3) + n] = (n < m || n == 0) ? 0.0 : std::sqrt(((double)n * n - (double)m * m) / (4.0 * n * n - 1.0));
  // internal row offsets
  p->h_rowoff.resize(N + 2);
  int ro = 0;
  for (int m = 0; m <= N; ++m) { p->h_rowoff[m] = ro; ro += N + 2 - m; }
  p->h_rowoff[N + 1] = ro;
  // twiddles (long double on the host, rounded once)
  std::vector<double2> tw(NC), twI(NC);
  const long double pi = 3.141592653589793238462643383279502884L;
  for (int k = 0; k < NC; ++k) {
    long double t = -2.0L * pi * k / NC;
    tw[k] = make_double2((double)cosl(t), (double)sinl(t));
    long double u = -2.0L * pi * k / I;
    twI[k] = make_double2((double)cosl(u), (double)sinl(u));
  }
  // Laplacian eigenvalues rn(l,1) = -n(n+1) (zonal layout: l = n)
  std::vector<double> rn(p->L);
  for (int n = 0; n <= N; ++n)
    for (int m = -n; m <= n; ++m)
      if (!p->zonal) rn[n * (n + 1) + m] = -(double)n * (n + 1);
      else if (m == 0) rn[n] = -(double)n * (n + 1);
  // tiles (n, m0) of the spectral layout conversions, n ascending
  std::vector<int2> tiles;
  for (int n = 0; n <= N + 1; ++n) {
    if (n == N + 1) p->n_pack_tiles = (int)tiles.size();
    const int mmax = p->zonal ? 0 : (n < N ? n : N);
    for (int m0 = 0; m0 <= mmax; m0 += 32) tiles.push_back(make_int2(n, m0));
  }
  p->n_spec_tiles = (int)tiles.size();
  // band pairs (m, N-m) with N+4 degrees each, plus the middle band of even N
  std::vector<int2> pairs;
  if (p->zonal) {
    pairs.push_back(make_int2(0, -1));  // the m = 0 band alone
  } else {
    for (int m = 0; m < N - m; ++m) pairs.push_back(make_int2(m, N - m));
    if (N % 2 == 0) pairs.push_back(make_int2(N / 2, -1));
  }
  p->n_pairs = (int)pairs.size();
  // items and block offsets of the band kernels
  std::vector<long long> boff;
  std::vector<BandItem> items;
  int rc = plan_band_items(p, boff, items);
  if (rc) return rc;

  // --- one allocation: the host image's parts, then the device-built tables
  TableArena ar;
  const size_t o_eps = ar.reserve<double>(eps.size());
  const size_t o_row = ar.reserve<int>(p->h_rowoff.size()), o_tw = ar.reserve<double2>(NC), o_twI = ar.reserve<double2>(NC);
  const size_t o_rn = ar.reserve<double>(rn.size()), o_tiles = ar.reserve<int2>(tiles.size());
  const size_t o_pairs = ar.reserve<int2>(pairs.size()), o_boff = ar.reserve<long long>(boff.size());
  const size_t o_items = ar.reserve<BandItem>(items.size()), o_rs = ar.reserve<double>((size_t)RS_COUNT * J);
  ar.host_bytes = ar.bytes;
  const size_t o_mu = ar.reserve<double>(J), o_wgt = ar.reserve<double>(J);
  const bool small = small_supported(p);  // reads row-major rows
  const size_t o_P = ar.reserve<double>(small ? (size_t)p->R * JH : 0);
  const size_t o_bP = ar.reserve<double>(64 * (size_t)boff.back());
  if ((e = cudaMalloc(&p->d_tables, ar.bytes)) != cudaSuccess) return cuda_fail(e, "cudaMalloc(plan tables)");
  char *const base = static_cast<char *>(p->d_tables);
  auto at = [&](size_t o, auto *&ptr) { ptr = reinterpret_cast<std::remove_reference_t<decltype(ptr)>>(base + o); };
  at(o_eps, p->d_eps); at(o_row, p->d_rowoff); at(o_tw, p->d_tw); at(o_twI, p->d_twI);
  at(o_rn, p->d_rn); at(o_tiles, p->d_spec_tiles); at(o_pairs, p->d_pairs); at(o_boff, p->d_band_off);
  at(o_items, p->d_band_items); at(o_rs, p->d_rowscale); at(o_mu, p->d_mu); at(o_wgt, p->d_wgt);
  at(o_bP, p->d_band_P);
  if (small) at(o_P, p->d_P);

  // --- Gauss nodes and weights on the device, read back for the row scales
  k_gauss_nodes<<<(J / 2 + 127) / 128, 128, 0, p->stream>>>(J, p->d_mu, p->d_wgt);
  count_launch();
  if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(e, "k_gauss_nodes");
  p->h_mu.resize(J);
  p->h_wgt.resize(J);
  if ((e = cudaMemcpyAsync(p->h_mu.data(), p->d_mu, sizeof(double) * J, cudaMemcpyDeviceToHost, p->stream)) != cudaSuccess ||
      (e = cudaMemcpyAsync(p->h_wgt.data(), p->d_wgt, sizeof(double) * J, cudaMemcpyDeviceToHost, p->stream)) != cudaSuccess ||
      (e = cudaStreamSynchronize(p->stream)) != cudaSuccess)
    return cuda_fail(e, "gauss nodes readback");
  // row scales
  std::vector<double> rs((size_t)RS_COUNT * J);
  for (int j = 0; j < J; ++j) {
    const double mu = p->h_mu[j], w = p->h_wgt[j];
    const double c2 = (1.0 - mu) * (1.0 + mu), c = std::sqrt(c2);
    rs[RS_FWD_PLAIN * J + j] = w / I;
    rs[RS_FWD_INV1MMU2 * J + j] = w / (I * c2);
    rs[RS_INV_PLAIN * J + j] = 1.0;
    rs[RS_INV_INVCOS * J + j] = 1.0 / c;
    rs[RS_INV_INVA1MMU2 * J + j] = 1.0 / (p->radius * c2);
    rs[RS_INV_INVACOS * J + j] = 1.0 / (p->radius * c);
    rs[RS_FWD_INVCOS * J + j] = w / (I * c);
  }
  std::vector<char> image(ar.host_bytes);
  auto put = [&](size_t o, const auto &v) { std::memcpy(image.data() + o, v.data(), sizeof(v[0]) * v.size()); };
  put(o_eps, eps); put(o_row, p->h_rowoff); put(o_tw, tw); put(o_twI, twI); put(o_rn, rn);
  put(o_tiles, tiles); put(o_pairs, pairs); put(o_boff, boff); put(o_items, items); put(o_rs, rs);
  if ((e = cudaMemcpyAsync(base, image.data(), ar.host_bytes, cudaMemcpyHostToDevice, p->stream)) != cudaSuccess)
    return cuda_fail(e, "plan table upload");

  // --- Legendre table on the device
  dim3 grid((JH + 127) / 128, p->M);
  k_legendre_table<<<grid, 128, 0, p->stream>>>(N, J, JH, p->d_mu, p->d_eps, p->d_band_off, p->d_band_P, p->d_P);
  count_launch();
  if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(e, "k_legendre_table");
  if ((e = cudaDeviceGetAttribute(&p->num_sms, cudaDevAttrMultiProcessorCount, p->device)) != cudaSuccess)
    return cuda_fail(e, "SM count");
  if ((e = cudaStreamSynchronize(p->stream)) != cudaSuccess) return cuda_fail(e, "plan tables");
  return SHT_OK;
}

}  // namespace sht
