// Host side shared by a single solver handle (ssfft.cu) and a batched group of slots
// (group.cuh): the grid plan (FFT factorisations, tiles, twiddle and tangent tables),
// the device buffers of one slot, and the launches of every kernel over a slot list with
// persistent, occupancy-sized grids.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/ssfft.h"
#include "common.cuh"
#include "constitutive.cuh"
#include "dif.cuh"
#include "fft.cuh"
#include "fields.cuh"
#include "krylov.cuh"
#include "launch.cuh"
#include "projector.cuh"
#include "slots.cuh"

#define ALLOC(ptr, bytes)                                                                 \
  do {                                                                                    \
    cudaError_t e_ = cudaMalloc((void **)&(ptr), (bytes));                                \
    if (e_ != cudaSuccess) {                                                              \
      cudaGetLastError();                                                                 \
      return ssfft_internal_fail(SSFFT_E_NOMEM, std::string("cudaMalloc ") + #ptr + ": " + \
                                                    cudaGetErrorString(e_));              \
    }                                                                                     \
  } while (0)

static int div_up(long long a, long long b) { return (int)((a + b - 1) / b); }

// ---------------------------------------------------------------------------------------
// grid plan
// ---------------------------------------------------------------------------------------
static const size_t SMEM_LIMIT = 200 * 1024;
#define PLANE_SMEM_LIMIT (200 * 1024)
#define CLUSTER_MAX 8  // largest portable cluster
#define MAX_ITEMS_PER_SLOT 65536

struct GridPlan {
  int dev;
  bool fp64;                  // solve precision
  int nx, ny, nz, hz;
  long long V, S;             // points; stored half-spectrum points
  AxisPlan px, py, pz;
  int lz, ky, kx;
  int kx_f;                   // kz columns per x-pass tile of the float transforms
  bool use_plane;             // plane-fused passes allowed (SSFFT_NO_PLANE=1 forbids)
  void *tw[2][3], *tn[2][3];  // [0]: float, [1]: double tables per axis
  Grid<float> gf;
  Grid<double> gd;
  DifPlane dplane[2][2];      // register-tiled passes: [0] float, [1] double; forward, inverse
  DifXPlan dx[2];
  DifXPlan dy[2];             // passes of planes too large for a block: y (tiles as the x pass's)
  DifZPlan dz[2][2];          // and z, forward and inverse
  bool few[2];                // given fields' projections in clusters although one block would do
  int cl_blocks[2], cl_threads[2];  // cluster passes: blocks a cluster (0: not used), their threads
  int x_threads[2];           // threads of a Stockham x-pass block
  size_t partial_doubles;     // reduction partials per slot
};

template <typename T> static std::vector<T> twiddles(int n) {
  std::vector<T> tw(2 * (size_t)n);
  for (int k = 0; k < n; ++k) {
    const long double a = -2.0L * 3.14159265358979323846264338327950288L * k / n;
    tw[2 * k] = (T)std::cos(a);
    tw[2 * k + 1] = (T)std::sin(a);
  }
  return tw;
}

// tan(pi f) for numpy's fftfreq ordering (first `count` entries).
template <typename T> static std::vector<T> tan_table(int n, int count) {
  std::vector<T> t(count);
  for (int k = 0; k < count; ++k) {
    const int kk = (k < (n + 1) / 2) ? k : k - n;  // fftfreq index
    const long double f = (long double)kk / n;
    if (2 * kk == -n || 2 * kk == n)
      t[k] = (T)0;  // Nyquist plane: operator is zeroed there
    else
      t[k] = (T)std::tan(3.14159265358979323846264338327950288L * f);
  }
  return t;
}

template <typename T> static Grid<T> &grid_of(GridPlan &p);
template <> Grid<float> &grid_of<float>(GridPlan &p) { return p.gf; }
template <> Grid<double> &grid_of<double>(GridPlan &p) { return p.gd; }
template <typename T> static const Grid<T> &grid_of(const GridPlan &p) {
  return grid_of<T>(const_cast<GridPlan &>(p));
}

template <typename T> static void fill_grid(GridPlan &p) {
  Grid<T> &g = grid_of<T>(p);
  memset(&g, 0, sizeof(g));
  g.nx = p.nx;
  g.ny = p.ny;
  g.nz = p.nz;
  g.hz = p.hz;
  g.V = p.V;
  g.S = p.S;
  // float transforms take radix 16 and 12 butterflies (two stages for every length up to
  // 256 the solver uses); double ones stop at radix 8, whose registers fit 64 a thread
  const int maxrad = sizeof(T) == 4 ? 16 : 8;
  make_axis_plan(p.nx, g.px, maxrad);
  make_axis_plan(p.ny, g.py, maxrad);
  make_axis_plan(p.nz, g.pz, maxrad);
  const int k = sizeof(T) == 8 ? 1 : 0;
  g.twx = (const cplx<T> *)p.tw[k][0];
  g.twy = (const cplx<T> *)p.tw[k][1];
  g.twz = (const cplx<T> *)p.tw[k][2];
  g.tanx = (const T *)p.tn[k][0];
  g.tany = (const T *)p.tn[k][1];
  g.tanz = (const T *)p.tn[k][2];
  g.scale = (T)(1.0 / (double)p.V);
  g.lz = p.lz;
  g.ky = p.ky;
  g.kx = sizeof(T) == 4 ? p.kx_f : p.kx;
  grid_divisors(g);
}

template <typename T> static bool plane_ok(const GridPlan &p) {
  return p.use_plane && smem_plane_bytes<T>(p.ny, p.nz) <= PLANE_SMEM_LIMIT;
}

// Blocks per cluster of the cluster plane passes (0: not used), for grids whose plane does
// not fit one block: the smallest C in 2, 4, 8 whose blocks fit two to an SM, else the
// smallest whose blocks fit at all (a single block per SM leaves its loads and its
// transforms without overlap).  SSFFT_CLUSTER=C asks for clusters of at least C blocks,
// also where one block would hold the plane.
static int env_int(const char *name) {
  const char *v = getenv(name);
  return v ? atoi(v) : 0;
}

template <typename T> static int cluster_size(const GridPlan &p) {
  if (!p.use_plane) return 0;
  const int want = env_int("SSFFT_CLUSTER");
  if (want <= 0 && plane_ok<T>(p)) return 0;
  const int hs = (p.nz % 2 == 0) ? p.nz / 2 : p.hz;
  auto fits = [&](int C, size_t lim) {
    return p.ny % C == 0 && (2 * hs) % C == 0 && C >= want &&
           smem_cplane_bytes<T>(p.ny, p.nz, hs, C) <= lim;
  };
  // the smallest cluster whose blocks fit two to an SM (512 threads each), else the
  // smallest whose blocks fit at all
  for (int C = 2; C <= CLUSTER_MAX; C *= 2)
    if (fits(C, 113 * 1024)) return C;
  for (int C = 2; C <= CLUSTER_MAX; C *= 2)
    if (fits(C, PLANE_SMEM_LIMIT)) return C;
  return 0;
}

template <typename T> static ClusterGeo cluster_geo(const GridPlan &p, int C) {
  ClusterGeo q;
  const int hs = (p.nz % 2 == 0) ? p.nz / 2 : p.hz;
  q.C = C;
  q.R = p.ny / C;
  q.Lq = 2 * hs / C;
  q.cap = cplane_buf_elems(p.ny, p.nz, hs, C);
  q.fd_R = make_fastdiv((uint32_t)q.R);
  q.fd_Lq = make_fastdiv((uint32_t)q.Lq);
  return q;
}

// Threads of a cluster block: for float transforms 256 when three blocks fit an SM's
// shared memory (128^3 on 4-block clusters: each radix-16 stage then has one butterfly per
// thread, where 512 threads left half of them idle; measured 7-8% faster per pass), else
// 512 when two fit, else 1024 (SSFFT_CLUSTER_THREADS=256, 512 or 1024 overrides).
template <typename T> static int cluster_threads(const GridPlan &p, int C) {
  const int hs = (p.nz % 2 == 0) ? p.nz / 2 : p.hz;
  const size_t bytes = smem_cplane_bytes<T>(p.ny, p.nz, hs, C);
  const int want = env_int("SSFFT_CLUSTER_THREADS");
  if (want == 1024 || want == 512 || want == 256) return want;
  if (sizeof(T) == 4 && bytes <= 75 * 1024) return 256;
  return bytes <= 113 * 1024 ? 512 : 1024;
}

// Threads of an x-pass block: 256, or 192 / 384 on float grids when SSFFT_XPASS_THREADS
// asks for them.
template <typename T> static int xpass_threads() {
  if (sizeof(T) != 4) return XPASS_THREADS;
  const int want = env_int("SSFFT_XPASS_THREADS");
  return (want == 192 || want == 384) ? want : XPASS_THREADS;
}

template <typename T, typename TF, bool KRY>
static int launch_xpass(const Grid<T> &g, int pt, size_t sx, long long items, int dev,
                        cudaStream_t stream, const SlotDev<TF> *tab, SlotList list) {
  if constexpr (sizeof(T) == 4) {
    if (pt == 384) {
      auto k = xpass_kernel<T, TF, KRY, 384>;
      return launch_kernel(false, k, persistent_grid(k, 384, sx, items, dev), 384, sx, stream, g, tab, list);
    }
    if (pt == 192) {
      auto k = xpass_kernel<T, TF, KRY, 192>;
      return launch_kernel(false, k, persistent_grid(k, 192, sx, items, dev), 192, sx, stream, g, tab, list);
    }
  }
  auto k = xpass_kernel<T, TF, KRY>;
  return launch_kernel(false, k, persistent_grid(k, XPASS_THREADS, sx, items, dev), XPASS_THREADS, sx,
                       stream, g, tab, list);
}

// Threads of a plane block: 1024 when a single block fits an SM (228 KB of shared memory),
// else 512.
template <typename T> static int plane_threads(const GridPlan &p) {
  return smem_plane_bytes<T>(p.ny, p.nz) > 113 * 1024 ? 1024 : 512;
}

// ---------------------------------------------------------------------------------------
// plans of the register-tiled passes (dif.cuh)
// ---------------------------------------------------------------------------------------
// Factor n into two or three stages with the first radix in `first`, the middle one at most
// 8 and the last one in `last` (bit r: radix r).  Fewest stages, then the smallest widest
// radix, then the larger first one.
#define DIF_RADICES 0x117feu     // 1 .. 10, 12, 16
#define DIF_RADICES_PAIR 0x1feu  // 1 .. 8: stages that hold two lines a thread
static bool dif_axis(int n, unsigned first, unsigned last, DifAxis &A) {
  memset(&A, 0, sizeof(A));
  int best = 1 << 30;
  auto ok = [](unsigned set, int r) { return r <= 16 && ((set >> r) & 1u); };
  auto take = [&](int ns, int r0, int r1, int r2) {
    const int widest = std::max(r0, std::max(r1, r2));
    const int cost = ns * 1000 + 4 * widest - (r0 >= r1 ? 1 : 0);
    if (cost >= best) return;
    best = cost;
    A.ns = ns;
    A.r0 = r0;
    A.r1 = r1;
    A.r2 = r2;
  };
  for (int r0 = 1; r0 <= 16; ++r0) {
    if (!ok(first, r0) || n % r0) continue;
    const int m = n / r0;
    if (ok(last, m)) take(2, r0, m, 1);
    for (int r1 = 2; r1 <= 8; ++r1)
      if (m % r1 == 0 && ok(last, m / r1)) take(3, r0, r1, m / r1);
  }
  if (A.ns == 0) return false;
  A.n = n;
  A.m = n / A.r0;
  const int rl = A.ns == 2 ? A.r1 : A.r2;
  A.fd_m = make_fastdiv((uint32_t)A.m);
  A.fd_r0 = make_fastdiv((uint32_t)A.r0);
  A.fd_nb = make_fastdiv((uint32_t)(n / rl));
  A.fd_nb1 = make_fastdiv((uint32_t)(A.r0 * A.r2));
  return true;
}

#define DIF_SMEM_LIMIT (224 * 1024)
// Smaller planes stay on the Stockham passes, whose kernels start faster: a 16^3 projection
// takes 36 us there and 40 us in the register-tiled passes; 30 x 28 x 27 takes 52 and 41.
#define DIF_MIN_PLANE 512

static int dif_last_radix_host(const DifAxis &A) { return A.ns == 2 ? A.r1 : A.r2; }

// z axis and row layout of a forward (inv = false) or inverse pass.
static bool dif_zrow(int nz, bool inv, DifPlane &P) {
  memset(&P, 0, sizeof(P));
  if (!dif_axis(nz, inv ? DIF_RADICES_PAIR : DIF_RADICES, inv ? DIF_RADICES : DIF_RADICES_PAIR, P.z))
    return false;
  P.z.a = P.z.r0 | 1;  // odd
  P.z.b = 1;
  P.ls = P.z.m * P.z.a;
  const int nb = nz / dif_last_radix_host(P.z);
  P.z.fd_un = make_fastdiv((uint32_t)((inv ? P.z.m : nb) / 2 + 1));
  return true;
}

// Plan of the forward (inv = false) or inverse plane pass in one block's buffer (ok = 0 where
// an axis has no plan or the plane is too large).
template <typename T> static DifPlane dif_plane(int ny, int nz, int hs, bool inv) {
  DifPlane P;
  if (!dif_zrow(nz, inv, P) || !dif_axis(ny, DIF_RADICES, DIF_RADICES, P.y)) return P;
  // column (1, 0): the padding slot of n' = 0, or one more slot a row where there is none
  P.xslot = (P.z.r0 & 1) ? P.ls++ : P.z.r0;
  P.elems = ny * P.ls;
  P.y.a = P.ls;
  P.y.b = P.y.m * P.ls;
  P.y.fd_un = make_fastdiv((uint32_t)P.ls);  // slots to rows
  const size_t bytes = DifTables<T, false>::bytes(P, ny, nz, hs);
  P.ok = bytes <= DIF_SMEM_LIMIT && P.ls < 65536 ? 1 : 0;
  // about one radix-8 butterfly a thread and stage
  // (up to 1024 in float where one block fills an SM: 32 warps instead of 16)
  const int most = sizeof(T) == 4 && bytes > 112 * 1024 ? 1024 : 512;
  P.threads = std::max(64, std::min(most, (ny * nz / 8 + 63) / 64 * 64));
  return P;
}

// x pass: tiles take 64-byte runs of a spectrum row, halved (down to a 32-byte sector) while
// the grid then has fewer than four tiles an SM and while a tile exceeds 40 KB (five blocks an
// SM).
template <typename T> static DifXPlan dif_xplan(int nx, int ny, int hs) {
  DifXPlan P;
  memset(&P, 0, sizeof(P));
  DifAxis &X = P.x;
  if (!dif_axis(nx, DIF_RADICES, DIF_RADICES, X)) return P;
  const int sector = 32 / (int)sizeof(cplx<T>);
  const int w = 128 / (int)sizeof(cplx<T>);
  P.kx = 64 / (int)sizeof(cplx<T>);
  auto layout = [&]() {
    const int run = X.r0 * P.kx;
    X.a = run + ((P.kx - run) % w + w) % w;
    X.b = P.kx;
    P.cs = X.m * X.a;
    P.elems = 6 * P.cs;
    P.nkx = (hs + P.kx - 1) / P.kx;
    return ((size_t)P.elems + nx) * sizeof(cplx<T>);
  };
  while (P.kx > sector && ((long long)((hs + P.kx - 1) / P.kx) * ny < 4 * 148 || P.kx >= 2 * hs)) P.kx /= 2;
  while (layout() > 40 * 1024 && P.kx > sector) P.kx /= 2;
  while (layout() > SMEM_LIMIT && P.kx > 1) P.kx /= 2;
  if (layout() > SMEM_LIMIT) return P;
  while ((1 << P.lkx) < P.kx) ++P.lkx;
  P.fd_mid = make_fastdiv((uint32_t)(X.r0 * P.kx));
  P.fd_r2 = make_fastdiv((uint32_t)X.r2);
  P.fd_items = make_fastdiv((uint32_t)(P.nkx * ny));
  P.fd_nkx = make_fastdiv((uint32_t)P.nkx);
  P.ok = 1;
  return P;
}

// y pass of planes too large for a block, one component a tile: 128-byte runs of a spectrum row,
// halved (down to a 32-byte sector) while a tile exceeds 40 KB (five blocks an SM), while the
// grid then has fewer than four tiles an SM, and while half of it is past the row's end.
template <typename T> static DifXPlan dif_yplan(int nx, int ny, int hs) {
  DifXPlan P;
  memset(&P, 0, sizeof(P));
  DifAxis &Y = P.x;
  if (!dif_axis(ny, DIF_RADICES, DIF_RADICES, Y)) return P;
  const int sector = 32 / (int)sizeof(cplx<T>);
  const int w = 128 / (int)sizeof(cplx<T>);
  P.kx = w;
  auto layout = [&]() {
    const int run = Y.r0 * P.kx;
    Y.a = run + ((P.kx - run) % w + w) % w;
    Y.b = P.kx;
    P.cs = 0;
    P.elems = Y.m * Y.a;
    P.nkx = (hs + P.kx - 1) / P.kx;
    return ((size_t)P.elems + ny) * sizeof(cplx<T>);
  };
  while (P.kx > sector && (layout() > 40 * 1024 || 6LL * nx * P.nkx < 4 * 148 || P.kx >= 2 * hs)) P.kx /= 2;
  if (layout() > SMEM_LIMIT) return P;
  while ((1 << P.lkx) < P.kx) ++P.lkx;
  P.fd_mid = make_fastdiv((uint32_t)(Y.r0 * P.kx));
  P.fd_r2 = make_fastdiv((uint32_t)Y.r2);
  P.fd_items = make_fastdiv((uint32_t)(6 * nx * P.nkx));
  P.fd_nkx = make_fastdiv((uint32_t)P.nkx);
  P.ok = 1;
  return P;
}

// z pass of such planes: tiles of as many lines as give each thread one pair of butterflies in
// the paired stage (the slowest: two lines' registers a thread), of at most 100 KB in double and
// 50 KB in float (as many blocks an SM as the registers allow).
template <typename T> static DifZPlan dif_zplan(long long lines, int nz, bool inv) {
  DifZPlan P;
  memset(&P, 0, sizeof(P));
  if (!dif_zrow(nz, inv, P.p)) return P;
  const int un = (inv ? P.p.z.m : nz / dif_last_radix_host(P.p.z)) / 2 + 1;
  const int most = (sizeof(T) == 8 ? 100 : 50) * 1024 / (int)(P.p.ls * sizeof(cplx<T>));
  P.lz = (int)std::min<long long>(lines, std::max(1, std::min(DIFZ_THREADS / un, most)));
  P.ntiles = (int)((lines + P.lz - 1) / P.lz);
  P.p.elems = P.lz * P.p.ls;
  P.fd_items = make_fastdiv((uint32_t)(3 * P.ntiles));
  P.ok = ((size_t)P.p.elems + nz) * sizeof(cplx<T>) <= SMEM_LIMIT ? 1 : 0;
  return P;
}

// Sum of the factors 5 and 7 of a length, which the Stockham passes transform by direct sums.
static int direct_sum_weight(int n) {
  int w = 0;
  for (int f : {5, 7})
    for (; n % f == 0; n /= f) w += f;
  return w;
}

// Small long planes keep the Stockham passes where the register-tiled ones have a plan too: a
// register-tiled block has a thread for eight points, and its chain of stages along a long axis
// is longer.  Projections in us, register-tiled / Stockham: 8 x 1 x 512 FP64 37.9 / 30.5,
// 8 x 512 x 1 39.0 / 33.5, 64 x 8 x 64 36.7 / 32.8, 8 x 8 x 256 mixed 35.0 / 32.6; Krylov
// iterations 5 to 20% faster.  Near-square planes of as many points lose or draw (30 x 20 1.2
// times slower), as do planes of twice the points (8 x 8 x 512 FP64 42.3 / 51.2), axes with direct
// sums, and grids of more than about 1024 points an SM in double and 2048 in float (128 x 8 x 128
// FP64 42.7 / 48.9, 160 x 16 x 128 mixed 50.6 / 53.9).  The rule follows from the grid alone, so
// a solve's arithmetic does not depend on its batch.
template <typename T> static bool long_plane(const GridPlan &p) {
  const bool pow2 = (p.ny & (p.ny - 1)) == 0 && (p.nz & (p.nz - 1)) == 0;
  const bool lng = p.nz >= (pow2 ? 4 : 8) * p.ny || p.ny >= 128 * p.nz;
  const int pts = p.ny * p.nz, most = sizeof(T) == 4 ? 2048 : 1024;
  return lng && direct_sum_weight(p.ny) + direct_sum_weight(p.nz) == 0 && pts <= most &&
         3LL * p.nx * pts <= 148LL * most;
}

// Projections of a given field on grids of few planes, each of 96 KB and more in float or of the
// size that clusters of four split in double: one block an SM leaves most of the chip idle where
// a cluster takes four SMs a plane.  In us, one block / cluster: 8 x 144 x 144 mixed 65.5 / 50.4,
// 8 x 128 x 128 mixed 53 / 47, 8 x 384 x 32 FP64 73.4 / 55.0, 8 x 640 x 20 FP64 80 / 74.  With
// direct sums the clusters lose (8 x 100 x 100 FP64 62 / 71, 6 x 160 x 160 mixed 72 / 76), and
// past 33 of them they share SMs (12 x 640 x 20 FP64 82 / 113, 24 x 144 x 144 mixed 71 / 84).
// Krylov iterations stay in one block: a group runs them for many slots at once, and a solve's
// arithmetic must not depend on its batch.
template <typename T> static bool few_planes(const GridPlan &p) {
  if (3 * p.nx > 33) return false;
  const int w = direct_sum_weight(p.ny) + direct_sum_weight(p.nz), C = cluster_size<T>(p);
  if (sizeof(T) == 8) return w <= 10 && C >= 4;
  return w == 0 && p.ny * p.nz >= 12288 &&
         (C ? smem_cplane_bytes<T>(p.ny, p.nz, p.gd.hs, C) <= 113 * 1024 : plane_ok<T>(p));
}

// The register-tiled x pass of lines of nx points.
template <typename T>
static void (*difx_of(int nx))(Grid<T>, DifXPlan, const SlotDev<T> *, SlotList, int) {
  if constexpr (sizeof(T) == 4)
    return difx_kernel<T, 5>;
  else
    return nx <= DIFX_THREE_MOST ? difx_kernel<T, 3> : difx_kernel<T, 2>;
}

// x pass of a launch: the register-tiled one where nx has a plan for it (unless a tile shape
// of the Stockham pass is asked for), else the Stockham one.
template <typename T, typename TF, bool KRY>
static int launch_x(const GridPlan &p, const Grid<T> &g, long long cap, cudaStream_t stream,
                     const SlotDev<TF> *tab, SlotList list) {
  const DifXPlan &P = p.dx[sizeof(T) == 8 ? 1 : 0];
  if (!P.ok)
    return launch_xpass<T, TF, KRY>(g, p.x_threads[sizeof(T) == 8 ? 1 : 0], smem_x_bytes<T>(g.kx, p.nx),
                                    cap * items_x(g), p.dev, stream, tab, list);
  auto k = difx_of<T>(p.nx);
  const size_t sm = ((size_t)P.elems + p.nx) * sizeof(cplx<T>);
  const int grid = persistent_grid(k, DIFX_THREADS, sm, cap * P.nkx * p.ny, p.dev);
  return launch_kernel(true, k, grid, DIFX_THREADS, sm, stream, g, P,
                       reinterpret_cast<const SlotDev<T> *>(tab), list, KRY ? 1 : 0);
}

// y pass of planes too large for a block: the register-tiled one where ny has a plan for it,
// else the Stockham one.
template <typename T, typename TF, bool INV, bool KRY>
static int launch_y(const GridPlan &p, const Grid<T> &g, long long cap, cudaStream_t stream,
                     const SlotDev<TF> *tab, SlotList list) {
  const DifXPlan &P = p.dy[sizeof(T) == 8 ? 1 : 0];
  if (!P.ok) {
    const size_t sy = smem_y_bytes<T>(p.ky, p.ny);
    auto ky = ypass_kernel<T, TF, INV, KRY>;
    return launch_kernel(false, ky, persistent_grid(ky, SSFFT_THREADS, sy, cap * items_y(g), p.dev),
                         SSFFT_THREADS, sy, stream, g, tab, list);
  }
  auto k = dify_kernel<T, INV>;
  const size_t sm = ((size_t)P.elems + p.ny) * sizeof(cplx<T>);
  const int grid = persistent_grid(k, DIFY_THREADS, sm, cap * 6 * p.nx * P.nkx, p.dev);
  return launch_kernel(true, k, grid, DIFY_THREADS, sm, stream, g, P,
                       reinterpret_cast<const SlotDev<T> *>(tab), list, KRY ? 1 : 0);
}

static int validate_config(const ssfft_config *cfg) {
  if (!cfg) return ssfft_internal_fail(SSFFT_E_INVALID, "null config");
  for (int d = 0; d < 3; ++d)
    if (cfg->n[d] < 1 || cfg->n[d] > 1024)
      return ssfft_internal_fail(SSFFT_E_UNSUPPORTED, "grid size out of range");
  if (cfg->precision != SSFFT_FP64 && cfg->precision != SSFFT_MIXED)
    return ssfft_internal_fail(SSFFT_E_INVALID, "precision must be SSFFT_FP64 or SSFFT_MIXED");
  for (int c = 0; c < 6; ++c)
    if (cfg->stress_mask[c] != 0.0 && cfg->stress_mask[c] != 1.0)
      return ssfft_internal_fail(SSFFT_E_INVALID, "stress mask can only have zeros and ones");
  if (!(cfg->krylov_floor >= 0.0 && cfg->krylov_floor < 1.0))
    return ssfft_internal_fail(SSFFT_E_INVALID, "krylov_floor must be in [0, 1)");
  if (!(cfg->krylov_forcing >= 0.0 && cfg->krylov_forcing < 1.0))
    return ssfft_internal_fail(SSFFT_E_INVALID, "krylov_forcing must be in [0, 1)");
  AxisPlan p;
  for (int d = 0; d < 3; ++d)
    if (!make_axis_plan(cfg->n[d], p))
      return ssfft_internal_fail(SSFFT_E_UNSUPPORTED, "grid size has a prime factor above 32");
  return 0;
}

// Tiles are sized for double-precision transforms, which both modes run (the mixed mode
// computes its equilibrium residual in double).
static int plan_tiles(GridPlan &p) {
  p.lz = std::max(1, std::min(32, 2048 / (3 * p.nz)));
  p.lz = (int)std::min<long long>(p.lz, (long long)p.nx * p.ny);
  p.ky = std::min(p.hz, 16);
  while (p.ky > 1 && smem_y_bytes<double>(p.ky, p.ny) > 96 * 1024) p.ky /= 2;
  // kz columns per x-pass tile: 8 (64-byte runs of the spectrum per x), 4 on grids of up
  // to 64 points along x, where 8 would leave about two blocks per SM
  p.kx = std::min(p.hz, p.nx <= 64 ? 4 : 8);
  while (p.kx > 1 && smem_x_bytes<double>(p.kx, p.nx) > 100 * 1024) p.kx /= 2;
  // float x tiles: the double tile unless SSFFT_XPASS_KX asks for another power of two
  // that fits
  p.kx_f = p.kx;
  const int want_kx = env_int("SSFFT_XPASS_KX");
  if (want_kx >= 1 && want_kx <= 32 && (want_kx & (want_kx - 1)) == 0 &&
      smem_x_bytes<float>(std::min(want_kx, p.hz), p.nx) <= SMEM_LIMIT)
    p.kx_f = std::min(want_kx, p.hz);
  if (smem_z_bytes<double>(p.lz, p.nz) > SMEM_LIMIT || smem_y_bytes<double>(p.ky, p.ny) > SMEM_LIMIT ||
      smem_x_bytes<double>(p.kx, p.nx) > SMEM_LIMIT)
    return ssfft_internal_fail(SSFFT_E_UNSUPPORTED, "grid too large for the shared-memory FFT passes");
  return 0;
}

static void plan_free(GridPlan &p) {
  for (int k = 0; k < 2; ++k)
    for (int a = 0; a < 3; ++a) {
      if (p.tw[k][a]) cudaFree(p.tw[k][a]);
      if (p.tn[k][a]) cudaFree(p.tn[k][a]);
      p.tw[k][a] = p.tn[k][a] = nullptr;
    }
}

// The z and y passes of a projection: fused in one block (register-tiled or Stockham) or in a
// cluster of C blocks, or passes of their own (z register-tiled where dif_z).
enum { ROUTE_DIF_PLANE, ROUTE_CLUSTER, ROUTE_PLANE, ROUTE_LINES };
struct Route {
  int kind, C;
  bool dif_z;
};

template <typename T, typename TF, int PRO, int EPI> static Route route_of(const GridPlan &p) {
  const int k = sizeof(T) == 8 ? 1 : 0;
  const bool few = PRO == PRO_INPUT && p.few[k];
  if (p.dplane[k][0].ok && p.dplane[k][1].ok && !few) return {ROUTE_DIF_PLANE, 0, false};
  // register-tiled z passes where nz has a plan and a pass only moves planes (the residual
  // and the re-projection, one each a Newton iteration, keep the Stockham ones)
  constexpr bool PLANES = sizeof(T) == sizeof(TF) && (PRO == PRO_INPUT || PRO == PRO_TAU) &&
                          (EPI == EPI_STORE || EPI == EPI_PTAU);
  const bool dif_z = PLANES && p.dz[k][0].ok && p.dz[k][1].ok;
  // Five register-tiled passes beat three on clusters wherever both run (projections, us,
  // clusters / five passes: 128^3 FP64 451 / 305, 64 x 128 x 144 FP64 280 / 190, 160^3 FP64
  // 1203 / 615, 192^3 FP64 1725 / 1007 and float 830 / 580, 256^3 float 2201 / 1262).
  if (!(dif_z && p.dy[k].ok) || few) {
    if (p.cl_blocks[k]) return {ROUTE_CLUSTER, p.cl_blocks[k], false};
    if (plane_ok<T>(p)) return {ROUTE_PLANE, 0, false};
  }
  return {ROUTE_LINES, 0, dif_z};
}

static int set_kernel_attrs(const GridPlan &p);

static int plan_create(GridPlan &p, const ssfft_config *cfg, cudaStream_t stream) {
  memset(&p, 0, sizeof(p));
  p.dev = cfg->device;
  p.fp64 = cfg->precision == SSFFT_FP64;
  p.nx = cfg->n[0];
  p.ny = cfg->n[1];
  p.nz = cfg->n[2];
  p.hz = p.nz / 2 + 1;
  p.V = (long long)p.nx * p.ny * p.nz;
  // stored half-spectrum columns: the Nyquist column of an even grid is not stored
  p.S = (long long)p.nx * p.ny * ((p.nz % 2 == 0) ? p.nz / 2 : p.hz);
  make_axis_plan(p.nx, p.px);
  make_axis_plan(p.ny, p.py);
  make_axis_plan(p.nz, p.pz);
  p.use_plane = env_int("SSFFT_NO_PLANE") != 1;
  CKR(plan_tiles(p));
  // FFT tables: float ones for the mixed-mode Krylov transforms, double ones for every
  // double-precision transform
  const int dims[3] = {p.nx, p.ny, p.nz};
  const int tcount[3] = {p.nx, p.ny, p.hz};
  for (int k = (p.fp64 ? 1 : 0); k < 2; ++k)
    for (int a = 0; a < 3; ++a) {
      const size_t es = k ? 8 : 4;
      ALLOC(p.tw[k][a], (size_t)dims[a] * 2 * es);
      ALLOC(p.tn[k][a], (size_t)tcount[a] * es);
      if (k) {
        auto tw = twiddles<double>(dims[a]);
        auto tn = tan_table<double>(dims[a], tcount[a]);
        CK(cudaMemcpyAsync(p.tw[k][a], tw.data(), tw.size() * es, cudaMemcpyHostToDevice, stream));
        CK(cudaMemcpyAsync(p.tn[k][a], tn.data(), tn.size() * es, cudaMemcpyHostToDevice, stream));
        CK(cudaStreamSynchronize(stream));  // the host vectors go out of scope
      } else {
        auto tw = twiddles<float>(dims[a]);
        auto tn = tan_table<float>(dims[a], tcount[a]);
        CK(cudaMemcpyAsync(p.tw[k][a], tw.data(), tw.size() * es, cudaMemcpyHostToDevice, stream));
        CK(cudaMemcpyAsync(p.tn[k][a], tn.data(), tn.size() * es, cudaMemcpyHostToDevice, stream));
        CK(cudaStreamSynchronize(stream));
      }
    }
  fill_grid<double>(p);
  if (!p.fp64) fill_grid<float>(p);
  if (p.use_plane && env_int("SSFFT_CLUSTER") <= 0 && p.ny * p.nz >= DIF_MIN_PLANE) {
    for (int d = 0; d < 2; ++d) {
      p.dplane[0][d] = dif_plane<float>(p.ny, p.nz, p.gd.hs, d == 1);
      p.dplane[1][d] = dif_plane<double>(p.ny, p.nz, p.gd.hs, d == 1);
    }
  }
  if (p.ny * p.nz >= DIF_MIN_PLANE && env_int("SSFFT_XPASS_KX") <= 0 && env_int("SSFFT_XPASS_THREADS") <= 0) {
    // two kinds of grid are short of work in the tiles and keep the Stockham pass: a single
    // column on long lines without direct sums in float, whose tiles are four wide (768 x 768 x 1:
    // the projection takes 289 us, 198 there; 800 x 800 x 1 227 and 287; at 48 points along x
    // up to 10% more there), and in double "lines" of one point, which fill 24 of 192 threads
    // (1 x 512 x 512: 170 us, 119)
    if (p.gd.hs > 1 || p.nx < 256 || direct_sum_weight(p.nx)) p.dx[0] = dif_xplan<float>(p.nx, p.ny, p.gd.hs);
    if (p.nx > 1) p.dx[1] = dif_xplan<double>(p.nx, p.ny, p.gd.hs);
    // SSFFT_NO_PLANE and SSFFT_CLUSTER choose among the Stockham z and y passes
    if (p.use_plane && env_int("SSFFT_CLUSTER") <= 0) {
      p.dy[0] = dif_yplan<float>(p.nx, p.ny, p.gd.hs);
      p.dy[1] = dif_yplan<double>(p.nx, p.ny, p.gd.hs);
      for (int d = 0; d < 2; ++d) {
        p.dz[0][d] = dif_zplan<float>((long long)p.nx * p.ny, p.nz, d == 1);
        p.dz[1][d] = dif_zplan<double>((long long)p.nx * p.ny, p.nz, d == 1);
      }
    }
  }
  for (int k = 0; k < 2; ++k) {
    if (!p.dplane[k][0].ok || !p.dplane[k][1].ok) continue;
    p.few[k] = k ? few_planes<double>(p) : few_planes<float>(p);
    if (k ? long_plane<double>(p) : long_plane<float>(p))
      p.dplane[k][0].ok = p.dy[k].ok = p.dz[k][0].ok = 0;
  }
  p.cl_blocks[0] = cluster_size<float>(p);
  p.cl_blocks[1] = cluster_size<double>(p);
  if (p.cl_blocks[0]) p.cl_threads[0] = cluster_threads<float>(p, p.cl_blocks[0]);
  if (p.cl_blocks[1]) p.cl_threads[1] = cluster_threads<double>(p, p.cl_blocks[1]);
  p.x_threads[0] = xpass_threads<float>();
  p.x_threads[1] = xpass_threads<double>();
  // items of one slot per reduction, times the values each stores
  const Grid<double> &g = p.gd;
  size_t need = 0;
  need = std::max(need, (size_t)3 * items_z(g));
  need = std::max(need, (size_t)3 * CLUSTER_MAX * items_plane(g));
  need = std::max(need, (size_t)NORM_VALS * vec_items(p.V));
  need = std::max(need, (size_t)21 * vec_items(p.V));
  need = std::max(need, (size_t)vec_items(6 * p.V));
  if (items_z(g) > MAX_ITEMS_PER_SLOT || vec_items(6 * p.V) > MAX_ITEMS_PER_SLOT ||
      items_y(g) > (1 << 30) / 2)
    return ssfft_internal_fail(SSFFT_E_UNSUPPORTED, "grid too large for the reduction partials");
  p.partial_doubles = need;
  return set_kernel_attrs(p);
}

// ---------------------------------------------------------------------------------------
// kernel attributes
// ---------------------------------------------------------------------------------------
template <typename F> static int smem_attr(F f, int m) {
  CK(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, m));
  return 0;
}

// Opt the kernels of one projection into the shared memory they may ask for.  Nothing else is
// named here: a kernel's first touch loads its code, and every kernel named is compiled.
template <typename T, typename TF, int PRO, int EPI> static int projector_attrs(const GridPlan &p) {
  const int m = (int)SMEM_LIMIT;
  constexpr bool KRY = PRO_IS_KRYLOV(PRO) || PRO == PRO_TAU;
  const int k = sizeof(T) == 8 ? 1 : 0;
  const Route r = route_of<T, TF, PRO, EPI>(p);
  if (p.dx[k].ok) {
    CKR(smem_attr(difx_of<T>(p.nx), m));
  } else {
    const int pt = p.x_threads[k];
    if constexpr (sizeof(T) == 4) {
      if (pt == 192) CKR((smem_attr(xpass_kernel<T, TF, KRY, 192>, m)));
      if (pt == 384) CKR((smem_attr(xpass_kernel<T, TF, KRY, 384>, m)));
    }
    if (pt == XPASS_THREADS) CKR((smem_attr(xpass_kernel<T, TF, KRY>, m)));
  }
  if (r.kind == ROUTE_DIF_PLANE) {
    if constexpr (PRO == PRO_RESIDUAL)
      CKR((smem_attr(dif_zyfwd_kernel<double, double, DIF_RESIDUAL>, DIF_SMEM_LIMIT)));
    else
      CKR((smem_attr(dif_zyfwd_kernel<T, TF, DIF_PLANES>, DIF_SMEM_LIMIT)));
    return smem_attr(dif_yzinv_kernel<T, TF, dif_kind(EPI)>, DIF_SMEM_LIMIT);
  }
  if (r.kind == ROUTE_CLUSTER) {
    const int pt = p.cl_threads[k];
    if (pt == 1024) {
      CKR((smem_attr(zyfwd_cl_kernel<T, TF, PRO, 1024>, m)));
      return smem_attr(yzinv_cl_kernel<T, TF, EPI, 1024>, m);
    }
    if (pt == 256) {
      CKR((smem_attr(zyfwd_cl_kernel<T, TF, PRO, 256>, m)));
      return smem_attr(yzinv_cl_kernel<T, TF, EPI, 256>, m);
    }
    CKR((smem_attr(zyfwd_cl_kernel<T, TF, PRO, 512>, m)));
    return smem_attr(yzinv_cl_kernel<T, TF, EPI, 512>, m);
  }
  if (r.kind == ROUTE_PLANE) {
    if (plane_threads<T>(p) == 1024) {
      CKR((smem_attr(zyfwd_kernel<T, TF, PRO, 1024>, m)));
      return smem_attr(yzinv_kernel<T, TF, EPI, 1024>, m);
    }
    CKR((smem_attr(zyfwd_kernel<T, TF, PRO, 512>, m)));
    return smem_attr(yzinv_kernel<T, TF, EPI, 512>, m);
  }
  if (p.dy[k].ok) {
    CKR((smem_attr(dify_kernel<T, false>, m)));
    CKR((smem_attr(dify_kernel<T, true>, m)));
  } else {
    CKR((smem_attr(ypass_kernel<T, TF, false, KRY>, m)));
    CKR((smem_attr(ypass_kernel<T, TF, true, KRY>, m)));
  }
  if constexpr (sizeof(T) == sizeof(TF)) {
    if (r.dif_z) {
      CKR(smem_attr(dif_zfwd_kernel<T>, m));
      return smem_attr(dif_zinv_kernel<T>, m);
    }
  }
  CKR(smem_attr(zfwd_kernel<T, TF, PRO>, m));
  return smem_attr(zinv_kernel<T, TF, EPI>, m);
}

// The projections of a plan: of a given field, of a Krylov iteration, of the residual, and in
// mixed precision of the Newton correction.
template <typename T> static int solve_attrs(const GridPlan &p) {
  CKR(smem_attr(constitutive_kernel<T>, (int)constitutive_smem_bytes()));
  CKR((projector_attrs<T, T, PRO_INPUT, EPI_STORE>(p)));
  CKR((projector_attrs<T, T, PRO_TAU, EPI_PTAU>(p)));
  CKR((projector_attrs<double, T, PRO_RESIDUAL, EPI_RESIDUAL>(p)));
  if constexpr (sizeof(T) == 4) CKR((projector_attrs<double, T, PRO_REPROJECT, EPI_REPROJECT>(p)));
  return 0;
}
static int set_kernel_attrs(const GridPlan &p) {
  return p.fp64 ? solve_attrs<double>(p) : solve_attrs<float>(p);
}

// ---------------------------------------------------------------------------------------
// one slot's device buffers
// ---------------------------------------------------------------------------------------
// Allocations are owned here (freed by slot_free); the descriptor mirror holds the same
// pointers in their current roles, which swaps change.
struct SlotBufs {
  bool fp64;
  size_t rs;                   // sizeof(real)
  long long V;
  void *field[14];             // 6-plane fields: eps, eps_old, dfl, sig x3 (double), b, kr[7]
  void *spec;
  double *partials;
  unsigned int *tickets;
  double *results;
  MinresState *st;
  bool st_shared;              // st is the caller's
  int *citers;
  // microstructure (capacities grow on rebinding)
  PhaseParams hparams[SSFFT_MAX_PHASES];
  bool phase_set[SSFFT_MAX_PHASES];
  PhaseParams *dparams;
  int32_t *orient, *phase, *gid;
  double *rm_tab;
  size_t cap_rm, cap_ktab;
  void *ktab;
  void *kvox_buf[2];
  double *slip_buf[5];         // g_in, g_out, g_old, gam (two)
  int cap_nslip;
  double *ep_buf[2], *Gam_buf[2];
  bool micro_set, have_phase_buf, voxel_mode, any_evp, any_j2;
  int nslip_max, n_orient, n_gid;
  SlotDev<float> mf;           // descriptor mirror (the one of the solve precision is used)
  SlotDev<double> md;
};

template <typename T> static SlotDev<T> &mirror(SlotBufs &b);
template <> SlotDev<float> &mirror<float>(SlotBufs &b) { return b.mf; }
template <> SlotDev<double> &mirror<double>(SlotBufs &b) { return b.md; }

static size_t field_bytes(const SlotBufs &b, int planes) {
  return (size_t)planes * (size_t)b.V * b.rs;
}

// Bytes of field[i]: the strain and stress fields (0..5) are double in both precisions.
static size_t field_bytes_of(const SlotBufs &b, int i) {
  return i < 6 ? (size_t)6 * (size_t)b.V * sizeof(double) : field_bytes(b, 6);
}

// st: the slot's MINRES state where the caller owns it (a group keeps its slots' states in
// one array), else one is allocated.
static int slot_alloc(SlotBufs &b, const GridPlan &p, cudaStream_t stream, MinresState *st = nullptr) {
  memset((void *)&b, 0, sizeof(b));
  b.fp64 = p.fp64;
  b.rs = p.fp64 ? 8 : 4;
  b.V = p.V;
  for (int i = 0; i < 14; ++i) {
    ALLOC(b.field[i], field_bytes_of(b, i));
    CK(cudaMemsetAsync(b.field[i], 0, field_bytes_of(b, i), stream));
  }
  ALLOC(b.spec, (size_t)6 * p.S * 16);  // sized for double-precision transforms
  ALLOC(b.partials, p.partial_doubles * sizeof(double));
  ALLOC(b.tickets, 16 * sizeof(unsigned int));
  CK(cudaMemsetAsync(b.tickets, 0, 16 * sizeof(unsigned int), stream));
  ALLOC(b.results, 64 * sizeof(double));
  CK(cudaMemsetAsync(b.results, 0, 64 * sizeof(double), stream));
  if (st) {
    b.st = st;
    b.st_shared = true;
  } else {
    ALLOC(b.st, sizeof(MinresState));
  }
  CK(cudaMemsetAsync(b.st, 0, sizeof(MinresState), stream));
  ALLOC(b.citers, 4 * sizeof(int));
  CK(cudaMemsetAsync(b.citers, 0, 4 * sizeof(int), stream));
  ALLOC(b.dparams, SSFFT_MAX_PHASES * sizeof(PhaseParams));
  return 0;
}

static void slot_free(SlotBufs &b) {
  void *ptrs[] = {b.spec, b.partials, b.tickets, b.results, b.st_shared ? nullptr : b.st, b.citers, b.dparams,
                  b.orient, b.phase, b.gid, b.rm_tab, b.ktab, b.kvox_buf[0], b.kvox_buf[1],
                  b.slip_buf[0], b.slip_buf[1], b.slip_buf[2], b.slip_buf[3], b.slip_buf[4],
                  b.ep_buf[0], b.ep_buf[1], b.Gam_buf[0], b.Gam_buf[1]};
  for (void *q : ptrs)
    if (q) cudaFree(q);
  for (int i = 0; i < 14; ++i)
    if (b.field[i]) cudaFree(b.field[i]);
  memset((void *)&b, 0, sizeof(b));
}

// The descriptor in its initial roles (after allocation or rebinding), with the solve
// options of cfg.
template <typename T> static void mirror_init(SlotBufs &b, const ssfft_config &cfg) {
  SlotDev<T> &m = mirror<T>(b);
  memset((void *)&m, 0, sizeof(m));
  T **f = reinterpret_cast<T **>(b.field);
  double **fd = reinterpret_cast<double **>(b.field);
  m.eps = fd[0];
  m.eps_old = fd[1];
  m.dfl = fd[2];
  m.sig = fd[3];
  m.sig_next = fd[4];
  m.sig_old = fd[5];
  m.b = f[6];
  for (int i = 0; i < 7; ++i) m.kr[i] = f[7 + i];
  m.spec = b.spec;
  m.gid = b.gid;
  m.ktab = (const T *)b.ktab;
  m.kvox = (T *)b.kvox_buf[0];
  m.kvox_old = (T *)b.kvox_buf[1];
  m.voxel_mode = b.voxel_mode ? 1 : 0;
  m.phase = b.have_phase_buf ? b.phase : nullptr;
  m.orient = b.orient;
  m.rm_tab = b.rm_tab;
  m.params = b.dparams;
  m.n_params = 1;
  for (int k = 0; k < SSFFT_MAX_PHASES; ++k)
    if (b.phase_set[k]) m.n_params = k + 1;
  m.nslip = b.nslip_max;
  m.any_evp = b.any_evp ? 1 : 0;
  m.any_j2 = b.any_j2 ? 1 : 0;
  m.g_in = b.slip_buf[0];
  m.g_out = b.slip_buf[1];
  m.g_old = b.slip_buf[2];
  m.gam_old = b.slip_buf[3];
  m.gam_trial = b.slip_buf[4];
  m.ep_old = b.ep_buf[0];
  m.ep_trial = b.ep_buf[1];
  m.Gam_old = b.Gam_buf[0];
  m.Gam_trial = b.Gam_buf[1];
  m.st = b.st;
  m.partials = b.partials;
  m.tickets = b.tickets;
  m.results = b.results;
  m.citers = b.citers;
  for (int c = 0; c < 6; ++c) m.mask[c] = (cfg.stress_mask[c] != 0.0) ? 1.0 : 0.0;
  m.fluct_scale = 1.0;
  m.dt = 1.0;
}

// Commit of a converged increment (update_state_variables; old_* <- current,
// small_strain_fft.py:213-218): roles swap; the slip resistances are copied by
// commit_slip_kernel.
template <typename T> static void mirror_commit(SlotDev<T> &m) {
  std::swap(m.sig_old, m.sig);
  std::swap(m.eps_old, m.eps);
  std::swap(m.kvox_old, m.kvox);
  std::swap(m.gam_old, m.gam_trial);
  std::swap(m.ep_old, m.ep_trial);
  std::swap(m.Gam_old, m.Gam_trial);
}

// Mandel form of a rotation (materialite/tensor.py:1668-1700).
static void rotation_mandel(const double *R, double *M) {
  const double r2 = SQRT2_D;
  auto r = [&](int i, int j) { return R[i * 3 + j]; };
  const int pr[3][2] = {{1, 2}, {0, 2}, {0, 1}};
  for (int a = 0; a < 3; ++a) {
    for (int b = 0; b < 3; ++b) M[a * 6 + b] = r(a, b) * r(a, b);
    for (int s = 0; s < 3; ++s) M[a * 6 + 3 + s] = r2 * r(a, pr[s][0]) * r(a, pr[s][1]);
  }
  for (int s = 0; s < 3; ++s) {
    const int i = pr[s][0], j = pr[s][1];
    for (int b = 0; b < 3; ++b) M[(3 + s) * 6 + b] = r2 * r(i, b) * r(j, b);
    for (int t = 0; t < 3; ++t) {
      const int k = pr[t][0], l = pr[t][1];
      M[(3 + s) * 6 + 3 + t] = r(i, k) * r(j, l) + r(i, l) * r(j, k);
    }
  }
}

template <typename T>
static void build_ktab(const SlotBufs &b, const std::vector<double> &Rm,
                       const std::vector<int> &gid_orient, const std::vector<int> &gid_phase,
                       std::vector<T> &tab) {
  const int n = (int)gid_orient.size();
  tab.assign((size_t)n * 21, (T)0);
  for (int g = 0; g < n; ++g) {
    const double *R = &Rm[(size_t)gid_orient[g] * 36];
    const double *C = b.hparams[gid_phase[g]].C;
    double CR[36];
    for (int i = 0; i < 6; ++i)
      for (int c = 0; c < 6; ++c) {
        double acc = 0.0;
        for (int j = 0; j < 6; ++j) acc += C[i * 6 + j] * R[j * 6 + c];
        CR[i * 6 + c] = acc;
      }
    for (int a = 0; a < 6; ++a)
      for (int c = a; c < 6; ++c) {
        double acc = 0.0;
        for (int i = 0; i < 6; ++i) acc += R[i * 6 + a] * CR[i * 6 + c];
        tab[(size_t)g * 21 + sym_idx(a, c)] = (T)acc;
      }
  }
}

// (Re)allocate *p to hold `bytes` unless its capacity *cap already does.
static int ensure_buffer(void **p, size_t *cap, size_t bytes) {
  if (*p && *cap >= bytes) return 0;
  if (*p) cudaFree(*p);
  *p = nullptr;
  *cap = 0;
  cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaSuccess) {
    cudaGetLastError();
    *p = nullptr;
    return ssfft_internal_fail(SSFFT_E_NOMEM, std::string("cudaMalloc: ") + cudaGetErrorString(e));
  }
  *cap = bytes;
  return 0;
}

// Bind a microstructure to a slot whose phases are set (Elastic/ElasticViscoplastic/
// Multiphase initialize, small_strain_fft.py:94): rotations, orientation and phase per
// point, and the tangent table (elastic phases only) or per-voxel tangent and plastic
// state buffers.  Host pointers are read during the call (uploads are synchronised).
static int slot_bind(SlotBufs &b, const ssfft_config &cfg, int n_orient, const double *rotations,
                     const int32_t *orient_of_point, const int32_t *phase_of_point,
                     cudaStream_t stream) {
  if (n_orient < 1 || !rotations || !orient_of_point)
    return ssfft_internal_fail(SSFFT_E_INVALID, "rotations and orientation indices are required");
  const long long V = b.V;
  int max_phase = 0;
  for (long long v = 0; v < V; ++v) {
    const int o = orient_of_point[v];
    const int ph = phase_of_point ? phase_of_point[v] : 0;
    if (o < 0 || o >= n_orient)
      return ssfft_internal_fail(SSFFT_E_INVALID, "orientation index out of range");
    if (ph < 0 || ph >= SSFFT_MAX_PHASES || !b.phase_set[ph])
      return ssfft_internal_fail(SSFFT_E_INVALID, "point refers to an undefined phase");
    max_phase = std::max(max_phase, ph);
  }
  b.any_evp = false;
  b.any_j2 = false;
  b.nslip_max = 0;
  for (int ph = 0; ph < SSFFT_MAX_PHASES; ++ph) {
    if (!b.phase_set[ph]) continue;
    if (b.hparams[ph].kind == PHASE_EVP) {
      b.any_evp = true;
      b.nslip_max = std::max(b.nslip_max, b.hparams[ph].nslip);
    } else if (b.hparams[ph].kind == PHASE_J2) {
      b.any_evp = true;
      b.any_j2 = true;
      b.nslip_max = std::max(b.nslip_max, 1);
    }
  }
  b.micro_set = false;
  b.voxel_mode = b.any_evp;
  b.n_orient = n_orient;
  std::vector<double> Rm((size_t)n_orient * 36);
  for (int o = 0; o < n_orient; ++o) rotation_mandel(rotations + (size_t)o * 9, &Rm[(size_t)o * 36]);
  CKR(ensure_buffer((void **)&b.rm_tab, &b.cap_rm, Rm.size() * sizeof(double)));
  CK(cudaMemcpyAsync(b.rm_tab, Rm.data(), Rm.size() * sizeof(double), cudaMemcpyHostToDevice, stream));
  if (!b.orient) ALLOC(b.orient, V * sizeof(int32_t));
  CK(cudaMemcpyAsync(b.orient, orient_of_point, V * sizeof(int32_t), cudaMemcpyHostToDevice, stream));
  if (phase_of_point) {
    if (!b.phase) ALLOC(b.phase, V * sizeof(int32_t));
    CK(cudaMemcpyAsync(b.phase, phase_of_point, V * sizeof(int32_t), cudaMemcpyHostToDevice, stream));
  }
  b.have_phase_buf = phase_of_point != nullptr;
  CK(cudaMemcpyAsync(b.dparams, b.hparams, sizeof(b.hparams), cudaMemcpyHostToDevice, stream));
  if (!b.voxel_mode) {
    // tangent table over the distinct (orientation, phase) pairs present
    std::vector<int> key_to_gid((size_t)n_orient * (max_phase + 1), -1);
    std::vector<int> g_or, g_ph;
    std::vector<int32_t> gid(V);
    for (long long v = 0; v < V; ++v) {
      const int o = orient_of_point[v], ph = phase_of_point ? phase_of_point[v] : 0;
      int &slot = key_to_gid[(size_t)ph * n_orient + o];
      if (slot < 0) {
        slot = (int)g_or.size();
        g_or.push_back(o);
        g_ph.push_back(ph);
      }
      gid[v] = slot;
    }
    b.n_gid = (int)g_or.size();
    if (!b.gid) ALLOC(b.gid, V * sizeof(int32_t));
    CK(cudaMemcpyAsync(b.gid, gid.data(), V * sizeof(int32_t), cudaMemcpyHostToDevice, stream));
    if (b.fp64) {
      std::vector<double> tab;
      build_ktab<double>(b, Rm, g_or, g_ph, tab);
      CKR(ensure_buffer(&b.ktab, &b.cap_ktab, tab.size() * sizeof(double)));
      CK(cudaMemcpyAsync(b.ktab, tab.data(), tab.size() * sizeof(double), cudaMemcpyHostToDevice, stream));
      CK(cudaStreamSynchronize(stream));
    } else {
      std::vector<float> tab;
      build_ktab<float>(b, Rm, g_or, g_ph, tab);
      CKR(ensure_buffer(&b.ktab, &b.cap_ktab, tab.size() * sizeof(float)));
      CK(cudaMemcpyAsync(b.ktab, tab.data(), tab.size() * sizeof(float), cudaMemcpyHostToDevice, stream));
      CK(cudaStreamSynchronize(stream));
    }
  } else {
    if (!b.kvox_buf[0]) {
      ALLOC(b.kvox_buf[0], field_bytes(b, 21));
      ALLOC(b.kvox_buf[1], field_bytes(b, 21));
    }
    const int S = b.nslip_max;
    if (b.cap_nslip < S) {
      for (double *&q : b.slip_buf) {
        if (q) cudaFree(q);
        q = nullptr;
      }
      for (double *&q : b.slip_buf) ALLOC(q, (size_t)S * V * 8);
      b.cap_nslip = S;
    }
    if (!b.ep_buf[0]) {
      ALLOC(b.ep_buf[0], (size_t)6 * V * 8);
      ALLOC(b.ep_buf[1], (size_t)6 * V * 8);
      ALLOC(b.Gam_buf[0], (size_t)V * 8);
      ALLOC(b.Gam_buf[1], (size_t)V * 8);
    }
  }
  CK(cudaStreamSynchronize(stream));  // host arrays of this call go out of scope
  b.micro_set = true;
  if (b.fp64)
    mirror_init<double>(b, cfg);
  else
    mirror_init<float>(b, cfg);
  return 0;
}

// Solve state at t = start: zero strain, stress and fluctuation, initial tangents and
// slip resistances (the descriptor returns to its initial roles).
static int slot_reset(SlotBufs &b, const ssfft_config &cfg, cudaStream_t stream) {
  if (!b.micro_set) return ssfft_internal_fail(SSFFT_E_INVALID, "microstructure not set");
  if (b.fp64)
    mirror_init<double>(b, cfg);
  else
    mirror_init<float>(b, cfg);
  for (int i = 0; i < 7; ++i) CK(cudaMemsetAsync(b.field[i], 0, field_bytes_of(b, i), stream));
  const long long V = b.V;
  const int eb = std::max(1, std::min(div_up(V, SSFFT_THREADS), 148 * 16));
  const int32_t *ph = b.have_phase_buf ? b.phase : nullptr;
  if (b.voxel_mode) {
    if (b.fp64)
      init_kvox_kernel<double><<<eb, SSFFT_THREADS, 0, stream>>>(V, ph, b.orient, b.dparams,
                                                               b.rm_tab, (double *)b.kvox_buf[0]);
    else
      init_kvox_kernel<float><<<eb, SSFFT_THREADS, 0, stream>>>(V, ph, b.orient, b.dparams,
                                                              b.rm_tab, (float *)b.kvox_buf[0]);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(b.kvox_buf[1], b.kvox_buf[0], field_bytes(b, 21), cudaMemcpyDeviceToDevice,
                       stream));
  }
  if (b.any_evp) {
    const int S = b.nslip_max;
    evp_init_kernel<<<eb, SSFFT_THREADS, 0, stream>>>(V, S, ph, b.dparams, b.slip_buf[0],
                                                      b.slip_buf[1], b.slip_buf[2]);
    CK(cudaGetLastError());
    CK(cudaMemsetAsync(b.slip_buf[3], 0, (size_t)S * V * 8, stream));
    CK(cudaMemsetAsync(b.slip_buf[4], 0, (size_t)S * V * 8, stream));
    for (int k = 0; k < 2; ++k) {
      CK(cudaMemsetAsync(b.ep_buf[k], 0, (size_t)6 * V * 8, stream));
      CK(cudaMemsetAsync(b.Gam_buf[k], 0, (size_t)V * 8, stream));
    }
  }
  return 0;
}

// Slot options (stress mask) into the descriptor.
template <typename T> static void mirror_options(SlotDev<T> &m, const ssfft_config &cfg) {
  for (int c = 0; c < 6; ++c) m.mask[c] = (cfg.stress_mask[c] != 0.0) ? 1.0 : 0.0;
}

// ---------------------------------------------------------------------------------------
// launches over a slot list (cap: slots the list can hold; the grid is sized for it)
// ---------------------------------------------------------------------------------------
struct LaunchCtx {
  const GridPlan *p;
  SlotList list;
  int cap;
  cudaStream_t stream;
  long long *launches;
};

// The register-tiled plane passes of one projection around the x pass.
template <typename T, typename TF, int PRO, int EPI, typename REC>
static int launch_dif_planes(const LaunchCtx &c, const SlotDev<TF> *tab, const ExtIO<TF> &io,
                              const REC &rec) {
  constexpr bool KRY = PRO == PRO_TAU;
  const GridPlan &p = *c.p;
  const DifPlane *PP = p.dplane[sizeof(T) == 8 ? 1 : 0], &P = PP[0], &Q = PP[1];
  const Grid<T> &g = grid_of<T>(p);
  const size_t sp = DifTables<T, false>::bytes(P, p.ny, p.nz, g.hs);
  const size_t sq = DifTables<T, true>::bytes(Q, p.ny, p.nz, g.hs);
  const long long it = (long long)c.cap * items_plane(g);
  const int pt = P.threads;
  if constexpr (PRO == PRO_RESIDUAL) {
    // the residual reads the stress alone, which is double for either storage type
    auto kf = dif_zyfwd_kernel<double, double, DIF_RESIDUAL>;
    CKR(launch_kernel(false, kf, persistent_grid(kf, pt, sp, it, p.dev), pt, sp, c.stream, g, P,
                      reinterpret_cast<const SlotDev<double> *>(tab), c.list, ExtIO<double>{}, (int)PRO));
  } else {
    auto kf = dif_zyfwd_kernel<T, TF, DIF_PLANES>;
    CKR(launch_kernel(KRY, kf, persistent_grid(kf, pt, sp, it, p.dev), pt, sp, c.stream, g, P, tab,
                      c.list, io, (int)PRO));
  }
  rec(1);
  rec(2);
  CKR((launch_x<T, TF, KRY>(p, g, c.cap, c.stream, tab, c.list)));
  rec(3);
  rec(4);
  auto ki = dif_yzinv_kernel<T, TF, dif_kind(EPI)>;
  return launch_kernel(true, ki, persistent_grid(ki, pt, sq, it, p.dev), pt, sq, c.stream, g, Q, tab,
                       c.list, io, (int)EPI);
}

// The passes of one projection.  ev (optional, 6 events) is recorded before the first pass
// and after each of the five pass slots z-fwd, y-fwd, x, y-inv, z-inv; with the
// plane-fused passes the y slots are empty (zero time).
template <typename T, typename TF, int PRO, int EPI>
static int launch_projector(const LaunchCtx &c, const SlotDev<TF> *tab, ExtIO<TF> io = {},
                            cudaEvent_t *ev = nullptr) {
  const GridPlan &p = *c.p;
  const Grid<T> &g = grid_of<T>(p);
  // the middle passes of a Krylov matvec skip finished solves as the outer ones do (a
  // device-side loop runs its chunk of iterations to the end after a solve finishes)
  constexpr bool KRY = PRO_IS_KRYLOV(PRO) || PRO == PRO_TAU;
  auto rec = [&](int k) {
    if (ev) cudaEventRecord(ev[k], c.stream);
  };
  const int dev = p.dev;
  const Route r = route_of<T, TF, PRO, EPI>(p);
  rec(0);
  if (r.kind == ROUTE_DIF_PLANE) {
    CKR((launch_dif_planes<T, TF, PRO, EPI>(c, tab, io, rec)));
    rec(5);
    if (c.launches) *c.launches += 3;
  } else if (r.kind == ROUTE_CLUSTER) {
    const int C = r.C;
    const ClusterGeo q = cluster_geo<T>(p, C);
    const size_t sp = smem_cplane_bytes<T>(p.ny, p.nz, g.hs, C);
    const long long it = (long long)c.cap * items_plane(g);
    const int pt = p.cl_threads[sizeof(T) == 8 ? 1 : 0];
    if (pt == 1024)
      CKR(launch_clustered(zyfwd_cl_kernel<T, TF, PRO, 1024>, C, 1024, sp, it, dev, c.stream, g, q, tab, c.list, io));
    else if (pt == 256)
      CKR(launch_clustered(zyfwd_cl_kernel<T, TF, PRO, 256>, C, 256, sp, it, dev, c.stream, g, q, tab, c.list, io));
    else
      CKR(launch_clustered(zyfwd_cl_kernel<T, TF, PRO, 512>, C, 512, sp, it, dev, c.stream, g, q, tab, c.list, io));
    rec(1);
    rec(2);
    CKR((launch_x<T, TF, KRY>(p, g, c.cap, c.stream, tab, c.list)));
    rec(3);
    rec(4);
    if (pt == 1024)
      CKR(launch_clustered(yzinv_cl_kernel<T, TF, EPI, 1024>, C, 1024, sp, it, dev, c.stream, g, q, tab, c.list, io));
    else if (pt == 256)
      CKR(launch_clustered(yzinv_cl_kernel<T, TF, EPI, 256>, C, 256, sp, it, dev, c.stream, g, q, tab, c.list, io));
    else
      CKR(launch_clustered(yzinv_cl_kernel<T, TF, EPI, 512>, C, 512, sp, it, dev, c.stream, g, q, tab, c.list, io));
    rec(5);
    if (c.launches) *c.launches += 3;
  } else if (r.kind == ROUTE_PLANE) {
    const size_t sp = smem_plane_bytes<T>(p.ny, p.nz);
    const long long it = (long long)c.cap * items_plane(g);
    if (plane_threads<T>(p) == 1024) {
      auto kf = zyfwd_kernel<T, TF, PRO, 1024>;
      CKR(launch_kernel(false, kf, persistent_grid(kf, 1024, sp, it, dev), 1024, sp, c.stream, g, tab, c.list, io));
    } else {
      auto kf = zyfwd_kernel<T, TF, PRO, 512>;
      CKR(launch_kernel(false, kf, persistent_grid(kf, 512, sp, it, dev), 512, sp, c.stream, g, tab, c.list, io));
    }
    rec(1);
    rec(2);
    CKR((launch_x<T, TF, KRY>(p, g, c.cap, c.stream, tab, c.list)));
    rec(3);
    rec(4);
    if (plane_threads<T>(p) == 1024) {
      auto ki = yzinv_kernel<T, TF, EPI, 1024>;
      CKR(launch_kernel(false, ki, persistent_grid(ki, 1024, sp, it, dev), 1024, sp, c.stream, g, tab, c.list, io));
    } else {
      auto ki = yzinv_kernel<T, TF, EPI, 512>;
      CKR(launch_kernel(false, ki, persistent_grid(ki, 512, sp, it, dev), 512, sp, c.stream, g, tab, c.list, io));
    }
    rec(5);
    if (c.launches) *c.launches += 3;
  } else {
    const size_t sz = smem_z_bytes<T>(p.lz, p.nz);
    const long long itz = (long long)c.cap * items_z(g);
    const DifZPlan *dz = p.dz[sizeof(T) == 8 ? 1 : 0];
    if constexpr (sizeof(T) == sizeof(TF)) {
      if (r.dif_z) {
        auto k = dif_zfwd_kernel<T>;
        const size_t sm = ((size_t)dz[0].p.elems + p.nz) * sizeof(cplx<T>);
        const int grid = persistent_grid(k, DIFZ_THREADS, sm, (long long)c.cap * 3 * dz[0].ntiles, dev);
        CKR(launch_kernel(KRY, k, grid, DIFZ_THREADS, sm, c.stream, g, dz[0], tab, c.list, io, KRY ? 1 : 0));
      }
    }
    if (!r.dif_z) {
      auto kz = zfwd_kernel<T, TF, PRO>;
      CKR(launch_kernel(false, kz, persistent_grid(kz, SSFFT_THREADS, sz, itz, dev), SSFFT_THREADS, sz,
                        c.stream, g, tab, c.list, io));
    }
    rec(1);
    CKR((launch_y<T, TF, false, KRY>(p, g, c.cap, c.stream, tab, c.list)));
    rec(2);
    CKR((launch_x<T, TF, KRY>(p, g, c.cap, c.stream, tab, c.list)));
    rec(3);
    CKR((launch_y<T, TF, true, KRY>(p, g, c.cap, c.stream, tab, c.list)));
    rec(4);
    if constexpr (sizeof(T) == sizeof(TF)) {
      if (r.dif_z) {
        auto k = dif_zinv_kernel<T>;
        const size_t sm = ((size_t)dz[1].p.elems + p.nz) * sizeof(cplx<T>);
        const int grid = persistent_grid(k, DIFZ_THREADS, sm, (long long)c.cap * 3 * dz[1].ntiles, dev);
        CKR(launch_kernel(true, k, grid, DIFZ_THREADS, sm, c.stream, g, dz[1], tab, c.list, io, KRY ? 1 : 0));
      }
    }
    if (!r.dif_z) {
      auto kzi = zinv_kernel<T, TF, EPI>;
      CKR(launch_kernel(false, kzi, persistent_grid(kzi, SSFFT_THREADS, sz, itz, dev), SSFFT_THREADS, sz,
                        c.stream, g, tab, c.list, io));
    }
    rec(5);
    if (c.launches) *c.launches += 5;
  }
  CK(cudaGetLastError());
  return 0;
}

// One MINRES iteration on every listed slot whose solve is not done: the projector passes
// with the pending vector update in the forward prologue and the scalar recurrence in the
// inverse epilogue.
// ev (optional, 8 events): ev[7] before the update kernel, ev[0..5] by the projector (the
// epilogue kernel follows ev[5]).
template <typename T>
static int launch_krylov_iteration(const LaunchCtx &c, const SlotDev<T> *tab, bool voxel,
                                   cudaEvent_t *ev = nullptr, bool pdl_first = false) {
  if (ev) cudaEventRecord(ev[7], c.stream);
  const long long it = (long long)c.cap * vec_items(c.p->V);
  const bool many = c.cap > 1;
  if (voxel) {
    auto k = many ? krylov_update_kernel<T, PRO_TANGENT_VOXEL, true> : krylov_update_kernel<T, PRO_TANGENT_VOXEL, false>;
    CKR(launch_kernel(pdl_first, k, persistent_grid(k, SSFFT_THREADS, 0, it, c.p->dev), SSFFT_THREADS, 0,
                      c.stream, tab, c.list, c.p->V));
  } else {
    auto k = many ? krylov_update_kernel<T, PRO_TANGENT_TABLE, true> : krylov_update_kernel<T, PRO_TANGENT_TABLE, false>;
    CKR(launch_kernel(pdl_first, k, persistent_grid(k, SSFFT_THREADS, 0, it, c.p->dev), SSFFT_THREADS, 0,
                      c.stream, tab, c.list, c.p->V));
  }
  if (c.launches) *c.launches += 1;
  CKR((launch_projector<T, T, PRO_TAU, EPI_PTAU>(c, tab, {}, ev)));
  auto ke = many ? krylov_epilogue_kernel<T, true> : krylov_epilogue_kernel<T, false>;
  CKR(launch_kernel(true, ke, persistent_grid(ke, SSFFT_THREADS, 0, it, c.p->dev), SSFFT_THREADS, 0,
                    c.stream, tab, c.list, c.p->V));
  if (c.launches) *c.launches += 1;
  return 0;
}

// b = P(Sbar - sigma) into each slot's b, max|b| into results[40].  The transform always
// runs in double: in the mixed mode the float stress field is read and b is stored as
// float, but the equilibrium residual and its norm are double-precision quantities.
template <typename T> static int launch_residual(const LaunchCtx &c, const SlotDev<T> *tab) {
  return launch_projector<double, T, PRO_RESIDUAL, EPI_RESIDUAL>(c, tab);
}

// Mixed mode: project each slot's Newton correction x back onto compatible strain fields
// with a double-precision transform (x <- Gamma-hat : x, an identity in exact arithmetic),
// then strain += x and fluctuation += x.  Float Krylov iterates pick up round-off in the
// null space of Gamma-hat K, which the equilibrium test cannot see; this removes it.
template <typename T> static int launch_reproject_update(const LaunchCtx &c, const SlotDev<T> *tab) {
  if constexpr (sizeof(T) == 4)
    return launch_projector<double, T, PRO_REPROJECT, EPI_REPROJECT>(c, tab);
  else
    return ssfft_internal_fail(SSFFT_E_INVALID, "double solves are not re-projected");
}

template <typename T>
static int launch_minres_init(const LaunchCtx &c, const SlotDev<T> *tab) {
  auto k = c.cap > 1 ? minres_init_kernel<T, true> : minres_init_kernel<T, false>;
  const long long it = (long long)c.cap * vec_items(6 * c.p->V);
  k<<<persistent_grid(k, SSFFT_THREADS, 0, it, c.p->dev), SSFFT_THREADS, 0, c.stream>>>(tab, c.list, c.p->V);
  if (c.launches) *c.launches += 1;
  CK(cudaGetLastError());
  return 0;
}

template <typename T> static int launch_strain_guess(const LaunchCtx &c, const SlotDev<T> *tab) {
  auto k = strain_guess_kernel<T>;
  const long long it = (long long)c.cap * vec_items(c.p->V);
  k<<<persistent_grid(k, SSFFT_THREADS, 0, it, c.p->dev), SSFFT_THREADS, 0, c.stream>>>(tab, c.list, c.p->V);
  if (c.launches) *c.launches += 1;
  CK(cudaGetLastError());
  return 0;
}

template <typename T> static int launch_update_strain(const LaunchCtx &c, const SlotDev<T> *tab) {
  auto k = update_strain_kernel<T>;
  const long long it = (long long)c.cap * vec_items(6 * c.p->V);
  k<<<persistent_grid(k, SSFFT_THREADS, 0, it, c.p->dev), SSFFT_THREADS, 0, c.stream>>>(tab, c.list, c.p->V);
  if (c.launches) *c.launches += 1;
  CK(cudaGetLastError());
  return 0;
}

template <typename T> static int launch_norms(const LaunchCtx &c, const SlotDev<T> *tab) {
  auto k = c.cap > 1 ? newton_norms_kernel<T, true> : newton_norms_kernel<T, false>;
  const long long it = (long long)c.cap * vec_items(c.p->V);
  k<<<persistent_grid(k, SSFFT_THREADS, 0, it, c.p->dev), SSFFT_THREADS, 0, c.stream>>>(tab, c.list, c.p->V);
  if (c.launches) *c.launches += 1;
  CK(cudaGetLastError());
  return 0;
}

template <typename T> static int launch_tangent_sum(const LaunchCtx &c, const SlotDev<T> *tab) {
  auto k = c.cap > 1 ? tangent_sum_kernel<T, true> : tangent_sum_kernel<T, false>;
  const long long it = (long long)c.cap * vec_items(c.p->V);
  k<<<persistent_grid(k, SSFFT_THREADS, 0, it, c.p->dev), SSFFT_THREADS, 0, c.stream>>>(tab, c.list, c.p->V);
  if (c.launches) *c.launches += 1;
  CK(cudaGetLastError());
  return 0;
}

// Constitutive update of every listed slot (j2: with the J2 counting pass first).  Each
// slot's citers must be cleared before.
template <typename T>
static int launch_constitutive(const LaunchCtx &c, const SlotDev<T> *tab, bool j2) {
  const long long it = (long long)c.cap * const_items(c.p->V);
  if (j2) {
    auto kj = j2_count_kernel<T>;
    kj<<<persistent_grid(kj, SSFFT_THREADS, 0, it, c.p->dev), SSFFT_THREADS, 0, c.stream>>>(tab, c.list, c.p->V,
                                                                                            c.cap > 1);
    if (c.launches) *c.launches += 1;
    CK(cudaGetLastError());
  }
  const size_t sm = constitutive_smem_bytes();
  auto k = constitutive_kernel<T>;
  k<<<persistent_grid(k, CONST_THREADS, sm, it, c.p->dev), CONST_THREADS, sm, c.stream>>>(tab, c.list, c.p->V, c.cap > 1);
  if (c.launches) *c.launches += 1;
  CK(cudaGetLastError());
  return 0;
}

template <typename T>
static int launch_commit_slip(const LaunchCtx &c, const SlotDev<T> *tab, int nslip_max) {
  if (nslip_max < 1) return 0;
  auto k = commit_slip_kernel<T>;
  const long long it = (long long)c.cap * vec_items((long long)nslip_max * c.p->V);
  k<<<persistent_grid(k, SSFFT_THREADS, 0, it, c.p->dev), SSFFT_THREADS, 0, c.stream>>>(
      tab, c.list, c.p->V, nslip_max);
  if (c.launches) *c.launches += 1;
  CK(cudaGetLastError());
  return 0;
}


// 6x6 inverse by Gauss-Jordan with partial pivoting (host and device, double).
__host__ __device__ inline bool inv6(const double *A, double *Ainv) {
  double a[6][12];
  for (int i = 0; i < 6; ++i)
    for (int j = 0; j < 12; ++j) a[i][j] = (j < 6) ? A[i * 6 + j] : (j - 6 == i ? 1.0 : 0.0);
  for (int c = 0; c < 6; ++c) {
    int p = c;
    for (int r = c + 1; r < 6; ++r)
      if (fabs(a[r][c]) > fabs(a[p][c])) p = r;
    if (a[p][c] == 0.0) return false;
    if (p != c)
      for (int j = 0; j < 12; ++j) {
        const double t = a[p][j];
        a[p][j] = a[c][j];
        a[c][j] = t;
      }
    const double d = a[c][c];
    for (int j = 0; j < 12; ++j) a[c][j] /= d;
    for (int r = 0; r < 6; ++r)
      if (r != c) {
        const double f = a[r][c];
        if (f != 0.0)
          for (int j = 0; j < 12; ++j) a[r][j] -= mul_rn(f, a[c][j]);
      }
  }
  for (int i = 0; i < 6; ++i)
    for (int j = 0; j < 6; ++j) Ainv[i * 6 + j] = a[i][j + 6];
  return true;
}

