// Register-tiled transform passes for axes whose length factors into two or three radices up
// to 16 (primes up to 7): the x pass with Gamma-hat, the fused z and y passes of one x plane, and
// separate z and y passes for planes too large for a block.
//
// Every line is transformed in place in one shared-memory buffer by decimation in frequency.
// A length N = r_0 r_1 .. r_s line is viewed as digits: stage 0 takes, for each
// n' < m = N / r_0, the r_0 points n' + m q, transforms them in registers, multiplies output q
// by w_N^(n' q) and stores it in the slot of input q; the next stage treats the remaining
// m-point lines in the same way, and so on.  Frequency k = q_0 + r_0 (q_1 + r_1 q_2) then sits
// in the slot of digits (q_0, q_1, q_2).  Run backwards, the same digits give the inverse, so
// a thread of the x pass's last stage owns the very slots it filled in the first.
//
// The first stage of a pass reads global memory into registers and the last one writes it from
// there, and the paired-line split is folded into a z stage.  With two stages an axis an element
// crosses shared memory four times in the x pass and three times in a plane pass, where the
// Stockham passes (projector.cuh) take six or seven crossings, two buffers, and a padded index
// computation per element.  Both are bound by instruction issue and, on small grids, by the
// chain of dependent reads at a kernel's start, not by memory.  Measured per Krylov iteration,
// Stockham against these (forward plane, x, inverse plane; events, about 2.5 us each of them
// the event's): 64^3 float 17.0 / 17.4 / 16.9 -> 15.7 / 15.0 / 15.0 us, 96^3 float 34.9 / 37.3 /
// 33.3 -> 27 / 29 / 25, 128^3 float 67.7 / 74.2 / 77.2 -> 60 / 52 / 58, 45 x 50 x 63 double
// 31.0 / 23.4 / 31.2 -> 18 / 20 / 17 (radices 5 and 7 were direct sums in local memory).
#pragma once

#include <cstddef>
#include <type_traits>
#include <utility>

#include "common.cuh"
#include "fft.cuh"
#include "projector.cuh"
#include "slots.cuh"

// ---- transforms in registers ----------------------------------------------------------

// cos and sin of 2 pi m / r at compile time: Taylor series after reduction to an octant.
__host__ __device__ constexpr double dif_series(double x, int first) {
  double term = first ? x : 1.0, sum = term;
  for (int k = first; k < 24; k += 2) {
    term *= -x * x / ((k + 1) * (k + 2));
    sum += term;
  }
  return sum;
}
__host__ __device__ constexpr double dif_cos(int m, int r) {
  m = ((m % r) + r) % r;
  if (2 * m > r) m = r - m;
  double sign = 1.0;
  if (4 * m > r) {
    sign = -1.0;
    m = r - 2 * m;
    r = 2 * r;
  }
  const double pi2 = 6.28318530717958647693;
  return sign * (8 * m <= r ? dif_series(pi2 * m / r, 0) : dif_series(pi2 * (r - 4 * m) / (4 * r), 1));
}
template <int M, int R> struct DifW {
  static constexpr double c = dif_cos(M, R);
  static constexpr double s = dif_cos(4 * M - R, 4 * R);
};

template <class F, int... I>
__device__ __forceinline__ void dif_for_impl(F &&f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F> __device__ __forceinline__ void dif_for(F &&f) {
  dif_for_impl(f, std::make_integer_sequence<int, N>{});
}

// v <- DFT_R v (exponent -, or + for the inverse; unscaled).
template <typename T, bool INV, int R> __device__ __forceinline__ void dft(cplx<T> *v);

// Odd prime lengths: sums and differences of mirrored points, (R-1)/2 products each.
template <typename T, bool INV, int R> __device__ __forceinline__ void dft_odd(cplx<T> *v) {
  constexpr int H = (R - 1) / 2;
  cplx<T> t[H], d[H], sum = v[0];
#pragma unroll
  for (int j = 0; j < H; ++j) {
    t[j] = cadd<T>(v[j + 1], v[R - 1 - j]);
    d[j] = csub<T>(v[j + 1], v[R - 1 - j]);
    sum = cadd<T>(sum, t[j]);
  }
  cplx<T> o[R];
  o[0] = sum;
  dif_for<H>([&](auto kc) {
    constexpr int k = decltype(kc)::value + 1;
    cplx<T> a = v[0], b = mk<T>((T)0, (T)0);
    dif_for<H>([&](auto jc) {
      constexpr int j = decltype(jc)::value;
      constexpr T c = (T)DifW<((j + 1) * k) % R, R>::c, s = (T)DifW<((j + 1) * k) % R, R>::s;
      a = mk<T>(a.x + c * t[j].x, a.y + c * t[j].y);
      b = mk<T>(b.x + s * d[j].x, b.y + s * d[j].y);
    });
    const cplx<T> r = mul_mi<T, INV>(b);
    o[k] = cadd<T>(a, r);
    o[R - k] = csub<T>(a, r);
  });
#pragma unroll
  for (int k = 0; k < R; ++k) v[k] = o[k];
}

// R = A B: DFT_A over x[B n1 + n2] for each n2, twiddles w_R^(n2 k1), DFT_B over n2.
template <typename T, bool INV, int A, int B> __device__ __forceinline__ void dft_ab(cplx<T> *v) {
  constexpr int R = A * B;
  cplx<T> a[R];
  dif_for<B>([&](auto n2c) {
    constexpr int n2 = decltype(n2c)::value;
    cplx<T> t[A];
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) t[n1] = v[B * n1 + n2];
    dft<T, INV, A>(t);
    dif_for<A>([&](auto k1c) {
      constexpr int k1 = decltype(k1c)::value;
      constexpr T c = (T)DifW<n2 * k1, R>::c, s = (T)(INV ? DifW<n2 * k1, R>::s : -DifW<n2 * k1, R>::s);
      if constexpr (n2 * k1 == 0)
        a[B * k1 + n2] = t[k1];
      else
        a[B * k1 + n2] = cmul<T>(t[k1], mk<T>(c, s));
    });
  });
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) {
    dft<T, INV, B>(a + B * k1);
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2) v[k1 + A * k2] = a[B * k1 + k2];
  }
}

template <typename T, bool INV, int R> __device__ __forceinline__ void dft(cplx<T> *v) {
  if constexpr (R == 2) bfly2<T, INV>(v);
  if constexpr (R == 3) bfly3<T, INV>(v);
  if constexpr (R == 4) bfly4<T, INV>(v);
  if constexpr (R == 5 || R == 7) dft_odd<T, INV, R>(v);
  if constexpr (R == 6) dft_ab<T, INV, 2, 3>(v);
  if constexpr (R == 8) bfly8<T, INV>(v);
  if constexpr (R == 9) dft_ab<T, INV, 3, 3>(v);
  if constexpr (R == 10) dft_ab<T, INV, 2, 5>(v);
  if constexpr (R == 12) bfly12<T, INV>(v);
  if constexpr (R == 16) bfly16<T, INV>(v);
}

// Run a statement with the constant R set to the run-time radix r (block-uniform): 1 to 10, 12
// or 16.  A macro rather than a generic lambda: where a lambda was not inlined, the buffers it
// captured became generic pointers in local memory, and the plane passes took twice as long.
#define DIF_CASE(N, ...)     \
  case N: {                  \
    constexpr int R = N;     \
    __VA_ARGS__              \
  } break;
#define DIF_RADIX8_CASES(...)                                                              \
  DIF_CASE(1, __VA_ARGS__)                                                                 \
  DIF_CASE(2, __VA_ARGS__)                                                                 \
  DIF_CASE(3, __VA_ARGS__)                                                                 \
  DIF_CASE(4, __VA_ARGS__)                                                                 \
  DIF_CASE(5, __VA_ARGS__)                                                                 \
  DIF_CASE(6, __VA_ARGS__)                                                                 \
  DIF_CASE(7, __VA_ARGS__)                                                                 \
  DIF_CASE(8, __VA_ARGS__)
#define DIF_RADIX(r, ...)                                                                  \
  switch (r) {                                                                             \
    DIF_RADIX8_CASES(__VA_ARGS__)                                                          \
    DIF_CASE(9, __VA_ARGS__)                                                               \
    DIF_CASE(10, __VA_ARGS__)                                                              \
    DIF_CASE(12, __VA_ARGS__)                                                              \
    DIF_CASE(16, __VA_ARGS__)                                                              \
  }
// The same for middle stages and stages of paired lines, whose radix is at most 8.
#define DIF_RADIX8(r, ...) \
  switch (r) { DIF_RADIX8_CASES(__VA_ARGS__) }

// Shared memory by 32-bit address.  The buffers are reached through helper functions and
// structures, where the compiler does not always recover that a pointer is to shared memory
// and falls back to generic accesses with 64-bit addresses.
template <typename T> struct SPtr {
  unsigned a;
  __device__ __forceinline__ SPtr operator+(int i) const { return SPtr{a + (unsigned)(i * (int)sizeof(cplx<T>))}; }
  __device__ __forceinline__ cplx<T> ld(int i) const {
    const unsigned p = a + (unsigned)(i * (int)sizeof(cplx<T>));
    cplx<T> v;
    if constexpr (sizeof(T) == 4)
      asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(p) : "memory");
    else
      asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(p) : "memory");
    return v;
  }
  __device__ __forceinline__ void st(int i, cplx<T> v) const {
    const unsigned p = a + (unsigned)(i * (int)sizeof(cplx<T>));
    if constexpr (sizeof(T) == 4)
      asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(p), "f"(v.x), "f"(v.y) : "memory");
    else
      asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(p), "d"(v.x), "d"(v.y) : "memory");
  }
};
struct SPtr16 {
  unsigned a;
  __device__ __forceinline__ int operator[](int i) const {
    unsigned short v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a + 2u * (unsigned)i) : "memory");
    return v;
  }
};
template <typename T, bool INV> __device__ __forceinline__ cplx<T> dif_tw(SPtr<T> tw, int i) {
  const cplx<T> w = tw.ld(i);
  return INV ? cconj<T>(w) : w;
}

// An axis's plan: stages, slot strides and the divisors of its index arithmetic.
struct DifAxis {
  int n, ns;           // length, stages (2 or 3)
  int r0, r1, r2;      // radices (r2 = 1: two stages)
  int m;               // n / r0
  int a, b;            // slot strides of n' and q_0
  FastDiv fd_m, fd_r0;
  FastDiv fd_nb;       // butterflies of the last stage, n / r_last
  FastDiv fd_nb1;      // butterflies of stage 1
  FastDiv fd_un;       // paired butterflies of the last (forward) or first (inverse) stage
};

__device__ __forceinline__ int dif_last_radix(const DifAxis &A) { return A.ns == 2 ? A.r1 : A.r2; }

// Slots of butterfly j of the last stage: base + q a holds frequency (or point) j + nb q,
// nb = n / r_last.
__device__ __forceinline__ int dif_last_base(const DifAxis &A, int j) {
  if (A.ns == 2) return j * A.b;
  const int h = udiv(j, A.fd_r0);
  return h * A.r2 * A.a + (j - h * A.r0) * A.b;
}

// ---- x pass -----------------------------------------------------------------------------
//
// An item is (slot, y, tile of kx kz columns).  Element (n', q_0) of component c, column col
// sits at c cs + n' a + q_0 kx + col, a padded so that the lanes of the first stage (columns,
// then n') touch distinct banks; the other stages read along (q_0, col), which is contiguous.
// Gamma-hat is a pass of its own over the slots: fused with the last forward and first inverse
// stages it saves two crossings, but holds 6 r components a thread, which left a third of the
// threads busy and 8 warps an SM (measured at 64^3 float: 21.0 us fused, 15.0 split;
// 128^3: 80 and 51.6).

struct DifXPlan {
  int ok;
  int kx, lkx, nkx;   // columns per tile (a power of two), its logarithm, tiles
  int cs, elems;      // component stride and buffer elements
  DifAxis x;
  FastDiv fd_mid, fd_r2, fd_items, fd_nkx;
};

// MB blocks an SM: five in float.  In double three (96 registers, 32 bytes spilled), which hide
// more of the latency than two (168), up to 200 points along x, and two for longer lines, whose
// tiles take 46 KB and more.  Both run the same stages; the line is where the sweep crosses.
// Projections in FP64, us, two / three blocks: 45 x 50 x 63 47.3 / 44.7, 96 x 80 x 60 82.0 / 76.8,
// 135 x 175 x 189 771 / 723, 128^3 305 / 297, 192^3 1007 / 1008, 200 x 225 x 64 469 / 460;
// 240 x 96 x 250 977 / 1051, 256^3 2177 / 2320.
#define DIFX_THREADS 192
#define DIFX_THREE_MOST 200

// Gamma-hat of one frequency on the six components m[], with t = (t0, t1, t2) = tan(pi f) not
// normalised: s = t / |t|^2, u = T t, O = s (x) u + u (x) s - (s . u) s (x) t, times the
// transform's scale.
template <typename T>
__device__ __forceinline__ void dif_green(T t0, T t1, T t2, T scale, cplx<T> *m) {
  const T inv = (T)1 / (t0 * t0 + t1 * t1 + t2 * t2);
  const T s0 = t0 * inv, s1 = t1 * inv, s2 = t2 * inv;
  const T h = (T)INV_SQRT2_D, r2 = (T)SQRT2_D;
  const T a0 = scale * s0, a1 = scale * s1, a2 = scale * s2;
#pragma unroll
  for (int ri = 0; ri < 2; ++ri) {
    T v[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) v[c] = ri ? m[c].y : m[c].x;
    const T u0 = v[0] * t0 + h * (v[5] * t1 + v[4] * t2);
    const T u1 = v[1] * t1 + h * (v[5] * t0 + v[3] * t2);
    const T u2 = v[2] * t2 + h * (v[4] * t0 + v[3] * t1);
    const T su = s0 * u0 + s1 * u1 + s2 * u2;
    T o[6];
    o[0] = a0 * (2 * u0 - su * t0);
    o[1] = a1 * (2 * u1 - su * t1);
    o[2] = a2 * (2 * u2 - su * t2);
    o[3] = r2 * (a1 * u2 + a2 * (u1 - su * t1));
    o[4] = r2 * (a0 * u2 + a2 * (u0 - su * t0));
    o[5] = r2 * (a0 * u1 + a1 * (u0 - su * t0));
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      if (ri)
        m[c].y = o[c];
      else
        m[c].x = o[c];
    }
  }
}

// The descriptors of the two storage types differ in pointer targets only; the x pass and the
// residual's forward pass read none of the typed fields, so they run on either.
static_assert(sizeof(SlotDev<float>) == sizeof(SlotDev<double>) &&
                  offsetof(SlotDev<float>, spec) == offsetof(SlotDev<double>, spec) &&
                  offsetof(SlotDev<float>, st) == offsetof(SlotDev<double>, st) &&
                  offsetof(SlotDev<float>, sig) == offsetof(SlotDev<double>, sig) &&
                  offsetof(SlotDev<float>, sbar) == offsetof(SlotDev<double>, sbar) &&
                  offsetof(SlotDev<float>, mask) == offsetof(SlotDev<double>, mask),
              "slot descriptors must have one layout");

// Middle stage of NC components' lines (three-stage axes): butterflies (c, n'', q_0, column).
template <typename T, bool INV, int NC = 6>
__device__ __forceinline__ void difx_middle(SPtr<T> buf, const DifXPlan &P, SPtr<T> tw) {
  const DifAxis &X = P.x;
  const int inner = X.r0 << P.lkx;            // contiguous (q_0, column)
  const int total = NC * X.r2 * inner;
  DIF_RADIX8(X.r1,
_Pragma("unroll 1")
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
      const int g = udiv(t, P.fd_mid), in = t - g * inner;
      const int c = NC == 1 ? 0 : udiv(g, P.fd_r2), n2 = g - c * X.r2;
      const SPtr<T> b = buf + c * P.cs + n2 * X.a + in;
      const int step = X.r2 * X.a;
      cplx<T> v[R];
_Pragma("unroll")
      for (int q = 0; q < R; ++q) v[q] = b.ld(q * step);
      dft<T, INV, R>(v);
      /* forward: w^(r_0 n" q); inverse: w^-(q_0 n_2 r_2) */
      const int e = INV ? (in >> P.lkx) * X.r2 : n2 * X.r0;
_Pragma("unroll")
      for (int q = 1; q < R; ++q) v[q] = cmul<T>(v[q], dif_tw<T, INV>(tw, q * e));
_Pragma("unroll")
      for (int q = 0; q < R; ++q) b.st(q * step, v[q]);
    }
    )
  __syncthreads();
}

// Last forward stage, or first inverse one, of the x lines: butterflies (c, j, column).
template <typename T, bool INV>
__device__ __forceinline__ void difx_last(SPtr<T> buf, const DifXPlan &P, int nx, SPtr<T> tw) {
  const DifAxis &X = P.x;
  DIF_RADIX(dif_last_radix(X),
    const int nb = nx / R, total = 6 * nb << P.lkx;
_Pragma("unroll 1")
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
      const int r = t >> P.lkx, c = udiv(r, X.fd_nb), j = r - c * nb;
      const SPtr<T> b = buf + c * P.cs + dif_last_base(X, j) + (t & (P.kx - 1));
      cplx<T> v[R];
_Pragma("unroll")
      for (int q = 0; q < R; ++q) v[q] = b.ld(q * X.a);
      dft<T, INV, R>(v);
_Pragma("unroll")
      for (int q = 0; q < R; ++q)
        b.st(q * X.a, INV && q ? cmul<T>(v[q], dif_tw<T, true>(tw, q * j)) : v[q]);
    }
    )
  __syncthreads();
}

template <typename T, int MB>
__global__ void __launch_bounds__(DIFX_THREADS, MB)
    difx_kernel(Grid<T> g, DifXPlan P, const SlotDev<T> *__restrict__ tab, SlotList list, int kry) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const DifAxis &X = P.x;
  const int nx = g.nx, ny = g.ny, hs = g.hs;
  pdl_begin();
  load_table<T>(reinterpret_cast<cplx<T> *>(smem_raw) + P.elems, g.twx, nx);
  const SPtr<T> buf{smem_u32(smem_raw)}, tw = buf + P.elems;
  __syncthreads();
  const int per = P.nkx * ny;
  pdl_wait();
  const int slot0 = list.ids[udiv(blockIdx.x, P.fd_items)];
  const int n_items = list_items(list, per);
  const int kxm = P.kx - 1;
  const long long rowx = (long long)ny * hs;      // spectrum step of one x
  for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
    const int ks = udiv(item, P.fd_items);
    const int local = item - ks * per;
    const int slot = item == (int)blockIdx.x ? slot0 : list.ids[ks];
    const SlotDev<T> &S = tab[slot];
    const bool done = kry && slot_done(list.st + slot);
    if (done) continue;
    const int y = udiv(local, P.fd_nkx);
    const int k0 = (local - y * P.nkx) << P.lkx;
    const int nk = min(P.kx, hs - k0);
    cplx<T> *spec = reinterpret_cast<cplx<T> *>(S.spec) + (long long)y * hs + k0;
    // first stage: global memory to slots.  The slots a thread fills are those its own last
    // stage of the previous item read, so no barrier is needed before.
    const int total0 = (6 * X.m) << P.lkx;
    DIF_RADIX(X.r0,
_Pragma("unroll 1")
      for (int t = threadIdx.x; t < total0; t += blockDim.x) {
        const int col = t & kxm, r = t >> P.lkx;
        const int c = udiv(r, X.fd_m), n = r - c * X.m;
        cplx<T> v[R];
        const cplx<T> *src = spec + c * g.S + n * rowx + col;
        const long long step = X.m * rowx;
_Pragma("unroll")
        for (int q = 0; q < R; ++q) v[q] = col < nk ? src[q * step] : mk<T>((T)0, (T)0);
        dft<T, false, R>(v);
_Pragma("unroll")
        for (int q = 1; q < R; ++q) v[q] = cmul<T>(v[q], tw.ld(q * n));
        const SPtr<T> b = buf + c * P.cs + n * X.a + col;
_Pragma("unroll")
        for (int q = 0; q < R; ++q) b.st(q << P.lkx, v[q]);
      }
    )
    __syncthreads();
    if (X.ns == 3) difx_middle<T, false>(buf, P, tw);
    difx_last<T, false>(buf, P, nx, tw);
    // Gamma-hat over the slots (n', q_0, column): frequency q_0 + r_0 (q_1 + r_1 q_2) with
    // n' = q_1 r_2 + q_2
    const T ty = g.tany[y];
#pragma unroll 1
    for (int t = threadIdx.x; t < nx << P.lkx; t += blockDim.x) {
      const int col = t & kxm, r = t >> P.lkx;
      const int n = udiv(r, X.fd_r0), q0 = r - n * X.r0;
      int kap = n;
      if (X.ns == 3) {
        const int q1 = udiv(n, P.fd_r2);
        kap = q1 + X.r1 * (n - q1 * X.r2);
      }
      const int k = q0 + X.r0 * kap, kz = min(k0 + col, hs - 1);
      const SPtr<T> b = buf + n * X.a + (q0 << P.lkx) + col;
      cplx<T> m[6];
#pragma unroll
      for (int c = 0; c < 6; ++c) m[c] = b.ld(c * P.cs);
      if (k == 0 && y == 0 && kz == 0) {
#pragma unroll
        for (int c = 0; c < 6; ++c) m[c] = cscale<T>(m[c], (T)S.mask[c] * g.scale);
      } else if (2 * y == ny || 2 * kz == g.nz || 2 * k == nx) {
#pragma unroll
        for (int c = 0; c < 6; ++c) m[c] = mk<T>((T)0, (T)0);
      } else {
        dif_green<T>(g.tanx[k], ty, g.tanz[kz], g.scale, m);
      }
#pragma unroll
      for (int c = 0; c < 6; ++c) b.st(c * P.cs, m[c]);
    }
    __syncthreads();
    difx_last<T, true>(buf, P, nx, tw);
    if (X.ns == 3) difx_middle<T, true>(buf, P, tw);
    // last inverse stage: slots to global memory
    DIF_RADIX(X.r0,
_Pragma("unroll 1")
      for (int t = threadIdx.x; t < total0; t += blockDim.x) {
        const int col = t & kxm, r = t >> P.lkx;
        const int c = udiv(r, X.fd_m), n = r - c * X.m;
        const SPtr<T> b = buf + c * P.cs + n * X.a + col;
        cplx<T> v[R];
_Pragma("unroll")
        for (int q = 0; q < R; ++q) v[q] = b.ld(q << P.lkx);
        dft<T, true, R>(v);
        cplx<T> *dst = spec + c * g.S + n * rowx + col;
        const long long step = X.m * rowx;
        if (col < nk) {
_Pragma("unroll")
          for (int q = 0; q < R; ++q) dst[q * step] = v[q];
        }
      }
    )
  }
}

// ---- y pass of planes too large for a block -----------------------------------------------
//
// An item is (slot, component, x, tile of kx kz columns), transformed in place like the x
// pass's tiles, one component at a time: a tile's rows are then 128-byte runs where the x
// pass, which needs all six components of a frequency, can hold 32.  Both outer stages touch
// global memory from registers, so an element of a two-stage axis crosses shared memory twice
// (the Stockham pass: five times, in two buffers).  Bound by HBM: the spectrum in and out.
// 128 x 256 x 256: 132 us in FP64 (0.94 of the rate of a copy), 90 in float.
#define DIFY_THREADS 128
#define DIFY_MIN_BLOCKS(T) (sizeof(T) == 4 ? 7 : 4)

template <typename T, bool INV>
__global__ void __launch_bounds__(DIFY_THREADS, DIFY_MIN_BLOCKS(T))
    dify_kernel(Grid<T> g, DifXPlan P, const SlotDev<T> *__restrict__ tab, SlotList list, int kry) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const DifAxis &Y = P.x;
  const int ny = g.ny, hs = g.hs;
  pdl_begin();
  load_table<T>(reinterpret_cast<cplx<T> *>(smem_raw) + P.elems, g.twy, ny);
  const SPtr<T> buf{smem_u32(smem_raw)}, tw = buf + P.elems;
  const int per = 6 * g.nx * P.nkx;
  pdl_wait();
  const int n_items = list_items(list, per);
  const int kxm = P.kx - 1, total0 = Y.m << P.lkx;
  for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
    const int ks = udiv(item, P.fd_items);
    const int local = item - ks * per;
    const int slot = list.ids[ks];
    if (kry && slot_done(list.st + slot)) continue;
    const int cx = udiv(local, P.fd_nkx), c = udiv(cx, g.fd_nx), x = cx - c * g.nx;
    const int k0 = (local - cx * P.nkx) << P.lkx;
    const int nk = min(P.kx, hs - k0);
    cplx<T> *spec = reinterpret_cast<cplx<T> *>(tab[slot].spec) + c * g.S + (long long)x * ny * hs + k0;
    __syncthreads();  // table ready; the previous item is done with the buffer
    if constexpr (INV) {
      // first inverse stage: frequencies j + nb q from global memory to their slots
      DIF_RADIX(dif_last_radix(Y),
        const int nb = ny / R;
_Pragma("unroll 1")
        for (int t = threadIdx.x; t < nb << P.lkx; t += blockDim.x) {
          const int j = t >> P.lkx, col = t & kxm;
          const cplx<T> *src = spec + j * hs + col;
          const int step = nb * hs;
          cplx<T> v[R];
_Pragma("unroll")
          for (int q = 0; q < R; ++q) v[q] = col < nk ? src[q * step] : mk<T>((T)0, (T)0);
          dft<T, true, R>(v);
          const SPtr<T> b = buf + dif_last_base(Y, j) + col;
_Pragma("unroll")
          for (int q = 0; q < R; ++q)
            b.st(q * Y.a, q ? cmul<T>(v[q], dif_tw<T, true>(tw, q * j)) : v[q]);
        }
      )
    } else {
      DIF_RADIX(Y.r0,
_Pragma("unroll 1")
        for (int t = threadIdx.x; t < total0; t += blockDim.x) {
          const int col = t & kxm, n = t >> P.lkx;
          const cplx<T> *src = spec + n * hs + col;
          const int step = Y.m * hs;
          cplx<T> v[R];
_Pragma("unroll")
          for (int q = 0; q < R; ++q) v[q] = col < nk ? src[q * step] : mk<T>((T)0, (T)0);
          dft<T, false, R>(v);
          const SPtr<T> b = buf + n * Y.a + col;
_Pragma("unroll")
          for (int q = 0; q < R; ++q) b.st(q << P.lkx, q ? cmul<T>(v[q], tw.ld(q * n)) : v[q]);
        }
      )
    }
    __syncthreads();
    if (Y.ns == 3) difx_middle<T, INV, 1>(buf, P, tw);
    if constexpr (INV) {
      DIF_RADIX(Y.r0,
_Pragma("unroll 1")
        for (int t = threadIdx.x; t < total0; t += blockDim.x) {
          const int col = t & kxm, n = t >> P.lkx;
          const SPtr<T> b = buf + n * Y.a + col;
          cplx<T> v[R];
_Pragma("unroll")
          for (int q = 0; q < R; ++q) v[q] = b.ld(q << P.lkx);
          dft<T, true, R>(v);
          cplx<T> *dst = spec + n * hs + col;
          const int step = Y.m * hs;
          if (col < nk) {
_Pragma("unroll")
            for (int q = 0; q < R; ++q) dst[q * step] = v[q];
          }
        }
      )
    } else {
      DIF_RADIX(dif_last_radix(Y),
        const int nb = ny / R;
_Pragma("unroll 1")
        for (int t = threadIdx.x; t < nb << P.lkx; t += blockDim.x) {
          const int j = t >> P.lkx, col = t & kxm;
          const SPtr<T> b = buf + dif_last_base(Y, j) + col;
          cplx<T> v[R];
_Pragma("unroll")
          for (int q = 0; q < R; ++q) v[q] = b.ld(q * Y.a);
          dft<T, false, R>(v);
          cplx<T> *dst = spec + j * hs + col;
          const int step = nb * hs;
          if (col < nk) {
_Pragma("unroll")
            for (int q = 0; q < R; ++q) dst[q * step] = v[q];
          }
        }
      )
    }
  }
}

// ---- plane passes ------------------------------------------------------------------------
//
// An item is (x plane, component pair).  The pair's plane sits in one buffer of ny rows of
// ls slots; along z the slot of digits (n', q_0) is n' a + q_0 (a odd: conflict-free first
// stage), along y rows are q_0 m + n'.  A thread of the last forward z stage takes the
// butterflies of frequencies k and nz - k, splits them into the half spectra of the pair's two
// components, and stores column (0, k) in the slot of k and column (1, k) in that of nz - k
// (column (1, 0) in an extra slot), so the plane is transformed along y in the same buffer.
// The inverse joins them again in its first z stage; its rows come out in digit order, undone
// by a row table when they are written.

struct DifPlane {
  int ok, threads;
  int ls, elems;       // row stride and buffer elements
  int xslot;           // slot of column (1, 0)
  DifAxis z, y;
};

// Slot of frequency k after the forward stages, and of frequency k before the inverse ones.
__device__ __forceinline__ int dif_pos_fwd(const DifAxis &A, int k) {
  const int kap = udiv(k, A.fd_r0), q0 = k - kap * A.r0;
  int q1 = kap, q2 = 0;
  if (A.ns == 3) {
    q2 = kap / A.r1;
    q1 = kap - q2 * A.r1;
  }
  return (q1 * A.r2 + q2) * A.a + q0 * A.b;
}
__device__ __forceinline__ int dif_pos_inv(const DifAxis &A, int k) {
  const int q = udiv(k, A.fd_m);
  return (k - q * A.m) * A.a + q * A.b;
}

// Tables of a plane block: twiddles, the slots of the 2 hs half-spectrum columns, and (for
// the inverse) the y of each row.
template <typename T, bool INV> struct DifTables {
  SPtr<T> buf, twz, twy;
  SPtr16 col, row;
  __device__ __forceinline__ DifTables(unsigned char *raw, const Grid<T> &g, const DifPlane &P) {
    cplx<T> *tz = reinterpret_cast<cplx<T> *>(raw) + P.elems, *ty = tz + g.nz;
    unsigned short *cl = reinterpret_cast<unsigned short *>(ty + g.ny), *rw = cl + 2 * g.hs;
    buf.a = smem_u32(raw);
    twz.a = smem_u32(tz);
    twy.a = smem_u32(ty);
    col.a = smem_u32(cl);
    row.a = smem_u32(rw);
    load_table<T>(tz, g.twz, g.nz);
    load_table<T>(ty, g.twy, g.ny);
    for (int k = threadIdx.x; k < g.hs; k += blockDim.x) {
      cl[k] = (unsigned short)(INV ? dif_pos_inv(P.z, k) : dif_pos_fwd(P.z, k));
      const int kb = k == 0 ? 0 : g.nz - k;
      cl[g.hs + k] = (unsigned short)(k == 0 ? P.xslot : (INV ? dif_pos_inv(P.z, kb) : dif_pos_fwd(P.z, kb)));
    }
    if (INV)
      for (int y = threadIdx.x; y < g.ny; y += blockDim.x)
        // the row of digits (q_0, q_1, q_2) holds output y; a row is ls slots
        rw[udiv(dif_pos_fwd(P.y, y), P.y.fd_un)] = (unsigned short)y;
  }
  static __host__ __device__ size_t bytes(const DifPlane &P, int ny, int nz, int hs) {
    return ((size_t)P.elems + ny + nz) * sizeof(cplx<T>) + (size_t)(2 * hs + ny) * 2;
  }
};

// Stage 1 of a three-stage axis, in place: butterfly j = q_0 + r_0 n'' of a line.
template <typename T, bool INV>
__device__ __forceinline__ void dif_stage1(SPtr<T> line, const DifAxis &A, int j, SPtr<T> tw) {
  const int h = udiv(j, A.fd_r0), q0 = j - h * A.r0;
  const SPtr<T> b = line + h * A.a + q0 * A.b;
  const int step = A.r2 * A.a;
  DIF_RADIX8(A.r1,
    cplx<T> v[R];
_Pragma("unroll")
    for (int q = 0; q < R; ++q) v[q] = b.ld(q * step);
    dft<T, INV, R>(v);
_Pragma("unroll")
    for (int q = 1; q < R; ++q) v[q] = cmul<T>(v[q], dif_tw<T, INV>(tw, q * h * A.r0));
_Pragma("unroll")
    for (int q = 0; q < R; ++q) b.st(q * step, v[q]);
    )
}

// Stage 1 of every z line / of every half-spectrum column (three-stage axes).
template <typename T, bool INV>
__device__ __forceinline__ void dif_z_middle(const DifTables<T, INV> &tb, const DifPlane &P, int ny) {
  const int nb = P.z.r0 * P.z.r2;
#pragma unroll 1
  for (int t = threadIdx.x; t < ny * nb; t += blockDim.x) {
    const int y = udiv(t, P.z.fd_nb1);
    dif_stage1<T, INV>(tb.buf + y * P.ls, P.z, t - y * nb, tb.twz);
  }
  __syncthreads();
}
template <typename T, bool INV>
__device__ __forceinline__ void dif_y_middle(const DifTables<T, INV> &tb, const DifPlane &P,
                                             const Grid<T> &g) {
  const int nb = P.y.r0 * P.y.r2, w = 2 * g.hs;
#pragma unroll 1
  for (int t = threadIdx.x; t < w * nb; t += blockDim.x) {
    const int j = udiv(t, g.fd_2hs);
    dif_stage1<T, INV>(tb.buf + tb.col[t - j * w], P.y, j, tb.twy);
  }
  __syncthreads();
}

// What a plane pass reads: the planes of the caller's field, of tau (a Krylov iteration, which
// skips finished solves) or of the Newton correction, chosen at run time; or the residual's
// Sbar - sigma.  What it writes: planes likewise, or the residual's or re-projection's epilogue.
enum { DIF_PLANES = 0, DIF_RESIDUAL = 1, DIF_REPROJECT = 2 };
constexpr int dif_kind(int epi) {
  return epi == EPI_RESIDUAL ? DIF_RESIDUAL : (epi == EPI_REPROJECT ? DIF_REPROJECT : DIF_PLANES);
}

// tau of the component pair p at point v.
template <typename T, typename TF, int KIND>
__device__ __forceinline__ cplx<T> dif_pair(const SlotDev<TF> &S, const TF *s0, const TF *s1,
                                            long long v, int p) {
  if constexpr (KIND == DIF_RESIDUAL) {
    return mk<T>((T)S.sbar[2 * p] - (T)s0[v], (T)S.sbar[2 * p + 1] - (T)s1[v]);
  } else {
    return mk<T>((T)s0[v], (T)s1[v]);
  }
}

// 64 registers a thread in float (1024 threads an SM; the widest stage holds 32 registers of
// data), 128 in double.
#define DIF_PLANE_THREADS(T) (sizeof(T) == 4 ? 1024 : 512)

template <typename T, typename TF, int KIND>
__global__ void __launch_bounds__(DIF_PLANE_THREADS(T), 1)
    dif_zyfwd_kernel(Grid<T> g, DifPlane P, const SlotDev<TF> *__restrict__ tab, SlotList list,
                     ExtIO<TF> io, int pro) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(16) unsigned char sdesc[sizeof(SlotDev<TF>)];
  pdl_begin();
  const DifTables<T, false> tb(smem_raw, g, P);
  const SPtr<T> buf = tb.buf;
  const int ny = g.ny, nz = g.nz, hs = g.hs, ls = P.ls;
  const DifAxis &Z = P.z, &Y = P.y;
  const long long V = g.V;
  const int per = items_plane(g);
  pdl_wait();
  const int slot0 = list.ids[udiv(blockIdx.x, g.fd_it_plane)];
  const int n_items = list_items(list, per);
  int staged = -1;
  for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
    const int k = udiv(item, g.fd_it_plane);
    const int local = item - k * per;
    const int slot = item == (int)blockIdx.x ? slot0 : list.ids[k];
    const bool done = pro == PRO_TAU && slot_done(list.st + slot);
    const SlotDev<TF> &S = stage_slot<TF>(tab, slot, sdesc, staged);
    if (done) continue;
    const int x = udiv(local, g.fd_3);
    const int p = local - 3 * x;
    const TF *src;
    if constexpr (KIND == DIF_RESIDUAL)
      src = S.sig;
    else
      src = pro == PRO_TAU ? S.kr[6] : (pro == PRO_REPROJECT ? S.kr[5] : io.in);
    src += 2 * p * V + (long long)x * ny * nz;
    __syncthreads();  // tables ready; the previous item is done with the buffer
    DIF_RADIX(Z.r0,
_Pragma("unroll 1")
      for (int t = threadIdx.x; t < ny * Z.m; t += blockDim.x) {
        const int y = udiv(t, Z.fd_m), n = t - y * Z.m;
        const TF *s0 = src + (y * nz + n), *s1 = s0 + V;
        cplx<T> v[R];
_Pragma("unroll")
        for (int q = 0; q < R; ++q) v[q] = dif_pair<T, TF, KIND>(S, s0, s1, q * Z.m, p);
        dft<T, false, R>(v);
_Pragma("unroll")
        for (int q = 1; q < R; ++q) v[q] = cmul<T>(v[q], tb.twz.ld(q * n));
        const SPtr<T> b = buf + y * ls + n * Z.a;
_Pragma("unroll")
        for (int q = 0; q < R; ++q) b.st(q, v[q]);
      }
    )
    __syncthreads();
    if (Z.ns == 3) dif_z_middle<T, false>(tb, P, ny);
    // last z stage of frequencies j + nb q and their negatives, split into the two components
    DIF_RADIX8(dif_last_radix(Z),
      const int nb = nz / R, un = nb / 2 + 1;
_Pragma("unroll 1")
      for (int t = threadIdx.x; t < ny * un; t += blockDim.x) {
        const int y = udiv(t, Z.fd_un), u = t - y * un;
        const SPtr<T> row = buf + y * ls;
        const SPtr<T> b1 = row + dif_last_base(Z, u), b2 = row + dif_last_base(Z, u == 0 ? 0 : nb - u);
        cplx<T> v1[R], v2[R];
_Pragma("unroll")
        for (int q = 0; q < R; ++q) {
          v1[q] = b1.ld(q * Z.a);
          v2[q] = b2.ld(q * Z.a);
        }
        dft<T, false, R>(v1);
        dft<T, false, R>(v2);
        const bool self = u == 0 || 2 * u == nb;
_Pragma("unroll")
        for (int q = 0; q < R; ++q) {
          const cplx<T> Zk = v1[q], Zm = u == 0 ? v2[(R - q) % R] : v2[R - 1 - q];
          const cplx<T> A = mk<T>((T)0.5 * (Zk.x + Zm.x), (T)0.5 * (Zk.y - Zm.y));
          const cplx<T> B = mk<T>((T)0.5 * (Zk.y + Zm.y), (T)0.5 * (Zm.x - Zk.x));
          const int kf = u + nb * q;
          const int p2 = (u == 0 ? (R - q) % R : R - 1 - q) * Z.a;
          if (kf == 0) {
            b1.st(q * Z.a, A);
            row.st(P.xslot, B);
          } else if (2 * kf < nz) {
            b1.st(q * Z.a, A);
            b2.st(p2, B);
          } else if (2 * kf > nz && !self) {
            b2.st(p2, cconj<T>(A));
            b1.st(q * Z.a, cconj<T>(B));
          }
        }
      }
    )
    __syncthreads();
    DIF_RADIX(Y.r0,
_Pragma("unroll 1")
      for (int t = threadIdx.x; t < 2 * hs * Y.m; t += blockDim.x) {
        const int n = udiv(t, g.fd_2hs), c2 = t - n * 2 * hs;
        const SPtr<T> b = buf + n * ls + tb.col[c2];
        cplx<T> v[R];
_Pragma("unroll")
        for (int q = 0; q < R; ++q) v[q] = b.ld(q * Y.b);
        dft<T, false, R>(v);
_Pragma("unroll")
        for (int q = 1; q < R; ++q) v[q] = cmul<T>(v[q], tb.twy.ld(q * n));
_Pragma("unroll")
        for (int q = 0; q < R; ++q) b.st(q * Y.b, v[q]);
      }
    )
    __syncthreads();
    if (Y.ns == 3) dif_y_middle<T, false>(tb, P, g);
    cplx<T> *spec = reinterpret_cast<cplx<T> *>(S.spec) + 2 * p * g.S + (long long)x * ny * hs;
    DIF_RADIX(dif_last_radix(Y),
      const int nb = ny / R;
_Pragma("unroll 1")
      for (int t = threadIdx.x; t < 2 * hs * nb; t += blockDim.x) {
        const int j = udiv(t, g.fd_2hs), c2 = t - j * 2 * hs;
        const SPtr<T> b = buf + tb.col[c2] + dif_last_base(Y, j);
        cplx<T> v[R];
_Pragma("unroll")
        for (int q = 0; q < R; ++q) v[q] = b.ld(q * Y.a);
        dft<T, false, R>(v);
        cplx<T> *dst = spec + j * hs + (c2 < hs ? (long long)c2 : g.S + (c2 - hs));
        const int step = nb * hs;
_Pragma("unroll")
        for (int q = 0; q < R; ++q) dst[q * step] = v[q];
      }
    )
  }
}

template <typename T, typename TF, int KIND>
__global__ void __launch_bounds__(DIF_PLANE_THREADS(T), 1)
    dif_yzinv_kernel(Grid<T> g, DifPlane P, const SlotDev<TF> *__restrict__ tab, SlotList list,
                     ExtIO<TF> io, int epi) {
  constexpr int EPI = KIND == DIF_RESIDUAL ? EPI_RESIDUAL
                                           : (KIND == DIF_REPROJECT ? EPI_REPROJECT : EPI_STORE);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[32];
  __shared__ __align__(16) unsigned char sdesc[sizeof(SlotDev<TF>)];
  pdl_begin();
  const DifTables<T, true> tb(smem_raw, g, P);
  const SPtr<T> buf = tb.buf;
  const int ny = g.ny, nz = g.nz, hs = g.hs, ls = P.ls;
  const DifAxis &Z = P.z, &Y = P.y;
  const long long V = g.V;
  const int per = items_plane(g);
  pdl_wait();
  const int slot0 = list.ids[udiv(blockIdx.x, g.fd_it_plane)];
  const int n_items = list_items(list, per);
  int staged = -1;
  for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
    const int k = udiv(item, g.fd_it_plane);
    const int local = item - k * per;
    const int slot = item == (int)blockIdx.x ? slot0 : list.ids[k];
    const bool done = epi == EPI_PTAU && slot_done(list.st + slot);
    const SlotDev<TF> &S = stage_slot<TF>(tab, slot, sdesc, staged);
    if (done) continue;
    const int x = udiv(local, g.fd_3);
    const int p = local - 3 * x;
    const long long vbase = (long long)x * ny * nz;
    const cplx<T> *spec =
        reinterpret_cast<const cplx<T> *>(S.spec) + 2 * p * g.S + (long long)x * ny * hs;
    __syncthreads();  // tables ready; the previous item is done with the buffer
    DIF_RADIX(Y.r0,
_Pragma("unroll 1")
      for (int t = threadIdx.x; t < 2 * hs * Y.m; t += blockDim.x) {
        const int n = udiv(t, g.fd_2hs), c2 = t - n * 2 * hs;
        const cplx<T> *src = spec + n * hs + (c2 < hs ? (long long)c2 : g.S + (c2 - hs));
        const int step = Y.m * hs;
        cplx<T> v[R];
_Pragma("unroll")
        for (int q = 0; q < R; ++q) v[q] = src[q * step];
        dft<T, true, R>(v);
        const SPtr<T> b = buf + n * ls + tb.col[c2];
_Pragma("unroll")
        for (int q = 0; q < R; ++q)
          b.st(q * Y.b, q ? cmul<T>(v[q], dif_tw<T, true>(tb.twy, q * n)) : v[q]);
      }
    )
    __syncthreads();
    if (Y.ns == 3) dif_y_middle<T, true>(tb, P, g);
    DIF_RADIX(dif_last_radix(Y),
      const int nb = ny / R;
_Pragma("unroll 1")
      for (int t = threadIdx.x; t < 2 * hs * nb; t += blockDim.x) {
        const int j = udiv(t, g.fd_2hs), c2 = t - j * 2 * hs;
        const SPtr<T> b = buf + tb.col[c2] + dif_last_base(Y, j);
        cplx<T> v[R];
_Pragma("unroll")
        for (int q = 0; q < R; ++q) v[q] = b.ld(q * Y.a);
        dft<T, true, R>(v);
_Pragma("unroll")
        for (int q = 0; q < R; ++q) b.st(q * Y.a, v[q]);
      }
    )
    __syncthreads();
    // columns k of both components joined into frequencies k and nz - k of Z = A + iB
    // (Hermitian in z; the unstored Nyquist column is zero), first z stage of the butterflies
    // of frequencies n' + m q and their negatives
    DIF_RADIX8(Z.r0,
      const int m = Z.m, un = m / 2 + 1;
_Pragma("unroll 1")
      for (int t = threadIdx.x; t < ny * un; t += blockDim.x) {
        const int y = udiv(t, Z.fd_un), n = t - y * un, n2 = n == 0 ? 0 : m - n;
        const SPtr<T> row = buf + y * ls;
        const SPtr<T> b1 = row + n * Z.a, b2 = row + n2 * Z.a;
        cplx<T> v1[R], v2[R];
_Pragma("unroll")
        for (int q = 0; q < R; ++q) {
          const int kf = n + m * q;
          const cplx<T> c1 = b1.ld(q);
          const cplx<T> c2 = kf == 0 ? row.ld(P.xslot) : b2.ld(n == 0 ? (R - q) % R : R - 1 - q);
          const bool low = 2 * kf < nz, nyq = 2 * kf == nz;
          const cplx<T> A = low ? c1 : c2, B = low ? c2 : c1;
          const cplx<T> zl = mk<T>(A.x - B.y, A.y + B.x), zh = mk<T>(A.x + B.y, B.x - A.y);
          v1[q] = nyq ? mk<T>((T)0, (T)0) : (low ? zl : zh);
          v2[R - 1 - q] = nyq ? mk<T>((T)0, (T)0) : (low ? zh : zl);
        }
        dft<T, true, R>(v1);
_Pragma("unroll")
        for (int q = 0; q < R; ++q)
          b1.st(q, q ? cmul<T>(v1[q], dif_tw<T, true>(tb.twz, q * n)) : v1[q]);
        if (n != 0 && 2 * n != m) {
          dft<T, true, R>(v2);
_Pragma("unroll")
          for (int q = 0; q < R; ++q)
            b2.st(q, q ? cmul<T>(v2[q], dif_tw<T, true>(tb.twz, q * n2)) : v2[q]);
        }
      }
    )
    __syncthreads();
    if (Z.ns == 3) dif_z_middle<T, true>(tb, P, ny);
    const KRoles<TF> kr = kroles<TF>(S, 0);
    ExtIO<TF> dst = io;
    if (epi == EPI_PTAU) dst.out = kr.Y;
    double acc0 = 0.0, acc1 = 0.0, acc2 = 0.0;
    DIF_RADIX(dif_last_radix(Z),
      const int nb = nz / R;
_Pragma("unroll 1")
      for (int t = threadIdx.x; t < ny * nb; t += blockDim.x) {
        const int row = udiv(t, Z.fd_nb), j = t - row * nb;
        const SPtr<T> b = buf + row * ls + dif_last_base(Z, j);
        cplx<T> v[R];
_Pragma("unroll")
        for (int q = 0; q < R; ++q) v[q] = b.ld(q * Z.a);
        dft<T, true, R>(v);
        const long long v0 = vbase + (int)tb.row[row] * nz + j;
        if constexpr (KIND == DIF_REPROJECT) {
          /* one component at a time, all of its loads before its first store (each may alias
             the other as far as the compiler knows): 51 -> 32 us at 64^3 */
_Pragma("unroll")
          for (int c = 0; c < 2; ++c) {
            const long long i0 = (2 * p + c) * V + v0;
            double f[R];
_Pragma("unroll")
            for (int q = 0; q < R; ++q) {
              f[q] = S.eps[i0 + q * nb];
            }
_Pragma("unroll")
            for (int q = 0; q < R; ++q) kr.X[i0 + q * nb] = (TF)(c ? v[q].y : v[q].x);
_Pragma("unroll")
            for (int q = 0; q < R; ++q) S.eps[i0 + q * nb] = f[q] + (double)(c ? v[q].y : v[q].x);
_Pragma("unroll")
            for (int q = 0; q < R; ++q) f[q] = S.dfl[i0 + q * nb];
_Pragma("unroll")
            for (int q = 0; q < R; ++q) S.dfl[i0 + q * nb] = f[q] + (double)(c ? v[q].y : v[q].x);
          }
        } else {
_Pragma("unroll")
          for (int q = 0; q < R; ++q) {
            const T r[2] = {v[q].x, v[q].y};
            epilogue_point<T, TF, EPI, 2>(S, dst, kr, V, v0 + q * nb, 2 * p, r, acc0);
          }
        }
      }
    )
    finish_inverse<TF, EPI>(S, acc0, acc1, acc2, local, per, red);
  }
}

// ---- z pass of planes too large for a block -----------------------------------------------
//
// An item is (slot, tile of lz consecutive (x, y) lines, component pair).  The stages are the
// plane passes' z stages; the split (or join) of the pair's two half spectra happens in
// registers beside the access to global memory, so a line crosses shared memory twice a
// two-stage axis and four times a three-stage one.  Bound by the FP64 pipe and by latency (two
// blocks an SM) before HBM: 128 x 256 x 256 takes 192 us forward and 258 back in FP64, 103 and
// 114 in float, of 123 and 62 for the bytes alone; with eight lines a tile, which left half of
// the threads idle in the paired stage, 201 / 351 and 117 / 143.  The 256^3 FP64 projection:
// 3430 us with Stockham passes, 2771 with the register-tiled x pass, 2177 with all five.
#define DIFZ_THREADS 256
#define DIFZ_MIN_BLOCKS(T) (sizeof(T) == 4 ? 4 : 2)

struct DifZPlan {
  int ok, lz, ntiles;  // lines a tile, tiles
  DifPlane p;          // row layout and z axis (ls, elems, z)
  FastDiv fd_items;
};

// Stage 1 of the tile's lines (three-stage axes).
template <typename T, bool INV>
__device__ __forceinline__ void difz_middle(SPtr<T> buf, const DifPlane &P, SPtr<T> tw, int nl) {
  const int nb = P.z.r0 * P.z.r2;
#pragma unroll 1
  for (int t = threadIdx.x; t < nl * nb; t += blockDim.x) {
    const int l = udiv(t, P.z.fd_nb1);
    dif_stage1<T, INV>(buf + l * P.ls, P.z, t - l * nb, tw);
  }
  __syncthreads();
}

template <typename T>
__global__ void __launch_bounds__(DIFZ_THREADS, DIFZ_MIN_BLOCKS(T))
    dif_zfwd_kernel(Grid<T> g, DifZPlan P, const SlotDev<T> *__restrict__ tab, SlotList list,
                    ExtIO<T> io, int kry) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const DifAxis &Z = P.p.z;
  const int nz = g.nz, hs = g.hs, ls = P.p.ls;
  const long long V = g.V, lines = (long long)g.nx * g.ny;
  pdl_begin();
  load_table<T>(reinterpret_cast<cplx<T> *>(smem_raw) + P.p.elems, g.twz, nz);
  const SPtr<T> buf{smem_u32(smem_raw)}, tw = buf + P.p.elems;
  const int per = 3 * P.ntiles;
  pdl_wait();
  const int n_items = list_items(list, per);
  for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
    const int ks = udiv(item, P.fd_items);
    const int local = item - ks * per;
    const int slot = list.ids[ks];
    if (kry && slot_done(list.st + slot)) continue;
    const SlotDev<T> &S = tab[slot];
    const int tile = udiv(local, g.fd_3), p = local - 3 * tile;
    const long long line0 = (long long)tile * P.lz;
    const int nl = (int)min((long long)P.lz, lines - line0);
    const T *src = (kry ? S.kr[6] : io.in) + 2 * p * V + line0 * nz;
    __syncthreads();  // table ready; the previous item is done with the buffer
    DIF_RADIX(Z.r0,
_Pragma("unroll 1")
      for (int t = threadIdx.x; t < nl * Z.m; t += blockDim.x) {
        const int l = udiv(t, Z.fd_m), n = t - l * Z.m;
        const T *s0 = src + (l * nz + n), *s1 = s0 + V;
        cplx<T> v[R];
_Pragma("unroll")
        for (int q = 0; q < R; ++q) v[q] = mk<T>(s0[q * Z.m], s1[q * Z.m]);
        dft<T, false, R>(v);
        const SPtr<T> b = buf + l * ls + n * Z.a;
_Pragma("unroll")
        for (int q = 0; q < R; ++q) b.st(q, q ? cmul<T>(v[q], tw.ld(q * n)) : v[q]);
      }
    )
    __syncthreads();
    if (Z.ns == 3) difz_middle<T, false>(buf, P.p, tw, nl);
    // last stage of frequencies j + nb q and their negatives, split into the two components
    cplx<T> *spec = reinterpret_cast<cplx<T> *>(S.spec) + 2 * p * g.S + line0 * hs;
    DIF_RADIX8(dif_last_radix(Z),
      const int nb = nz / R, un = nb / 2 + 1;
_Pragma("unroll 1")
      for (int t = threadIdx.x; t < nl * un; t += blockDim.x) {
        const int l = udiv(t, Z.fd_un), u = t - l * un;
        const SPtr<T> row = buf + l * ls;
        const SPtr<T> b1 = row + dif_last_base(Z, u), b2 = row + dif_last_base(Z, u == 0 ? 0 : nb - u);
        cplx<T> v1[R], v2[R];
_Pragma("unroll")
        for (int q = 0; q < R; ++q) {
          v1[q] = b1.ld(q * Z.a);
          v2[q] = b2.ld(q * Z.a);
        }
        dft<T, false, R>(v1);
        dft<T, false, R>(v2);
        const bool self = u == 0 || 2 * u == nb;
        cplx<T> *dst = spec + l * hs;
_Pragma("unroll")
        for (int q = 0; q < R; ++q) {
          const cplx<T> Zk = v1[q], Zm = u == 0 ? v2[(R - q) % R] : v2[R - 1 - q];
          const cplx<T> A = mk<T>((T)0.5 * (Zk.x + Zm.x), (T)0.5 * (Zk.y - Zm.y));
          const cplx<T> B = mk<T>((T)0.5 * (Zk.y + Zm.y), (T)0.5 * (Zm.x - Zk.x));
          const int kf = u + nb * q;
          if (2 * kf < nz) {
            dst[kf] = A;
            dst[g.S + kf] = B;
          } else if (2 * kf > nz && !self) {
            dst[nz - kf] = cconj<T>(A);
            dst[g.S + nz - kf] = cconj<T>(B);
          }
        }
      }
    )
  }
}

template <typename T>
__global__ void __launch_bounds__(DIFZ_THREADS, DIFZ_MIN_BLOCKS(T))
    dif_zinv_kernel(Grid<T> g, DifZPlan P, const SlotDev<T> *__restrict__ tab, SlotList list,
                    ExtIO<T> io, int kry) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const DifAxis &Z = P.p.z;
  const int nz = g.nz, hs = g.hs, ls = P.p.ls;
  const long long V = g.V, lines = (long long)g.nx * g.ny;
  pdl_begin();
  load_table<T>(reinterpret_cast<cplx<T> *>(smem_raw) + P.p.elems, g.twz, nz);
  const SPtr<T> buf{smem_u32(smem_raw)}, tw = buf + P.p.elems;
  const int per = 3 * P.ntiles;
  pdl_wait();
  const int n_items = list_items(list, per);
  for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
    const int ks = udiv(item, P.fd_items);
    const int local = item - ks * per;
    const int slot = list.ids[ks];
    if (kry && slot_done(list.st + slot)) continue;
    const SlotDev<T> &S = tab[slot];
    const int tile = udiv(local, g.fd_3), p = local - 3 * tile;
    const long long line0 = (long long)tile * P.lz;
    const int nl = (int)min((long long)P.lz, lines - line0);
    const cplx<T> *spec = reinterpret_cast<const cplx<T> *>(S.spec) + 2 * p * g.S + line0 * hs;
    __syncthreads();  // table ready; the previous item is done with the buffer
    // frequencies n' + m q of Z = A + iB and their negatives from the stored halves
    // (Hermitian in z; the unstored Nyquist column is zero)
    DIF_RADIX8(Z.r0,
      const int m = Z.m, un = m / 2 + 1;
_Pragma("unroll 1")
      for (int t = threadIdx.x; t < nl * un; t += blockDim.x) {
        const int l = udiv(t, Z.fd_un), n = t - l * un, n2 = n == 0 ? 0 : m - n;
        const cplx<T> *src = spec + l * hs;
        cplx<T> v1[R], v2[R];
_Pragma("unroll")
        for (int q = 0; q < R; ++q) {
          const int kf = n + m * q;
          const bool low = 2 * kf < nz, nyq = 2 * kf == nz;
          const int kh = nyq ? 0 : (low ? kf : nz - kf);
          const cplx<T> A = src[kh], B = src[g.S + kh];
          const cplx<T> zl = mk<T>(A.x - B.y, A.y + B.x), zh = mk<T>(A.x + B.y, B.x - A.y);
          v1[q] = nyq ? mk<T>((T)0, (T)0) : (low ? zl : zh);
          v2[R - 1 - q] = nyq ? mk<T>((T)0, (T)0) : (low ? zh : zl);
        }
        dft<T, true, R>(v1);
        const SPtr<T> b1 = buf + l * ls + n * Z.a, b2 = buf + l * ls + n2 * Z.a;
_Pragma("unroll")
        for (int q = 0; q < R; ++q)
          b1.st(q, q ? cmul<T>(v1[q], dif_tw<T, true>(tw, q * n)) : v1[q]);
        if (n != 0 && 2 * n != m) {
          dft<T, true, R>(v2);
_Pragma("unroll")
          for (int q = 0; q < R; ++q)
            b2.st(q, q ? cmul<T>(v2[q], dif_tw<T, true>(tw, q * n2)) : v2[q]);
        }
      }
    )
    __syncthreads();
    if (Z.ns == 3) difz_middle<T, true>(buf, P.p, tw, nl);
    T *out = (kry ? S.kr[6] : io.out) + 2 * p * V + line0 * nz;
    DIF_RADIX(dif_last_radix(Z),
      const int nb = nz / R;
_Pragma("unroll 1")
      for (int t = threadIdx.x; t < nl * nb; t += blockDim.x) {
        const int l = udiv(t, Z.fd_nb), j = t - l * nb;
        const SPtr<T> b = buf + l * ls + dif_last_base(Z, j);
        cplx<T> v[R];
_Pragma("unroll")
        for (int q = 0; q < R; ++q) v[q] = b.ld(q * Z.a);
        dft<T, true, R>(v);
        T *d0 = out + (l * nz + j), *d1 = d0 + V;
_Pragma("unroll")
        for (int q = 0; q < R; ++q) {
          d0[q * nb] = v[q].x;
          d1[q * nb] = v[q].y;
        }
      }
    )
  }
}
