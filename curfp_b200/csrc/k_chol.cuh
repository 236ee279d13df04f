// k_chol.cuh — tile Cholesky of a lower-triangular matrix, with the rows below
// it, in one launch.
//
// The matrix is cut into 64 x 64 tiles that hand their results on through
// flags in L2, so the time is the chain of diagonal tiles.  (A recursion down
// to single-CTA 128-row tiles instead pays a chain of small launches: tile,
// inverses, solve, update, ~100 us per 128 columns.)
//
// Tickets (atomic counter) go out in the order: the first diagonal tile, then
// for each tile column c the tiles (c+1, c), (c+2, c), ...  A CTA waits only
// on smaller tickets, which are running or done, so no co-residency is needed
// and the scheme cannot deadlock.  CTA (i, c):
//   acc  = sum_{k<c} L_ik L_ck^T as the tiles are published,
//   X    = L_ic = (A_ic - acc) W_c^T once W_c = inv(L_cc) is published;
// and, when i = c + 1, it also factors the next diagonal tile,
//   S    = A_ii - sum_{k<c} L_ik L_ik^T - X X^T = L_ii L_ii^T,  W_i = inv(L_ii).
//
// The sums run on 8 x 8 register tiles (k_micro.cuh): 64 threads cover a tile,
// the CTA's groups of 64 split k and their partial sums meet once per CTA.  In
// a diagonal CTA half of the groups sum for X and half for S.
//
// The chain from one W to the next is ordered so that only what the next
// pivot needs is on it: X's upper 32 rows, S's upper-left quarter, its factor
// by warp 0 (factor32); meanwhile warp 1 follows column by column with the
// quarter's inverse and a further set of warps forms X's lower rows and the
// rest of S.
//
// Published tiles live in a packed workspace (k-major 64 x 64, element (a, b)
// at b * 64 + a), whatever the matrix's strides: consumers fetch them by
// 16-byte L2-only cp.async (cp.async.cg), and the matrix itself is read and
// written once, by the tile's owner.  Partial tiles are padded with the
// identity.
//
// The matrix is given as the logical lower blocks V11 (n1 x n1), V21
// (n2 x n1) and V22 (n2 x n2) of an RFP array.  The first nbf tile columns
// are factored: all of them, or only the first block's (then V21 becomes
// V21 L11^-T and V22 is not touched; a plain matrix has n2 = 0).
// Bound by the chain: a 64-column step takes 12.9 us in FP32 and 24.7 us in
// FP64 (n = 2000; 5.8 us of it the two 32-column factors, 180 cycles a column:
// one warp's instruction issue, which paired FMAs relieve and pairs of columns
// with their extra products do not), against ~50 us per 64 columns of the
// recursion with 128-row tiles.  RFP factorizations on B200, recursion -> this:
// n = 250 0.19 -> 0.055 ms, n = 4095 4.3 -> 1.02 ms (with one tensor-core
// update), FP64 n = 3000 4.8 -> 1.3 ms.
// Waits are bounded; a CTA that gives up (or whose diagonal tile has a
// non-positive pivot) publishes poisoned flags so that its dependents stop.
#pragma once
#include <climits>
#include <cstdint>
#include <type_traits>

#include "engine.h"
#include "k_micro.cuh"
#include "k_trsv.cuh"

namespace rfp {
namespace kchol {

using namespace kmicro;

constexpr int LDW = NB + 4;  // column stride of W in shared memory (conflict-free 16-byte columns)

// 64 threads per group; FP32 has 512 threads, FP64 256 (registers).
template <typename T> constexpr int threads() { return sizeof(T) == 4 ? 512 : 256; }
template <typename T> constexpr int groups() { return threads<T>() / 64; }
// two double-buffered operand tiles, T, S, W
template <typename T> constexpr int smem_bytes() { return (6 * TILE + NB * LDW) * (int)sizeof(T); }

template <typename T>
struct Args {
  ViewT<T> v11, v21, v22;
  int n1, n2, nb1, nb;  // orders, tiles of the first block, tiles in all
  int nbf;              // tile columns factored: nb, or nb1
  T* ws;                // published tiles (tile_index; W_i at (i, i))
  int* sync;            // [0] ticket, [1 + tile] flags (0 not ready, 1 ready, -1 poisoned);
                        // nullptr for a single CTA
  int* info;            // pivot failures (INT_MAX: none)
  int* err;             // wait timeouts
  int info_base;
};

// Index of published tile (i, k): packed lower triangle, then full rows of
// nbf tiles below the factored columns.
__host__ __device__ __forceinline__ int tile_index(int nbf, int i, int k) {
  return i < nbf ? i * (i + 1) / 2 + k : nbf * (nbf + 1) / 2 + (i - nbf) * nbf + k;
}
inline int64_t tile_count(int nb, int nbf) {
  return (int64_t)nbf * (nbf + 1) / 2 + (int64_t)(nb - nbf) * nbf;
}
// CTAs of a launch: the first diagonal tile and the tiles below the diagonal
// of the factored columns.
inline int cta_count(int nb, int nbf) {
  int t = 1;
  for (int c = 0; c < nbf; ++c) t += nb - 1 - c;
  return t;
}

template <typename T>
__device__ __forceinline__ void fetch_tile(T* s, const T* g) {
  constexpr int VW = 16 / (int)sizeof(T);
#pragma unroll
  for (int u = 0; u < TILE / VW / threads<T>(); ++u) {
    const int e = (threadIdx.x + threads<T>() * u) * VW;
    cp16(s + e, g + e);
  }
}
template <int COUNT>
__device__ __forceinline__ void bar_sync_id(int id) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(COUNT) : "memory");
}
template <int COUNT>
__device__ __forceinline__ void bar_arrive_id(int id) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(COUNT) : "memory");
}

// 1/sqrt(d): the hardware estimate r and one Newton step for y = x^-1/2 in
// the form r + r/2 (1 - d r^2), whose last rounding dominates its error.
__device__ __forceinline__ float rsqrt_newton(float d) {
  const float r = rsqrtf(d);
  return fmaf(0.5f * r, fmaf(-d * r, r, 1.0f), r);
}
__device__ __forceinline__ double rsqrt_newton(double d) {
  const double r = rsqrt(d);
  return fma(0.5 * r, fma(-d * r, r, 1.0), r);
}

// x_k += f l_k for K0 <= k < 32, two at a time in FP32 (one warp issues these
// alone, so their number is what counts).
template <int K0, typename T>
__device__ __forceinline__ void axpy(T (&x)[32], T f, const T (&l)[32]) {
  if constexpr (sizeof(T) == 4) {
    if constexpr (K0 < 32 && K0 % 2 == 1) x[K0] = fma(f, l[K0], x[K0]);
#pragma unroll
    for (int k = (K0 + 1) & ~1; k < 32; k += 2) fma2(x[k], x[k + 1], l[k], l[k + 1], f, f);
  } else {
#pragma unroll
    for (int k = K0; k < 32; ++k) x[k] = fma(f, l[k], x[k]);
  }
}
// The compile-time index of an unrolled loop.
template <int J, typename F>
__device__ __forceinline__ void each_column(F f) {
  if constexpr (J < 32) {
    f(std::integral_constant<int, J>{});
    each_column<J + 1>(f);
  }
}

// One warp, lane = row: Cholesky factor of a 32 x 32 block s (column-major,
// stride 64; lower triangle read, overwritten by the factor; garbage above
// the diagonal).  The chain of a column is: update the next column, its pivot
// by shuffle, rsqrt, scale.  The column goes to raw (32 x 32, column-major)
// unscaled: it comes back as 16-byte broadcast reads behind the rsqrt, and
// drives the inverse in another warp, which is let on every 8 columns
// (barriers bar0 .. bar0 + 3).  Returns 0, or 1 + the failing column.
template <typename T>
__device__ __forceinline__ int factor32(T* s, T* raw, int bar0) {
  const int lane = threadIdx.x & 31;
  T a[32];
#pragma unroll
  for (int k = 0; k < 32; ++k) a[k] = s[k * NB + lane];
  int fail = 0;
  raw[lane] = a[0];
  T d = __shfl_sync(0xffffffffu, a[0], 0);
  __syncwarp();
  each_column<0>([&](auto jc) {
    constexpr int j = decltype(jc)::value;
    // No branch on the pivot: straight-line code lets a column's updates fill
    // the next one's chain.  From a failed pivot on, r = 0 leaves everything
    // as it is.
    fail = fail == 0 && !(d > T(0)) ? j + 1 : fail;  // the same value in every lane
    const T r = fail ? T(0) : rsqrt_newton(d);
    T lk[32];
#pragma unroll
    for (int v4 = (j + 1) / 4; v4 < 8; ++v4)
      lds4(raw + j * 32 + 4 * v4, *reinterpret_cast<T(*)[4]>(lk + 4 * v4));
    const T l = a[j] * r, t = l * r, dj = d;
    if constexpr (j + 1 < 32) {
      a[j + 1] = fma(-t, lk[j + 1], a[j + 1]);
      d = __shfl_sync(0xffffffffu, a[j + 1], j + 1);
      raw[(j + 1) * 32 + lane] = a[j + 1];
      __syncwarp();
    }
    // the diagonal element: sqrt(d) = d r corrected by its residual
    a[j] = fail ? a[j] : (lane == j ? fma(T(0.5) * r, fma(-l, l, dj), l) : l);
    axpy<j + 2>(a, -t, lk);
    if ((j & 7) == 7) bar_arrive_id<64>(bar0 + (j >> 3));
  });
#pragma unroll
  for (int k = 0; k < 32; ++k) s[k * NB + lane] = a[k];
  return fail;
}
// The pivots whose reciprocal is a normal number.
template <typename T> struct Pivot;
template <> struct Pivot<float> { static constexpr float lo = 0x1p-126f, hi = 0x1p125f; };
template <> struct Pivot<double> { static constexpr double lo = 0x1p-1022, hi = 0x1p1021; };

// inverse32 for pivots of any size: 1 / d_j, infinite for a subnormal d_j, is
// never formed; 2^64 or 2^-64 of it goes to the column instead.
template <typename T>
__device__ __noinline__ void inverse32_any(T* w, const T* raw) {
  T* x = w + (threadIdx.x & 31) * LDW;
  for (int k = 0; k < 32; ++k) x[k] = k == (threadIdx.x & 31) ? T(1) : T(0);
  for (int j = 0; j < 32; ++j) {
    const T d = raw[j * 32 + j], r = rsqrt_newton(d), u = x[j] * r;
    const T s = d < T(1) ? T(0x1p64) : T(0x1p-64), v = u * (T(1) / s) * r;
    x[j] = u;
    for (int k = j + 1; k < 32; ++k) x[k] = fma(raw[j * 32 + k] * s, -v, x[k]);
  }
}
// The warp that follows factor32: lane = column of the inverse, written to w
// (column-major, stride LDW, zeros above the diagonal).  Column j of the
// factor is raw_j / sqrt(d_j), so x_j /= sqrt(d_j), then
// x_i -= raw_ij (x_j / sqrt(d_j)).  Returns whether a pivot asks for
// inverse32_any instead.
template <typename T>
__device__ __forceinline__ bool inverse32(T* w, const T* raw, int bar0) {
  const int lane = threadIdx.x & 31;
  T x[32];
#pragma unroll
  for (int k = 0; k < 32; ++k) x[k] = k == lane ? T(1) : T(0);
  bool any = false;
  each_column<0>([&](auto jc) {
    constexpr int j = decltype(jc)::value;
    if ((j & 7) == 0) bar_sync_id<64>(bar0 + (j >> 3));
    if (j == 24) {  // every pivot is there
      const T d = raw[lane * 33];
      any = __any_sync(0xffffffffu, !(d >= Pivot<T>::lo && d <= Pivot<T>::hi));
    }
    T lk[32];
#pragma unroll
    for (int v4 = j / 4; v4 < 8; ++v4)
      lds4(raw + j * 32 + 4 * v4, *reinterpret_cast<T(*)[4]>(lk + 4 * v4));
    const T r = rsqrt_newton(lk[j]);
    const T u = x[j] * r, v = u * r;
    x[j] = u;
    axpy<j + 1>(x, -v, lk);
  });
#pragma unroll
  for (int k = 0; k < 32; k += 4) {
    const T v[4] = {x[k], x[k + 1], x[k + 2], x[k + 3]};
    sts4(w + lane * LDW + k, v);
  }
  return any;
}

// Tile (row tile i, column tile j) of the matrix as a view and its extents.
template <typename T>
__device__ __forceinline__ ViewT<T> tile_view(const Args<T>& g, int i, int j, int& rows,
                                              int& cols) {
  const bool r2 = i >= g.nb1, c2 = j >= g.nb1;
  const int li = (r2 ? i - g.nb1 : i) * NB, lj = (c2 ? j - g.nb1 : j) * NB;
  rows = min(NB, (r2 ? g.n2 : g.n1) - li);
  cols = min(NB, (c2 ? g.n2 : g.n1) - lj);
  return sub(c2 ? g.v22 : (r2 ? g.v21 : g.v11), li, lj);
}

// Visits the tile's elements in groups of four rows of a column: group (b, q)
// holds rows 4q .. 4q + 3 of column b, one 16-byte shared-memory access.  For
// row-contiguous views a warp takes 8 columns x 4 groups (whole 32-byte
// sectors in memory, 8 banks apart in shared memory, where lanes along a row
// would all fall in one bank), else 16 groups x 2 columns.
template <typename T, typename F>
__device__ __forceinline__ void for_groups(bool rowcont, F f) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int NW = threads<T>() / 32;
#pragma unroll
  for (int u = 0; u < 32 / NW; ++u) {
    const int w = warp + NW * u;
    if (rowcont) f((w & 7) * 8 + (lane & 7), (w >> 3) * 4 + (lane >> 3));
    else f(w * 2 + (lane >> 4), lane & 15);
  }
}

// Matrix tile -> k-major shared tile, zeros (diag: identity) outside; of a
// diagonal tile only the lower triangle is read and zeros stand above it.
template <typename T>
__device__ __forceinline__ void load_matrix(T* s, ViewT<T> v, int rows, int cols, bool diag) {
  const bool rowcont = (v.cs == 1 || v.cs == -1) && !(v.rs == 1 || v.rs == -1);
  for_groups<T>(rowcont, [&](int b, int q) {
    T x[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int a = 4 * q + e;
      x[e] = diag && a == b ? T(1) : T(0);
      if (a < rows && b < cols && (!diag || a >= b))
        x[e] = __ldcg(v.p + (int64_t)a * v.rs + (int64_t)b * v.cs);
    }
    sts4(s + b * NB + 4 * q, x);
  });
}
template <typename T>
__device__ __forceinline__ void store_matrix(const T* s, ViewT<T> v, int rows, int cols,
                                             bool diag) {
  const bool rowcont = (v.cs == 1 || v.cs == -1) && !(v.rs == 1 || v.rs == -1);
  for_groups<T>(rowcont, [&](int b, int q) {
    T x[4];
    lds4(s + b * NB + 4 * q, x);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int a = 4 * q + e;
      if (a < rows && b < cols && (!diag || a >= b))
        v.p[(int64_t)a * v.rs + (int64_t)b * v.cs] = x[e];
    }
  });
}

// Both flags ready: 1; either poisoned: -1; else 0.
__device__ __forceinline__ int peek2(const int* f, const int* g) {
  const int a = ktrsv::ld_acquire(f), b = ktrsv::ld_acquire(g);
  return a < 0 || b < 0 ? -1 : (a > 0 && b > 0 ? 1 : 0);
}

template <typename T>
__global__ void __launch_bounds__(threads<T>(), 1) chol_wave(const Args<T> g) {
  extern __shared__ __align__(16) unsigned char chol_raw[];
  T* A0 = reinterpret_cast<T*>(chol_raw);  // L_ik, double-buffered
  T* B0 = A0 + 2 * TILE;                   // L_ck, double-buffered
  T* Ts = B0 + 2 * TILE;
  T* Ss = Ts + TILE;
  T* Ws = Ss + TILE;  // W_i, column stride LDW
  __shared__ int sh_ticket, sh_known[3], sh_state;
  __shared__ int2 sh_odd;  // 1 + a failing column of the diagonal tile, pivots out of range
  constexpr int THR = threads<T>(), G = groups<T>();
  const int tid = threadIdx.x, grp = tid >> 6, u = tid & 63;
  const int warp = tid >> 5, lane = tid & 31;
  constexpr int NW = THR / 32;
  if (tid == 0) {
    sh_ticket = g.sync ? atomicAdd(g.sync, 1) : 0;
    sh_odd = make_int2(0, 0);
  }
  const bool abort = g.info && *g.info != INT_MAX;
  __syncthreads();
  int* flags = g.sync + 1;
  auto tidx = [&](int r, int k) { return tile_index(g.nbf, r, k); };
  // ticket 0: diagonal tile 0; then column by column (c+1, c), (c+2, c), ...
  int c = -1, i = 0;
  if (sh_ticket > 0) {
    int rem = sh_ticket - 1;
    c = 0;
    while (rem >= g.nb - 1 - c) rem -= g.nb - 1 - c++;
    i = c + 1 + rem;
  }
  const bool diag = i == c + 1 && i < g.nbf;

  auto poison = [&]() {
    __syncthreads();
    if (tid == 0) {
      if (c >= 0) ktrsv::st_release(&flags[tidx(i, c)], -1);
      if (diag && g.sync) ktrsv::st_release(&flags[tidx(i, i)], -1);
    }
  };
  if (__syncthreads_or(abort)) return poison();  // a pivot failed earlier

  int xr = 0, xc = 0, sr = 0, scols = 0;
  ViewT<T> xv{}, sv{};
  if (c >= 0) {
    xv = tile_view(g, i, c, xr, xc);
    load_matrix(Ts, xv, xr, xc, false);
  }
  if (diag) {
    sv = tile_view(g, i, i, sr, scols);
    load_matrix(Ss, sv, sr, sr, true);
  }

  auto ready = [&](int k) { return peek2(&flags[tidx(i, k)], &flags[tidx(c, k)]); };
  // Warp 0: how far from k on the tiles are published (32 flags in one round
  // trip), into *known.
  auto scan = [&](int k, int* known) {
    const int st = k + lane < c ? ready(k + lane) : 0;
    const unsigned m = __ballot_sync(0xffffffffu, st > 0);
    if (lane == 0) *known = k + (m == 0xffffffffu ? 32 : __ffs(~m) - 1);
  };
  // Warp 0: waits for tile k, then scans on.
  auto wait2 = [&](int k, int* known) {
    if (lane == 0) {
      int st = ktrsv::wait_flag(&flags[tidx(i, k)], g.err);
      if (st > 0) st = ktrsv::wait_flag(&flags[tidx(c, k)], g.err);
      sh_state = st;
    }
    __syncwarp();
    scan(k, known);
  };
  auto fetch = [&](int k) {
    fetch_tile(A0 + (k & 1) * TILE, g.ws + (int64_t)tidx(i, k) * TILE);
    fetch_tile(B0 + (k & 1) * TILE, g.ws + (int64_t)tidx(c, k) * TILE);
  };

  if (c > 0) {
    T acc[8][8];
#pragma unroll
    for (int p = 0; p < 8; ++p)
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[p][q] = T(0);
    if (warp == 0) wait2(0, &sh_known[2]);
    __syncthreads();
    if (sh_state < 0) return poison();
    int known = sh_known[2];  // tiles k < known are published
    fetch(0);
    ktrsv::cp_commit();
    for (int k = 0; k < c; ++k) {
      const bool more = k + 1 < c, ask = more && k + 1 >= known;
      if (ask && warp == 0) scan(k + 1, &sh_known[k & 1]);
      ktrsv::cp_wait_all();
      __syncthreads();  // tile k landed; every thread is done with the other buffers
      if (ask) known = sh_known[k & 1];
      const bool now = more && k + 1 < known;
      if (now) fetch(k + 1);
      ktrsv::cp_commit();
      const T* Ak = A0 + (k & 1) * TILE;
      const T* Bk = B0 + (k & 1) * TILE;
      if (!diag) product8<NB, NB, NB / G>(acc, Ak, Bk, grp * (NB / G), u);
      else
        product8<NB, NB, 2 * NB / G>(acc, Ak, grp < G / 2 ? Bk : Ak, (grp % (G / 2)) * (2 * NB / G), u);
      if (more && !now) {
        if (warp == 0) wait2(k + 1, &sh_known[2]);
        __syncthreads();
        if (sh_state < 0) return poison();
        known = sh_known[2];
        fetch(k + 1);
        ktrsv::cp_commit();
      }
    }
    // T := A_ic - acc, S := A_ii - sum L_ik L_ik^T (both still ahead of W_c);
    // the partial sums meet in the operand buffers (4 tiles)
    __syncthreads();
    if constexpr (G == 8) {
      if (!diag) {
        if (grp >= 4) store8(A0 + (grp - 4) * TILE, acc, u);
        __syncthreads();
        if (grp < 4) {
          add8(acc, A0 + grp * TILE, u);
          store8(A0 + grp * TILE, acc, u);
        }
        __syncthreads();
        subtract<4, THR>(Ts, A0);
      } else {
        if (grp < 4) store8(A0 + grp * TILE, acc, u);
        __syncthreads();
        subtract<4, THR>(Ts, A0);
        __syncthreads();
        if (grp >= 4) store8(A0 + (grp - 4) * TILE, acc, u);
        __syncthreads();
        subtract<4, THR>(Ss, A0);
      }
    } else {
      store8(A0 + grp * TILE, acc, u);
      __syncthreads();
      if (!diag) {
        subtract<4, THR>(Ts, A0);
      } else {
        subtract<2, THR>(Ts, A0);
        subtract<2, THR>(Ss, A0 + 2 * TILE);
      }
    }
  }

  T* Xs = A0;                // L_ic, k-major
  T* Wc = A0 + TILE;         // W_c
  T* red = B0;               // partial sums of the chain's products
  T* Lb = B0 + TILE;         // L10, column-major, stride 32
  T* Pb = Lb + 32 * 32;      // L10 inv(D0), column-major, stride 36
  T* raw = Pb + 32 * 36;     // factor32's unscaled columns
  T* out = g.ws + (c >= 0 ? (int64_t)tidx(i, c) * TILE : 0);
  if (c >= 0) {
    if (tid == 0) sh_state = ktrsv::wait_flag(&flags[tidx(c, c)], g.err);
    __syncthreads();
    if (sh_state < 0) return poison();
    fetch_tile(Wc, g.ws + (int64_t)tidx(c, c) * TILE);
    ktrsv::cp_commit();
    ktrsv::cp_wait_all();
    __syncthreads();
    // X = T W_c^T, rows 0-31 (diagonal CTAs) or all rows: 4 x 4 per thread,
    // groups of threads split k (W_c(c, k) = 0 for k > c)
    T o[4][4];
    if (!diag) {
      constexpr int XG = THR / 256, KX = NB / XG;
      const int xg = tid >> 8, v = tid & 255, tr = v & 15, tc = v >> 4;
      product4<NB, NB>(o, Ts, Wc, xg * KX, min(xg * KX + KX, tc * 4 + 4), tr, tc);
      reduce4<XG, 256, 1>(o, red, xg, v);
      if (xg == 0) {
        put4<NB, false>(Xs, o, tr, tc);
        put4<NB, false>(out, o, tr, tc);
      }
      __syncthreads();
      if (tid == 0) ktrsv::st_release(&flags[tidx(i, c)], 1);
      store_matrix(Xs, xv, xr, xc, false);
      return;
    }
    {
      constexpr int XG = THR / 128, KX = NB / XG;
      const int xg = tid >> 7, v = tid & 127, tr = v & 7, tc = v >> 3;
      product4<NB, NB>(o, Ts, Wc, xg * KX, min(xg * KX + KX, tc * 4 + 4), tr, tc);
      reduce4<XG, 128, 1>(o, red, xg, v);
      if (xg == 0) {
        put4<NB, false>(Xs, o, tr, tc);
        put4<NB, false>(out, o, tr, tc);
      }
    }
    __syncthreads();
    // S00 -= X0 X0^T
    {
      constexpr int SG = THR / 64, KS = NB / SG;
      const int tr = u & 7, tc = u >> 3;
      product4<NB, NB>(o, Xs, Xs, grp * KS, grp * KS + KS, tr, tc);
      reduce4<SG, 64, 1>(o, red, grp, u);
      if (grp == 0) put4<NB, true>(Ss, o, tr, tc);
    }
  }
  __syncthreads();

  // Diagonal tile by 32 x 32 quarters: D0 and its inverse by warps 0 and 1,
  // while the last quarter of the warps on the SMSPs that hold neither form
  // X's lower rows and S10 (FP64 S11 too).
  constexpr int SH = THR / 2;  // threads of the shadow work: warps w with w % 4 >= 2
  // In FP32 the shadow work is the longer side, so S11's product with X goes
  // beside L10 (n = 2000: 414 against 440 us); in FP64 the factor is longer and
  // both ways take the same time, so its order stays.
  constexpr bool kBeside = sizeof(T) == 4;
  // A tile of up to 32 rows has no second half: zeros and the identity in W.
  const bool half = sr <= 32;
  const bool shadow = (warp & 3) >= 2;
  int fail = 0;  // 1 + the failing column
  const int st = ((warp >> 2) * 2 + (warp & 1)) * 32 + lane;
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {  // one copy of the code (instruction cache)
    if (warp == 0) {
      const int f = factor32(Ss + h * (32 * NB + 32), raw, 2 + 4 * h);
      // (an infinite last pivot makes the padding's NaN: no failure)
      if (lane == 0 && f && 32 * h + f <= sr) sh_odd.x = 32 * h + f;
    } else if (warp == 1) {
      const bool any = inverse32(Ws + h * (32 * LDW + 32), raw, 2 + 4 * h);
      if (lane == 0) sh_odd.y = any;
    } else if (h == 0 && shadow) {
      if (c >= 0) {
        T o[4][4];
        {
          constexpr int XG = SH / 128, KX = NB / XG;
          const int xg = st >> 7, v = st & 127, tr = v & 7, tc = v >> 3;
          product4<NB, NB>(o, Ts + 32, Wc, xg * KX, min(xg * KX + KX, tc * 4 + 4), tr, tc);
          reduce4<XG, 128, 10>(o, red, xg, v);
          if (xg == 0) {
            put4<NB, false>(Xs + 32, o, tr, tc);
            put4<NB, false>(out + 32, o, tr, tc);
          }
        }
        bar_sync<10, SH>();
        if constexpr (kBeside) {
          // S10 -= X1 X0^T (S11's share follows beside L10)
          constexpr int SG = SH / 64, KS = NB / SG;
          const int sg = st >> 6, v = st & 63, tr = v & 7, tc = v >> 3;
          product4<NB, NB>(o, Xs + 32, Xs, sg * KS, sg * KS + KS, tr, tc);
          reduce4<SG, 64, 10>(o, red, sg, v);
          if (sg == 0) put4<NB, true>(Ss + 32, o, tr, tc);
        } else {
          // S10 -= X1 X0^T and S11 -= X1 X1^T, 64 threads each
          const int v = st & 63, q11 = st >> 6, tr = v & 7, tc = v >> 3;
          product4<NB, NB>(o, Xs + 32, Xs + 32 * q11, 0, NB, tr, tc);
          put4<NB, true>(Ss + 32 * q11 * NB + 32, o, tr, tc);
        }
        if (st == SH - 1) ktrsv::st_release(&flags[tidx(i, c)], 1);  // X, ordered by the barriers
      }
      for (int e = st; e < 32 * 32; e += SH) Ws[(32 + (e >> 5)) * LDW + (e & 31)] = T(0);
    } else if (h == 1 && shadow) {
      // off the chain: L10 into S's lower-left quarter, P = L10 inv(D0)
      for (int cc = st >> 5; cc < 32; cc += SH / 32) {
        Ss[cc * NB + 32 + lane] = Lb[cc * 32 + lane];
        T o = T(0);
#pragma unroll 4
        for (int k = 0; k < 32; k += 4) {
          T b[4];
          lds4(Ws + cc * LDW + k, b);
#pragma unroll
          for (int q = 0; q < 4; ++q) o = fma(Lb[(k + q) * 32 + lane], b[q], o);
        }
        Pb[cc * 36 + lane] = o;
      }
    }
    __syncthreads();
    const int2 odd = sh_odd;
    fail = odd.x;
    if (odd.y) {
      if (warp == 1) inverse32_any(Ws + h * (32 * LDW + 32), raw);
      __syncthreads();
    }
    if (fail || h == 1 || half) break;
    // Half of the groups: L10 = S10 inv(D0)^T; with kBeside the others
    // S11 -= X1 X1^T.  Then S11 -= L10 L10^T.
    T o[4][4];
    const int tr = u & 7, tc = u >> 3;
    constexpr int HG = G / 2, KL = 32 / HG, KX = NB / HG;
    if (grp < HG) {
      product4<NB, LDW>(o, Ss + 32, Ws, grp * KL, min(grp * KL + KL, tc * 4 + 4), tr, tc);
      reduce4<HG, 64, 1>(o, red, grp, u);
      if (grp == 0) put4<32, false>(Lb, o, tr, tc);
    } else if (kBeside && c >= 0) {
      const int xg = grp - HG;
      product4<NB, NB>(o, Xs + 32, Xs + 32, xg * KX, xg * KX + KX, tr, tc);
      reduce4<HG, 64, 11>(o, Wc, xg, u);  // W_c has served
      if (xg == 0) put4<NB, true>(Ss + 32 * NB + 32, o, tr, tc);
    }
    __syncthreads();
    if (grp < HG) {
      product4<32, 32>(o, Lb, Lb, grp * KL, grp * KL + KL, tr, tc);
      reduce4<HG, 64, 1>(o, red, grp, u);
      if (grp == 0) put4<NB, true>(Ss + 32 * NB + 32, o, tr, tc);
    }
    __syncthreads();
  }
  if (half) {
    for (int e = tid; e < 32 * 64; e += THR) {
      const int cc = e & 63, r = 32 + (e >> 6);
      Ws[cc * LDW + r] = cc == r ? T(1) : T(0);
    }
    __syncthreads();
  }
  if (!fail) {
    // W10 = -inv(D1) P
    for (int c0 = half ? 32 : warp * 2; c0 < 32; c0 += NW * 2) {
      T o[2] = {T(0), T(0)};
#pragma unroll
      for (int k = 0; k < 32; k += 4) {
        T p0[4], p1[4];
        lds4(Pb + c0 * 36 + k, p0);
        lds4(Pb + (c0 + 1) * 36 + k, p1);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const T a = Ws[(32 + k + q) * LDW + 32 + lane];
          o[0] = fma(-a, p0[q], o[0]);
          o[1] = fma(-a, p1[q], o[1]);
        }
      }
      Ws[c0 * LDW + 32 + lane] = o[0];
      Ws[(c0 + 1) * LDW + 32 + lane] = o[1];
    }
    __syncthreads();
    T* wout = g.ws + (int64_t)tidx(i, i) * TILE;
#pragma unroll
    for (int w = 0; w < TILE / 4 / THR; ++w) {
      const int e = tid + THR * w;
      T v[4];
      lds4(Ws + (e >> 4) * LDW + (e & 15) * 4, v);
      sts4(wout + e * 4, v);
    }
    __syncthreads();
    if (tid == 0 && g.sync) ktrsv::st_release(&flags[tidx(i, i)], 1);
  } else if (tid == 0) {
    const int col0 = i >= g.nb1 ? g.n1 + (i - g.nb1) * NB : i * NB;
    atomicMin(g.info, g.info_base + col0 + fail);
    if (g.sync) ktrsv::st_release(&flags[tidx(i, i)], -1);
  }
  if (c >= 0) store_matrix(Xs, xv, xr, xc, false);
  store_matrix(Ss, sv, sr, sr, true);
}

}  // namespace kchol
}  // namespace rfp
