// k_tri.cuh — inverse of a lower triangular block, and solves with many
// right-hand sides (solve_tiles), by waves of 64 x 64 tiles.
//
// M = L^-1 in one launch (and one that stores it): tickets in row order, so a
// CTA waits only on smaller tickets and no co-residency is needed.  CTA (i, c),
// c <= i:
//   M_ic = W_i (I_ic - sum_{c<=k<i} L_ik M_kc),   W_i = inv(L_ii).
// The term k = c, which holds M's dominant diagonal tile, is subtracted by
// itself: a running sum that starts with it rounds every later term against it
// (inverse at n = 2000: error 2.0e-7 so, 1.7e-7 apart, at 1% of the time).
// Other CTAs read L throughout, so the result stays in the published tiles
// until store_inverse writes it over L.
//
// The sums run on 8 x 8 register tiles (k_micro.cuh): four groups of 64
// threads split k, two CTAs per SM in FP32.  Tiles are published row-major
// (element (a, b) at a * 64 + b) in a packed workspace and fetched by 16-byte
// L2-only cp.async.
//
// Bound by the chain of block rows: n = 1536 takes 0.14 ms, where the
// recursion down to 64-row tiles took ~100 launches of ~14 us.
// Waits are bounded; a CTA that gives up publishes a poisoned flag (-1).
#pragma once
#include <climits>
#include <cstdint>

#include "engine.h"
#include "k_micro.cuh"
#include "k_trsv.cuh"

namespace rfp {
namespace ktri {

using namespace kmicro;

constexpr int THR = 256, G = THR / 64;
constexpr int LDL = ktrsv::LDL;  // column stride of L tiles and row stride of T
template <typename T>
constexpr int smem_bytes() {
  // L double-buffered | X double-buffered (both: the partial sums) | W | T
  return (2 * NB * LDL + 2 * TILE + TILE + NB * LDL) * (int)sizeof(T);
}

template <typename T>
struct Args {
  ViewT<T> L;
  int n;
  const T* W;  // kInvStride elements per block row, W_i first (column-major)
  T* ws;       // published tiles
  int* sync;   // [0] ticket, [1 + tile] flags
  int* err;
  const int* abort_flag;
};

// Row i holds the tiles (i, 0) .. (i, i).
__device__ __forceinline__ int tile_at(int i, int c) { return i * (i + 1) / 2 + c; }
__device__ __forceinline__ void tile_of(int t, int& i, int& c) {
  i = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
  while (tile_at(i + 1, 0) <= t) ++i;
  while (tile_at(i, 0) > t) --i;
  c = t - tile_at(i, 0);
}

template <typename T>
__global__ void __launch_bounds__(THR, sizeof(T) == 4 ? 2 : 1) inverse_wave(const Args<T> g) {
  if (g.abort_flag && *g.abort_flag != INT_MAX) return;
  extern __shared__ __align__(16) unsigned char tri_raw[];
  T* Ls = reinterpret_cast<T*>(tri_raw);
  T* Xs = Ls + 2 * NB * LDL;
  T* Ws = Xs + 2 * TILE;
  T* Ts = Ws + TILE;
  __shared__ int sh_ticket, sh_known[3], sh_state;
  const int tid = threadIdx.x, grp = tid >> 6, u = tid & 63;
  if (tid == 0) sh_ticket = atomicAdd(g.sync, 1);
  __syncthreads();
  int* flags = g.sync + 1;
  int i, c;
  tile_of(sh_ticket, i, c);
  const int rows = min(NB, g.n - i * NB);
  constexpr int VW = 16 / (int)sizeof(T);

  auto load_l = [&](int k) {
    ktrsv::load_tile<LDL>(Ls + ((k - c) & 1) * NB * LDL, sub(g.L, (int64_t)i * NB, (int64_t)k * NB),
                          rows, NB);
  };
  auto load_x = [&](int k) {
    T* s = Xs + ((k - c) & 1) * TILE;
    const T* x = g.ws + (int64_t)tile_at(k, c) * TILE;
#pragma unroll
    for (int w = 0; w < TILE / VW / THR; ++w) {
      const int e = (tid + THR * w) * VW;
      cp16(s + e, x + e);
    }
  };
  auto flag = [&](int k) { return &flags[tile_at(k, c)]; };
  const int warp = tid >> 5, lane = tid & 31;
  // Warp 0: how far from k on the column's tiles are published (32 flags in
  // one round trip), into *known; and the same after waiting for tile k.
  auto scan = [&](int k, int* known) {
    const int st = k + lane < i ? ktrsv::ld_acquire(flag(k + lane)) : 0;
    const unsigned m = __ballot_sync(0xffffffffu, st > 0);
    if (lane == 0) *known = k + (m == 0xffffffffu ? 32 : __ffs(~m) - 1);
  };
  auto wait = [&](int k, int* known) {
    if (lane == 0) sh_state = ktrsv::wait_flag(flag(k), g.err);
    __syncwarp();
    scan(k, known);
  };
  auto poison = [&]() {
    ktrsv::cp_wait_all();
    __syncthreads();
    if (tid == 0) ktrsv::st_release(flag(i), -1);
  };

  // What depends on no other CTA: W_i, I_ic, the first L tile.
  {
    const T* w = g.W + (int64_t)i * kInvStride;
#pragma unroll
    for (int q = 0; q < TILE / VW / THR; ++q) {
      const int e = (tid + THR * q) * VW;
      cp16(Ws + e, w + e);
    }
  }
#pragma unroll 4
  for (int q = 0; q < TILE / THR; ++q) {
    const int e = tid + THR * q, a = e / NB, b = e % NB;
    Ts[a * LDL + b] = i == c && a == b ? T(1) : T(0);
  }
  if (i > c) {
    load_l(c);
    if (warp == 0) wait(c, &sh_known[2]);
    __syncthreads();
    if (sh_state < 0) return poison();
    int known = sh_known[2];  // tiles k < known are published
    load_x(c);
    ktrsv::cp_commit();
    T acc[8][8];
#pragma unroll
    for (int p = 0; p < 8; ++p)
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[p][q] = T(0);
    for (int k = c; k < i; ++k) {
      const bool more = k + 1 < i, ask = more && k + 1 >= known;
      const int par = (k - c) & 1;
      if (ask && warp == 0) scan(k + 1, &sh_known[par]);
      ktrsv::cp_wait_all();
      __syncthreads();  // tile k landed; every thread is done with the other buffers
      if (ask) known = sh_known[par];
      const bool ready = more && k + 1 < known;
      if (more) load_l(k + 1);
      if (ready) load_x(k + 1);
      ktrsv::cp_commit();
      // rows of the register tile: M's columns, columns: L's rows
      if (k == c) {  // the dominant term goes to T by itself
        const int tr = tid & 15, tc = tid >> 4;
        T s[4][4];
        product4<NB, LDL>(s, Xs, Ls, 0, NB / 4, tr, tc);
#pragma unroll 1
        for (int q = 1; q < 4; ++q) {
          T o[4][4];
          product4<NB, LDL>(o, Xs, Ls, q * (NB / 4), (q + 1) * (NB / 4), tr, tc);
#pragma unroll
          for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) s[a][b] += o[a][b];
        }
        put4<LDL, true>(Ts, s, tr, tc);
      } else {
        product8<NB, LDL, NB / G>(acc, Xs + par * TILE, Ls + par * NB * LDL, grp * (NB / G), u);
      }
      if (more && !ready) {
        if (warp == 0) wait(k + 1, &sh_known[2]);
        __syncthreads();
        if (sh_state < 0) return poison();
        known = sh_known[2];
        load_x(k + 1);
        ktrsv::cp_commit();
      }
    }
    // T -= the groups' partial sums, which meet in the operand buffers
    if (i > c + 1) {
      __syncthreads();
      store8(Ls + grp * TILE, acc, u);
      __syncthreads();
#pragma unroll
      for (int w = 0; w < TILE / 4 / THR; ++w) {
        const int e = (tid + THR * w) * 4;
        T* t = Ts + (e / NB) * LDL + e % NB;
        T s[4], v[4];
        lds4(Ls + e, s);
#pragma unroll
        for (int q = 1; q < G; ++q) {
          lds4(Ls + q * TILE + e, v);
#pragma unroll
          for (int r = 0; r < 4; ++r) s[r] += v[r];
        }
        lds4(t, v);
#pragma unroll
        for (int r = 0; r < 4; ++r) v[r] -= s[r];
        sts4(t, v);
      }
    }
  }
  ktrsv::cp_commit();
  ktrsv::cp_wait_all();
  __syncthreads();
  // M = W_i T: W_i(a, k) = 0 for k > a
  {
    T o[4][4];
    const int tr = tid & 15, tc = tid >> 4;
    product4<LDL, NB>(o, Ts, Ws, 0, tc * 4 + 4, tr, tc);
    put4<NB, false>(g.ws + (int64_t)tile_at(i, c) * TILE, o, tr, tc);
  }
  __syncthreads();
  if (tid == 0) ktrsv::st_release(flag(i), 1);
}

// L X = alpha B (B n x m view, X over B) by a wave of 64 x 64 tiles: CTA (i, c),
// tickets in row order,
//   X_ic = W_i (alpha B_ic - sum_{k<i} L_ik X_kc),
// for the many right-hand sides of the recursion's leaves, where throughput
// counts and not the chain: 8 x 8 register products, two CTAs per SM, L packed
// beforehand (pack_lower) and X published in the workspace so that both are
// fetched 16 bytes at a time.  The products' shared-memory reads take half
// of the time, the CTAs' starts, reductions and stores the rest.  512 rows and 16384 / 8192 / 4096 columns take 148 / 91 / 79 us
// with the packing; with 4-byte copies of L from the matrix 172 / 100 / 81 us;
// ktrsv::trsm_wave (4 x 4 register products) 208 / 118 / 88 us.
template <typename T>
struct SolveArgs {
  ViewT<T> B;
  const T* Lp;  // pack_lower's tiles
  int n, m, nblk, nchunk;
  T alpha;
  const T* W;
  T* ws;
  int* sync;  // [0] ticket, [1 + i * nchunk + c] flags
  int* err;
  const int* abort_flag;
};

// The tiles (i, k), k < i, of L, k-major, at tile_at(i - 1, k) of ws.
template <typename T>
__global__ void __launch_bounds__(THR) pack_lower(ViewT<T> L, int n, T* ws,
                                                  const int* abort_flag) {
  if (abort_flag && *abort_flag != INT_MAX) return;
  __shared__ T s[NB * (NB + 1)];
  int i, k;
  tile_of((int)blockIdx.x, i, k);
  const int rows = min(NB, n - (i + 1) * NB);
  ktrsv::load_tile<NB + 1>(s, sub(L, (int64_t)(i + 1) * NB, (int64_t)k * NB), rows, NB);
  ktrsv::cp_commit();
  ktrsv::cp_wait_all();
  __syncthreads();
#pragma unroll 4
  for (int q = 0; q < TILE / THR; ++q) {
    const int e = threadIdx.x + THR * q;
    ws[(int64_t)blockIdx.x * TILE + e] = s[(e / NB) * (NB + 1) + e % NB];
  }
}

template <typename T>
__global__ void __launch_bounds__(THR, sizeof(T) == 4 ? 2 : 1) solve_tiles(const SolveArgs<T> g) {
  if (g.abort_flag && *g.abort_flag != INT_MAX) return;
  extern __shared__ __align__(16) unsigned char tri_raw[];
  T* Ls = reinterpret_cast<T*>(tri_raw);
  T* Xs = Ls + 2 * NB * LDL;
  T* Ws = Xs + 2 * TILE;
  T* Ts = Ws + TILE;
  __shared__ int sh_ticket, sh_state[2];  // tile k's state at k & 1
  const int tid = threadIdx.x, grp = tid >> 6, u = tid & 63;
  if (tid == 0) sh_ticket = atomicAdd(g.sync, 1);
  __syncthreads();
  const int i = sh_ticket / g.nchunk, c = sh_ticket % g.nchunk;
  const int rows = min(NB, g.n - i * NB), cols = min(NB, g.m - c * NB);
  int* const flags = g.sync + 1 + c;  // tile (k, c) at k * nchunk
  T* const xs = g.ws + (int64_t)c * TILE;
  constexpr int VW = 16 / (int)sizeof(T);

  auto load_l = [&](int k) {
    T* s = Ls + (k & 1) * NB * LDL;
    const T* l = g.Lp + (int64_t)tile_at(i - 1, k) * TILE;
#pragma unroll
    for (int w = 0; w < TILE / VW / THR; ++w) {
      const int e = (tid + THR * w) * VW;
      cp16(s + (e / NB) * LDL + e % NB, l + e);
    }
  };
  auto load_x = [&](int k) {
    T* s = Xs + (k & 1) * TILE;
    const T* x = xs + (int64_t)k * g.nchunk * TILE;
#pragma unroll
    for (int w = 0; w < TILE / VW / THR; ++w) {
      const int e = (tid + THR * w) * VW;
      cp16(s + e, x + e);
    }
  };
  // Thread 0 waits for tile k; the block barrier that follows tells the rest.
  auto wait = [&](int k) {
    if (tid == 0) sh_state[k & 1] = ktrsv::wait_flag(&flags[(int64_t)k * g.nchunk], g.err);
  };

  if (i > 0) load_l(0);
  {
    const T* w = g.W + (int64_t)i * kInvStride;
#pragma unroll
    for (int q = 0; q < TILE / VW / THR; ++q) {
      const int e = (tid + THR * q) * VW;
      cp16(Ws + e, w + e);
    }
  }
  // T = alpha B_ic, read along B's contiguous index
  const ViewT<T> Bv = sub(g.B, (int64_t)i * NB, (int64_t)c * NB);
  const bool rowcont = (Bv.cs == 1 || Bv.cs == -1) && !(Bv.rs == 1 || Bv.rs == -1);
#pragma unroll 8
  for (int q = 0; q < TILE / THR; ++q) {
    const int e = tid + THR * q, a = rowcont ? e / NB : e % NB, b = rowcont ? e % NB : e / NB;
    Ts[a * LDL + b] = a < rows && b < cols ? g.alpha * Bv.p[a * Bv.rs + b * Bv.cs] : T(0);
  }
  if (i > 0) {
    wait(0);
    __syncthreads();
    bool good = sh_state[0] >= 0;
    if (good) load_x(0);
    ktrsv::cp_commit();
    T acc[8][8];
#pragma unroll
    for (int p = 0; p < 8; ++p)
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[p][q] = T(0);
    for (int k = 0; good && k < i; ++k) {
      const bool more = k + 1 < i;
      ktrsv::cp_wait_all();
      if (more) wait(k + 1);
      __syncthreads();  // tile k landed; every thread is done with the other buffers
      if (more) {
        good = sh_state[(k + 1) & 1] >= 0;
        load_l(k + 1);
        if (good) load_x(k + 1);
        ktrsv::cp_commit();
      }
      // rows of the register tile: X's columns, columns: L's rows
      product8<NB, LDL, NB / G>(acc, Xs + (k & 1) * TILE, Ls + (k & 1) * NB * LDL,
                                grp * (NB / G), u);
    }
    if (!good) {  // the same in every thread
      ktrsv::cp_wait_all();
      __syncthreads();
      if (tid == 0) ktrsv::st_release(&flags[(int64_t)i * g.nchunk], -1);
      return;
    }
    // T -= the groups' partial sums, which meet in the operand buffers
    __syncthreads();
    store8(Ls + grp * TILE, acc, u);
    __syncthreads();
#pragma unroll
    for (int w = 0; w < TILE / 4 / THR; ++w) {
      const int e = (tid + THR * w) * 4;
      T* t = Ts + (e / NB) * LDL + e % NB;
      T s[4], v[4];
      lds4(Ls + e, s);
#pragma unroll
      for (int q = 1; q < G; ++q) {
        lds4(Ls + q * TILE + e, v);
#pragma unroll
        for (int r = 0; r < 4; ++r) s[r] += v[r];
      }
      lds4(t, v);
#pragma unroll
      for (int r = 0; r < 4; ++r) v[r] -= s[r];
      sts4(t, v);
    }
  }
  ktrsv::cp_commit();
  ktrsv::cp_wait_all();
  __syncthreads();
  // X = W_i T: W_i(a, k) = 0 for k > a
  T o[4][4];
  const int tr = tid & 15, tc = tid >> 4;
  product4<LDL, NB>(o, Ts, Ws, 0, tc * 4 + 4, tr, tc);
  if (i + 1 < g.nblk) {
    put4<NB, false>(xs + (int64_t)i * g.nchunk * TILE, o, tr, tc);
    __syncthreads();
    if (tid == 0) ktrsv::st_release(&flags[(int64_t)i * g.nchunk], 1);
  } else {
    __syncthreads();
  }
  put4<LDL, false>(Ts, o, tr, tc);
  __syncthreads();
#pragma unroll 8
  for (int q = 0; q < TILE / THR; ++q) {
    const int e = tid + THR * q, a = rowcont ? e / NB : e % NB, b = rowcont ? e % NB : e / NB;
    if (a < rows && b < cols) Bv.p[a * Bv.rs + b * Bv.cs] = Ts[a * LDL + b];
  }
}

// The inverse's published tiles -> the lower triangle of L.
template <typename T>
__global__ void __launch_bounds__(THR) store_inverse(ViewT<T> L, int n, const T* ws,
                                                     const int* abort_flag) {
  if (abort_flag && *abort_flag != INT_MAX) return;
  __shared__ T s[NB][NB + 1];
  int i, c;
  tile_of((int)blockIdx.x, i, c);
  const ViewT<T> V = sub(L, (int64_t)i * NB, (int64_t)c * NB);
  const int rows = min(NB, n - i * NB), cols = min(NB, n - c * NB);
  const T* t = ws + (int64_t)blockIdx.x * TILE;
  const bool rowcont = (V.cs == 1 || V.cs == -1) && !(V.rs == 1 || V.rs == -1);
#pragma unroll 4
  for (int q = 0; q < TILE / THR; ++q) {
    const int e = threadIdx.x + THR * q;
    s[e / NB][e % NB] = t[e];
  }
  __syncthreads();
#pragma unroll 4
  for (int q = 0; q < TILE / THR; ++q) {
    const int e = threadIdx.x + THR * q;
    const int a = rowcont ? e / NB : e % NB, b = rowcont ? e % NB : e / NB;
    if (a < rows && b < cols && (i != c || a >= b))
      V.p[(int64_t)a * V.rs + (int64_t)b * V.cs] = s[a][b];
  }
}

}  // namespace ktri
}  // namespace rfp
