// k_tile.cuh — single-CTA kernels on small triangular tiles held in shared
// memory: the diagonal Cholesky tile (the only place pivots are checked), the
// inverses of diagonal blocks used by the blocked TRSM, the in-place
// inverse / L^T L tiles of the blocked spftri and the diagonal tiles of the
// Cholesky adjoint.
#pragma once
#include <climits>
#include <cstdint>
#include <type_traits>

#include "engine.h"

namespace rfp {
namespace ktile {

// Copy the lower triangle of an n x n view tile into shared memory s[i][j]
// (zeros above the diagonal).  The warp runs along the view's contiguous
// dimension and each thread keeps 8 loads in flight.  n <= 32 * RW.
template <int LDS, typename E>
__device__ __forceinline__ void load_lower(ViewT<E> L, int n, E* s) {
  const bool rcont = (L.cs == 1 || L.cs == -1);
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32, nw = blockDim.x / 32;
  for (int base = warp; base < n; base += 8 * nw) {
    E v[8][4];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int a = base + u * nw;  // row (rcont) or column (!rcont)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int b = lane + 32 * q;
        const int i = rcont ? a : b, j = rcont ? b : a;
        v[u][q] = (a < n && b < n && i >= j) ? L.p[(int64_t)i * L.rs + (int64_t)j * L.cs] : E(0);
      }
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int a = base + u * nw;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int b = lane + 32 * q;
        const int i = rcont ? a : b, j = rcont ? b : a;
        if (a < n && b < n) s[i * LDS + j] = v[u][q];
      }
    }
  }
}

// Store the lower triangle of s back to the view (same thread mapping).
template <int LDS, typename E>
__device__ __forceinline__ void store_lower(ViewT<E> L, int n, const E* s) {
  const bool rcont = (L.cs == 1 || L.cs == -1);
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32, nw = blockDim.x / 32;
  for (int a = warp; a < n; a += nw) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int b = lane + 32 * q;
      const int i = rcont ? a : b, j = rcont ? b : a;
      if (b < n && i >= j) L.p[(int64_t)i * L.rs + (int64_t)j * L.cs] = s[i * LDS + j];
    }
  }
}

constexpr int T = 64;        // trtri / lauum / TRSM-leaf tile (== kTrsmLeaf == kTriTile)
constexpr int LD = T + 1;    // padded shared-memory leading dimension

static_assert(T == kTrsmLeaf && T == kTriTile, "tile kernels assume one tile size");

// Inverse of lower-triangular diagonal blocks.  Block b = blockIdx.x covers
// rows/cols [b*64, min(n, b*64+64)); 256 threads.  The two 32 x 32 diagonal
// quarters are inverted in registers by warps 0 and 1 (lane = column of the
// inverse, right-looking: element j is final once scaled by 1/D_jj, then
// updates the elements below with broadcast reads of D's column; by row and
// shuffle a launch took 20 us, so 18 us for four matrices), and the off-diagonal quarter
// follows as
// inv([D0 0; B D1]) = [inv(D0) 0; -inv(D1) (B inv(D0))  inv(D1)] by two
// 32 x 32 products over all threads.  W != nullptr: block b writes the record
// W + b*kInvStride = [W_b | M_b], both 64 x 64 column-major (ld 64, zeros
// outside the block): W_b = inv(L_bb) and, for b >= 1, M_b = W_b L_{b,b-1}
// (the block left of the diagonal block), which lets the wavefront solve
// finish a block row with one product after its predecessor is published.
// W == nullptr: the inverse replaces the lower triangle in place.
constexpr int TRTRI_THREADS = 256;
template <typename E>
constexpr int trtri_smem() { return 2 * T * LD * (int)sizeof(E); }

// Several matrices in one launch: matrix i's blocks are begin[i] .. of the
// grid, and their records follow each other at W.
template <typename E>
struct TriBatch {
  static constexpr int MAX = 4;
  ViewT<E> L[MAX];
  int n[MAX], begin[MAX], count;
  E* W;
};

template <typename E>
__global__ void __launch_bounds__(TRTRI_THREADS) trtri_blocks(const TriBatch<E> batch,
                                                              const int* abort_flag) {
  if (abort_flag && *abort_flag != INT_MAX) return;
  int mi = 0;
  while (mi + 1 < batch.count && (int)blockIdx.x >= batch.begin[mi + 1]) ++mi;
  const ViewT<E> L = batch.L[mi];
  const int n = batch.n[mi];
  E* const W = batch.W ? batch.W + (int64_t)batch.begin[mi] * kInvStride : nullptr;
  extern __shared__ __align__(16) unsigned char trtri_raw[];
  __shared__ E rinv[T];
  E (*s)[LD] = reinterpret_cast<E (*)[LD]>(trtri_raw);  // L_bb, later the block left of it
  E (*x)[LD] = s + T;  // the inverse (upper-right quarter: scratch)
  const int b = blockIdx.x - batch.begin[mi], r0 = b * T;
  const int sz = min(T, n - r0);
  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const ViewT<E> Lb = sub(L, r0, r0);
  // both buffers start at zero: the quarter products read whole 32 x 32
  // quarters, also rows beyond a partial last block
  for (int e = tid; e < T * LD; e += TRTRI_THREADS) {
    (&x[0][0])[e] = E(0);
    (&s[0][0])[e] = E(0);
  }
  __syncthreads();
  load_lower<LD>(Lb, sz, &s[0][0]);
  __syncthreads();
  if (tid < T) rinv[tid] = tid < sz ? E(1) / s[tid][tid] : E(0);
  __syncthreads();
  if (warp < 2) {
    const int q0 = warp * 32;
    E xc[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) xc[k] = k == lane && q0 + lane < sz ? E(1) : E(0);
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      xc[j] *= rinv[q0 + j];
#pragma unroll
      for (int k = j + 1; k < 32; ++k) xc[k] = fma(-s[q0 + k][q0 + j], xc[j], xc[k]);
    }
#pragma unroll
    for (int k = 0; k < 32; ++k) x[q0 + k][q0 + lane] = xc[k];
  }
  __syncthreads();
  if (sz > 32) {
    // T = B inv(D0) into the upper-right quarter (inv(D0) zero above its
    // diagonal, so the sums may run over all k)
    for (int e = tid; e < 1024; e += TRTRI_THREADS) {
      const int i = e >> 5, j = e & 31;
      E a0 = E(0), a1 = E(0);
#pragma unroll
      for (int k = 0; k < 32; k += 2) {
        a0 = fma(s[32 + i][k], x[k][j], a0);
        a1 = fma(s[32 + i][k + 1], x[k + 1][j], a1);
      }
      x[i][32 + j] = a0 + a1;
    }
    __syncthreads();
    // lower-left = -inv(D1) T
    for (int e = tid; e < 1024; e += TRTRI_THREADS) {
      const int i = e >> 5, j = e & 31;
      E a0 = E(0), a1 = E(0);
#pragma unroll
      for (int k = 0; k < 32; k += 2) {
        a0 = fma(x[32 + i][32 + k], x[k][32 + j], a0);
        a1 = fma(x[32 + i][33 + k], x[k + 1][32 + j], a1);
      }
      x[32 + i][j] = -(a0 + a1);
    }
    __syncthreads();
    for (int e = tid; e < 1024; e += TRTRI_THREADS) x[e >> 5][32 + (e & 31)] = E(0);
    __syncthreads();
  }
  if (!W) {
    store_lower<LD>(Lb, sz, &x[0][0]);
    return;
  }
  E* Wb = W + (int64_t)b * kInvStride;
  for (int e = tid; e < T * T; e += TRTRI_THREADS) Wb[e] = x[e & 63][e >> 6];
  if (b == 0) return;
  // M_b = W_b L_{b,b-1}: the 64 x 64 block left of the diagonal block (rows
  // beyond sz are zero), 4 x 4 outputs per thread.
  const ViewT<E> Lp = sub(L, r0, r0 - T);
  for (int e = tid; e < T * T; e += TRTRI_THREADS) {
    const int i = e >> 6, c = e & 63;
    s[i][c] = i < sz ? Lp.p[(int64_t)i * Lp.rs + (int64_t)c * Lp.cs] : E(0);
  }
  __syncthreads();
  const int ri = (tid >> 4) * 4, ci = (tid & 15) * 4;
  E acc[4][4];
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[p][q] = E(0);
#pragma unroll 4
  for (int k = 0; k < T; ++k) {
    E x4[4], s4[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      x4[p] = x[ri + p][k];
      s4[p] = s[k][ci + p];
    }
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[p][q] = fma(x4[p], s4[q], acc[p][q]);
  }
  E* Mb = Wb + T * T;
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) Mb[(int64_t)(ci + q) * T + ri + p] = acc[p][q];
}

// In-place L := L^T L (lower part) for an n x n tile, n <= 64.
// (L^T L)(i,j) = sum_{k >= i} L(k,i) L(k,j) for i >= j.
template <typename E>
__global__ void __launch_bounds__(256) lauum_tile(ViewT<E> L, int n) {
  __shared__ E s[T][LD];
  const int tid = threadIdx.x;
  load_lower<LD>(L, n, &s[0][0]);
  __syncthreads();
  E out[16];
  const int j = tid % T, i0 = tid / T;
#pragma unroll
  for (int r = 0; r < 16; ++r) {
    const int i = i0 + 4 * r;
    E acc = E(0);
    if (i < n && j < n && i >= j)
      for (int k = i; k < n; ++k) acc = fma(s[k][i], s[k][j], acc);
    out[r] = acc;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < 16; ++r) {
    const int i = i0 + 4 * r;
    if (i < n && j < n && i >= j)
      L.p[(int64_t)i * L.rs + (int64_t)j * L.cs] = out[r];
  }
}

// Adjoint of the Cholesky factorization of one diagonal tile (n <= T), in
// place on G's lower triangle.  Column j = n-1 .. 0 reverses the forward
// step that produced column j of L (l = L(j,j), v = L(j+1:, j)) once the
// trailing block's cotangent G(j+1:, j+1:) is final:
//   w = (tril(G_t) + tril(G_t)^T) v      (G_t's diagonal counted twice)
//   G(j+1:, j) = (G(j+1:, j) - w) / l
//   G(j, j)    = (G(j, j) - G(j+1:, j)^T v) / (2 l)
// Four threads share a row of w (strided k, shuffle sum); warp 0 forms the
// diagonal dot product.  Two block barriers per column.
constexpr int ADJ_THREADS = 256;
template <typename E>
constexpr int adj_smem() { return 2 * T * LD * (int)sizeof(E); }

template <typename E>
__global__ void __launch_bounds__(ADJ_THREADS) potrf_adj_tile(ViewT<E> L, ViewT<E> G, int n) {
  extern __shared__ __align__(16) unsigned char adj_raw[];
  E* Ls = reinterpret_cast<E*>(adj_raw);
  E* Gs = Ls + T * LD;
  load_lower<LD>(L, n, Ls);
  load_lower<LD>(G, n, Gs);
  __syncthreads();
  const int tid = threadIdx.x, r = tid >> 2, sl = tid & 3;
  for (int j = n - 1; j >= 0; --j) {
    const E l = Ls[j * LD + j];
    const int p = j + 1 + r;
    E w = E(0);
    if (p < n) {
      for (int q = j + 1 + sl; q < n; q += 4) {
        const E g = q < p ? Gs[p * LD + q] : (q > p ? Gs[q * LD + p] : E(2) * Gs[p * LD + p]);
        w += g * Ls[q * LD + j];
      }
    }
    w += __shfl_xor_sync(0xffffffffu, w, 1);
    w += __shfl_xor_sync(0xffffffffu, w, 2);
    // column j is not read above (q, p > j), so it is updated in place
    if (p < n && sl == 0) Gs[p * LD + j] = (Gs[p * LD + j] - w) / l;
    __syncthreads();
    if (tid < 32) {
      E d = E(0);
      for (int i = j + 1 + tid; i < n; i += 32) d += Gs[i * LD + j] * Ls[i * LD + j];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
      if (tid == 0) Gs[j * LD + j] = (Gs[j * LD + j] - d) / (E(2) * l);
    }
    __syncthreads();
  }
  store_lower<LD>(G, n, Gs);
}

}  // namespace ktile
}  // namespace rfp
