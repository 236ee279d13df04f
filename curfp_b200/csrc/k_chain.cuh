// k_chain.cuh — triangular solve with few right-hand sides: the chain of block
// rows runs inside thread-block clusters.
//
// L X = alpha B (L n x n lower, any strided view; B n x m view), X over B.
// 64-row blocks; a cluster of CS = 8 CTAs takes eight consecutive block rows
// of one NC-column chunk, CTA rank r the block row j = 8 q + r:
//   Y_j = W_j (alpha B_j - sum_{k<j-2} L_jk X_k),
//   X_j = Y_j - N_j X_{j-2} - M_j X_{j-1},
// with W_j = inv(L_jj), M_j = W_j L_{j,j-1} from trtri_blocks and
// N_j = W_j L_{j,j-2} formed at the start, so one 64 x NC x 64 product is on
// the chain per block row, and what follows X_{j-2} is one product too (with
// L_{j,j-2} in the sum, the sums over groups and the product with W_j behind
// it set the pace: 179 against 166 us).  Inside the cluster X_j
// goes to the later ranks by st.async into their shared memory, data and
// arrival (mbarrier transaction bytes) in one; only every eighth hand-off
// passes through L2 and a flag.  Handing every X_j on through L2 (stores,
// release, polled flag, reload) cost 2.5 us per block row with one right-hand
// side and 6.4 us with 64; inside a cluster a row takes 0.85 us with 8 columns
// (0.2 us of it between the CTAs), and every eighth hand-off 2.9 us.  A solve
// with 8192 rows: one column 318 -> 166 us, 64 columns 700 -> 385 us.
//
// Clusters take tickets in (cluster row, chunk) order and wait only on smaller
// tickets.  L streams through a ring of tiles by cp.async, two products ahead;
// X_k of earlier clusters comes from a packed workspace (row-major 64 x NC).
// A thread sums 4 rows x 8 columns over its share of k; the shares meet once
// per CTA in the ring's space.
//
// Waits are bounded (~2 s); a CTA that gives up records an error code,
// publishes a poisoned flag (-1), and every CTA passes the same two cluster
// barriers on all paths.
#pragma once
#include <climits>
#include <cstdint>

#include "engine.h"
#include "k_micro.cuh"
#include "k_trsv.cuh"

namespace rfp {
namespace kchain {

using namespace kmicro;

constexpr int CS = 8;     // cluster size: block rows per cluster
constexpr int THR = 256;
constexpr int LDL = NB + 4;

template <typename T, int NC>
struct Cfg {
  static constexpr int RING = sizeof(T) == 4 ? 4 : 2;  // L tiles in shared memory
  static constexpr int XT = NB * NC;                   // elements of an X tile
  static constexpr int TPG = 2 * NC;                   // threads of a k group (4 x 8 each)
  static constexpr int KG = THR / TPG, KD = NB / KG;   // k groups, depth of each
  static constexpr int UNITS = XT / 4;                 // 4-column pieces of an X tile
  static constexpr int UPT = (UNITS + THR - 1) / THR;  // per thread
  // ring (later the partial sums: KG X tiles) | W | M | N | X ring | X of the
  // cluster's earlier rows | T
  static constexpr int SMEM =
      (RING * NB * LDL + 3 * TILE + 2 * XT + (CS - 1) * XT + XT) * (int)sizeof(T);
  static_assert(KG * XT <= RING * NB * LDL, "partial sums fit the ring");
};

template <typename T>
struct Args {
  ViewT<T> L, B;
  int n, m, nblk, nchunk;
  T alpha;
  const T* W;  // kInvStride elements per block row: [W_j | M_j]
  T* ws;       // published X tiles, (block row, chunk)
  int* sync;   // [0] ticket, [1 + block row * nchunk + chunk] flags
  int* err;
  const int* abort_flag;
};

__device__ __forceinline__ uint32_t su32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// Every thread of the cluster (converged warps).
__device__ __forceinline__ void cluster_barrier() {
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ bool bar_try(uint32_t bar) {  // phase 0 complete?
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool bar_wait(uint32_t bar) {
  if (bar_try(bar)) return true;
  const uint64_t t0 = ktrsv::gtimer();
  do {
    if (bar_try(bar)) return true;
  } while (ktrsv::gtimer() - t0 < ktrsv::WAIT_NS);
  return false;
}
// 16 bytes to another CTA of the cluster, counted on its barrier.
__device__ __forceinline__ void send16(uint32_t addr, uint32_t bar, const uint32_t (&v)[4]) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, "
      "[%5];" ::"r"(addr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(bar)
      : "memory");
}

// acc(4 x 8) += A X over the group's share of k: A k-major with stride LDA,
// X row-major (64 x NC).
template <int LDA, int NC, typename T>
__device__ __forceinline__ void mac(T (&acc)[4][8], const T* A, const T* X, int kg, int tr,
                                    int tc) {
  constexpr int KD = Cfg<T, NC>::KD;
  const T* a0 = A + kg * KD * LDA + tr * 4;
  const T* x0 = X + kg * KD * NC + tc * 8;
#pragma unroll 4
  for (int k = 0; k < KD; ++k) {
    T a[4], x[8];
    lds4(a0 + k * LDA, a);
    lds4(x0 + k * NC, *reinterpret_cast<T(*)[4]>(x));
    lds4(x0 + k * NC + 4, *reinterpret_cast<T(*)[4]>(x + 4));
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      if constexpr (sizeof(T) == 4) {
#pragma unroll
        for (int q = 0; q < 8; q += 2) fma2(acc[p][q], acc[p][q + 1], x[q], x[q + 1], a[p], a[p]);
      } else {
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[p][q] = fma(a[p], x[q], acc[p][q]);
      }
    }
  }
}
// The shares' partial sums: piece (row r, columns 4h..) of a group at
// ((h * 64 + (r % 4) * 16 + r / 4) * 4), so that a warp's stores are contiguous.
template <int NC, typename T>
__device__ __forceinline__ void put_share(T* red, const T (&acc)[4][8], int kg, int tr, int tc) {
  T* p = red + kg * Cfg<T, NC>::XT;
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const T v[4] = {acc[r][4 * h], acc[r][4 * h + 1], acc[r][4 * h + 2], acc[r][4 * h + 3]};
      sts4(p + (((tc * 2 + h) * NB + r * 16 + tr) * 4), v);
    }
}
template <int NC, typename T>
__device__ __forceinline__ void sum_shares(T (&v)[4], const T* red, int unit) {
  lds4(red + unit * 4, v);
#pragma unroll
  for (int g = 1; g < Cfg<T, NC>::KG; ++g) {
    T w[4];
    lds4(red + g * Cfg<T, NC>::XT + unit * 4, w);
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] += w[e];
  }
}

template <typename T, int NC>
__global__ void __cluster_dims__(CS, 1, 1) __launch_bounds__(THR, 1)
    trsm_chain(const Args<T> g) {
  using C = Cfg<T, NC>;
  if (g.abort_flag && *g.abort_flag != INT_MAX) return;  // the same for every CTA
  extern __shared__ __align__(16) unsigned char chain_raw[];
  T* Lr = reinterpret_cast<T*>(chain_raw);
  T* Ws = Lr + C::RING * NB * LDL;
  T* Ms = Ws + TILE;
  T* Ns = Ms + TILE;
  T* Xr = Ns + TILE;           // X of earlier clusters, two tiles
  T* Xin = Xr + 2 * C::XT;     // X of this cluster's rows
  T* Ts = Xin + (CS - 1) * C::XT;
  T* red = Lr;
  __shared__ __align__(8) uint64_t full[CS - 1];
  __shared__ int sh_ticket, sh_known[3], sh_state;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int kg = tid / C::TPG, tg = tid % C::TPG, tr = tg & 15, tc = tg >> 4;
  const int rank = (int)cluster_rank();
  if (tid == 0) {
    for (int s = 0; s < CS - 1; ++s)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(su32(&full[s])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int s = 0; s < rank; ++s)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(su32(&full[s])),
                   "r"((uint32_t)(C::XT * sizeof(T)))
                   : "memory");
    if (rank == 0) sh_ticket = atomicAdd(g.sync, 1);
  }
  cluster_barrier();
  int* flags = g.sync + 1;
  int ticket;  // rank 0's
  asm volatile("ld.shared::cluster.u32 %0, [%1];"
               : "=r"(ticket)
               : "r"(map_rank(su32(&sh_ticket), 0))
               : "memory");
  const int q0 = (ticket / g.nchunk) * CS, c = ticket % g.nchunk;  // first row, chunk
  const int j = q0 + rank;
  const int rows = min(NB, g.n - j * NB), cols = min(NC, g.m - c * NC);
  const ViewT<T> Bt = sub(g.B, (int64_t)j * NB, (int64_t)c * NC);
  const bool bcont = (Bt.cs == 1 || Bt.cs == -1) && !(Bt.rs == 1 || Bt.rs == -1);
  const bool lcont = (g.L.cs == 1 || g.L.cs == -1) && !(g.L.rs == 1 || g.L.rs == -1);
  constexpr int VW = 16 / (int)sizeof(T);
  const int kend = j - 2;  // products of the loop: k < kend
  bool ok = j < g.nblk, bad = false;

  // L_jk -> ring slot k % RING, element (a, b) at b * LDL + a; pointer steps
  // along the view's outer dimension.
  auto load_l = [&](int k) {
    T* s = Lr + (k % C::RING) * NB * LDL;
    const ViewT<T> v = sub(g.L, (int64_t)j * NB, (int64_t)k * NB);
    const int inner = tid & 63, outer = tid >> 6;
    const int64_t step = 4 * (lcont ? v.rs : v.cs);
    const T* p = v.p + (int64_t)outer * (lcont ? v.rs : v.cs) + (int64_t)inner * (lcont ? v.cs : v.rs);
    T* t = s + (lcont ? inner * LDL + outer : outer * LDL + inner);
    const int tstep = lcont ? 4 : 4 * LDL;
#pragma unroll 8
    for (int u = 0; u < 16; ++u, p += step, t += tstep) {
      const bool in = (lcont ? outer + 4 * u : inner) < rows;
      ktrsv::cp1(t, in ? p : v.p, in);
    }
  };
  auto load_x = [&](int k, T* s) {
    const T* x = g.ws + ((int64_t)k * g.nchunk + c) * C::XT;
    for (int e = tid * VW; e < C::XT; e += THR * VW) cp16(s + e, x + e);
  };
  auto flag = [&](int k) { return &flags[k * g.nchunk + c]; };
  // Warp 0: how far from k on earlier clusters' rows are published; the same
  // after waiting for row k.
  auto scan = [&](int k, int* known) {
    const int st = k + lane < min(kend, q0) ? ktrsv::ld_acquire(flag(k + lane)) : 0;
    const unsigned m = __ballot_sync(0xffffffffu, st > 0);
    if (lane == 0) *known = k + (m == 0xffffffffu ? 32 : __ffs(~m) - 1);
  };
  auto wait = [&](int k, int* known) {
    if (lane == 0) sh_state = ktrsv::wait_flag(flag(k), g.err);
    __syncwarp();
    scan(k, known);
  };

  if (ok) {
    const T* w = g.W + (int64_t)j * kInvStride;
    for (int e = tid * VW; e < 2 * TILE; e += THR * VW) cp16(Ws + e, w + e);  // W_j, M_j
    ktrsv::cp_commit();
    // alpha B_j -> T (row-major, zeros outside)
    for (int e = tid; e < C::XT; e += THR) {
      const int a = bcont ? e / NC : e % NB, b = bcont ? e % NC : e / NB;
      T v = T(0);
      if (a < rows && b < cols) v = g.alpha * __ldcg(Bt.p + (int64_t)a * Bt.rs + (int64_t)b * Bt.cs);
      Ts[a * NC + b] = v;
    }
    T acc[4][8];
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[p][q] = T(0);
    // N_j = W_j L_{j,j-2}, the tile row-major in the ring's first slot
    if (j > 1) {
      const ViewT<T> v = sub(g.L, (int64_t)j * NB, (int64_t)(j - 2) * NB);
      const int inner = tid & 63, outer = tid >> 6;
      for (int u = 0; u < 16; ++u) {
        const int a = lcont ? outer + 4 * u : inner, b = lcont ? inner : outer + 4 * u;
        ktrsv::cp1(Lr + a * LDL + b, a < rows ? v.p + (int64_t)a * v.rs + (int64_t)b * v.cs : v.p,
                   a < rows);
      }
      ktrsv::cp_commit();
      ktrsv::cp_wait_all();
      __syncthreads();
      T o[4][4];
      const int ar = tid & 15, ac = tid >> 4;
      product4<NB, LDL>(o, Ws, Lr, 0, NB, ar, ac);
      put4<NB, false>(Ns, o, ar, ac);
      __syncthreads();
    }
    constexpr int AHEAD = C::RING - 1;  // L tiles in flight or landed ahead of the product
    int known = 0;
    bool loaded = false;  // X_k is in the X ring (or on its way)
    for (int k = 0; k < AHEAD; ++k) {
      if (k < kend) load_l(k);
      ktrsv::cp_commit();
    }
    for (int k = 0; k < kend && !bad; ++k) {
      const bool glob = k < q0;
      if (glob && !loaded) {  // at the front: wait for the row, then fetch it
        if (warp == 0) wait(k, &sh_known[2]);
        __syncthreads();
        bad = sh_state < 0;
        if (bad) break;
        known = sh_known[2];
        load_x(k, Xr + (k & 1) * C::XT);
        ktrsv::cp_commit();
        ktrsv::cp_wait_all();
      } else {
        // everything but the last L tile asked for, where it is not this one
        asm volatile("cp.async.wait_group %0;\n" ::"n"(AHEAD > 1 ? 1 : 0) : "memory");
      }
      const bool next = k + 1 < kend && k + 1 < q0, ask = next && k + 1 >= known;
      if (ask && warp == 0) scan(k + 1, &sh_known[k & 1]);
      __syncthreads();  // tile k landed; every thread is done with product k - 1
      if (ask) known = sh_known[k & 1];
      loaded = next && k + 1 < known;
      if (loaded) load_x(k + 1, Xr + ((k + 1) & 1) * C::XT);
      ktrsv::cp_commit();
      if (k + AHEAD < kend) load_l(k + AHEAD);
      ktrsv::cp_commit();
      const T* X = Xr + (k & 1) * C::XT;
      if (!glob) {
        X = Xin + (k - q0) * C::XT;
        bad = __syncthreads_or(!bar_wait(su32(&full[k - q0])));
        if (bad) break;
      }
      mac<LDL, NC>(acc, Lr + (k % C::RING) * NB * LDL, X, kg, tr, tc);
    }
    ktrsv::cp_wait_all();
    __syncthreads();
    T y[C::UPT][4];
    if (!bad) {
      // T -= the sum, Y = W T
      put_share<NC>(red, acc, kg, tr, tc);
      __syncthreads();
#pragma unroll
      for (int w2 = 0; w2 < C::UPT; ++w2) {
        const int unit = tid + THR * w2;
        if (C::UNITS % THR == 0 || unit < C::UNITS) {
          T v[4], t[4];
          sum_shares<NC>(v, red, unit);
          const int h = unit >> 6, slot = unit & 63, r = (slot & 15) * 4 + (slot >> 4);
          lds4(Ts + r * NC + 4 * h, t);
#pragma unroll
          for (int e = 0; e < 4; ++e) t[e] -= v[e];
          sts4(Ts + r * NC + 4 * h, t);
        }
      }
      __syncthreads();
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[p][q] = T(0);
      mac<NB, NC>(acc, Ws, Ts, kg, tr, tc);
      put_share<NC>(red, acc, kg, tr, tc);
      __syncthreads();
#pragma unroll
      for (int w2 = 0; w2 < C::UPT; ++w2) {
        const int unit = tid + THR * w2;
        if (C::UNITS % THR == 0 || unit < C::UNITS) sum_shares<NC>(y[w2], red, unit);
      }
      __syncthreads();
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[p][q] = T(0);
#pragma unroll 1
      for (int back = 2; back >= 1; --back) {  // N_j X_{j-2}, M_j X_{j-1}
        const int k = j - back;
        if (k < 0) continue;
        const T* X = Xin + (k - q0) * C::XT;
        if (k < q0) {  // an earlier cluster's
          if (tid == 0) sh_state = ktrsv::wait_flag(flag(k), g.err);
          __syncthreads();
          bad = sh_state < 0;
          if (bad) break;
          T* x = Xr + (back & 1) * C::XT;
          load_x(k, x);
          ktrsv::cp_commit();
          ktrsv::cp_wait_all();
          __syncthreads();
          X = x;
        } else {
          // every thread waits for itself: no block barrier on the chain
          bad = bad || !bar_wait(su32(&full[k - q0]));
        }
        mac<NB, NC>(acc, back == 2 ? Ns : Ms, X, kg, tr, tc);
      }
      put_share<NC>(red, acc, kg, tr, tc);
      bad = __syncthreads_or(bad);
    }
    if (bad) {
      if (tid == 0) {
        atomicExch(g.err, 5);
        ktrsv::st_release(flag(j), -1);
      }
    } else {
      // X_j: to the later ranks (the next one first), the workspace and B
#pragma unroll
      for (int w2 = 0; w2 < C::UPT; ++w2) {
        const int unit = tid + THR * w2;
        if (C::UNITS % THR != 0 && unit >= C::UNITS) continue;
        const int h = unit >> 6, slot = unit & 63, r = (slot & 15) * 4 + (slot >> 4);
        if (j > 0) {
          T v[4];
          sum_shares<NC>(v, red, unit);
#pragma unroll
          for (int e = 0; e < 4; ++e) y[w2][e] -= v[e];
        }
        const uint32_t at = su32(Xin + rank * C::XT + r * NC + 4 * h), bar = su32(&full[rank]);
        const uint32_t* bits = reinterpret_cast<const uint32_t*>(&y[w2][0]);
        for (int d = rank + 1; d < CS && q0 + d < g.nblk; ++d) {
#pragma unroll
          for (int p = 0; p < (int)sizeof(T) / 4; ++p) {
            const uint32_t v4[4] = {bits[4 * p], bits[4 * p + 1], bits[4 * p + 2], bits[4 * p + 3]};
            send16(map_rank(at + 16 * p, d), map_rank(bar, d), v4);
          }
        }
        sts4(g.ws + ((int64_t)j * g.nchunk + c) * C::XT + r * NC + 4 * h, y[w2]);
        sts4(Ts + r * NC + 4 * h, y[w2]);
      }
      __syncthreads();
      if (tid == 0) ktrsv::st_release(flag(j), 1);
      for (int e = tid; e < C::XT; e += THR) {
        const int a = bcont ? e / NC : e % NB, b = bcont ? e % NC : e / NB;
        if (a < rows && b < cols) Bt.p[(int64_t)a * Bt.rs + (int64_t)b * Bt.cs] = Ts[a * NC + b];
      }
    }
  }
  // No CTA leaves while another may still write to its shared memory: the
  // barrier follows every send, and a CTA that gave up early still takes in
  // (bounded) what was sent to it.
  cluster_barrier();
  if (bad && tid == 0) {
    const uint64_t t0 = ktrsv::gtimer();
    for (int s = 0; s < rank; ++s)
      while (!bar_try(su32(&full[s])) && ktrsv::gtimer() - t0 < 1000000ull) {}
  }
  __syncthreads();
}

}  // namespace kchain
}  // namespace rfp
