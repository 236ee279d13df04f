// k_chain1.cuh — triangular solve with one right-hand side (FP32), the chain of
// k_chain.cuh with everything a row needs in registers.
//
// L x = alpha b: a cluster of eight CTAs takes eight consecutive 64-row blocks,
//   y_j = W_j (alpha b_j - sum_{k<j-2} L_jk x_k),
//   x_j = y_j - N_j x_{j-2} - M_j x_{j-1}.
// Four lanes share a row: lane s holds the elements k = 4 i + s (i < 16) of the
// row in each tile, so a product is 16 FMAs and two shuffles, with no shared
// memory but the 64 elements of x and no block barrier on the chain.  The tiles
// of L go straight to registers, four ahead.  x_j reaches the later ranks by
// st.async; to later clusters it travels as 8-byte words {bits, 1} that two
// fetching warps poll (data and flag in one L2 round trip) and pass on through
// a ring in shared memory.  A step inside a cluster
// takes 0.35 us, a hand-off between clusters 2 us; 8192 rows 166 us with the
// 8-column kernel, 108 us so, 2048 rows 48 and 30 us.
//
// Waits are bounded (~2 s); a wait that runs out records an error code and the
// CTA goes on with what it has, so that every hand-off still takes place.  No
// word is poisoned: the error word alone says that the result is void.
#pragma once
#include <climits>
#include <cstdint>

#include "k_chain.cuh"

namespace rfp {
namespace kchain1 {

using namespace kmicro;
using kchain::CS;
using kchain::su32;

constexpr int THR = 320;   // eight computing warps, two fetching
constexpr int XR = 8;      // x blocks in the fetch ring
constexpr int LDR = NB + 4;

struct Args {
  View L, B;
  int n, nblk;
  float alpha;
  const float* W;         // kInvStride elements per block row: [W_j | M_j]
  unsigned long long* ws; // published words, 64 per block row, zero at launch
  int* sync;              // ticket
  int* err;
  const int* abort_flag;
};

__device__ __forceinline__ bool try_parity(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// *late: a wait of this CTA ran out before; it does not wait again.
__device__ __forceinline__ void wait_parity(uint32_t bar, uint32_t parity, int* err,
                                            volatile int* late) {
  if (try_parity(bar, parity) || *late) return;
  const uint64_t t0 = ktrsv::gtimer();
  while (!try_parity(bar, parity))
    if (ktrsv::gtimer() - t0 > ktrsv::WAIT_NS) {
      atomicExch(err, 5);
      *late = 1;
      return;
    }
}
__device__ __forceinline__ void arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(bar)), "r"(count));
}
__device__ __forceinline__ unsigned long long ld_word(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
// Element k of an x block sits at perm(k), so that a lane's 16 are contiguous.
__device__ __forceinline__ int perm(int k) { return (k & 3) * 16 + (k >> 2); }

__global__ void __cluster_dims__(CS, 1, 1) __launch_bounds__(THR, 1) chain1(const Args g) {
  if (g.abort_flag && *g.abort_flag != INT_MAX) return;  // the same for every CTA
  __shared__ __align__(16) float Ws[TILE];       // W_j, then N_j (column-major)
  __shared__ __align__(16) float Lt[NB * LDR];   // L_{j,j-2}, row-major
  __shared__ __align__(16) float Xr[XR][NB], Xin[CS - 1][NB], Ts[NB];
  __shared__ __align__(8) uint64_t full[XR], empty[XR], in[CS - 1];
  __shared__ int sh_ticket;
  __shared__ volatile int sh_late;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = (int)kchain::cluster_rank();
  if (tid == 0) {
    for (int s = 0; s < XR; ++s) {
      init(&full[s], 64);
      init(&empty[s], 8);
    }
    for (int s = 0; s < CS - 1; ++s) init(&in[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int s = 0; s < rank; ++s)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(su32(&in[s])),
                   "r"((uint32_t)(NB * sizeof(float)))
                   : "memory");
    sh_late = 0;
    if (rank == 0) sh_ticket = atomicAdd(g.sync, 1);
  }
  kchain::cluster_barrier();
  int q0;  // the cluster's first block row
  asm volatile("ld.shared::cluster.u32 %0, [%1];"
               : "=r"(q0)
               : "r"(kchain::map_rank(su32(&sh_ticket), 0))
               : "memory");
  q0 *= CS;
  const int j = q0 + rank;
  if (j < g.nblk) {
    const int rows = min(NB, g.n - j * NB);
    const View Lj = sub(g.L, (int64_t)j * NB, 0);
    // N_j = W_j L_{j,j-2}
    const float* w = g.W + (int64_t)j * kInvStride;
    const bool lcont = (g.L.cs == 1 || g.L.cs == -1) && !(g.L.rs == 1 || g.L.rs == -1);
    for (int e = tid * 4; e < TILE; e += THR * 4) cp16(Ws + e, w + e);
    if (j > 1)
      for (int e = tid; e < TILE; e += THR) {
        const int a = lcont ? e >> 6 : e & 63, b = lcont ? e & 63 : e >> 6;
        const float* p = Lj.p + (int64_t)a * Lj.rs + (int64_t)((j - 2) * NB + b) * Lj.cs;
        ktrsv::cp1(Lt + a * LDR + b, a < rows ? p : Lj.p, a < rows);
      }
    ktrsv::cp_commit();
    ktrsv::cp_wait_all();
    __syncthreads();
    const int r = (tid >> 2) & 63, s = tid & 3;  // computing warps: row, share of k
    float wr[16], mr[16], nr[16];
    if (warp < 8) {
#pragma unroll
      for (int i = 0; i < 16; ++i) wr[i] = Ws[(4 * i + s) * NB + r];
    }
    float o[4][4];
    const int ar = tid & 15, ac = (tid >> 4) & 15;
    if (warp < 8 && j > 1) product4<NB, LDR>(o, Ws, Lt, 0, NB, ar, ac);
    __syncthreads();
    if (warp < 8 && j > 1) put4<NB, false>(Ws, o, ar, ac);
    __syncthreads();
    if (warp < 8) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        nr[i] = j > 1 ? Ws[(4 * i + s) * NB + r] : 0.f;
        mr[i] = j > 0 ? w[TILE + (4 * i + s) * NB + r] : 0.f;
      }
    }
    const int nglob = min(q0, j);  // blocks that come through the ring, in order
    if (warp >= 8) {
      // ---------------- fetching warps ----------------
      const int e = tid - 256;
      const unsigned long long* p = g.ws + e;
      for (int k0 = 0; k0 < nglob; k0 += 4) {
        unsigned long long v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = k0 + u < nglob ? ld_word(p + (int64_t)(k0 + u) * NB) : 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int k = k0 + u;
          if (k >= nglob) break;
          if (!(v[u] >> 32) && !sh_late) {
            const uint64_t t0 = ktrsv::gtimer();
            while (!((v[u] = ld_word(p + (int64_t)k * NB)) >> 32))
              if (ktrsv::gtimer() - t0 > ktrsv::WAIT_NS) {
                atomicExch(g.err, 5);
                sh_late = 1;
                break;
              }
          }
          const int slot = k % XR, use = k / XR;
          if (use > 0) wait_parity(su32(&empty[slot]), (use - 1) & 1, g.err, &sh_late);
          Xr[slot][perm(e)] = __uint_as_float((unsigned)v[u]);
          arrive(su32(&full[slot]));
        }
      }
    } else {
      // ---------------- computing warps ----------------
      const bool live = r < rows;
      const float* lp = Lj.p + (live ? (int64_t)r * Lj.rs : 0) + (int64_t)s * Lj.cs;
      const int64_t cs4 = 4 * Lj.cs;
      const float b = live ? g.alpha * __ldcg(g.B.p + (int64_t)(j * NB + r) * g.B.rs) : 0.f;
      auto load = [&](float (&l)[16], int k) {
        const float* p = lp + (int64_t)k * NB * Lj.cs;
#pragma unroll
        for (int i = 0; i < 16; ++i) l[i] = live ? __ldg(p + i * cs4) : 0.f;
      };
      // the row's product with x_k: waits for the block and releases it
      auto mul = [&](const float (&l)[16], int k, float (&acc)[4]) {
        const float* x;
        const bool ring = k < nglob;
        if (ring) {
          wait_parity(su32(&full[k % XR]), (k / XR) & 1, g.err, &sh_late);
          x = Xr[k % XR];
        } else {
          wait_parity(su32(&in[k - q0]), 0, g.err, &sh_late);
          x = Xin[k - q0];
        }
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          float v[4];
          lds4(x + s * 16 + 4 * h, v);
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[e] = fmaf(l[4 * h + e], v[e], acc[e]);
        }
        if (ring) {
          __syncwarp();
          if (lane == 0) arrive(su32(&empty[k % XR]));
        }
      };
      auto row_sum = [&](const float (&acc)[4]) {
        float t = (acc[0] + acc[1]) + (acc[2] + acc[3]);
        t += __shfl_xor_sync(0xffffffffu, t, 1);
        return t + __shfl_xor_sync(0xffffffffu, t, 2);
      };
      const int kend = j - 2;
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
      float l0[16], l1[16], l2[16], l3[16];
      if (0 < kend) load(l0, 0);
      if (1 < kend) load(l1, 1);
      if (2 < kend) load(l2, 2);
      if (3 < kend) load(l3, 3);
#pragma unroll 1
      for (int k = 0; k < kend; k += 4) {
        mul(l0, k, acc);
        if (k + 4 < kend) load(l0, k + 4);
        if (k + 1 < kend) mul(l1, k + 1, acc);
        if (k + 5 < kend) load(l1, k + 5);
        if (k + 2 < kend) mul(l2, k + 2, acc);
        if (k + 6 < kend) load(l2, k + 6);
        if (k + 3 < kend) mul(l3, k + 3, acc);
        if (k + 7 < kend) load(l3, k + 7);
      }
      const float t = b - row_sum(acc);
      if (s == 0) Ts[perm(r)] = t;
      bar_sync<1, 256>();
      float y4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        float v[4];
        lds4(Ts + s * 16 + 4 * h, v);
#pragma unroll
        for (int e = 0; e < 4; ++e) y4[e] = fmaf(wr[4 * h + e], v[e], y4[e]);
      }
      const float y = row_sum(y4);
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[e] = 0.f;
      if (j > 1) mul(nr, j - 2, acc);
      if (j > 0) mul(mr, j - 1, acc);
      const float xj = y - row_sum(acc);
      if (s == 0) {
        const uint32_t bits = __float_as_uint(xj);
        const uint32_t at = su32(&Xin[0][0]) + (rank * NB + perm(r)) * 4, bar = su32(&in[0]) + 8 * rank;
        for (int d = rank + 1; d < CS && q0 + d < g.nblk; ++d)
          asm volatile(
              "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(
                  kchain::map_rank(at, d)),
              "r"(bits), "r"(kchain::map_rank(bar, d))
              : "memory");
        asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(g.ws + (int64_t)j * NB + r),
                     "l"((1ull << 32) | bits)
                     : "memory");
        if (live) g.B.p[(int64_t)(j * NB + r) * g.B.rs] = xj;
      }
    }
  }
  // No CTA leaves while another may still write to its shared memory: every
  // send precedes the barrier, and every block sent here has been waited for.
  // The barrier orders a send, not its arrival, so a CTA that stopped waiting
  // waits (bounded) for what was sent now.
  kchain::cluster_barrier();
  if (sh_late && j < g.nblk) {
    const uint64_t t0 = ktrsv::gtimer();
    for (int s = 0; s < rank; ++s)
      while (!try_parity(su32(&in[s]), 0) && ktrsv::gtimer() - t0 < 1000000ull) {}
  }
}

}  // namespace kchain1
}  // namespace rfp
