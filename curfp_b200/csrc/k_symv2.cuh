// k_symv2.cuh — y := alpha A x + beta y for a symmetric FP32 A held in RFP (any
// variant), one right-hand side (ssfmv).
//
// Bandwidth-bound, and every stored element is read exactly once, for both
// halves of the product.  Each RFP block is walked along its contiguous
// index: with l the contiguous and o the other index of a block, CTA (g, s)
// takes 64 o's and a strip of l's, 128 at a time; a warp owns 8 o's, a lane
// the l's lane + 32 a:
//   * the sums over l (y_o += a x_l) stay in 8 registers per lane over the
//     whole strip and leave once per strip, after one shuffle reduction;
//   * the sums over o (y_l += a x_o) of each 128 l's meet over the warps in
//     shared memory and leave as one vector per o group.
// So an element costs a load, two FMAs and little else, and 32 loads are in
// flight per thread.  (Walking 64 x 64 tiles whatever the layout, half of them
// across the contiguous index, took 25 instructions per 128-byte load and ran
// at 3.1 TB/s at 58% issue.)  symv2_reduce adds the partial vectors in a fixed
// order, so the result is bitwise repeatable; they take 3 n^2 / 256 elements and a
// little for the strips.
//
// n = 16001: 179 -> 113 us, 512 MB stored (78 us at the measured copy rate);
// n = 32768 620 -> 381 us.
#pragma once
#include <cstdint>

#include "k_symv.cuh"
#include "symv2_layout.h"

namespace rfp {
namespace ksymv2 {

constexpr int THR = 256;

// grid (groups, strips)
__global__ void __launch_bounds__(THR, 3)
    symv2_strips(const Args args, const float* __restrict__ arf, const float* __restrict__ x,
                 int64_t incx, float* __restrict__ part) {
  __shared__ float ls[2][8][LT];
  int bi = 0;
  while (bi + 1 < args.nblocks && (int)blockIdx.x >= args.b[bi + 1].g0) ++bi;
  const Block& b = args.b[bi];
  const int g = blockIdx.x - b.g0;
  int lo, hi;
  l_range(b, g, lo, hi);
  lo += blockIdx.y * args.span;
  hi = min(hi, lo + args.span);
  if (lo >= hi) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int o0 = g * OG + 8 * w;
  const int ll = b.ll, nlo = b.lo, tri = b.tri;
  float xo[8], so[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    xo[q] = o0 + q < nlo ? __ldg(x + (int64_t)(b.obase + o0 + q) * incx) : 0.f;
    so[q] = 0.f;
  }
  const float* base = arf + b.off + (int64_t)o0 * b.so + lane;
  const float* xl0 = x + (int64_t)b.lbase * incx;
  float* lp = part + b.lpart + (int64_t)g * ll;
  int par = 0;
  for (int l0 = lo; l0 < hi; l0 += LT, par ^= 1) {
    float v[8][4], xl[4], sl[4];
    // whole step inside the stored part, off the diagonal
    const bool full = l0 + LT <= hi && g * OG + OG <= nlo &&
                      (tri == 0 || (tri == 1 ? l0 >= g * OG + OG : l0 + LT <= g * OG));
    if (full) {
      const float* p = base + l0;
#pragma unroll
      for (int q = 0; q < 8; ++q, p += b.so)
#pragma unroll
        for (int a = 0; a < 4; ++a) v[q][a] = __ldg(p + 32 * a);
    }
    unsigned in = 0xffffffffu;  // bit 4 q + a: the element is stored
    if (!full) {
      const float* p = base + l0;
      in = 0;
#pragma unroll
      for (int q = 0; q < 8; ++q, p += b.so)
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          const int l = l0 + lane + 32 * a, o = o0 + q;
          const bool ok = l < hi && o < nlo && (tri == 0 || (tri == 1 ? l >= o : l <= o));
          in |= ok ? 1u << (4 * q + a) : 0u;
          v[q][a] = ok ? __ldg(p + 32 * a) : 0.f;
        }
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int l = l0 + lane + 32 * a;
      xl[a] = l < ll ? __ldg(xl0 + (int64_t)l * incx) : 0.f;
      sl[a] = 0.f;
    }
    if (full) {
#pragma unroll
      for (int q = 0; q < 8; ++q)
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          sl[a] = fmaf(v[q][a], xo[q], sl[a]);
          so[q] = fmaf(v[q][a], xl[a], so[q]);
        }
    } else {  // x at an element that is not stored does not count, infinite or not
#pragma unroll
      for (int q = 0; q < 8; ++q)
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          const bool ok = in >> (4 * q + a) & 1u;
          if (ok) sl[a] = fmaf(v[q][a], xo[q], sl[a]);
          // a diagonal element belongs to the sums over o alone
          if (ok && !(tri && l0 + lane + 32 * a == o0 + q)) so[q] = fmaf(v[q][a], xl[a], so[q]);
        }
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) ls[par][w][lane + 32 * a] = sl[a];
    __syncthreads();  // the other buffer is free again after the next one
    if (threadIdx.x < LT && l0 + (int)threadIdx.x < hi) {
      float t = ls[par][0][threadIdx.x];
#pragma unroll
      for (int q = 1; q < 8; ++q) t += ls[par][q][threadIdx.x];
      lp[l0 + threadIdx.x] = t;
    }
  }
  const float t = ksymv::warp_sum8(so, lane);
  if ((lane & 3) == 0 && o0 + (lane >> 2) < nlo)
    part[b.opart + (int64_t)blockIdx.y * nlo + o0 + (lane >> 2)] = t;
}

// 32 y's per CTA, the partial vectors dealt to 8 warps (lane = y): their sums
// meet in warp order.
__global__ void __launch_bounds__(THR)
    symv2_reduce(const Args args, const float* __restrict__ part, float* y, int64_t incy,
                 float alpha, float beta) {
  __shared__ float ws[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane;
  float t = 0.f;
  for (int bi = 0; bi < args.nblocks; ++bi) {
    const Block& b = args.b[bi];
    const int l = i - b.lbase, o = i - b.obase;
    if (l >= 0 && l < b.ll) {
      const float* p = part + b.lpart + l;
      const int ga = b.tri == 2 ? l / OG : 0, gb = b.tri == 1 ? l / OG + 1 : b.groups;
#pragma unroll 4
      for (int g = ga + w; g < gb; g += 8) t += p[(int64_t)g * b.ll];
    }
    if (o >= 0 && o < b.lo) {
      int lo, hi;
      l_range(b, o / OG, lo, hi);
      const int ns = (hi - lo + args.span - 1) / args.span;
      for (int s = w; s < ns; s += 8) t += part[b.opart + (int64_t)s * b.lo + o];
    }
  }
  ws[w][lane] = t;
  __syncthreads();
  if (w == 0 && i < args.n) {
#pragma unroll
    for (int q = 1; q < 8; ++q) t += ws[q][lane];
    float* yi = y + (int64_t)i * incy;
    *yi = beta == 0.f ? alpha * t : fmaf(beta, *yi, alpha * t);
  }
}

}  // namespace ksymv2
}  // namespace rfp
