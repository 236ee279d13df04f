// k_micro.cuh — 64 x 64 tile products in shared memory, shared by the tile
// Cholesky and the wavefront solves.
//
// Operands are k-major (element (row a, k) at s[k * LD + a]), so that a thread
// reads four rows of a k with one 16-byte load.  Shared memory returns 128
// bytes a cycle whether lanes share an address or not: a 4 x 4 register tile
// (8 loads for 16 FMAs) runs at half the FMA rate, and 8 x 8 is where loads
// and FMAs meet, so long sums take product8 with k split over groups of 64
// threads, short ones on a latency chain product4.
#pragma once
#include <cstdint>

namespace rfp {
namespace kmicro {

constexpr int NB = 64;
constexpr int TILE = NB * NB;

// 16 bytes by cp.async, L2 only (the data was written by CTAs of this launch).
__device__ __forceinline__ void cp16(void* smem, const void* g) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(g) : "memory");
}
template <int ID, int COUNT>
__device__ __forceinline__ void bar_sync() {
  asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(COUNT) : "memory");
}
__device__ __forceinline__ void lds4(const float* p, float (&v)[4]) {
  const float4 x = *reinterpret_cast<const float4*>(p);
  v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}
__device__ __forceinline__ void lds4(const double* p, double (&v)[4]) {
  const double2 x = reinterpret_cast<const double2*>(p)[0];
  const double2 y = reinterpret_cast<const double2*>(p)[1];
  v[0] = x.x; v[1] = x.y; v[2] = y.x; v[3] = y.y;
}
__device__ __forceinline__ void sts4(float* p, const float (&v)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void sts4(double* p, const double (&v)[4]) {
  reinterpret_cast<double2*>(p)[0] = make_double2(v[0], v[1]);
  reinterpret_cast<double2*>(p)[1] = make_double2(v[2], v[3]);
}

// Two FP32 FMAs in one instruction, each rounded as by fmaf.
__device__ __forceinline__ void fma2(float& d0, float& d1, float a0, float a1, float b0, float b1) {
  asm("{\n\t.reg .b64 a, b, d;\n\t"
      "mov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 d, {%0, %1};\n\t"
      "fma.rn.f32x2 d, a, b, d;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "+f"(d0), "+f"(d1)
      : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}
// acc += A B^T over k in [k0, k0 + KG), A and B k-major with column strides
// LDA, LDB; thread u of 64: rows 4 (u % 8) + {0, 32}.., columns
// 4 (u / 8) + {0, 32}..  FP32 rows go in pairs (a 64^3 product 3030 -> 2650
// cycles: the issue slots of 64 FMAs, 4 loads and the loop are what bounds it).
template <int LDA, int LDB, int KG, typename T>
__device__ __forceinline__ void product8(T (&acc)[8][8], const T* A, const T* B, int k0, int u) {
  const T* a0 = A + k0 * LDA + (u & 7) * 4;
  const T* b0 = B + k0 * LDB + (u >> 3) * 4;
#pragma unroll 4
  for (int k = 0; k < KG; ++k) {
    T a[8], b[8];
    lds4(a0 + k * LDA, *reinterpret_cast<T(*)[4]>(a));
    lds4(a0 + k * LDA + 32, *reinterpret_cast<T(*)[4]>(a + 4));
    lds4(b0 + k * LDB, *reinterpret_cast<T(*)[4]>(b));
    lds4(b0 + k * LDB + 32, *reinterpret_cast<T(*)[4]>(b + 4));
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      if constexpr (sizeof(T) == 4) {
#pragma unroll
        for (int p = 0; p < 8; p += 2) fma2(acc[p][q], acc[p + 1][q], a[p], a[p + 1], b[q], b[q]);
      } else {
#pragma unroll
        for (int p = 0; p < 8; ++p) acc[p][q] = fma(a[p], b[q], acc[p][q]);
      }
    }
  }
}
template <typename T>
__device__ __forceinline__ void store8(T* s, const T (&acc)[8][8], int u) {
#pragma unroll
  for (int q = 0; q < 8; ++q)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const T v[4] = {acc[4 * h][q], acc[4 * h + 1][q], acc[4 * h + 2][q], acc[4 * h + 3][q]};
      sts4(s + ((u >> 3) * 4 + (q >> 2) * 32 + (q & 3)) * NB + (u & 7) * 4 + 32 * h, v);
    }
}
template <typename T>
__device__ __forceinline__ void add8(T (&acc)[8][8], const T* s, int u) {
#pragma unroll
  for (int q = 0; q < 8; ++q)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      T v[4];
      lds4(s + ((u >> 3) * 4 + (q >> 2) * 32 + (q & 3)) * NB + (u & 7) * 4 + 32 * h, v);
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[4 * h + e][q] += v[e];
    }
}
// dst -= the sum of N partial tiles at src, src + TILE, ... (THR threads).
template <int N, int THR, typename T>
__device__ __forceinline__ void subtract(T* dst, const T* src) {
#pragma unroll
  for (int w = 0; w < TILE / 4 / THR; ++w) {
    const int e = (threadIdx.x + THR * w) * 4;
    T s[4], v[4];
    lds4(src + e, s);
#pragma unroll
    for (int i = 1; i < N; ++i) {
      lds4(src + i * TILE + e, v);
#pragma unroll
      for (int q = 0; q < 4; ++q) s[q] += v[q];
    }
    lds4(dst + e, v);
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] -= s[q];
    sts4(dst + e, v);
  }
}

// out(4 x 4 at rows 4 tr, columns 4 tc) = sum_{k0 <= k < k1} A B^T, column
// strides LDA, LDB.
template <int LDA, int LDB, typename T>
__device__ __forceinline__ void product4(T (&o)[4][4], const T* A, const T* B, int k0, int k1,
                                         int tr, int tc) {
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) o[p][q] = T(0);
#pragma unroll 4
  for (int k = k0; k < k1; ++k) {
    T a[4], b[4];
    lds4(A + k * LDA + tr * 4, a);
    lds4(B + k * LDB + tc * 4, b);
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int q = 0; q < 4; ++q) o[p][q] = fma(a[p], b[q], o[p][q]);
  }
}
// The sum over G groups of CNT threads each (thread u of group g; COUNT =
// G * CNT threads meet at barrier ID) into group 0; red: (G - 1) * CNT * 16.
template <int G, int CNT, int ID, typename T>
__device__ __forceinline__ void reduce4(T (&o)[4][4], T* red, int g, int u) {
  if constexpr (G > 1) {
    if (g > 0) {
#pragma unroll
      for (int p = 0; p < 4; ++p) sts4(red + (((g - 1) * 4 + p) * CNT + u) * 4, o[p]);
    }
    bar_sync<ID, G * CNT>();
    if (g == 0) {
#pragma unroll
      for (int i = 0; i < G - 1; ++i)
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          T v[4];
          lds4(red + ((i * 4 + p) * CNT + u) * 4, v);
#pragma unroll
          for (int q = 0; q < 4; ++q) o[p][q] += v[q];
        }
    }
  }
}
// s(rows 4 tr.., columns 4 tc..; column stride LD) = o, or -= o.
template <int LD, bool kSub, typename T>
__device__ __forceinline__ void put4(T* s, const T (&o)[4][4], int tr, int tc) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    T* p = s + (tc * 4 + q) * LD + tr * 4;
    T v[4] = {o[0][q], o[1][q], o[2][q], o[3][q]};
    if (kSub) {
      T w[4];
      lds4(p, w);
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = w[e] - v[e];
    }
    sts4(p, v);
  }
}

}  // namespace kmicro
}  // namespace rfp
