// solve_route.h — which kernel solves a lower triangle of n rows with m
// right-hand sides; host code, shared by the planner, the CUDA executor and
// the host tests.  Times below are whole RFP solves of order 2n (two triangles
// forward, two backward, a rectangle product each way) on one B200.
#pragma once
#include <cstdint>

#include "engine.h"

namespace rfp {

// Elements of X from which the SMs are busy with one launch whatever its chain
// of block rows does: the products' rate counts from here on.
constexpr int64_t kSolveBusy = int64_t(9) << 18;

// The whole triangle as one launch, or the recursion whose rectangle updates
// are products on the tensor cores (math != 0): a launch does n^2 m operations
// on the SIMT cores, so above 8192 rows and kSolveBusy elements the recursion
// wins from 128 columns on (order 20000, 256 columns 7.6 ms in one launch, 7.5;
// 24000, 200 9.2 / 7.5; 32768, 200 / 512 15.4 / 28 and 11.1 / 16.9; 65536, 128 / 512
// 35 / 103 and 28 / 49).  Below it loses (17000, 128 / 256 3.4 / 5.8 and 4.8 / 6.1;
// 24000, 128 5.9 / 6.7), and with fewer columns always (65536, 64 / 127 24 / 45 and
// 27 / 48).
inline bool solve_in_one_launch(int n, int m, int math) {
  return m <= kTrsvMaxRhs && !(math && m >= 128 && n > 8192 && (int64_t)n * m >= kSolveBusy);
}
// Rows that the recursion leaves to one launch: small blocks, so that most of
// the work is in the updates, but with few columns a launch of 512 rows is
// bound by its chain (order 65536, 256 columns: 40 ms with 512 rows, 38 with
// 1024, 35 with 2048).
inline int solve_leaf_rows(int m) { return m > kTrsvMaxRhs ? 512 : 2048; }

enum SolveKernel {
  SOLVE_CHAIN1,   // k_chain1.cuh, one FP32 column
  SOLVE_CHAIN8,   // k_chain.cuh, chunks of 8, 16 and 32 columns
  SOLVE_CHAIN16,
  SOLVE_CHAIN32,
  SOLVE_WAVE64,   // k_trsv.cuh, chunks of 64 columns
  SOLVE_TILES     // k_tri.cuh solve_tiles, 64 x 64 tiles
};

// FP32: the chain inside clusters, in chunks as narrow as the throughput
// allows, since the chain's step shrinks with the chunk while the products'
// cost per column grows: 8 columns up to 256 (block row, chunk) pairs, 16 up to
// 512, else 32 (8192 rows, 16 / 64 / 128 columns: 8 wide 190 / 510 / 970 us, 16
// wide 262 / 390 / 690 us, 32 wide 400 / 420 / 600 us), and 32 from 256 columns on
// where the triangle is one row of clusters (order 500, 256 / 480 columns: 8 wide
// 248 / 299 us, 32 wide 199 / 198).  Chunks of 64 columns (k_trsv.cuh) win above
// 480 columns, where 32-column chunks need another turn of clusters (order 500,
// 480 / 481 / 512: 198 / 250 / 265 us, 64 wide 221 / 222 / 222; order 8192: 2.59 / 3.00
// / 3.01 ms, 64 wide 2.78), and above 256 from kSolveBusy elements on (order 12000,
// 440: 5.11 ms, 64 wide 4.62; order 16384, 384: 7.19 and 6.97; order 32768 in FP32
// mode, 200 / 320 / 400: 21.6 / 30.5 / 38.7, 64 wide 22.9 / 29.5 / 37.4).  From 4096
// columns on, 64 x 64 tiles with 8 x 8 register products (512 rows, 2048 / 4096 / 16384 columns: 64
// wide 70 / 88 / 208 us, tiles 77 / 79 / 148).
// FP64: 8 columns a chunk, up to 2048 (block row, chunk) pairs and 128 columns,
// then 64 a chunk (order 16384, 65 / 100 / 128 columns: 7.1 / 8.8 / 10.7 ms
// against 8.7 / 8.8 / 8.8; order 32768, 33 / 64 / 100: 14.4 / 19.5 / 32.6 against
// 17.2 / 17.5 / 27.7), unless that leaves nearly half of the columns empty (order
// 32768, 65: 26.2 against 27.5).
inline SolveKernel solve_kernel(bool fp32, int n, int m) {
  const int64_t nblk = (n + kTrsmLeaf - 1) / kTrsmLeaf;
  if (!fp32)
    return (m <= 128 && nblk * ((m + 7) / 8) < 2048) || (m > 64 && m <= 72) ? SOLVE_CHAIN8
                                                                            : SOLVE_WAVE64;
  if (m == 1) return SOLVE_CHAIN1;
  if (m >= 4096) return SOLVE_TILES;
  if (m > 480 || (m > 256 && (int64_t)n * m >= kSolveBusy)) return SOLVE_WAVE64;
  if (nblk * ((m + 15) / 16) > 512 || (m >= 256 && nblk <= 8)) return SOLVE_CHAIN32;
  return nblk * ((m + 7) / 8) > 256 ? SOLVE_CHAIN16 : SOLVE_CHAIN8;
}

}  // namespace rfp
