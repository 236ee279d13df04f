// solve_route.h — which kernel solves a lower triangle of n rows with m
// right-hand sides; host code, shared by the planner, the CUDA executor and
// the host tests.  Times below are whole RFP solves of order 2n (two triangles
// forward, two backward, a rectangle product each way) on one B200.
#pragma once
#include <cstdint>

#include "engine.h"

namespace rfp {

// The whole triangle as one launch, or the recursion whose rectangle updates
// are products on the tensor cores (math != 0): a launch does n^2 m operations
// on the SIMT cores, so above 8192 rows the recursion wins from 128 columns on
// (order 32768, 128 / 200 / 512 columns: 9.7 / 15.4 / 32.2 ms in one launch, 9.6 /
// 10.8 / 17.2; order 65536: 35 / 57 / 119 and 28 / 33 / 50) and loses below (order
// 65536, 64 / 100 columns: 24 / 45 and 27 / 47 ms; order 16384, 100 / 200 columns:
// 3.7 / 4.5 and 4.3 / 4.0).
inline bool solve_in_one_launch(int n, int m, int math) {
  return m <= kTrsvMaxRhs && !(math && m >= 128 && n > 8192);
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
// wide 262 / 390 / 690 us, 32 wide 400 / 420 / 600 us).  With more columns the
// SMs are busy whatever the chain does, and 64 columns a chunk win: above 448
// columns (order 2000, 400 / 512 columns: chain 535 / 642 us, here 611 / 534;
// order 16384: 7.7 / 9.2 ms, here 7.6 / 8.2), and from 256 on in up to four block
// rows, where half of each cluster is idle (order 250, 200 / 256 / 512: 167 / 183
// / 233 us, here 163 / 164 / 163), and above 8192 rows (order 32768 in FP32 mode,
// 200 / 320 / 400: 21.6 / 30.5 / 38.7 ms, here 22.9 / 29.5 / 37.4).  From 4096
// columns on, 64 x 64 tiles with 8 x 8 register products (512 rows, 2048 / 4096 /
// 16384 columns: 64 a chunk 70 / 88 / 208 us, tiles 77 / 79 / 148).
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
  if (m > 448 || (m >= 256 && (nblk <= 4 || n > 8192))) return SOLVE_WAVE64;
  if (nblk * ((m + 15) / 16) > 512) return SOLVE_CHAIN32;
  return nblk * ((m + 7) / 8) > 256 ? SOLVE_CHAIN16 : SOLVE_CHAIN8;
}

}  // namespace rfp
