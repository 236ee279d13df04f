// symv2_layout.h — blocks, groups, strips and partial sums of the ssfmv strips
// (k_symv2.cuh), host- and device-callable so that the host tests can
// enumerate them.
#pragma once
#include <cstdint>

#include "rfp.h"

namespace rfp {
namespace ksymv2 {

constexpr int OG = 64;    // o's per CTA
constexpr int LT = 128;   // l's per step

struct Block {
  int64_t off, so;       // element (l, o) at off + l + o * so
  int ll, lo;            // extents
  int lbase, obase;      // y index of l = 0 and o = 0
  int tri;               // 0 full; stored where l >= o (1) or l <= o (2), diagonal included
  int g0, groups;        // first group of the grid, groups
  int strips;            // most strips of a group
  int64_t lpart, opart;  // offsets of [group][l] and [strip][o] partial sums
};
struct Args {
  Block b[3];
  int nblocks, groups, strips, n;
  int span;  // l's per strip (a multiple of LT)
};

// The l range of group g: [lo, hi).
RFP_HD void l_range(const Block& b, int g, int& lo, int& hi) {
  lo = b.tri == 1 ? g * OG : 0;
  hi = b.tri == 2 ? (b.ll < g * OG + OG ? b.ll : g * OG + OG) : b.ll;
}

// The launch's blocks; returns the number of partial elements.
inline int64_t plan(const Geometry& g, Args* a) {
  const BlockGeom* bg[3] = {&g.b11, &g.b21, &g.b22};
  const int rows[3] = {g.n1, g.n2, g.n2}, cols[3] = {g.n1, g.n1, g.n2};
  const int pb[3] = {0, g.n1, g.n1}, qb[3] = {0, 0, g.n1};
  // strips of 1024 where that leaves several CTAs per SM, else shorter
  a->span = 1024;
  while (a->span > LT && (int64_t)g.n * g.n / 2 < (int64_t)OG * a->span * 148 * 8) a->span /= 2;
  int64_t total = 0;
  int cnt = 0, groups = 0, strips = 1;
  for (int i = 0; i < 3; ++i) {
    if (rows[i] <= 0 || cols[i] <= 0) continue;
    Block& b = a->b[cnt++];
    const bool rowfast = bg[i]->rs == 1;
    b.off = bg[i]->off;
    b.so = rowfast ? bg[i]->cs : bg[i]->rs;
    b.ll = rowfast ? rows[i] : cols[i];
    b.lo = rowfast ? cols[i] : rows[i];
    b.lbase = rowfast ? pb[i] : qb[i];
    b.obase = rowfast ? qb[i] : pb[i];
    b.tri = i == 1 ? 0 : (rowfast ? 1 : 2);
    b.g0 = groups;
    b.groups = (b.lo + OG - 1) / OG;
    groups += b.groups;
    b.strips = (b.ll + a->span - 1) / a->span;
    strips = strips > b.strips ? strips : b.strips;
    b.lpart = total;
    total += (int64_t)b.groups * b.ll;
    b.opart = total;
    total += (int64_t)b.strips * b.lo;
  }
  a->nblocks = cnt;
  a->groups = groups;
  a->strips = strips;
  a->n = g.n;
  return total;
}

}  // namespace ksymv2
}  // namespace rfp
