// layout_checks.cpp — TEST-ONLY host entry points for the index arithmetic
// of the single-read symmetric matrix-vector kernel (symv_layout.h), the
// routing of few-column products and the split of k (gemm_route.h), run
// without a GPU.
#include <cstdint>
#include <vector>

#include "engine.h"
#include "func_attr.h"
#include "gemm_route.h"
#include "solve_route.h"
#include "symv2_layout.h"
#include "symv_layout.h"

using namespace rfp;

extern "C" {

// Enumerates the CTAs of the ssfmv launch at order n the way the kernel maps
// them.  out: [0] CTAs, [1] lower tiles visited, [2] visits to a tile
// already visited or outside the lower triangle, [3] row_part entries past
// n_row, [4] col_part entries past n_col, [5] col_part entries written by two
// tiles, [6] strips with an empty tile range.
int hs_symv_layout(int n, int64_t* out) {
  const ksymv::Parts P = ksymv::parts(n);
  const int T = P.tiles;
  const int64_t ctas = ksymv::strips_before(T);
  std::vector<int> seen((size_t)T * T, 0);
  std::vector<int> col((size_t)(P.n_col / ksymv::TB), 0);
  int64_t visited = 0, dup = 0, row_over = 0, col_over = 0, col_dup = 0, empty = 0;
  for (int64_t b = 0; b < ctas; ++b) {
    int I, s;
    ksymv::strip_of(b, T, I, s);
    const int Jb = s * ksymv::S, Je = Jb + ksymv::S < I + 1 ? Jb + ksymv::S : I + 1;
    if (Jb >= Je) ++empty;
    if (((int64_t)I * P.strips + s + 1) * ksymv::TB > P.n_row) ++row_over;
    for (int J = Jb; J < Je; ++J) {
      if (J > I || J < 0 || seen[(size_t)I * T + J]++) ++dup;
      ++visited;
      const int64_t e = ksymv::col_base(J, T) + (I - J);
      if ((e + 1) * ksymv::TB > P.n_col) {
        ++col_over;
      } else if (col[(size_t)e]++) {
        ++col_dup;
      }
    }
  }
  out[0] = ctas;
  out[1] = visited;
  out[2] = dup;
  out[3] = row_over;
  out[4] = col_over;
  out[5] = col_dup;
  out[6] = empty;
  return 0;
}

// Enumerates the CTAs (g, s) of the ssfmv strips at order n the way the kernel
// walks them.  out: [0] partial elements, [1] stored elements visited, [2]
// visits outside the array or to an element already visited, [3] visits whose
// y indices are not the element's row and column, [4] partial sums outside the
// buffer or written twice, [5] steps not a multiple of the span.
int hs_symv2_layout(int n, int transr, int lower, int64_t* out) {
  const Geometry geo = geometry(n, transr, lower);
  ksymv2::Args a{};
  const int64_t total = ksymv2::plan(geo, &a);
  const int64_t nt = (int64_t)n * (n + 1) / 2;
  std::vector<int> row((size_t)nt, -1), col((size_t)nt, -1);  // logical indices of an offset
  const BlockGeom* bg[3] = {&geo.b11, &geo.b21, &geo.b22};
  const int pb[3] = {0, geo.n1, geo.n1}, qb[3] = {0, 0, geo.n1};
  const int rows[3] = {geo.n1, geo.n2, geo.n2}, cols[3] = {geo.n1, geo.n1, geo.n2};
  for (int i = 0; i < 3; ++i)
    for (int p = 0; p < rows[i]; ++p)
      for (int q = 0; q < cols[i]; ++q) {
        if (i != 1 && q > p) continue;
        const int64_t e = bg[i]->off + (int64_t)p * bg[i]->rs + (int64_t)q * bg[i]->cs;
        row[(size_t)e] = pb[i] + p;
        col[(size_t)e] = qb[i] + q;
      }
  std::vector<char> seen((size_t)nt, 0), part((size_t)total, 0);
  int64_t visited = 0, bad = 0, wrong = 0, slots = 0, span = 0;
  auto slot = [&](int64_t at) {
    if (at < 0 || at >= total || part[(size_t)at]++) ++slots;
  };
  for (int bi = 0; bi < a.nblocks; ++bi) {
    const ksymv2::Block& b = a.b[bi];
    for (int g = 0; g < b.groups; ++g)
      for (int s = 0; s < a.strips; ++s) {
        int lo, hi;
        ksymv2::l_range(b, g, lo, hi);
        lo += s * a.span;
        hi = hi < lo + a.span ? hi : lo + a.span;
        if (lo >= hi) continue;
        span += a.span % ksymv2::LT != 0;
        for (int l = lo; l < hi; ++l) slot(b.lpart + (int64_t)g * b.ll + l);
        for (int o = g * ksymv2::OG; o < b.lo && o < (g + 1) * ksymv2::OG; ++o) {
          slot(b.opart + (int64_t)s * b.lo + o);
          for (int l = lo; l < hi; ++l) {
            if (!(b.tri == 0 || (b.tri == 1 ? l >= o : l <= o))) continue;
            ++visited;
            const int64_t e = b.off + l + o * b.so;
            if (e < 0 || e >= nt || seen[(size_t)e]++) {
              ++bad;
              continue;
            }
            const int i = b.lbase + l, j = b.obase + o, r = row[(size_t)e], c = col[(size_t)e];
            if (!((i == r && j == c) || (i == c && j == r))) ++wrong;
          }
        }
      }
  }
  out[0] = total;
  out[1] = visited;
  out[2] = bad;
  out[3] = wrong;
  out[4] = slots;
  out[5] = span;
  return 0;
}

// skinny_route of a product C (m x n) = A (m x k, strides a_rs, a_cs) B
// (k x n, column-major) with the given flags.  out: use, transpose, rows,
// instantiation, and the routed m, n, k.
int hs_skinny_route(int m, int n, int k, int k2, int a_tri, int b_tri, int c_lower, int inplace,
                    int64_t a_rs, int64_t a_cs, int* out) {
  static float buf[1];
  GemmProb g{};
  g.A = View{buf, a_rs, a_cs};
  g.B = View{buf, 1, k};
  g.C = View{buf, 1, m};
  g.A2 = g.A;
  g.B2 = g.B;
  g.m = m;
  g.n = n;
  g.k = k;
  g.k2 = k2;
  g.alpha = -1.0f;
  g.beta = 1.0f;
  g.a_tri = a_tri;
  g.b_tri = b_tri;
  g.c_lower = c_lower;
  g.inplace = inplace;
  GemmProb r{};
  const SkinnyRoute s = skinny_route(g, &r);
  out[0] = s.use;
  out[1] = s.transpose;
  out[2] = s.rows;
  out[3] = s.inst;
  out[4] = s.use ? r.m : 0;
  out[5] = s.use ? r.n : 0;
  out[6] = s.use ? r.k : 0;
  return 0;
}

// The split of k for `tiles` 64 x 64 tiles (few = 0) or m rows of a few-column
// product (few = 1).  out: splits, columns per split.
int hs_k_split(int few, int size, int k, int* out) {
  const KSplit s = few ? skinny_split(size, k) : tile_split(size, k);
  out[0] = s.splits;
  out[1] = s.kseg;
  return 0;
}

// The solve of an n-row triangle with m right-hand sides.  out: one launch (or
// the recursion), rows of the recursion's leaves, kernel of a launch.
int hs_solve_route(int fp32, int n, int m, int math, int* out) {
  out[0] = solve_in_one_launch(n, m, math);
  out[1] = solve_leaf_rows(m);
  out[2] = solve_kernel(fp32 != 0, n, m);
  return 0;
}

// A setting made once per device: `calls` devices are asked for in order, the
// setter fails for the fail_at-th run (-1: never).  out[i]: result of call i,
// + 2 if the setter ran.
int hs_once_per_device(int calls, const int* device, int fail_at, int* out) {
  OncePerDevice once;
  int runs = 0;
  for (int i = 0; i < calls; ++i) {
    bool ran = false;
    const bool ok = once(device[i], [&] {
      ran = true;
      return runs++ != fail_at;
    });
    out[i] = (ok ? 1 : 0) + (ran ? 2 : 0);
  }
  return 0;
}

}  // extern "C"
