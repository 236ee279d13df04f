// exec_cuda.cu — CUDA executor: turns planner primitives into sm_100a kernel
// launches on the handle's stream.
#include <algorithm>
#include <climits>
#include <cstdint>
#include <type_traits>

#include "context.h"
#include "func_attr.h"
#include "k_chain.cuh"
#include "k_chain1.cuh"
#include "k_chol.cuh"
#include "k_gemm.cuh"
#include "gemm_route.h"
#include "k_skinny.cuh"
#include "k_tile.cuh"
#include "k_tri.cuh"
#include "k_trsv.cuh"
#include "solve_route.h"

namespace rfp {

void* grow_buffer(curfpContext* ctx, void** buf, size_t* cur, size_t bytes) {
  ctx->scratch_used = true;
  if (*buf && *cur >= bytes) return *buf;
  if (*buf) {
    cudaFreeAsync(*buf, ctx->stream);
    *buf = nullptr;
  }
  // grow geometrically so that a recursion of increasing sizes reallocates
  // O(log) times
  size_t want = bytes < 256 ? 256 : bytes;
  if (*cur && want < *cur + *cur / 2) want = *cur + *cur / 2;
  void* p = nullptr;
  if (cudaMallocFromPoolAsync(&p, want, ctx->pool, ctx->stream) != cudaSuccess) {
    cudaGetLastError();
    want = bytes;  // retry without the growth margin
    if (cudaMallocFromPoolAsync(&p, want, ctx->pool, ctx->stream) != cudaSuccess) {
      cudaGetLastError();
      *cur = 0;
      return nullptr;
    }
  }
  *buf = p;
  *cur = want;
  return p;
}

namespace {
// Work captured into a graph neither records nor waits: the event belongs to
// what has been launched, and a wait for it would break the capture.  (An error:
// the legacy stream while another one captures.)
bool capturing(cudaStream_t stream) {
  cudaStreamCaptureStatus status;
  if (cudaStreamIsCapturing(stream, &status) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return status != cudaStreamCaptureStatusNone;
}
}  // namespace

ScratchScope::~ScratchScope() {
  if (!ctx_->scratch_used) return;
  ctx_->scratch_used = false;
  if (capturing(ctx_->stream)) return;
  if ((ctx_->ev_scratch ||
       cudaEventCreateWithFlags(&ctx_->ev_scratch, cudaEventDisableTiming) == cudaSuccess) &&
      cudaEventRecord(ctx_->ev_scratch, ctx_->stream) == cudaSuccess) {
    ctx_->scratch_pending = true;
    return;
  }
  cudaGetLastError();
  cudaStreamSynchronize(ctx_->stream);
}

void order_after_scratch(curfpContext* ctx, cudaStream_t stream) {
  if (!ctx->scratch_pending || capturing(stream)) return;
  if (cudaStreamWaitEvent(stream, ctx->ev_scratch, 0) == cudaSuccess) return;
  cudaGetLastError();
  cudaEventSynchronize(ctx->ev_scratch);
}

template <typename T>
T* CudaExecT<T>::workspace(size_t count) {
  return static_cast<T*>(grow_buffer(ctx_, &ctx_->ws, &ctx_->ws_bytes, count * sizeof(T)));
}

namespace {

// Clears a waiting kernel's flags and its ticket counter, which the self-test
// starts behind the tickets it leaves out.
int clear_sync(curfpContext* ctx, void* flags, size_t bytes, int* ticket) {
  if (cudaMemsetAsync(flags, 0, bytes, ctx->stream) != cudaSuccess) return 4;
  if (ctx->skip_tickets &&
      cudaMemcpyAsync(ticket, &ctx->skip_tickets, sizeof(int), cudaMemcpyHostToDevice,
                      ctx->stream) != cudaSuccess)
    return 4;
  return 0;
}

template <typename T, int BM, int BN>
int launch_gemm(const GemmProbT<T>* p, int count, const int* abort_flag,
                curfpContext* ctx, bool alloc = false) {
  cudaStream_t st = ctx->stream;
  double flops = 0;
  kgemm::Batch<T> b{};
  int tiles = 0, cnt = 0;
  for (int i = 0; i < count; ++i) {
    const GemmProbT<T>& g = p[i];
    if (g.m <= 0 || g.n <= 0) continue;
    kgemm::Prob<T>& q = b.p[cnt];
    q.A = g.A.p; q.a_rs = g.A.rs; q.a_cs = g.A.cs;
    q.B = g.B.p; q.b_rs = g.B.rs; q.b_cs = g.B.cs;
    q.A2 = g.A2.p; q.a2_rs = g.A2.rs; q.a2_cs = g.A2.cs;
    q.B2 = g.B2.p; q.b2_rs = g.B2.rs; q.b2_cs = g.B2.cs;
    q.C = g.C.p; q.c_rs = g.C.rs; q.c_cs = g.C.cs;
    q.m = g.m; q.n = g.n; q.k = g.k; q.k2 = g.k2;
    q.alpha = g.alpha; q.beta = g.beta;
    q.c_lower = g.c_lower;
    q.a_tri = g.a_tri; q.b_tri = g.b_tri; q.a2_tri = g.a2_tri; q.b2_tri = g.b2_tri;
    q.tiles_m = (g.m + BM - 1) / BM;
    q.tiles_n = (g.n + BN - 1) / BN;
    if (g.inplace && q.tiles_m != 1) return 3;  // planner contract
    if (g.c_lower && (q.tiles_m != q.tiles_n || BM != BN || g.m != g.n))
      return 3;
    q.tile_begin = tiles;
    tiles += g.c_lower ? q.tiles_m * (q.tiles_m + 1) / 2 : q.tiles_m * q.tiles_n;
    flops += 2.0 * g.m * g.n * (double)(g.k + g.k2) * (g.c_lower ? 0.5 : 1.0);
    ++cnt;
  }
  if (cnt == 0) return 0;
  b.count = cnt;
  b.total_tiles = tiles;
  b.abort_flag = abort_flag;
  // One unmasked product with few tiles and a long k (the solves' rectangle
  // updates): k is split so that about two CTAs per SM run, their partial
  // tiles added in order by split_reduce (2048 x 64, k = 2048: 32 CTAs 170 us,
  // with the split 60 us).
  int splits = 1;
  const kgemm::Prob<T>& q0 = b.p[0];
  if (alloc && cnt == 1 && !q0.k2 && !q0.a_tri && !q0.b_tri && !q0.c_lower && !p[0].inplace) {
    const KSplit ks = tile_split(tiles, q0.k);
    splits = ks.splits;
    b.kseg = ks.kseg;
  }
  if (splits > 1) {
    b.part = static_cast<T*>(grow_buffer(ctx, &ctx->wst, &ctx->wst_bytes,
                                         (size_t)splits * tiles * BM * BN * sizeof(T)));
    if (!b.part) splits = 1;  // no memory: one range, no scratch
  }
  ProfScope ps(ctx->prof, st, K_SGEMM, flops, 0);
  ps.shape(b.p[0].m, b.p[0].n, b.p[0].k + b.p[0].k2, tiles);
  bool blocked = false;
  if constexpr (BM == 64) {
    blocked = cnt == 1 && !q0.k2 && (q0.a_tri || q0.b_tri);
    if (blocked) kgemm::sgemm_batch<T, BM, BN, true><<<tiles, kgemm::kThreads, 0, st>>>(b);
  }
  if (!blocked)
    kgemm::sgemm_batch<T, BM, BN><<<dim3(tiles, splits), kgemm::kThreads, 0, st>>>(b);
  ++ctx->launches;
  if (splits > 1) {
    kgemm::split_reduce<T, BM, BN><<<tiles, kgemm::kThreads, 0, st>>>(b, splits);
    ++ctx->launches;
  }
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

// The few-column kernels (k_skinny.cuh) for the products gemm_route.h
// routes to them; -1 when it does not.
template <typename T>
int launch_skinny(const GemmProbT<T>& g0, const int* abort_flag, curfpContext* ctx, bool alloc) {
  GemmProbT<T> g;
  const SkinnyRoute r = skinny_route(g0, &g);
  if (!r.use) return -1;
  kskinny::Args<T> a{g.A.p, g.A.rs, g.A.cs, g.B.p, g.B.rs, g.B.cs, g.C.p, g.C.rs, g.C.cs,
                     g.m, g.n, g.k, g.alpha, g.beta, g.k, nullptr};
  ProfScope ps(ctx->prof, ctx->stream, K_SGEMM, 2.0 * g.m * g.n * (double)g.k,
               (double)sizeof(T) * g.m * (double)g.k);
  int splits = 1;
  if (alloc) {
    const KSplit ks = skinny_split(g.m, g.k);
    splits = ks.splits;
    a.kseg = ks.kseg;
  }
  if (splits > 1) {
    a.part = static_cast<T*>(grow_buffer(ctx, &ctx->wst, &ctx->wst_bytes,
                                         (size_t)splits * g.n * g.m * sizeof(T)));
    if (!a.part) {  // no memory: one range, no scratch
      splits = 1;
      a.kseg = g.k;
    }
  }
  const dim3 grid((g.m + 31) / 32, splits);
  cudaStream_t st = ctx->stream;
  auto go = [&](auto ncols) {
    constexpr int N = decltype(ncols)::value;
    if (r.rows) kskinny::skinny_rows<T, N><<<grid, kskinny::kThreads, 0, st>>>(a, abort_flag);
    else kskinny::skinny_cols<T, N><<<grid, kskinny::kThreads, 0, st>>>(a, abort_flag);
  };
  switch (r.inst) {
    case 1: go(std::integral_constant<int, 1>{}); break;
    case 2: go(std::integral_constant<int, 2>{}); break;
    case 4: go(std::integral_constant<int, 4>{}); break;
    default: go(std::integral_constant<int, 8>{}); break;
  }
  ++ctx->launches;
  if (splits > 1) {
    kskinny::skinny_reduce<T><<<dim3((g.m + kskinny::kThreads - 1) / kskinny::kThreads, g.n),
                                kskinny::kThreads, 0, st>>>(a, splits, abort_flag);
    ++ctx->launches;
  }
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

}  // namespace

namespace {
// Dst (packed, Src's contiguous dimension first) := Src (rows x cols view);
// lower: only elements with row >= column.  The warp runs along the
// contiguous dimension.
template <typename T>
__global__ void __launch_bounds__(256) copy_view(ViewT<T> dst, ViewT<T> src, int rows, int cols,
                                                 int lower, const int* abort_flag) {
  if (abort_flag && *abort_flag != INT_MAX) return;
  const bool rowcont = (src.cs == 1 || src.cs == -1) && !(src.rs == 1 || src.rs == -1);
  const int64_t inner = rowcont ? cols : rows, total = (int64_t)rows * cols;
  for (int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * 256) {
    const int64_t o = e / inner, k = e % inner;
    const int64_t r = rowcont ? o : k, c = rowcont ? k : o;
    if (!lower || r >= c) dst.p[r * dst.rs + c * dst.cs] = src.p[r * src.rs + c * src.cs];
  }
}

// L(i, j) := s(i, i) s(i, j) on the lower triangle.
template <typename T>
__global__ void __launch_bounds__(256) scale_by_diagonal(ViewT<T> L, ViewT<T> s, int n,
                                                         const int* abort_flag) {
  if (abort_flag && *abort_flag != INT_MAX) return;
  const bool rowcont = (L.cs == 1 || L.cs == -1) && !(L.rs == 1 || L.rs == -1);
  const int64_t total = (int64_t)n * n;
  for (int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * 256) {
    const int64_t o = e / n, k = e % n;
    const int64_t i = rowcont ? o : k, j = rowcont ? k : o;
    if (i >= j) L.p[i * L.rs + j * L.cs] = s.p[i * (s.rs + s.cs)] * s.p[i * s.rs + j * s.cs];
  }
}

// A packed copy of a view in the handle's tile workspace.
template <typename T>
int packed_copy(curfpContext* ctx, const int* abort_flag, ViewT<T> src, int rows, int cols,
                int lower, ViewT<T>* out) {
  const int64_t total = (int64_t)rows * cols;
  T* p = static_cast<T*>(
      grow_buffer(ctx, &ctx->wst, &ctx->wst_bytes, (size_t)total * sizeof(T)));
  if (!p) return 2;
  const bool rowcont = (src.cs == 1 || src.cs == -1) && !(src.rs == 1 || src.rs == -1);
  *out = rowcont ? ViewT<T>{p, cols, 1} : ViewT<T>{p, 1, rows};
  const int64_t blocks = (total + 1023) / 1024;
  ProfScope ps(ctx->prof, ctx->stream, K_PACK, 0, 2.0 * sizeof(T) * total);
  copy_view<T><<<(int)(blocks < 148 * 8 ? blocks : 148 * 8), 256, 0, ctx->stream>>>(
      *out, src, rows, cols, lower, abort_flag);
  ++ctx->launches;
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

// An in-place SIMT problem of more than one tile row reads a copy of B.
template <typename T>
int unalias(curfpContext* ctx, const int* abort_flag, GemmProbT<T>* g) {
  if (!g->inplace || g->m <= 64) return 0;
  ViewT<T> b;
  const int rc = packed_copy(ctx, abort_flag, g->B, g->k, g->n, 0, &b);
  if (rc) return rc;
  g->B = g->B2 = b;
  g->inplace = 0;
  return 0;
}
}  // namespace

// Output written through a column-contiguous view keeps the tensor-core
// epilogue's warp-wide stores coalesced: C = A B^T is computed as
// C^T = B A^T when C's contiguous dimension is its column index.
// Returns whether it swapped the operands.
static bool orient(View& A, int& arows, View& B, int& brows, SharedTask& t) {
  const bool col_contig = (t.C.cs == 1 || t.C.cs == -1) && !(t.C.rs == 1 || t.C.rs == -1);
  if (!col_contig) return false;
  View tv = A; A = B; B = tv;
  int tr_ = arows; arows = brows; brows = tr_;
  int x = t.a_row0; t.a_row0 = t.b_row0; t.b_row0 = x;
  x = t.m; t.m = t.n; t.n = x;
  t.C = tr(t.C);
  t.c_lower = t.c_lower ? 2 : 0;  // 2 = upper mask after transposition
  return true;
}

template <>
int CudaExecT<double>::gemm_shared(ViewT<double> X, int rows, int k,
                                   const SharedTaskT<double>* t, int count, int math) {
  return ExecT<double>::gemm_shared(X, rows, k, t, count, math);  // SIMT FP64 only
}

template <>
int CudaExecT<float>::gemm_shared(View X, int rows, int k, const SharedTask* t, int count,
                                  int math) {
  bool tc = math != 0 && count <= kMaxBatch;
  for (int i = 0; tc && i < count; ++i)
    tc = tc_worthwhile(t[i].m, t[i].n, k);
  if (!tc) return Exec::gemm_shared(X, rows, k, t, count, math);
  SharedTask tt[kMaxBatch];
  for (int i = 0; i < count; ++i) {
    tt[i] = t[i];
    View A = X, B{nullptr, 0, 0};
    int ar = rows, br = rows;
    orient(A, ar, B, br, tt[i]);  // shared operand: swapping keeps B == A
  }
  return tc_contract(ctx_, abort_, X, rows, View{nullptr, 0, 0}, rows, k, tt, count);
}

template <>
int CudaExecT<double>::gemm_pair(ViewT<double> X, ViewT<double> Y, int rows, int k,
                                 const SharedTaskT<double>* t, int count, int math) {
  return ExecT<double>::gemm_pair(X, Y, rows, k, t, count, math);  // SIMT FP64 only
}

// Rank-2k blocks on the tensor cores: two split-BF16 contractions over all
// blocks.  Launch 0 contracts (X, Y), launch 1 (Y, X).  A task whose C is
// column-contiguous is written transposed (orient()): C^T = Y[b] X[a]^T +
// X[b] Y[a]^T takes its two products from the launches in the other order,
// which sums to the same result.  beta applies in launch 0 only.
template <>
int CudaExecT<float>::gemm_pair(View X, View Y, int rows, int k, const SharedTask* t, int count,
                                int math) {
  bool tc = math != 0 && count <= kMaxBatch;
  for (int i = 0; tc && i < count; ++i)
    tc = tc_worthwhile(t[i].m, t[i].n, k);
  if (!tc) return Exec::gemm_pair(X, Y, rows, k, t, count, math);
  SharedTask tt[kMaxBatch];
  for (int pass = 0; pass < 2; ++pass) {
    View P = pass ? Y : X, Q = pass ? X : Y;
    for (int i = 0; i < count; ++i) {
      tt[i] = t[i];
      if (pass) tt[i].beta = 1.0f;
      View a = P, b = Q;
      int r0 = rows, r1 = rows;
      orient(a, r0, b, r1, tt[i]);  // only the task's rows and C are used here
    }
    const int rc = tc_contract(ctx_, abort_, P, rows, Q, rows, k, tt, count);
    if (rc) return rc;
  }
  return 0;
}

template <>
int CudaExecT<double>::gemm(const GemmProbT<double>* p, int count) {
  if (count <= 0) return 0;
  if (count > kMaxBatch) return 3;
  if (count == 1) {
    const int rc = launch_skinny<double>(p[0], abort_, ctx_, may_allocate());
    if (rc >= 0) return rc;
  }
  GemmProbT<double> q;
  if (count == 1 && p[0].inplace) {
    q = p[0];
    const int rc = unalias(ctx_, abort_, &q);
    if (rc) return rc;
    p = &q;
  }
  // 128 x 128 tiles (64 accumulators per thread, one CTA per SM) when they
  // fill the machine, else 64 x 64
  int64_t t128 = 0;
  bool inplace = false;
  for (int i = 0; i < count; ++i) {
    const int64_t tm = (p[i].m + 127) / 128, tn = (p[i].n + 127) / 128;
    t128 += p[i].c_lower ? tm * (tm + 1) / 2 : tm * tn;
    inplace = inplace || p[i].inplace;
  }
  if (t128 >= 148 && !inplace) return launch_gemm<double, 128, 128>(p, count, abort_, ctx_);
  return launch_gemm<double, 64, 64>(p, count, abort_, ctx_, may_allocate());
}

template <>
int CudaExecT<float>::gemm(const GemmProb* p, int count) {
  if (count <= 0) return 0;
  if (count > kMaxBatch) return 3;
  if (count == 1) {
    const int rc = launch_skinny<float>(p[0], abort_, ctx_, may_allocate());
    if (rc >= 0) return rc;
  }
  // One problem, one or two products, on the tensor cores: the A operands
  // may be triangular (lower / upper, staged with zeros), the B operands
  // full; the second product accumulates with beta = 1.
  // An in-place problem (C aliases B) qualifies when its operands are staged
  // whole before the product runs (one slab, one product).
  if (count == 1 && p[0].math && p[0].b_tri == 0 && p[0].b2_tri == 0 &&
      p[0].a_tri <= 2 && p[0].a2_tri <= 2 && tc_worthwhile(p[0].m, p[0].n, p[0].k) &&
      (p[0].k2 == 0 || tc_worthwhile(p[0].m, p[0].n, p[0].k2)) &&
      (!p[0].inplace ||
       (p[0].k2 == 0 && tc_single_slab(p[0].m > p[0].n ? p[0].m : p[0].n, p[0].k)))) {
    const GemmProb& g = p[0];
    for (int prod = 0; prod < (g.k2 ? 2 : 1); ++prod) {
      View A = prod ? g.A2 : g.A, Bt = tr(prod ? g.B2 : g.B);  // A: m x k, Bt: n x k
      int ar = g.m, br = g.n;
      int amask = prod ? g.a2_tri : g.a_tri, bmask = 0;
      SharedTask t{0, 0, g.m, g.n, g.C, g.alpha, prod ? 1.0f : g.beta, g.c_lower};
      if (orient(A, ar, Bt, br, t)) {  // operands swapped: the mask moves with A
        bmask = amask;
        amask = 0;
      }
      const int rc = (amask || bmask)
                         ? tc_contract_masked(ctx_, abort_, A, ar, amask, Bt, br, bmask,
                                              prod ? g.k2 : g.k, &t, 1)
                         : tc_contract(ctx_, abort_, A, ar, Bt, br, prod ? g.k2 : g.k, &t, 1);
      if (rc) return rc;
    }
    return 0;
  }
  GemmProb q;
  if (count == 1 && p[0].inplace) {
    q = p[0];
    const int rc = unalias(ctx_, abort_, &q);
    if (rc) return rc;
    p = &q;
  }
  // Tile choice: 128 x 128 when it fills the machine, else 64 x 64.
  int64_t t128 = 0;
  int maxm = 0;
  for (int i = 0; i < count; ++i) {
    int64_t tm = (p[i].m + 127) / 128, tn = (p[i].n + 127) / 128;
    t128 += p[i].c_lower ? tm * (tm + 1) / 2 : tm * tn;
    if (p[i].inplace && p[i].m > maxm) maxm = p[i].m;
  }
  if (t128 >= 2 * 148 && maxm == 0)
    return launch_gemm<float, 128, 128>(p, count, abort_, ctx_);
  return launch_gemm<float, 64, 64>(p, count, abort_, ctx_, may_allocate());
}

template <typename T>
int CudaExecT<T>::potrf_adj_tile(ViewT<T> L, ViewT<T> G, int n) {
  if (n <= 0) return 0;
  if (n > ktile::T) return 3;
  ProfScope ps(ctx_->prof, ctx_->stream, K_POTRF, 2.0 * n * (double)n * n / 3.0, 0);
  constexpr int smem = ktile::adj_smem<T>();
  static OncePerDevice attr;
  if (!smem_attr(attr, ctx_->device, ktile::potrf_adj_tile<T>, smem)) return 4;
  ktile::potrf_adj_tile<T><<<1, ktile::ADJ_THREADS, smem, ctx_->stream>>>(L, G, n);
  ++ctx_->launches;
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

namespace {
// The tile Cholesky (k_chol.cuh) of the logical lower blocks V11, V21, V22,
// or with panel set of V11 and V21 alone.
template <typename T>
int launch_chol(curfpContext* ctx, ViewT<T> V11, ViewT<T> V21, ViewT<T> V22, int n1, int n2,
                bool panel, int info_base) {
  kchol::Args<T> a{};
  a.v11 = V11; a.v21 = V21; a.v22 = V22;
  a.n1 = n1; a.n2 = n2;
  a.nb1 = (n1 + kchol::NB - 1) / kchol::NB;
  a.nb = a.nb1 + (n2 + kchol::NB - 1) / kchol::NB;
  a.nbf = panel ? a.nb1 : a.nb;
  const size_t tiles = (size_t)kchol::tile_count(a.nb, a.nbf), words = 1 + tiles;
  a.ws = static_cast<T*>(
      grow_buffer(ctx, &ctx->ws, &ctx->ws_bytes, tiles * kchol::TILE * sizeof(T)));
  if (!a.ws) return 2;
  const int ctas = kchol::cta_count(a.nb, a.nbf) - ctx->skip_tickets;
  if (ctas > 1) {
    a.sync = static_cast<int*>(grow_buffer(ctx, &ctx->tsv, &ctx->tsv_bytes, words * sizeof(int)));
    if (!a.sync) return 2;
    if (clear_sync(ctx, a.sync, words * sizeof(int), a.sync)) return 4;
  }
  a.info = ctx->d_info;
  a.err = ctx->d_info + 1;
  a.info_base = info_base;
  constexpr int smem = kchol::smem_bytes<T>();
  static OncePerDevice attr;
  if (!smem_attr(attr, ctx->device, kchol::chol_wave<T>, smem)) return 4;
  const double n = (double)n1 + n2, m = panel ? n2 : 0;
  ProfScope ps(ctx->prof, ctx->stream, K_POTRF,
               panel ? (n1 / 3.0 + m) * n1 * n1 : n * n * n / 3.0, 0);
  ps.shape(n1, n2, panel ? 1 : 0, (int)tiles);
  kchol::chol_wave<T><<<ctas, kchol::threads<T>(), smem, ctx->stream>>>(a);
  ++ctx->launches;
  ++ctx->wait_launches;
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}
}  // namespace

template <typename T>
int CudaExecT<T>::potrf_tile(ViewT<T> L, int n, int info_base) {
  if (n <= 0) return 0;
  if (n > potrf_tile_rows()) return 3;
  return launch_chol<T>(ctx_, L, L, L, n, 0, false, info_base);
}

template <typename T>
int CudaExecT<T>::potrf_blocks(ViewT<T> V11, ViewT<T> V21, ViewT<T> V22, int n1, int n2) {
  if (n1 + n2 > kCholRfpRows || (sizeof(T) == 4 && tc_worthwhile(n2, n2, n1)))
    return kNotSupported;
  const int rc = after_first_block();
  return rc ? rc : launch_chol<T>(ctx_, V11, V21, V22, n1, n2, false, 0);
}

template <typename T>
bool CudaExecT<T>::has_panel(int n1, int n2) const {
  return n1 > 0 && n2 > 0 && n1 <= potrf_tile_rows() && n2 <= kCholPanelRows;
}

template <typename T>
int CudaExecT<T>::potrf_panel(ViewT<T> L, ViewT<T> A21, int n1, int n2, int info_base) {
  return launch_chol<T>(ctx_, L, A21, A21, n1, n2, true, info_base);
}

template <typename T>
int CudaExecT<T>::trtri_batch(const ViewT<T>* L, const int* n, int count, T* W) {
  ktile::TriBatch<T> b{};
  if (count > ktile::TriBatch<T>::MAX) return 3;
  int blocks = 0;
  double flops = 0;
  for (int i = 0; i < count; ++i) {
    b.L[i] = L[i];
    b.n[i] = n[i];
    b.begin[i] = blocks;
    blocks += n[i] > 0 ? (n[i] + ktile::T - 1) / ktile::T : 0;
    flops += (double)n[i] * ktile::T * ktile::T / 3.0;
  }
  if (blocks == 0) return 0;
  b.count = count;
  b.W = W;
  ProfScope ps(ctx_->prof, ctx_->stream, K_TRTRI, flops, 0);
  constexpr int smem = ktile::trtri_smem<T>();
  static OncePerDevice attr;
  if (!smem_attr(attr, ctx_->device, ktile::trtri_blocks<T>, smem)) return 4;
  ktile::trtri_blocks<T><<<blocks, ktile::TRTRI_THREADS, smem, ctx_->stream>>>(b, abort_);
  ++ctx_->launches;
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

template <typename T>
int CudaExecT<T>::trtri_blocks(ViewT<T> L, int n, int nb, T* W) {
  if (n <= 0) return 0;
  if (nb != ktile::T) return 3;
  return trtri_batch(&L, &n, 1, W);
}

template <typename T>
int CudaExecT<T>::trtri_tile(ViewT<T> L, int n) {
  if (n <= 0) return 0;
  if (n > ktile::T) return 3;
  return trtri_batch(&L, &n, 1, nullptr);
}

template <typename T>
int CudaExecT<T>::trtri_block(ViewT<T> L, int n) {
  if (n <= 0) return 0;
  if (n <= ktile::T) return trtri_tile(L, n);
  const int nblk = (n + kTrsmLeaf - 1) / kTrsmLeaf;
  T* W = workspace((size_t)nblk * kInvStride);
  if (!W) return 2;
  const int rc = trtri_blocks(L, n, kTrsmLeaf, W);
  if (rc) return rc;
  ktri::Args<T> a{};
  a.L = L;
  a.n = n;
  a.W = W;
  const int tiles = nblk * (nblk + 1) / 2;
  const size_t words = 1 + (size_t)tiles;
  a.ws = static_cast<T*>(grow_buffer(ctx_, &ctx_->wst, &ctx_->wst_bytes,
                                     (size_t)tiles * ktri::TILE * sizeof(T)));
  a.sync = static_cast<int*>(grow_buffer(ctx_, &ctx_->tsv, &ctx_->tsv_bytes, words * sizeof(int)));
  if (!a.ws || !a.sync) return 2;
  if (clear_sync(ctx_, a.sync, words * sizeof(int), a.sync)) return 4;
  a.err = ctx_->d_info + 1;
  a.abort_flag = abort_;
  constexpr int smem = ktri::smem_bytes<T>();
  static OncePerDevice attr;
  if (!smem_attr(attr, ctx_->device, ktri::inverse_wave<T>, smem)) return 4;
  ProfScope ps(ctx_->prof, ctx_->stream, K_TRTRI, (double)n * n * n / 3, 0);
  ps.shape(n, n, n, tiles);
  ktri::inverse_wave<T><<<tiles - ctx_->skip_tickets, ktri::THR, smem, ctx_->stream>>>(a);
  ktri::store_inverse<T><<<tiles, ktri::THR, 0, ctx_->stream>>>(L, n, a.ws, abort_);
  ctx_->launches += 2;
  ++ctx_->wait_launches;
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

template <typename T>
int CudaExecT<T>::lauum_tile(ViewT<T> L, int n) {
  if (n <= 0) return 0;
  if (n > ktile::T) return 3;
  ProfScope ps(ctx_->prof, ctx_->stream, K_LAUUM, (double)n * n * n / 3.0, 0);
  ktile::lauum_tile<T><<<1, 256, 0, ctx_->stream>>>(L, n);
  ++ctx_->launches;
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

// L := L^T L (lower) as one product: with L = D + N,
// (L^T L)(i, j) = d_i L(i, j) + (N^T N)(i, j) for i >= j, masked operands read
// from a packed copy of L.  (A sum that starts at a dominant d_i^2 rounds every
// later term against it: diagonal error 2.4e-6 against 7e-7 at n = 6001.)
template <typename T>
int CudaExecT<T>::lauum_block(ViewT<T> L, int n) {
  if (n <= ktile::T) return lauum_tile(L, n);
  ViewT<T> c;
  const int rc = packed_copy(ctx_, abort_, L, n, n, 1, &c);
  if (rc) return rc;
  GemmProbT<T> p{};
  p.A = p.A2 = tr(c);
  p.B = p.B2 = c;
  p.C = L;
  p.m = p.n = p.k = n;
  p.alpha = p.beta = T(1);
  p.c_lower = 1;
  p.a_tri = 3;
  p.b_tri = 1;
  {
    ProfScope ps(ctx_->prof, ctx_->stream, K_LAUUM, 0, 0);
    const int64_t blocks = ((int64_t)n * n + 1023) / 1024;
    scale_by_diagonal<T><<<(int)(blocks < 148 * 8 ? blocks : 148 * 8), 256, 0, ctx_->stream>>>(
        L, c, n, abort_);
    ++ctx_->launches;
  }
  return gemm(&p, 1);
}

namespace {
// The wavefront solve, 64 right-hand-side columns per CTA.
template <typename T>
int launch_wave(curfpContext* ctx, const int* abort_flag, ViewT<T> L, int n, ViewT<T> B, int m,
                T alpha, const T* W) {
  const int nblk = (n + ktrsv::NB - 1) / ktrsv::NB, nchunk = (m + ktrsv::NB - 1) / ktrsv::NB;
  const size_t words = 1 + (size_t)nblk * nchunk;
  int* sync = static_cast<int*>(grow_buffer(ctx, &ctx->tsv, &ctx->tsv_bytes, words * 4));
  if (!sync) return 2;
  if (clear_sync(ctx, sync, words * 4, sync)) return 4;
  constexpr int smem = ktrsv::smem_bytes<T>();
  static OncePerDevice attr;
  if (!smem_attr(attr, ctx->device, ktrsv::trsm_wave<T>, smem)) return 4;
  ProfScope ps(ctx->prof, ctx->stream, K_TRSV, (double)n * n * m,
               (double)n * n * sizeof(T) / 2.0);
  ps.shape(n, m, n, nblk * nchunk);
  ktrsv::trsm_wave<T><<<nblk * nchunk - ctx->skip_tickets, 256, smem, ctx->stream>>>(
      L, n, B, m, alpha, W, sync, ctx->d_info + 1, abort_flag);
  ++ctx->launches;
  ++ctx->wait_launches;
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}
}  // namespace

namespace {
// The solve whose chain runs inside clusters (k_chain.cuh), NC columns a chunk.
template <typename T, int NC>
int launch_chain(curfpContext* ctx, const int* abort_flag, ViewT<T> L, int n, ViewT<T> B, int m,
                 T alpha, const T* W) {
  using C = kchain::Cfg<T, NC>;
  kchain::Args<T> a{};
  a.L = L; a.B = B;
  a.n = n; a.m = m;
  a.nblk = (n + kchain::NB - 1) / kchain::NB;
  a.nchunk = (m + NC - 1) / NC;
  a.alpha = alpha;
  a.W = W;
  const size_t tiles = (size_t)a.nblk * a.nchunk, words = 1 + tiles;
  a.ws = static_cast<T*>(
      grow_buffer(ctx, &ctx->wst, &ctx->wst_bytes, tiles * C::XT * sizeof(T)));
  a.sync = static_cast<int*>(grow_buffer(ctx, &ctx->tsv, &ctx->tsv_bytes, words * sizeof(int)));
  if (!a.ws || !a.sync) return 2;
  if (clear_sync(ctx, a.sync, words * sizeof(int), a.sync)) return 4;
  a.err = ctx->d_info + 1;
  a.abort_flag = abort_flag;
  static OncePerDevice attr;
  if (!smem_attr(attr, ctx->device, kchain::trsm_chain<T, NC>, C::SMEM)) return 4;
  ProfScope ps(ctx->prof, ctx->stream, K_TRSV, (double)n * n * m, (double)n * n * sizeof(T) / 2.0);
  ps.shape(n, m, n, (int)tiles);
  const int clusters = (a.nblk + kchain::CS - 1) / kchain::CS * a.nchunk - ctx->skip_tickets;
  kchain::trsm_chain<T, NC><<<clusters * kchain::CS, kchain::THR, C::SMEM, ctx->stream>>>(a);
  ++ctx->launches;
  ++ctx->wait_launches;
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}
// One FP32 right-hand side (k_chain1.cuh).
int launch_chain1(curfpContext* ctx, const int* abort_flag, View L, int n, View B, float alpha,
                  const float* W) {
  kchain1::Args a{};
  a.L = L; a.B = B;
  a.n = n;
  a.nblk = (n + kchain::NB - 1) / kchain::NB;
  a.alpha = alpha;
  a.W = W;
  const size_t words = (size_t)a.nblk * kchain::NB + 1;  // the ticket follows the words
  a.ws = static_cast<unsigned long long*>(
      grow_buffer(ctx, &ctx->tsv, &ctx->tsv_bytes, words * sizeof(unsigned long long)));
  if (!a.ws) return 2;
  a.sync = reinterpret_cast<int*>(a.ws + words - 1);
  if (clear_sync(ctx, a.ws, words * sizeof(unsigned long long), a.sync)) return 4;
  a.err = ctx->d_info + 1;
  a.abort_flag = abort_flag;
  ProfScope ps(ctx->prof, ctx->stream, K_TRSV, (double)n * n, (double)n * n * 2.0);
  ps.shape(n, 1, n, a.nblk);
  const int clusters = (a.nblk + kchain::CS - 1) / kchain::CS - ctx->skip_tickets;
  kchain1::chain1<<<clusters * kchain::CS, kchain1::THR, 0, ctx->stream>>>(a);
  ++ctx->launches;
  ++ctx->wait_launches;
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}
}  // namespace

namespace {
// Many right-hand sides: 64 x 64 tiles handed on through the workspace (k_tri.cuh).
template <typename T>
int launch_solve_tiles(curfpContext* ctx, const int* abort_flag, ViewT<T> L, int n, ViewT<T> B,
                       int m, T alpha, const T* W) {
  ktri::SolveArgs<T> a{};
  a.B = B;
  a.n = n; a.m = m;
  a.nblk = (n + ktri::NB - 1) / ktri::NB;
  a.nchunk = (m + ktri::NB - 1) / ktri::NB;
  a.alpha = alpha;
  a.W = W;
  const size_t tiles = (size_t)a.nblk * a.nchunk, words = 1 + tiles;
  const int lower = a.nblk * (a.nblk - 1) / 2;  // packed tiles of L, then X's
  T* const ws = static_cast<T*>(grow_buffer(
      ctx, &ctx->wst, &ctx->wst_bytes,
      (lower + tiles - a.nchunk + 1) * ktri::TILE * sizeof(T)));
  a.Lp = ws;
  a.ws = ws + (size_t)lower * ktri::TILE;
  a.sync = static_cast<int*>(grow_buffer(ctx, &ctx->tsv, &ctx->tsv_bytes, words * sizeof(int)));
  if (!ws || !a.sync) return 2;
  if (clear_sync(ctx, a.sync, words * sizeof(int), a.sync)) return 4;
  a.err = ctx->d_info + 1;
  a.abort_flag = abort_flag;
  constexpr int smem = ktri::smem_bytes<T>();
  static OncePerDevice attr;
  if (!smem_attr(attr, ctx->device, ktri::solve_tiles<T>, smem)) return 4;
  ProfScope ps(ctx->prof, ctx->stream, K_TRSV, (double)n * n * m, (double)n * n * sizeof(T) / 2.0);
  ps.shape(n, m, n, (int)tiles);
  if (lower > 0) {
    ktri::pack_lower<T><<<lower, ktri::THR, 0, ctx->stream>>>(L, n, ws, abort_flag);
    ++ctx->launches;
  }
  ktri::solve_tiles<T><<<(int)tiles - ctx->skip_tickets, ktri::THR, smem, ctx->stream>>>(a);
  ++ctx->launches;
  ++ctx->wait_launches;
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}
}  // namespace

// The kernels' choice: solve_route.h.  The wavefront solve needs the least
// scratch (its flags); it stands in where another kernel's does not fit (rc 2:
// nothing was launched).
template <typename T>
int CudaExecT<T>::trsm_wave(ViewT<T> L, int n, ViewT<T> B, int m, T alpha, const T* W) {
  if (n <= 0 || m <= 0) return 0;
  const SolveKernel kernel = solve_kernel(sizeof(T) == 4, n, m);
  int rc = 2;
  if constexpr (sizeof(T) == 4) {
    switch (kernel) {
      case SOLVE_CHAIN1: rc = launch_chain1(ctx_, abort_, L, n, B, alpha, W); break;
      case SOLVE_CHAIN16: rc = launch_chain<T, 16>(ctx_, abort_, L, n, B, m, alpha, W); break;
      case SOLVE_CHAIN32: rc = launch_chain<T, 32>(ctx_, abort_, L, n, B, m, alpha, W); break;
      case SOLVE_TILES: rc = launch_solve_tiles<T>(ctx_, abort_, L, n, B, m, alpha, W); break;
      default: break;
    }
  }
  if (kernel == SOLVE_CHAIN8) rc = launch_chain<T, 8>(ctx_, abort_, L, n, B, m, alpha, W);
  return rc == 2 ? launch_wave<T>(ctx_, abort_, L, n, B, m, alpha, W) : rc;
}

template class CudaExecT<float>;
template class CudaExecT<double>;

// Bounded-wait self-test of one waiting kernel through its ordinary launch, the
// CTAs of its first ticket (the first tile; in the two cluster chains the first
// eight block rows) left out.  The operands are zeros and live in a buffer
// that no launch takes scratch from.
int wait_selftest(curfpContext* ctx, int kind) {
  constexpr int n = 1024, m = 4096, nblk = n / kTrsmLeaf;
  constexpr size_t nb = (size_t)192 * m;  // right-hand sides: 1024 x 9, 192 x 600, 192 x 4096
  constexpr size_t fl = (size_t)n * n + nb + (size_t)nblk * kInvStride;
  float* L = static_cast<float*>(
      grow_buffer(ctx, &ctx->wsg, &ctx->wsg_bytes, fl * sizeof(float)));
  if (!L) return 2;
  if (cudaMemsetAsync(L, 0, fl * sizeof(float), ctx->stream) != cudaSuccess) return 4;
  float* B = L + (size_t)n * n;
  const float* W = B + nb;
  CudaExec ex(ctx);
  ctx->skip_tickets = 1;
  int rc = 3;
  switch (kind) {
    case 0: rc = ex.trsm_wave(View{L, n, 1}, n, View{B, 1, n}, 1, 1.0f, W); break;    // chain1
    case 1: rc = ex.trsm_wave(View{L, n, 1}, n, View{B, 1, n}, 9, 1.0f, W); break;    // trsm_chain
    case 2: rc = ex.trsm_wave(View{L, n, 1}, 192, View{B, 1, 192}, 600, 1.0f, W); break;  // trsm_wave
    case 3: rc = ex.trsm_wave(View{L, n, 1}, 192, View{B, 1, 192}, m, 1.0f, W); break;  // solve_tiles
    case 4: rc = ex.trtri_block(View{L, n, 1}, 192); break;                          // inverse_wave
    case 5: rc = ex.potrf_tile(View{L, n, 1}, 192, 0); break;                        // chol_wave
  }
  ctx->skip_tickets = 0;
  return rc;
}

int launch_trsm_wave_fixed(curfpContext* ctx, const int* abort_flag, View L, int n, View B,
                           int m, float alpha, const float* W, int* sync, size_t sync_words) {
  if (n <= 0 || m <= 0) return 0;
  const int nblk = (n + ktrsv::NB - 1) / ktrsv::NB, nchunk = (m + ktrsv::NB - 1) / ktrsv::NB;
  const size_t words = 1 + (size_t)nblk * nchunk;
  if (words > sync_words) return 3;
  if (cudaMemsetAsync(sync, 0, words * 4, ctx->stream) != cudaSuccess) return 4;
  constexpr int smem = ktrsv::smem_bytes<float>();
  static OncePerDevice attr;
  if (!smem_attr(attr, ctx->device, ktrsv::trsm_wave<float>, smem)) return 4;
  ProfScope ps(ctx->prof, ctx->stream, K_TRSV, (double)n * n * m, (double)n * n * 2.0);
  ktrsv::trsm_wave<float><<<nblk * nchunk, 256, smem, ctx->stream>>>(
      L, n, B, m, alpha, W, sync, ctx->d_info + 1, abort_flag);
  ++ctx->launches;
  ++ctx->wait_launches;
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

}  // namespace rfp
