// context.h — the library handle (struct curfpContext) and the CUDA executor.
//
// The reference context wraps a cuBLAS and a cuSOLVER handle
// (src/curfp_internal.h:11-14); this one holds what the native kernels need:
// the stream, the device, one device-side info word (pivot failures, also used
// as the abort flag that makes later kernels of a failed factorization return
// immediately), a kernel error word, grow-only stream-ordered workspaces and
// the staging buffers of the split-BF16 path.  Workspaces come from the
// handle's own memory pool (created with the handle, kept across calls), so
// the device's default pool and its settings are left to the caller.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

#include "engine.h"
#include "profile.h"

struct curfpContext {
  cudaStream_t stream = nullptr;
  int device = 0;
  cudaMemPool_t pool = nullptr;  // the handle's workspace pool
  int math = 1;            // contraction arithmetic of the drop-in routines (curfpSetMathMode)
  long long wait_launches = 0;  // kernels with bounded waits launched (status.cuh)
  int skip_tickets = 0;    // self-test: first tickets of a waiting kernel that no CTA takes
  int* d_info = nullptr;   // [0]: INT_MAX = no pivot failure; [1]: kernel error code
  void* ws = nullptr;      // TRSM diagonal-block inverses and other scratch
  size_t ws_bytes = 0;
  void* stage = nullptr;   // split-BF16 operand staging (first operand)
  size_t stage_bytes = 0;
  void* stage2 = nullptr;  // split-BF16 operand staging (second operand)
  size_t stage2_bytes = 0;
  void* ws2 = nullptr;     // refinement scratch (saved RHS, residual)
  size_t ws2_bytes = 0;
  void* ws3 = nullptr;     // FP64 accumulator of split symmetric multiplies
  size_t ws3_bytes = 0;
  long long launches = 0;  // kernels launched through this handle
  rfp::Profiler prof;      // optional per-class event timing
  void* tsv = nullptr;     // wavefront solve flags / tickets
  size_t tsv_bytes = 0;
  void* wst = nullptr;     // tiles published by the wavefront solves, packed operand copies
  size_t wst_bytes = 0;
  void* wsg = nullptr;     // adjoint scratch (solve adjoint n x 2nrhs, NLL gradient)
  size_t wsg_bytes = 0;
  // Workspaces are one set per handle, whatever its stream: an entry point that
  // returns with work on them still in flight records ev_scratch behind it, and
  // the stream that the handle is bound to next waits for it.
  bool scratch_used = false;     // a workspace was handed out since the last record or synchronisation
  bool scratch_pending = false;  // ev_scratch is recorded
  cudaEvent_t ev_scratch = nullptr;
  cudaStream_t copy_stream = nullptr;  // host-input factorization: the overlapped copy
  cudaEvent_t ev_start = nullptr, ev_rest = nullptr;
};

namespace rfp {

// What the tile Cholesky (k_chol.cuh) takes in one launch: a diagonal block
// of up to kCholRows, with up to kCholPanelRows rows below it, and a whole RFP
// matrix of up to kCholRfpRows (FP64), or up to where its trailing update is
// large enough for the tensor cores (FP32, order 1300, in both math modes).  The
// lines are where the launch has been proven, not where it stops winning.  One
// launch against panel and update: FP32 n = 1300 311 / 358 us, 3000 651 / 716, 4096
// 1097 / 1033 (FP32 mode 306 / 375, 651 / 853, 1098 / 1244); FP64 n = 5000 3.8 / 5.6
// ms, 8192 12.4 / 14.2.
constexpr int kCholRows = 2048;
constexpr int kCholPanelRows = 2048;
constexpr int kCholRfpRows = 4096;
// Triangular inverses of up to kTriRows are one wave; L^T L products and
// in-place triangular multiplies of up to kLeafRows are one masked product on
// the SIMT cores (on a copy of the operand).  Not on the tensor cores: a row's
// digits are relative to its largest element, and an inverse factor's rows
// have a dominant diagonal (n = 6001 inverse, error against FP64: 1.8e-5 with
// 2048-row blocks on the tensor cores, 5e-7 with the diagonal kept apart,
// 1.3e-7 this way, 1.8e-7 with 64-row leaves).  1024 against 512 rows: 6.2
// against 7.5 ms for that inverse (25.6 ms with 64-row leaves).
constexpr int kTriRows = 2048;
constexpr int kLeafRows = 1024;

// An entry point's use of the workspaces (exec_cuda.cu): records ev_scratch at
// its end unless it synchronised after the last use.
class ScratchScope {
 public:
  explicit ScratchScope(curfpContext* ctx) : ctx_(ctx) {}
  ScratchScope(const ScratchScope&) = delete;
  ScratchScope& operator=(const ScratchScope&) = delete;
  ~ScratchScope();

 private:
  curfpContext* ctx_;
};
// Orders `stream` after the recorded use of the workspaces.
void order_after_scratch(curfpContext* ctx, cudaStream_t stream);

// The CUDA executor for FP32 (SIMT and split-BF16 tensor-core contractions)
// and FP64 (SIMT DFMA) element types.
template <typename T>
class CudaExecT : public ExecT<T> {
 public:
  explicit CudaExecT(curfpContext* ctx, const int* abort_flag = nullptr)
      : ctx_(ctx), abort_(abort_flag), scratch_(ctx) {}
  int gemm(const GemmProbT<T>* p, int count) override;
  int potrf_tile(ViewT<T> L, int n, int info_base) override;
  int potrf_tile_rows() const override { return kCholRows; }
  int potrf_blocks(ViewT<T> V11, ViewT<T> V21, ViewT<T> V22, int n1, int n2) override;
  bool has_panel(int n1, int n2) const override;
  int potrf_panel(ViewT<T> L, ViewT<T> A21, int n1, int n2, int info_base) override;
  int trtri_blocks(ViewT<T> L, int n, int nb, T* W) override;
  int trtri_tile(ViewT<T> L, int n) override;
  int lauum_tile(ViewT<T> L, int n) override;
  T* workspace(size_t count) override;
  int trtri_rows() const override { return kTriRows; }
  int trtri_block(ViewT<T> L, int n) override;
  int lauum_rows() const override { return kLeafRows; }
  int lauum_block(ViewT<T> L, int n) override;
  int inplace_rows() const override { return kLeafRows; }
  int gemm_shared(ViewT<T> X, int rows, int k, const SharedTaskT<T>* t, int count,
                  int math) override;
  int gemm_pair(ViewT<T> X, ViewT<T> Y, int rows, int k, const SharedTaskT<T>* t, int count,
                int math) override;
  int trsm_wave(ViewT<T> L, int n, ViewT<T> B, int m, T alpha, const T* W) override;
  int potrf_adj_tile(ViewT<T> L, ViewT<T> G, int n) override;
  // Whether products may take scratch for split sums from the workspaces.
  virtual bool may_allocate() const { return true; }
  bool batch_inverses() const override { return may_allocate(); }
  int trtri_batch(const ViewT<T>* L, const int* n, int count, T* W) override;
  // When set, work after the first diagonal block waits for this event.
  int after_first_block() override {
    if (!rest_ready) return 0;
    return cudaStreamWaitEvent(ctx_->stream, rest_ready, 0) == cudaSuccess ? 0 : 4;
  }
  cudaEvent_t rest_ready = nullptr;

 protected:
  curfpContext* ctx_;
  const int* abort_;

 private:
  ScratchScope scratch_;
};
using CudaExec = CudaExecT<float>;
using CudaExecD = CudaExecT<double>;

// Grow a stream-ordered buffer to at least `bytes`; returns nullptr on failure.
void* grow_buffer(curfpContext* ctx, void** buf, size_t* cur, size_t bytes);

// Split-BF16 tensor-core contraction (tc_engine.cu).  C_t := alpha_t *
// A[a_row0:+m, :] B[b_row0:+n, :]^T + beta_t C_t with A (arows x k) and B
// (brows x k) FP32 views; B.p == nullptr means B is A.
int tc_contract(curfpContext* ctx, const int* abort_flag, View A, int arows, View B,
                int brows, int k, const SharedTask* tasks, int count);
// The same with triangular operand masks (0 full, 1 keep column <= row,
// 2 keep column >= row, columns counted over the whole k range): masked
// elements are staged as zeros and never read.  B.p must be set.
int tc_contract_masked(curfpContext* ctx, const int* abort_flag, View A, int arows, int amask,
                       View B, int brows, int bmask, int k, const SharedTask* tasks,
                       int count);
// The wavefront solve with a caller-provided flag buffer of sync_words words
// (cleared here on the stream); no allocation.
int launch_trsm_wave_fixed(curfpContext* ctx, const int* abort_flag, View L, int n, View B,
                           int m, float alpha, const float* W, int* sync, size_t sync_words);
// Bounded-wait self-tests (exec_cuda.cu), kind 0 to kWaitSelftests - 1: each
// launches one waiting kernel whose first ticket no CTA takes; the CTAs that
// depend on it time out (~2 s) and set error code 5 in ctx->d_info[1].
constexpr int kWaitSelftests = 6;
int wait_selftest(curfpContext* ctx, int kind);
// Whether a contraction of this size goes to the tensor-core path.
bool tc_worthwhile(int m, int n, int k);
// Whether a contraction with operands of at most `rows` rows stages its
// whole k range at once (no k slabs): every operand is then read before the
// product writes C, so C may alias an operand.
bool tc_single_slab(int rows, int k);

}  // namespace rfp
