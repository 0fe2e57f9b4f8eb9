// Launch sequences of a backward pass behind one call each: what a pass on one device launches anyway, in the same order on the same
// stream, without a return to Python between the launches. Between kernels of 3 to 15 us that return is what the device waits for: a
// call through Python takes 6 us in a tight loop and 14 among everything else that a step does, a launch from here 3. Forward and backward
// of 512 rows through a feed-forward of d 1024 in nine calls 236 us (the kernels take 115), attention of 2 x 512 tokens in four 190 (33).
#include "attn_api.h"
#include "common/host_util.h"

using namespace ra;

extern "C" int ra_gemm_bf16(const void* A, const void* B, void* C, const void* R, int M, int N, int K, long long lda, long long ldb,
                            long long ldc, long long ldr, int a_mn, int b_mn, int c_fp32, int group_m, int* status, void* stream);
extern "C" int ra_swiglu_fwd(const void* gu, void* h, long long rows, int F, void* stream);
extern "C" int ra_swiglu_bwd(const void* gu, const void* dh, void* dgu, long long rows, int F, void* stream);

// Attention backward: preparation (delta, log-sum-exp, zeroes dq_acc), the backward kernel, dQ to bf16. `bwd.lse2`, `bwd.delta` and
// `bwd.dq_acc` are scratch; out (B, Sq, H, D) bf16 with element strides, lse (B, H, Sq); dq rows of H * D values, dq_ld elements apart.
struct RaAttnBwdRun {
  RaAttnBwdArgs bwd;
  const void* out; long long o_sb, o_ss, o_sh;
  const float* lse;
  void* dq; long long dq_ld;
};

extern "C" int ra_attn_bwd_run(const RaAttnBwdRun* r) {
  const RaAttnBwdArgs& a = r->bwd;
  const int row = a.H * a.D;
  int rc = ra_attn_bwd_prep(r->out, r->o_sb, r->o_ss, r->o_sh, a.d_o, a.do_sb, a.do_ss, a.do_sh, r->lse, const_cast<float*>(a.lse2),
                            const_cast<float*>(a.delta), a.dq_acc, a.B, a.H, a.Sq, a.Sq_pad, a.D, a.stream);
  if (rc == kHostOk) rc = ra_attn_bwd(&a);
  if (rc == kHostOk) rc = ra_cast_f32_bf16(a.dq_acc, r->dq, static_cast<long long>(a.B) * a.Sq, row, row, r->dq_ld, a.stream);
  return rc;
}

// Backward of a SwiGLU feed-forward over one chunk of rows, all operands contiguous: x, dy, dx (rows, d), wgu (2F, d), wd (d, F), scratch gu
// (rows, 2F), act and da (rows, F). gu holds the pre-activations, or they are made here (`recompute`); it ends as their gradient. The
// weight gradients go to dwd (d, F) and dwgu (2F, d) with addends dwd_add and dwgu_add (or null); *_mode as ra_gemm_bf16's c_fp32.
extern "C" int ra_ffn_bwd_run(const void* x, const void* dy, void* dx, const void* wgu, const void* wd, void* gu, void* act, void* da,
                              void* dwd, const void* dwd_add, void* dwgu, const void* dwgu_add, int rows, int d, int F, int recompute,
                              int dwd_mode, int dwgu_mode, int* status, void* stream) {
  int rc = kHostOk;
  if (recompute) rc = ra_gemm_bf16(x, wgu, gu, nullptr, rows, 2 * F, d, d, d, 2 * F, 0, 0, 0, 0, 8, status, stream);
  if (rc == kHostOk) rc = ra_swiglu_fwd(gu, act, rows, F, stream);
  if (rc == kHostOk) rc = ra_gemm_bf16(dy, wd, da, nullptr, rows, F, d, d, F, F, 0, 0, 1, 0, 8, status, stream);
  if (rc == kHostOk) rc = ra_gemm_bf16(dy, act, dwd, dwd_add, d, F, rows, d, F, F, F, 1, 1, dwd_mode, 8, status, stream);
  if (rc == kHostOk) rc = ra_swiglu_bwd(gu, da, gu, rows, F, stream);
  if (rc == kHostOk) rc = ra_gemm_bf16(gu, x, dwgu, dwgu_add, 2 * F, d, rows, 2 * F, d, d, d, 1, 1, dwgu_mode, 8, status, stream);
  if (rc == kHostOk) rc = ra_gemm_bf16(gu, wgu, dx, nullptr, rows, d, 2 * F, 2 * F, d, d, 0, 0, 1, 0, 8, status, stream);
  return rc;
}

RA_PACKED(ra_ffn_bwd_run)
