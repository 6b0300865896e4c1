// One trunk layer's launches, forward and backward, issued from native code.
//
// A layer is six launches forward and sixteen backward.  Issued one by one from Python each costs 15-20 us of
// host time (argument marshalling, output allocation, stream lookup) against 5-60 us on the device, so small
// batches ran at the host's pace: 2.8 ms of host work for a 3.0 ms training step of 64 x 512 tokens, 1.0 ms
// for 0.41 ms of kernels in a block's forward and backward at 11 100 rows x 384.  Here a layer is one call
// each way: the caller hands in the saved activations, one bf16 and one fp32 workspace and the outputs.
// Nothing is allocated, kept or synchronised; every pointer belongs to the caller for this call only.
//
// The sequence is the trunk's (reference block: src/chaoscontrol/model.py:111-140, core.py:322-507):
//   P = rs1 (x Wp'^T); y, h = scan(P); x2 = x + y Wo^T; u, f = rs2 (x2 Wfc'^T), silu; x3 = x2 + f Wproj^T
#include "ccb_api.h"
#include "runtime.h"

extern "C" {
int ccb_scan_fwd(const void* P, int64_t ldp, const float* log_a, const float* h0, void* y, void* hout, float* hT,
                 int64_t B, int64_t T, int64_t D, int64_t la_bstride, void* stream);
int ccb_scan_bwd(const void* P, int64_t ldp, const float* log_a, const float* h0, const void* hstates, const void* dy,
                 const float* dhT, const float* rowss, float inv_dim, float eps, void* dP, int64_t lddp,
                 float* dloga_part, float* dh0, int64_t B, int64_t T, int64_t D, int64_t la_bstride, void* stream);
int ccb_splitk_reduce_parts(const float* part, int64_t S, int64_t split_stride, int64_t N, int64_t K,
                            const void* colscale, const void* W, const float* scale, void* const* outs, int64_t nout,
                            int64_t out_bf16, int64_t accumulate, float* colpart, void* colsum_out,
                            int64_t colsum_accumulate, void* stream);
int ccb_colsum_as(const float* part, int64_t NB, int64_t K, void* out, int64_t out_bf16, int64_t accumulate, void* stream);

typedef struct CcbLayerArgs {
  int64_t B, T, D, F;
  float eps;
  int64_t grad_bf16;                      // weight gradients and dlog_a: 1 bf16, 0 fp32
  // weights: folded (Wp_f, Wfc_f), plain, norm weights, fp32 log_a
  const void *Wp_f, *Wfc_f, *Wo, *Wproj, *Wp, *Wfc, *wn1, *wn2;
  const float *log_a, *h0;
  // activations [R, .]: forward writes all but x and ss1 (h may be null), backward reads them
  const void* x;
  const float* ss1;
  void *P, *y, *h, *x2, *u, *f;
  float* ss2;
  // forward outputs
  void* x3;
  float *ss3, *hT;
  // backward inputs, workspaces and outputs
  const void* dx3;
  const float* dhT;
  void* ws16;                             // ccb_layer_bwd_ws16 elements
  float* ws32;                            // ccb_layer_bwd_ws32 elements
  void *dx, *dWp[4];                      // one [4D, D] (dWp[1] null) or four [D, D]
  void *dWo, *dWfc, *dWproj, *dwn1, *dwn2, *dlog_a;
  float* dh0;
} CcbLayerArgs;
}

namespace ccb {

static CcbGemmArgs gemm_args(const void* A, int64_t lda, const void* B, int64_t ldb, void* C, int64_t M, int64_t N,
                             int64_t K) {
  CcbGemmArgs a = {};
  a.A = A; a.B = B; a.C = C;
  a.M = M; a.N = N; a.K = K;
  a.batch = 1; a.splits = 1;
  a.lda = lda; a.ldb = ldb; a.ldc = N;
  a.alpha = 1.f;
  return a;
}

static int64_t wgrad_splits(int64_t m, int64_t n, int64_t k) {
  const int64_t tall = ccb_gemm_wgrad_splits(m, n, k, 1);
  return tall > 0 ? tall : ccb_gemm_wgrad_splits(m, n, k, 0);
}

static int64_t max64(int64_t a, int64_t b) { return a > b ? a : b; }

// x + y W^T with the row sum of squares of the result
static int resid(const void* y, int64_t K, const void* W, const void* x, void* out, float* ss, int64_t R, int64_t D,
                 cudaStream_t s) {
  CcbGemmArgs a = gemm_args(y, K, W, K, out, R, D, K);
  a.epi = CCB_EPI_RESID_SS;
  a.R1 = x; a.ldr = D;
  a.ss_out = ss;
  if (D > 256) {
    // a row spans two column tiles: each adds its share (two addends, so their order does not matter)
    cudaError_t e = cudaMemsetAsync(ss, 0, sizeof(float) * (size_t)R, s);
    if (e != cudaSuccess) return set_error("layer: cudaMemsetAsync: %s", cudaGetErrorString(e));
    a.ss_atomic = 1;
  }
  return ccb_gemm(&a, s);
}

// out[N, K] = dy^T x over R rows, with the folded norm weight's gradient when wn is given
static int wgrad(const void* dy, int64_t N, const void* x, int64_t K, int64_t R, float* part, float* colpart,
                 const void* wn, const void* W, void* const* outs, int64_t nout, void* dwn, int64_t out_bf16,
                 cudaStream_t s) {
  CcbGemmArgs a = gemm_args(dy, N, x, K, part, N, K, R);
  a.a_mn = 1; a.b_mn = 1;
  a.out_fp32 = 1;
  a.splits = wgrad_splits(N, K, R);
  a.c_split = a.splits > 1 ? N * K : 0;
  if (int rc = ccb_gemm(&a, s)) return rc;
  return ccb_splitk_reduce_parts(part, a.splits, N * K, N, K, wn, W, nullptr, outs, nout, out_bf16, 0, colpart, dwn, 0, s);
}

}  // namespace ccb

using namespace ccb;

// Elements of the backward's bf16 workspace: du, dx2, dy, dP.
extern "C" int64_t ccb_layer_bwd_ws16(int64_t R, int64_t D, int64_t F) { return R * (F + 6 * D); }
// Elements of its fp32 workspace: split-K partials, their column sums, per-row d log_a.
extern "C" int64_t ccb_layer_bwd_ws32(int64_t B, int64_t T, int64_t D, int64_t F) {
  const int64_t R = B * T;
  int64_t part = max64(wgrad_splits(D, F, R) * D * F, wgrad_splits(F, D, R) * F * D);
  part = max64(part, max64(wgrad_splits(D, D, R) * D * D, wgrad_splits(4 * D, D, R) * 4 * D * D));
  return part + max64((F + 7) / 8, (4 * D + 7) / 8) * D + B * D;
}

extern "C" int ccb_layer_forward(const CcbLayerArgs* p, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  const int64_t R = p->B * p->T, D = p->D, F = p->F;
  if (R <= 0) return 0;
  const float inv_d = 1.f / (float)D;
  CcbGemmArgs a = gemm_args(p->x, D, p->Wp_f, D, p->P, R, 4 * D, D);
  a.epi = CCB_EPI_ROWSCALE;
  a.rowss = p->ss1; a.inv_dim = inv_d; a.eps = p->eps;
  if (int rc = ccb_gemm(&a, s)) return rc;
  if (int rc = ccb_scan_fwd(p->P, 4 * D, p->log_a, p->h0, p->y, p->h, p->hT, p->B, p->T, D, 0, s)) return rc;
  if (int rc = resid(p->y, D, p->Wo, p->x, p->x2, p->ss2, R, D, s)) return rc;
  a = gemm_args(p->x2, D, p->Wfc_f, D, p->u, R, F, D);
  a.epi = CCB_EPI_ROWSCALE_SILU;
  a.rowss = p->ss2; a.inv_dim = inv_d; a.eps = p->eps;
  a.C2 = p->f;
  if (int rc = ccb_gemm(&a, s)) return rc;
  return resid(p->f, F, p->Wproj, p->x2, p->x3, p->ss3, R, D, s);
}

extern "C" int ccb_layer_backward(const CcbLayerArgs* p, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  const int64_t R = p->B * p->T, D = p->D, F = p->F;
  if (R <= 0) return 0;
  const float inv_d = 1.f / (float)D;
  uint16_t* du = (uint16_t*)p->ws16;
  uint16_t *dx2 = du + R * F, *dy = dx2 + R * D, *dP = dy + R * D;
  float* dla = p->ws32;
  float* colpart = dla + p->B * D;
  float* part = colpart + max64((F + 7) / 8, (4 * D + 7) / 8) * D;
  // feed-forward half
  CcbGemmArgs a = gemm_args(p->dx3, D, p->Wproj, F, du, R, F, D);
  a.b_mn = 1;
  a.epi = CCB_EPI_DSILU;
  a.R1 = p->u; a.ldr = F;
  a.rowss = p->ss2; a.inv_dim = inv_d; a.eps = p->eps;
  if (int rc = ccb_gemm(&a, s)) return rc;
  if (int rc = wgrad(p->dx3, D, p->f, F, R, part, nullptr, nullptr, nullptr, &p->dWproj, 1, nullptr, p->grad_bf16, s)) return rc;
  a = gemm_args(du, F, p->Wfc_f, D, dx2, R, D, F);
  a.b_mn = 1;
  a.epi = CCB_EPI_RMSBWD;
  a.R1 = p->x2; a.R2 = p->dx3; a.ldr = D;
  a.rowss = p->ss2; a.inv_dim = inv_d; a.eps = p->eps;
  if (int rc = ccb_gemm(&a, s)) return rc;
  if (int rc = wgrad(du, F, p->x2, D, R, part, colpart, p->wn2, p->Wfc, &p->dWfc, 1, p->dwn2, p->grad_bf16, s)) return rc;
  // recurrence half
  a = gemm_args(dx2, D, p->Wo, D, dy, R, D, D);
  a.b_mn = 1;
  if (int rc = ccb_gemm(&a, s)) return rc;
  if (int rc = wgrad(dx2, D, p->y, D, R, part, nullptr, nullptr, nullptr, &p->dWo, 1, nullptr, p->grad_bf16, s)) return rc;
  if (int rc = ccb_scan_bwd(p->P, 4 * D, p->log_a, p->h0, p->h, dy, p->dhT, p->ss1, inv_d, p->eps, dP, 4 * D, dla, p->dh0,
                            p->B, p->T, D, 0, s)) return rc;
  if (int rc = ccb_colsum_as(dla, p->B, D, p->dlog_a, p->grad_bf16, 0, s)) return rc;
  a = gemm_args(dP, 4 * D, p->Wp_f, D, p->dx, R, D, 4 * D);
  a.b_mn = 1;
  a.epi = CCB_EPI_RMSBWD;
  a.R1 = p->x; a.R2 = dx2; a.ldr = D;
  a.rowss = p->ss1; a.inv_dim = inv_d; a.eps = p->eps;
  if (int rc = ccb_gemm(&a, s)) return rc;
  return wgrad(dP, 4 * D, p->x, D, R, part, colpart, p->wn1, p->Wp, p->dWp, p->dWp[1] ? 4 : 1, p->dwn1, p->grad_bf16, s);
}
