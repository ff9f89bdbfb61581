// Split-precision (FP16 fixed-point slices on tcgen05) form of the Zernike
// contractions and of the SH Legendre sums; see split.cu.
#pragma once

#include <vector>

struct zest_gpu_context;

namespace zgpu {

struct ZtPlan;
struct StPlan;
struct SplitState;  // per-context state of the split path, defined in split.cu
void destroy_split(SplitState* s);
struct SplitDeleter {
    void operator()(SplitState* s) const { destroy_split(s); }
};

// ZEST_GPU_OK when the split path is available on the current device.
int split_available();
int split_zt_forward(zest_gpu_context* ctx, ZtPlan& plan, int Lg, int Le, int Lm, int batch, const double* grids,
                     double* coeffs);
int split_zt_backward(zest_gpu_context* ctx, ZtPlan& plan, int Le, int Lg, int Lm, int batch, const double* coeffs,
                      double* grids);
// Legendre sums of the SH transforms in split precision (6 slices).  Forward:
// the spectra X[b][m][lat][2] of orders m < Lm -> coefficients of degrees < Lm.
// Backward: coefficients -> the parity sums E_p[b][m][j'][2] (in the context's
// scratch), conjugated, for the inverse longitude transform.
int split_st_forward(zest_gpu_context* ctx, StPlan& plan, int Lg, int Lm, int batch, const double* X, double* coeffs,
                     long long csz);
int split_st_backward(zest_gpu_context* ctx, StPlan& plan, int Lg, int Lm, int batch, const double* coeffs,
                      long long csz, double** E);
// C = A B^T (A: M x K, B: N x K, C: M x N, row-major FP64 device buffers)
int split_dense_gemm(zest_gpu_context* ctx, int M, int N, int K, const double* A, const double* B, double* C);
// FP16 tensor-core flops of the split GEMM launches since the last reset
// (counted while profiling is enabled): useful = valid rows x table rows x K,
// issued = whole 128-row tiles as executed.
void split_flops(zest_gpu_context* ctx, bool reset, double* useful, double* issued);
// Synchronizes the context stream and reports (and clears) a bounded-wait
// timeout recorded by the split GEMMs launched since the last check.
int split_check_flag(zest_gpu_context* ctx);
// End of a split-path call: split_check_flag, except while the stream is
// being captured into a graph (whose replays are checked by the caller).
int split_finish(zest_gpu_context* ctx);
// Makes one bounded mbarrier wait run out after limit_ns (nothing arrives on
// it) and reports it as the GEMMs' timeouts are reported: ZEST_GPU_ERR_TIMEOUT.
int split_wait_selftest(zest_gpu_context* ctx, long long limit_ns);

}  // namespace zgpu
