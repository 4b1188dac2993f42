// FP64 complex dense linear algebra used by the per-layer solve (dense_z.cu).
#pragma once

#include <cuda_runtime.h>
#include <algorithm>

#include "scw_internal.h"

namespace scw {

#ifdef __CUDACC__
// principal square root without cancellation: the larger of |Re|, |Im| of the root comes from
// sqrt((|Re a| + |a|) / 2), the other from Im a / (2 x)
__device__ __forceinline__ double2 zsqrt(double2 a) {
    if (a.x == 0.0 && a.y == 0.0) return make_double2(0.0, 0.0);
    const double t = sqrt(0.5 * (fabs(a.x) + hypot(a.x, a.y)));
    if (a.x >= 0.0) return make_double2(t, a.y / (2.0 * t));
    return make_double2(fabs(a.y) / (2.0 * t), copysign(t, a.y));
}
__device__ __forceinline__ float2 zsqrt(float2 a) {
    if (a.x == 0.0f && a.y == 0.0f) return make_float2(0.0f, 0.0f);
    const float t = sqrtf(0.5f * (fabsf(a.x) + hypotf(a.x, a.y)));
    if (a.x >= 0.0f) return make_float2(t, a.y / (2.0f * t));
    return make_float2(fabsf(a.y) / (2.0f * t), copysignf(t, a.y));
}
#endif

// The kernels are templates over the complex element type: double2 (FP64, the solve's
// precision) or float2 (FP32, the first stage of the mixed-precision eigen-solver).  A
// non-null skip[b] != 0 makes every kernel leave batch entry b untouched.

// Device workspace of the FP64 GEMM (gemm_tc.cu): any size that holds one matrix's operands; err is
// a device flag raised when a bounded wait gave up.
struct GemmWs {
    char* base = nullptr;
    size_t bytes = 0;
    int* err = nullptr;
    bool parts = false;                // every real and imaginary part as exact as an FP64 sum (see zgemm)
};
// cap on a workspace sized for a whole batch; larger batches go through it in parts
constexpr size_t kGemmWsCap = 1024ull << 20;
// the context's tensor-core error flag (cleared unless a check is pending) is in use from here on: the next scw_ctx_synchronize reads it
scw_status ctx_tc_flag(scw_ctx ctx);
// a context's own GEMM workspace of at least `one` bytes, `all` if that is below the cap; none (the
// products then run without one) while the context's stream is being captured
scw_status ctx_gemm_ws(scw_ctx ctx, size_t one, size_t all, GemmWs& ws);
// workspace that takes the whole batch in one pass
size_t zgemm_ws_bytes(int M, int N, int K, int batch);
// buf as a workspace for products of `one` bytes of operands a matrix: for the whole batch up to the cap, or for one
// matrix at a time where memory is short
scw_status reserve_gemm_ws(scw_ctx ctx, DevBuf& buf, size_t one, int batch, GemmWs& ws);
// C = alpha A op(B) + beta C + diag I (row-major, batched by strides in elements), FP64 on the tensor
// cores; op = identity, transpose or conjugate transpose.  Without a workspace
// by gemm<double2> (no conjugate transpose, no diagonal).
// The error is small against the largest |a_ik| |b_kj| of row i and column j (after the best scaling of the inner
// index; none where one A, sA = 0, serves several B), not against the sum of all |a_ik| |b_kj|: what the solve needs.
// With ws.parts it is small against the sums that make up each part of the result, as with FP64 arithmetic;
// C must then not overlap A or B, which it may be otherwise.
enum : int { kOpN = 0, kOpT = 1, kOpC = 2 };
scw_status zgemm(cudaStream_t st, int M, int N, int K, double2 alpha, const double2* A, int lda, long long sA,
                 const double2* B, int ldb, long long sB, double2 beta, double2* C, int ldc, long long sC, int batch,
                 const GemmWs& ws, const int* skip = nullptr, double diag = 0.0, int opB = kOpN);
// The same kernel with 30-bit operands, for corrections that need FP32 accuracy: n x n matrices back
// to back, C = alpha A op(B) + beta C + diag I.
template <typename TA, typename TB, typename TC>
scw_status gemm32(cudaStream_t st, int n, double alpha, const TA* A, const TB* B, int opB, double beta, double diag, TC* C,
                  int batch, const GemmWs& ws, const int* skip);
// FP32 product with a short side on the CUDA cores (cgemm32.cu): C = alpha op(A) op(B), added to C if add; alpha = +-1
scw_status cgemm(cudaStream_t st, int M, int N, int K, float alpha, const float2* A, int lda, long long sA, int opA,
                 const float2* B, int ldb, long long sB, int opB, bool add, float2* C, int ldc, long long sC, int batch);

// C = alpha A op(B) + beta C, op = identity or transpose (row-major, batched by strides in elements)
template <typename C>
scw_status gemm(cudaStream_t st, int M, int N, int K, C alpha, const C* A, int lda, long long sA, const C* B, int ldb,
                long long sB, C beta, C* Cm, int ldc, long long sC, int batch, const int* skip = nullptr, int opB = kOpN);
// in-place LU with partial pivoting of the first n columns of n x ncols matrices (leading dimension lda;
// further columns are carried along as right-hand sides); info[b] = first zero pivot + 1
scw_status zgetrf(cudaStream_t st, double2* A, int n, int ncols, int lda, long long sA, int* piv, long long sP, int* info,
                  int batch, const GemmWs& ws, const int* skip);
// B := U^-1 B with the upper factor of getrf
scw_status ztrsm_upper(cudaStream_t st, const double2* LU, int n, int lda, long long sA, double2* B, int nrhs, int ldb,
                       long long sB, int batch, const GemmWs& ws, const int* skip);
// B := A^-1 B using getrf's factors (leading dimension n; B: n x nrhs, leading dimension nrhs)
scw_status zgetrs(cudaStream_t st, const double2* LU, int n, long long sA, const int* piv, long long sP, double2* B,
                  int nrhs, long long sB, int batch, const GemmWs& ws, const int* skip);
// Schur form A = Q T Q^H in FP32 (T over A, eigenvalues W); work: hess32_ws_elems(n) per matrix; share:
// solves of this size that run at the same time (lanes of a batch)
scw_status schur32(cudaStream_t st, float2* A, float2* Q, float2* W, int n, int batch, float2* work, int* status, int share);
// its stages: Hessenberg form of A with Q (hess32.cu), then the QR iteration with vectors accumulated into Z
// (hqr32.cu; ctas: CTAs per matrix, 0 = chosen by size and batch)
size_t hess32_ws_elems(int n);
scw_status hess32(cudaStream_t st, float2* A, float2* Q, int n, int batch, float2* work, int share);
scw_status hqr32(cudaStream_t st, float2* H, float2* Z, int n, float2* W, int* status, int batch, int ctas, int share);
// eigenvectors of the triangular T as the rows of X (unit diagonal), and the inverse Z of the unit
// triangular matrix whose columns those are
template <typename C>
scw_status trevc(cudaStream_t st, const C* T, C* X, int n, int batch, const int* skip);
scw_status trtri_rows(cudaStream_t st, const float2* X, float2* Z, int n, int batch);
// the same in FP32 in blocks (tri32.cu)
scw_status trevc32(cudaStream_t st, const float2* T, float2* X, int n, int batch);
scw_status trtri32(cudaStream_t st, const float2* X, float2* Z, int n, int batch);
// eigenvalues W and right eigenvectors V (columns) of A (overwritten), FP64; work >= batch (n^2 + 3 n);
// status[b] = 1 when the QR iteration did not converge.  wide: the Hessenberg reduction of
// matrices with n >= kWideMinN is spread over the whole GPU (3 launches per column) instead of one
// CTA per matrix -- for batches too small to fill the SMs; a batch graph with many concurrent
// items keeps the one-CTA form (fewer nodes).
constexpr int kWideMinN = 128;
scw_status zgeev(cudaStream_t st, double2* A, double2* W, double2* V, int n, int batch, double2* work, int* status,
                 const int* skip, bool wide, const GemmWs& ws);
// the same in FP32 (the first stage of the mixed solver); work >= batch (n^2 + hess32_ws_elems(n))
scw_status cgeev(cudaStream_t st, float2* A, float2* W, float2* V, int n, int batch, float2* work, int* status, int share);
// Hessenberg form of A (in place, n x n per batch entry) and the unitary Q (A = Q H Q^H);
// work >= batch * 3 n
scw_status zgehrd(cudaStream_t st, double2* A, double2* Q, int n, int batch, double2* work);

}  // namespace scw
