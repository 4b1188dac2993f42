// FP32 triangular steps of the mixed-precision eigen-solver, blocked: eigenvectors of an upper triangular matrix
// and the inverse of a unit triangular one, batched.
//
// Element by element, a warp per vector or row walks a chain of n dot products (trevc_kernel, trtri_kernel in
// dense_z.cu: 3 us a step, most of it latency).  Here blocks of 32 rows or columns are taken at a time: their sums
// over the blocks done before are one product for all vectors (cgemm), then a warp per vector does 32
// steps of substitution in the block:
//   * eigenvectors, from the last block of rows up: S = T(I, > I) X(> I, :), each vector with its own diagonal;
//   * inverse, from the first block of columns on: S = Z(:, < J) M(< J, J).  (Doubling, Z12 = -Z11 M12 Z22, takes fewer
//     launches, but its left residual is not bounded like substitution's, and the refinement starts from it.)
// 20 matrices of n = 648: eigenvectors 1.60 -> 1.43 ms, inverse 1.96 -> 1.05 ms, 60 % of it in the products; 10 of n = 216: 190 -> 136
// and 175 -> 88 us.  Up to kTriSmall, where they have few blocks and launches count, the element-wise kernels
// are faster (n = 50: 26 and 18 us).
#include <algorithm>

#include "scw_complex.cuh"
#include "scw_dense.h"
#include "scw_launch.h"

namespace scw {
namespace z {

constexpr int kTriB = 32;

// Block [i0, i1) of x_k for every k; X(k, i0 ..) holds the sums over the blocks below.  As trevc_kernel: a warp
// per vector, lane l: row i0 + l.
__global__ void __launch_bounds__(256)
trevc_block_kernel(const float2* __restrict__ T, float2* __restrict__ X, int n, int i0, int i1) {
    chain_wait();
    T += (long long)n * n * blockIdx.y;
    X += (long long)n * n * blockIdx.y;
    __shared__ float2 B[kTriB][kTriB + 1];
    __shared__ float red[8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nb = i1 - i0;
    float deg = 0.f;
    for (int i = tid; i < n; i += 256) deg = fmaxf(deg, cabs1(T[(long long)i * n + i]));
    for (int o = 16; o > 0; o >>= 1) deg = fmaxf(deg, __shfl_xor_sync(0xffffffffu, deg, o));
    if (lane == 0) red[warp] = deg;
    for (int e = tid; e < nb * nb; e += 256) B[e / nb][e % nb] = T[(long long)(i0 + e / nb) * n + i0 + e % nb];
    __syncthreads();
    const int k = blockIdx.x * 8 + warp;
    if (k >= n) return;
    float2* x = X + (long long)k * n + i0 + lane;
    float2 v = make_float2(0.f, 0.f);
    if (k >= i0) {
#pragma unroll
        for (int w = 0; w < 8; w++) deg = fmaxf(deg, red[w]);
        const float ulp = CT<float2>::ulp;
        deg *= 16.f * ulp;
        const float2 lam = T[(long long)k * n + k];
        const float smin = fmaxf(ulp * cabs1(lam), CT<float2>::safmin * ((float)n / ulp));
        float2 s = v;
        int top = nb - 1;
        if (k >= i1) {
            if (lane < nb) s = *x;
        } else {                                     // the vector starts in this block, with x_k = 1
            top = k - i0 - 1;
            if (lane <= top) s = B[lane][k - i0];
            if (lane == k - i0) v = make_float2(1.f, 0.f);
        }
        for (int i = top; i >= 0; i--) {
            float2 xi = make_float2(0.f, 0.f);
            if (lane == i) {
                float2 d = csub(B[i][i], lam);
                if (cabs1(d) > deg || cabs1(s) > deg) {
                    if (cabs1(d) < smin) d = make_float2(smin, 0.f);
                    xi = cdiv(make_float2(-s.x, -s.y), d);
                }
                v = xi;
            }
            xi.x = __shfl_sync(0xffffffffu, xi.x, i);
            xi.y = __shfl_sync(0xffffffffu, xi.y, i);
            if (lane < i) s = cfma(B[lane][i], xi, s);
        }
    }
    if (lane < nb) *x = v;
}

// Columns [j0, j1) of every row r of the inverse; Z(r, j0 ..) holds the sums over the columns before.  A warp per row,
// lane l: column j0 + l.
__global__ void __launch_bounds__(256)
trtri_block_kernel(const float2* __restrict__ X, float2* __restrict__ Z, int n, int j0, int j1) {
    chain_wait();
    X += (long long)n * n * blockIdx.y;
    Z += (long long)n * n * blockIdx.y;
    __shared__ float2 B[kTriB][kTriB + 1];           // column j0 + j of the matrix in row j
    const int tid = threadIdx.x, lane = tid & 31, nb = j1 - j0, r = blockIdx.x * 8 + (tid >> 5);
    for (int e = tid; e < nb * nb; e += 256) B[e / nb][e % nb] = X[(long long)(j0 + e / nb) * n + j0 + e % nb];
    __syncthreads();
    if (r >= n || lane >= nb) return;
    const unsigned all = nb == 32 ? 0xffffffffu : (1u << nb) - 1u;
    float2 v = make_float2(0.f, 0.f);
    float2* z = Z + (long long)r * n + j0 + lane;
    if (r < j1) {
        float2 s = v;
        int first = 0;
        if (r < j0) {
            s = *z;
        } else {                                     // the row starts in this block, with z_r = 1
            first = r - j0 + 1;
            if (lane >= first) s = B[lane][first - 1];
            if (lane == first - 1) v = make_float2(1.f, 0.f);
        }
        for (int j = first; j < nb; j++) {
            const float2 zj = make_float2(-__shfl_sync(all, s.x, j), -__shfl_sync(all, s.y, j));
            if (lane == j) v = zj;
            if (lane > j) s = cfma(zj, B[lane][j], s);
        }
    }
    *z = v;
}

}  // namespace z

constexpr int kTriSmall = 96;

scw_status trevc32(cudaStream_t st, const float2* T, float2* X, int n, int batch) {
    if (n <= kTriSmall) return trevc<float2>(st, T, X, n, batch, nullptr);
    const long long nn = (long long)n * n;
    for (int i0 = (n - 1) / z::kTriB * z::kTriB; i0 >= 0; i0 -= z::kTriB) {
        const int i1 = std::min(n, i0 + z::kTriB), below = n - i1;
        const scw_status s = cgemm(st, below, i1 - i0, below, 1.f, X + (long long)i1 * n + i1, n, nn, kOpN, T + (long long)i0 * n + i1, n,
                                   nn, kOpT, false, X + (long long)i1 * n + i0, n, nn, batch);
        if (s != SCW_OK) return s;
        SCW_CUDA_TRY(launch_chained(true, st, dim3((n + 7) / 8, batch), 256, 0, z::trevc_block_kernel, T, X, n, i0, i1));
    }
    return SCW_OK;
}

scw_status trtri32(cudaStream_t st, const float2* X, float2* Z, int n, int batch) {
    if (n <= kTriSmall) return trtri_rows(st, X, Z, n, batch);
    const long long nn = (long long)n * n;
    for (int j0 = 0; j0 < n; j0 += z::kTriB) {
        const int j1 = std::min(n, j0 + z::kTriB);
        const scw_status s = cgemm(st, j0, j1 - j0, j0, 1.f, Z, n, nn, kOpN, X + (long long)j0 * n, n, nn, kOpT, false, Z + j0, n, nn, batch);
        if (s != SCW_OK) return s;
        SCW_CUDA_TRY(launch_chained(true, st, dim3((n + 7) / 8, batch), 256, 0, z::trtri_block_kernel, X, Z, n, j0, j1));
    }
    return SCW_OK;
}

}  // namespace scw
