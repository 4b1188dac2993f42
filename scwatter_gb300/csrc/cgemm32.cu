// FP32 complex products with a short side: C = alpha op(A) op(B) + beta C, batched, alpha = +-1, beta = 0 or 1.
//
// The rank-32 updates and 32-column products of the Hessenberg reduction are bound by memory about as much as by
// their multiply-adds on CUDA cores (20 matrices of n = 648: 26 us at the FP32 rate, 22 us of memory
// traffic), so cutting their operands into digits for the tensor core (gemm_tc.cu: two launches before the
// product, and an epilogue of fixed-point conversions) costs more than it saves.
//
// A thread holds 4 x 4 complex sums as register pairs (re, im): with A's parts doubled, (re, re) and (im, im), and B
// next to i B, (re, im) and (-im, re), in shared memory, a complex multiply-add is two packed FMAs and
// an operand is one 16-byte load.  The next 16 inner indices are fetched into registers meanwhile.  Sums of 16 terms go
// to a second set of registers, so that a long inner index rounds like a blocked sum.  Where one side
// of C is 32, two groups of threads share the inner index.
//
// The products of all panels, 20 matrices of n = 648: 5.5 ms, against 8.1 as digit products and 2.9 for their digits; 10
// of n = 216: 0.50 against 0.63 + 0.29 ms; 4 of n = 50: 76 against 152 + 75 us.  A rank-32 update of 616 columns takes
// 80 us (3 CTAs per SM; 88 with 2): the latency of its loads, two chunks and C is what bounds it.
#include <algorithm>

#include "scw_complex.cuh"
#include "scw_dense.h"
#include "scw_launch.h"

namespace scw {
namespace z {

constexpr int kCgK = 16;                         // inner indices per chunk

__device__ __forceinline__ unsigned long long cg_pair(float x, float y) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ unsigned long long cg_fma(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ unsigned long long cg_add(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

struct CgArgs {
    const float2 *A, *B;
    float2* C;
    int M, N, K, lda, ldb, ldc;
    long long sA, sB, sC;
    float alpha, conjA, conjB;         // conj: -1 for the conjugate
    int add;
};

// CA, CB: the transpose of the stored matrix.  KS groups of (TM / 4) (TN / 4) threads along the inner index.
// SHORT: at most two chunks, one set of sums.
template <int TM, int TN, int KS, bool CA, bool CB, bool SHORT>
__global__ void __launch_bounds__(TM / 4 * (TN / 4) * KS, SHORT ? 3 : 2)
cgemm_kernel(CgArgs p) {
    chain_wait();
    constexpr int kX = TN / 4, kG = TM / 4 * kX;         // threads along a row, of a group
    constexpr int nA = TM * kCgK / kG, nB = TN * kCgK / kG;
    extern __shared__ __align__(16) unsigned char cg_smem[];
    using RowsA = ulonglong2[kCgK][TM + 1];
    using RowsB = ulonglong2[kCgK][TN + 1];
    RowsA* sA = reinterpret_cast<RowsA*>(cg_smem);       // [KS]
    RowsB* sB = reinterpret_cast<RowsB*>(cg_smem + KS * sizeof(RowsA));
    const int group = threadIdx.x / kG, t = threadIdx.x - group * kG, tx = t % kX, ty = t / kX;
    const float2* A = p.A + p.sA * blockIdx.z;
    const float2* B = p.B + p.sB * blockIdx.z;
    const int i0 = blockIdx.y * TM, j0 = blockIdx.x * TN;
    const int chunks = (p.K + kCgK - 1) / kCgK;
    float2 ra[nA], rb[nB];
    auto fetch = [&](int ch) {
        const int k0 = ch * kCgK;
#pragma unroll
        for (int q = 0; q < nA; q++) {
            const int e = t + q * kG;
            const int k = CA ? e / TM : e % kCgK, i = CA ? e % TM : e / kCgK;
            const bool in = i0 + i < p.M && k0 + k < p.K;
            ra[q] = in ? A[CA ? (long long)(k0 + k) * p.lda + i0 + i : (long long)(i0 + i) * p.lda + k0 + k] : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int q = 0; q < nB; q++) {
            const int e = t + q * kG;
            const int k = CB ? e % kCgK : e / TN, j = CB ? e / kCgK : e % TN;
            const bool in = j0 + j < p.N && k0 + k < p.K;
            rb[q] = in ? B[CB ? (long long)(j0 + j) * p.ldb + k0 + k : (long long)(k0 + k) * p.ldb + j0 + j] : make_float2(0.f, 0.f);
        }
    };
    unsigned long long acc[4][4], tot[4][4];
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int c = 0; c < 4; c++) tot[r][c] = acc[r][c] = 0ull;
    fetch(group);
    for (int base = 0; base < chunks; base += KS) {
        // (a group past the last chunk has fetched zeros)
#pragma unroll
        for (int q = 0; q < nA; q++) {
            const int e = t + q * kG;
            const float y = p.conjA * ra[q].y;
            sA[group][CA ? e / TM : e % kCgK][CA ? e % TM : e / kCgK] =
                make_ulonglong2(cg_pair(ra[q].x, ra[q].x), cg_pair(y, y));
        }
#pragma unroll
        for (int q = 0; q < nB; q++) {
            const int e = t + q * kG;
            const float y = p.conjB * rb[q].y;
            sB[group][CB ? e % kCgK : e / TN][CB ? e / kCgK : e % TN] =
                make_ulonglong2(cg_pair(rb[q].x, y), cg_pair(-y, rb[q].x));
        }
        __syncthreads();
        if (base + KS < chunks) fetch(base + KS + group);
#pragma unroll
        for (int k = 0; k < kCgK; k++) {
            ulonglong2 a[4], b[4];
#pragma unroll
            for (int r = 0; r < 4; r++) a[r] = sA[group][k][4 * ty + r];
#pragma unroll
            for (int c = 0; c < 4; c++) b[c] = sB[group][k][tx + kX * c];
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int c = 0; c < 4; c++) acc[r][c] = cg_fma(a[r].y, b[c].y, cg_fma(a[r].x, b[c].x, acc[r][c]));
        }
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int c = 0; c < 4; c++)
                if (SHORT) {
                    tot[r][c] = acc[r][c];
                } else {
                    tot[r][c] = cg_add(tot[r][c], acc[r][c]);
                    acc[r][c] = 0ull;
                }
        __syncthreads();
    }
    // the other groups' sums through shared memory
    static_assert(KS == 1 || KS * sizeof(RowsB) >= sizeof(unsigned long long) * TM * TN, "sums of a group");
    if (KS == 2) {
        unsigned long long* s = reinterpret_cast<unsigned long long*>(sB);
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int c = 0; c < 4; c++)
                if (group == 1) s[(r * 4 + c) * kG + t] = tot[r][c];
        __syncthreads();
        if (group == 1) return;
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int c = 0; c < 4; c++) tot[r][c] = cg_add(tot[r][c], s[(r * 4 + c) * kG + t]);
    }
    float2* C = p.C + p.sC * blockIdx.z;
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const int i = i0 + 4 * ty + r;
        if (i >= p.M) break;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int j = j0 + tx + kX * c;
            if (j >= p.N) continue;
            float2* o = C + (long long)i * p.ldc + j;
            const float x = __uint_as_float((unsigned)tot[r][c]), y = __uint_as_float((unsigned)(tot[r][c] >> 32));
            float2 v = p.add ? *o : make_float2(0.f, 0.f);
            v.x = fmaf(p.alpha, x, v.x);
            v.y = fmaf(p.alpha, y, v.y);
            *o = v;
        }
    }
}

template <int TM, int TN, int KS, bool SHORT = false>
static scw_status cgemm_launch(cudaStream_t st, const CgArgs& p, bool ca, bool cb, int batch) {
    const dim3 grid((p.N + TN - 1) / TN, (p.M + TM - 1) / TM, batch);
    constexpr int threads = TM / 4 * (TN / 4) * KS;
    constexpr size_t smem = sizeof(ulonglong2) * KS * kCgK * (TM + 1 + TN + 1);
    auto kernel = ca ? (cb ? cgemm_kernel<TM, TN, KS, true, true, SHORT> : cgemm_kernel<TM, TN, KS, true, false, SHORT>)
                     : (cb ? cgemm_kernel<TM, TN, KS, false, true, SHORT> : cgemm_kernel<TM, TN, KS, false, false, SHORT>);
    if (smem > 48 * 1024) SCW_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    SCW_CUDA_TRY(launch_chained(true, st, grid, threads, smem, kernel, p));
    return SCW_OK;
}

}  // namespace z

scw_status cgemm(cudaStream_t st, int M, int N, int K, float alpha, const float2* A, int lda, long long sA, int opA,
                 const float2* B, int ldb, long long sB, int opB, bool add, float2* C, int ldc, long long sC, int batch) {
    if (M <= 0 || N <= 0 || batch <= 0) return SCW_OK;
    const bool ca = opA != kOpN, cb = opB != kOpN;
    const z::CgArgs p{A, B, C, M, N, K, lda, ldb, ldc, sA, sB, sC, alpha, opA == kOpC ? -1.f : 1.f, opB == kOpC ? -1.f : 1.f, add ? 1 : 0};
    // (a grid's z has 65 535 blocks at most)
    for (int b0 = 0; b0 < batch; b0 += 65535) {
        z::CgArgs q = p;
        q.A += sA * b0;
        q.B += sB * b0;
        q.C += sC * b0;
        const int nb = std::min(batch - b0, 65535);
        const scw_status s = M <= 32 ? z::cgemm_launch<32, 64, 2>(st, q, ca, cb, nb)
                           : N <= 32 ? z::cgemm_launch<64, 32, 2>(st, q, ca, cb, nb)
                           : K <= 2 * z::kCgK ? z::cgemm_launch<64, 64, 1, true>(st, q, ca, cb, nb)
                                              : z::cgemm_launch<64, 64, 1>(st, q, ca, cb, nb);
        if (s != SCW_OK) return s;
    }
    return SCW_OK;
}

}  // namespace scw
