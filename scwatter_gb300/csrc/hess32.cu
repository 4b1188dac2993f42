// FP32 Hessenberg reduction A -> Q^H A Q of batched complex matrices, blocked (zgehrd / zlahr2 of LAPACK
// restated): the first stage of the mixed-precision eigen-solver.
//
// A panel of nb columns is reduced by one thread-block cluster per matrix; the trailing matrix and Q
// then get its nb reflectors at once as products on the tensor cores (gemm32).  Per column j the
// cluster does
//   b = A(:, j) - Y V(j, :)^H, then b -= V T^H (V^H b)      (rows below the panel's top)
//   the reflector v of b below row j, and y = tau (A v - Y V^H v)
// with V, Y distributed over the CTAs by rows in shared memory, and two cluster barriers: one for
// V^H b, one for |b|^2 and V^H v (which follows from V^H b because v is b scaled but for its first
// entry).  The product A v reads the trailing matrix once per column; that read, from L2, bounds a
// column (n (n - j) values over the cluster's SMs), with the two barriers.  Reduced column by column,
// with three launches each, every column read A three times, wrote it once, and the same for Q: 84 ms
// for 20 matrices of n = 648, now 23 (12.6 of them in the panels).
//
// A column whose part below the diagonal is under ulp ||A||_F / sqrt(n) (ulp times the root-mean-square
// row norm) is set to zero instead of reflected.  That is a backward error of rounding size, and it
// keeps a (nearly) diagonal matrix, e.g. the reduced matrix of a homogeneous layer whose off-diagonal
// entries are DFT rounding, from being scrambled by reflectors built from noise.
#include <algorithm>

#include <cooperative_groups.h>

#include "scw_complex.cuh"
#include "scw_dense.h"

namespace scw {
namespace z {

constexpr int kHb = 32;                    // largest panel width
constexpr int kHessThreads = 512;
constexpr int kHessWarps = kHessThreads / 32;
constexpr int kHessMax = 8;                // CTAs per cluster

struct HessShared {
    float2 w[kHessMax][kHb];               // V^H b, one row per CTA
    float2 u[kHessMax][kHb];               // V(j+2.., :)^H b, one row per CTA
    float nrm[kHessMax];                   // |b(j+2..)|^2
    float2 alpha;                          // b(j+1)
    float2 T[kHb][kHb + 1];
    float2 VP[kHb + 1][kHb + 1];           // V(j0 + 1 + i, q)
    float2 w2[kHb], vv[kHb];
    float red[kHessWarps];
};

__device__ __forceinline__ float2 conjc(float2 a) { return make_float2(a.x, -a.y); }
__device__ __forceinline__ float2 wsum(float2 s) {
    for (int o = 16; o > 0; o >>= 1) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
        s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
    }
    return s;
}

// ||A||_F^2 per matrix (fro starts at zero)
__global__ void __launch_bounds__(256) fro32_kernel(const float2* __restrict__ A, long long per, float* __restrict__ fro) {
    A += per * blockIdx.y;
    float s = 0.f;
    for (long long e = blockIdx.x * 256ll + threadIdx.x; e < per; e += gridDim.x * 256ll) s += cabs2(A[e]);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(fro + blockIdx.y, s);
}

__global__ void eye32_kernel(float2* __restrict__ Q, int n, long long total) {
    const long long e = blockIdx.x * 256ll + threadIdx.x;
    if (e >= total) return;
    const long long r = e % ((long long)n * n);
    Q[e] = make_float2(r / n == r % n ? 1.f : 0.f, 0.f);
}

// Columns j0 .. j0 + ib - 1.  rows: rows per CTA.  Outputs V, Y, VT = V T, VTH = V T^H (n x nb each, back to
// back per matrix); the panel's columns of A are final.
__global__ void __launch_bounds__(kHessThreads)
hess_panel_kernel(float2* __restrict__ A, int n, long long sA, int j0, int ib, int nb, int rows, float2* __restrict__ out,
                  const float* __restrict__ fro) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int K = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int mat = blockIdx.x / K;
    A += sA * mat;
    out += 4ll * n * nb * mat;
    extern __shared__ __align__(16) unsigned char hess_smem[];
    HessShared& S = *reinterpret_cast<HessShared*>(hess_smem);
    const int ld = nb + 1;
    float2* V = reinterpret_cast<float2*>(hess_smem + sizeof(HessShared));    // [rows][ld]
    float2* Y = V + rows * ld;                                                // [rows][ld]
    float2* bs2 = Y + rows * ld;                                              // [2][rows]: b, by column parity
    float2* vf = bs2 + 2 * rows;                                              // [n]: v
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g0 = rank * rows, nr = max(0, min(rows, n - g0));
    for (int e = tid; e < rows * ld; e += kHessThreads) V[e] = Y[e] = make_float2(0.f, 0.f);
    for (int e = tid; e < kHb * (kHb + 1); e += kHessThreads) (&S.T[0][0])[e] = make_float2(0.f, 0.f);
    for (int e = tid; e < (kHb + 1) * (kHb + 1); e += kHessThreads) (&S.VP[0][0])[e] = make_float2(0.f, 0.f);
    const float neg2 = fro[mat] * CT<float2>::ulp * CT<float2>::ulp / (float)n;
    cluster.sync();                                  // every CTA runs before the first remote write
    for (int i = 0; i < ib; i++) {
        const int j = j0 + i;
        // (another CTA may still read the b of the column before)
        float2* bs = bs2 + (i & 1) * rows;
        // b = A(:, j) - Y V(j, :)^H on the rows below the panel's top; V(j, q) = VP[i - 1][q]
        for (int r = tid; r < nr; r += kHessThreads) {
            float2 b = make_float2(0.f, 0.f);
            if (g0 + r > j0) {
                b = A[(long long)(g0 + r) * n + j];
                for (int q = 0; q < i; q++) b = csub(b, cmul(Y[r * ld + q], conjc(S.VP[i - 1][q])));
            }
            bs[r] = b;
        }
        __syncthreads();
        for (int q = warp; q < i; q += kHessWarps) {
            float2 s = make_float2(0.f, 0.f);
            for (int r = lane; r < nr; r += 32) s = cfma(conjc(V[r * ld + q]), bs[r], s);
            s = wsum(s);
            if (lane < K) cluster.map_shared_rank(&S, lane)->w[rank][q] = s;
        }
        cluster.sync();
        // w2 = T^H w
        if (warp == 0) {
            float2 w = make_float2(0.f, 0.f);
            if (lane < i)
                for (int c = 0; c < K; c++) w = cadd(w, S.w[c][lane]);
            S.vv[lane] = w;
            __syncwarp();
            float2 s = make_float2(0.f, 0.f);
            if (lane < i)
                for (int p = 0; p <= lane; p++) s = cfma(conjc(S.T[p][lane]), S.vv[p], s);
            S.w2[lane] = s;
        }
        __syncthreads();
        float nn = 0.f;
        for (int r = tid; r < nr; r += kHessThreads) {
            const int gr = g0 + r;
            if (gr > j0) {
                float2 b = bs[r];
                for (int q = 0; q < i; q++) b = csub(b, cmul(V[r * ld + q], S.w2[q]));
                bs[r] = b;
                if (gr >= j + 2) nn += cabs2(b);
                if (gr == j + 1)
                    for (int c = 0; c < K; c++) cluster.map_shared_rank(&S, c)->alpha = b;
            }
        }
        for (int o = 16; o > 0; o >>= 1) nn += __shfl_xor_sync(0xffffffffu, nn, o);
        if (lane == 0) S.red[warp] = nn;
        __syncthreads();
        if (warp == 0) {
            nn = lane < kHessWarps ? S.red[lane] : 0.f;
            for (int o = 16; o > 0; o >>= 1) nn += __shfl_xor_sync(0xffffffffu, nn, o);
            if (lane < K) cluster.map_shared_rank(&S, lane)->nrm[rank] = nn;
        }
        for (int q = warp; q < i; q += kHessWarps) {
            float2 s = make_float2(0.f, 0.f);
            for (int r = max(0, j + 2 - g0) + lane; r < nr; r += 32) s = cfma(conjc(V[r * ld + q]), bs[r], s);
            s = wsum(s);
            if (lane < K) cluster.map_shared_rank(&S, lane)->u[rank][q] = s;
        }
        cluster.sync();
        // the reflector (zlarfg), the same in every CTA
        float x2 = 0.f;
        for (int c = 0; c < K; c++) x2 += S.nrm[c];
        const float2 alpha = S.alpha;
        float2 tau = make_float2(0.f, 0.f), scal = tau;
        float2 beta = alpha;
        const bool drop = x2 + cabs2(alpha) <= neg2;
        if (drop) {
            beta = make_float2(0.f, 0.f);
        } else if (!(x2 == 0.f && alpha.y == 0.f)) {
            const float bt = -copysignf(sqrtf(alpha.x * alpha.x + alpha.y * alpha.y + x2), alpha.x);
            tau = make_float2((bt - alpha.x) / bt, -alpha.y / bt);
            beta = make_float2(bt, 0.f);
            scal = cdiv(make_float2(1.f, 0.f), csub(alpha, beta));
        }
        const bool live = tau.x != 0.f || tau.y != 0.f;
        // column j of the Hessenberg form
        for (int r = tid; r < nr; r += kHessThreads) {
            const int gr = g0 + r;
            if (gr > j0) A[(long long)gr * n + j] = gr <= j ? bs[r] : gr == j + 1 ? beta : make_float2(0.f, 0.f);
        }
        if (live) {
            // v of all rows; V^H v = scal u + conj(V(j + 1, :))
            for (int r = j + 1 + tid; r < n; r += kHessThreads) {
                const int c = r / rows;
                const float2 b = cluster.map_shared_rank(bs, c)[r - c * rows];
                const float2 v = r == j + 1 ? make_float2(1.f, 0.f) : cmul(b, scal);
                vf[r] = v;
                if (r <= j0 + kHb) S.VP[r - j0 - 1][i] = v;
            }
            if (warp == 0) {
                float2 s = make_float2(0.f, 0.f);
                if (lane < i) {
                    for (int c = 0; c < K; c++) s = cadd(s, S.u[c][lane]);
                    s = cadd(cmul(scal, s), conjc(S.VP[i][lane]));
                }
                S.vv[lane] = s;
                __syncwarp();
                // T(:, i) = -tau T V^H v
                float2 t = make_float2(0.f, 0.f);
                if (lane < i)
                    for (int p = lane; p < i; p++) t = cfma(S.T[lane][p], S.vv[p], t);
                t = cmul(t, tau);
                if (lane < i) S.T[lane][i] = make_float2(-t.x, -t.y);
                if (lane == i) S.T[i][i] = tau;
            }
            __syncthreads();
            for (int r = tid; r < nr; r += kHessThreads)
                V[r * ld + i] = g0 + r > j ? vf[g0 + r] : make_float2(0.f, 0.f);
            // y = tau (A v - Y V^H v): a warp per pair of rows, lanes along the row
            for (int r = 2 * warp; r < nr; r += 2 * kHessWarps) {
                const bool two = r + 1 < nr;
                const float2* a0 = A + (long long)(g0 + r) * n;
                const float2* a1 = two ? a0 + n : a0;
                float2 s0 = make_float2(0.f, 0.f), s1 = s0;
#pragma unroll 4
                for (int c = j + 1 + lane; c < n; c += 32) {
                    const float2 v = vf[c];
                    s0 = cfma(a0[c], v, s0);
                    s1 = cfma(a1[c], v, s1);
                }
                if (lane < i) {
                    const float2 q = S.vv[lane];
                    s0 = csub(s0, cmul(Y[r * ld + lane], q));
                    if (two) s1 = csub(s1, cmul(Y[(r + 1) * ld + lane], q));
                }
                s0 = wsum(s0);
                s1 = wsum(s1);
                __syncwarp();
                if (lane == 0) {
                    Y[r * ld + i] = cmul(tau, s0);
                    if (two) Y[(r + 1) * ld + i] = cmul(tau, s1);
                }
            }
        }
        __syncthreads();
    }
    // rows above the panel in its columns, and the factors of the trailing update
    for (int e = tid; e < nr * nb; e += kHessThreads) {
        const int r = e / nb, q = e - r * nb, gr = g0 + r;
        if (gr <= j0 && q >= 1 && q < ib) {
            float2 a = A[(long long)gr * n + j0 + q];
            for (int p = 0; p < q; p++) a = csub(a, cmul(Y[r * ld + p], conjc(S.VP[q - 1][p])));
            A[(long long)gr * n + j0 + q] = a;
        }
        float2 vt = make_float2(0.f, 0.f), vth = vt;
        if (q < ib) {
            for (int p = 0; p <= q; p++) vt = cfma(V[r * ld + p], S.T[p][q], vt);
            for (int p = q; p < ib; p++) vth = cfma(V[r * ld + p], conjc(S.T[q][p]), vth);
        }
        const long long o = (long long)gr * nb + q, per = (long long)n * nb;
        out[o] = V[r * ld + q];
        out[per + o] = Y[r * ld + q];
        out[2 * per + o] = vt;
        out[3 * per + o] = vth;
    }
    cluster.sync();                                  // no CTA leaves while another may read its b
}

}  // namespace z

size_t hess32_ws_elems(int n) { return (size_t)n * (5 * z::kHb) + 1; }

scw_status hess32(cudaStream_t st, float2* A, float2* Q, int n, int batch, float2* work, const GemmWs& ws, int share) {
    if (n <= 0 || batch <= 0) return SCW_OK;
    const long long nn = (long long)n * n;
    float* fro = reinterpret_cast<float*>(work);
    float2* pan = work + batch;                      // V, Y, V T, V T^H of every matrix, then W
    z::eye32_kernel<<<(unsigned)((nn * batch + 255) / 256), 256, 0, st>>>(Q, n, nn * batch);
    SCW_CUDA_TRY(cudaGetLastError());
    if (n < 3) return SCW_OK;
    SCW_CUDA_TRY(cudaMemsetAsync(fro, 0, sizeof(float) * batch, st));
    z::fro32_kernel<<<dim3((unsigned)std::min<long long>((nn + 255) / 256, 64), batch), 256, 0, st>>>(A, nn, fro);
    SCW_CUDA_TRY(cudaGetLastError());
    int dev = 0, sms = 0;
    SCW_CUDA_TRY(cudaGetDevice(&dev));
    SCW_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    // CTAs per matrix: all clusters (of `share` such batches at a time) resident at once, at least 32 rows
    // in each; more where the panel would not fit, then a narrower panel
    constexpr size_t kLimit = 220 * 1024;
    auto smem_of = [&](int k, int nb) {
        const int rows = (n + k - 1) / k;
        return sizeof(z::HessShared) + sizeof(float2) * ((size_t)rows * (2 * (nb + 1) + 2) + n);
    };
    int k = std::max(1, std::min({z::kHessMax, sms / (batch * std::max(1, share)), (n + 31) / 32})), nb = z::kHb;
    while (k < z::kHessMax && smem_of(k, nb) > kLimit) k++;
    while (nb > 1 && smem_of(k, nb) > kLimit) nb /= 2;
    if (smem_of(k, nb) > kLimit) return fail(SCW_ERR_ARG, "hess32: matrix too large");
    SCW_CUDA_TRY(cudaFuncSetAttribute(z::hess_panel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLimit));
    const long long per = (long long)n * nb, sp = 4 * per, sw = (long long)nb * n;
    float2 *V = pan, *Y = pan + per, *VT = pan + 2 * per, *VTH = pan + 3 * per, *W = pan + sp * batch;
    for (int j0 = 0; j0 + 2 < n; j0 += nb) {
        const int ib = std::min(nb, n - 2 - j0), c = j0 + ib, rem = n - c;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)k;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3((unsigned)(k * batch));
        cfg.blockDim = dim3(z::kHessThreads);
        cfg.dynamicSmemBytes = smem_of(k, nb);
        cfg.stream = st;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        SCW_CUDA_TRY(cudaLaunchKernelEx(&cfg, z::hess_panel_kernel, A, n, nn, j0, ib, nb, (n + k - 1) / k, pan,
                                        (const float*)fro));
        // A(:, c..) -= Y V(c.., :)^H, then A(:, c..) -= V T^H (V^H A(:, c..)); Q -= (Q V T) V^H
        scw_status s = gemm32x(st, n, rem, ib, -1.0, Y, nb, sp, kOpN, V + (long long)c * nb, nb, sp, kOpC, 1.0, A + c, n, nn,
                               batch, ws);
        if (s == SCW_OK) s = gemm32x(st, ib, rem, n, 1.0, V, nb, sp, kOpC, A + c, n, nn, kOpN, 0.0, W, n, sw, batch, ws);
        if (s == SCW_OK) s = gemm32x(st, n, rem, ib, -1.0, VTH, nb, sp, kOpN, W, n, sw, kOpN, 1.0, A + c, n, nn, batch, ws);
        if (s == SCW_OK) s = gemm32x(st, n, ib, n, 1.0, Q, n, nn, kOpN, VT, nb, sp, kOpN, 0.0, W, nb, sw, batch, ws);
        if (s == SCW_OK) s = gemm32x(st, n, n, ib, -1.0, W, nb, sw, kOpN, V, nb, sp, kOpC, 1.0, Q, n, nn, batch, ws);
        if (s != SCW_OK) return s;
    }
    return SCW_OK;
}

}  // namespace scw
