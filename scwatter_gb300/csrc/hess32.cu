// FP32 Hessenberg reduction A -> Q^H A Q of batched complex matrices, blocked (zgehrd / zlahr2 of LAPACK
// restated): the first stage of the mixed-precision eigen-solver.
//
// A panel of nb columns is reduced by one thread-block cluster per matrix; the trailing matrix and Q
// then get its nb reflectors at once as FP32 products (cgemm32.cu).  Per column j the
// cluster does, on the rows below the panel's top,
//   b = A(:, j) - Y V(j, :)^H, then b -= V T^H (V^H b)
//   the reflector v of b below row j, and y = tau (A v - Y V^H v)
// with V, Y distributed over the CTAs by rows in shared memory, and two cluster barriers: one for
// V^H b, one for |b|^2 and V^H v (which follows from V^H b because v is b scaled but for its first
// entry).  The rows of Y above follow as one product, Y = A V T.
//
// What bounds a column: A v reads the whole trailing matrix, 480 KB per CTA at n = 648 on 6 or 7 CTAs; the columns
// that fit (200 KB; from 430 rows on all of them) are kept in shared memory for the panel, the others come from L2
// at 11 000 clocks a column.  The rest are short phases between barriers, about 7000 clocks.  All clusters
// have to be resident at once: 20 clusters of 7 CTAs are not (16 fit into the GPCs), and took two turns.
// 20 matrices of n = 648: the panels 12.6 ms with every row of A read from L2 in 7-CTA clusters, 5.1 now;
// 10 of n = 216: 1.27 -> 0.90 ms; 4 of n = 50: 254 -> 181 us.  The products leave out the zero rows of V above
// the panel.  (Reduced column by column, with three launches each, every
// column read A three times, wrote it once, and the same for Q: 84 ms.)
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

constexpr int kHessSub = 4;                // lanes per row in the row loops

struct HessShared {
    float2 w[kHessMax][kHb];               // V^H b, one row per CTA
    float2 u[kHessMax][kHb];               // V(j+2.., :)^H b, one row per CTA
    float nrm[kHessMax];                   // |b(j+2..)|^2
    float2 T[kHb][kHb + 1];
    float2 VP[kHb + 1][kHb + 1];           // V(j0 + 1 + i, q)
    float2 w2[kHb], vv[kHb];
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

// y = tau (A v - Y q) of this CTA's rows into column i of Y: a warp takes R rows at a time, lanes along the
// row.  Columns c0 .. cm - 1 come from global memory (Ar), those from cm on from shared memory (Ac).
template <int R>
__device__ __forceinline__ void hess_rows(const float2* __restrict__ Ar, int n, const float2* Ac, int cc, int cm, const float2* v,
                                          int c0, int m, int nr, float2* Y, const float2* q, float2 tau, int i) {
    constexpr int ld = kHb + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int r = R * warp; r < nr; r += R * kHessWarps) {
        float2 s[R];
        int row[R];
#pragma unroll
        for (int t = 0; t < R; t++) {
            s[t] = make_float2(0.f, 0.f);
            row[t] = min(r + t, nr - 1);
        }
#pragma unroll 4
        for (int c = c0 + lane; c < cm; c += 32) {
            const float2 x = v[c];
#pragma unroll
            for (int t = 0; t < R; t++) s[t] = cfma(Ar[(long long)row[t] * n + c], x, s[t]);
        }
#pragma unroll 2
        for (int c = max(cm, c0) + lane; c < m; c += 32) {
            const float2 x = v[c];
#pragma unroll
            for (int t = 0; t < R; t++) s[t] = cfma(Ac[row[t] * cc + c - cm], x, s[t]);
        }
        const float2 w = q[lane];                    // zero from i on
#pragma unroll
        for (int t = 0; t < R; t++) {
            s[t] = csub(s[t], cmul(Y[row[t] * ld + lane], w));
            s[t] = wsum(s[t]);
        }
        __syncwarp();
#pragma unroll
        for (int t = 0; t < R; t++)
            if (lane == t && r + t < nr) Y[(r + t) * ld + i] = cmul(tau, s[t]);
    }
}

// V, Y (rows each) and two b of m entries
__host__ __device__ constexpr long long hess_cta_elems(int rows, int m) { return 2ll * rows * (kHb + 1) + 2ll * m; }

// Columns j0 .. j0 + ib - 1 on the rows below j0, `rows` per CTA.  The last cc columns of A's rows are kept in
// shared memory.  Outputs V, Y, VT = V T, VTH = V T^H (n x nb each, back to back per matrix; rows j0 + 1 .. n - 1)
// and the panel's columns of A below row j0.
// big: where V, Y and b do not fit into shared memory, a place for them per CTA (hess_cta_elems each).
__global__ void __launch_bounds__(kHessThreads)
hess_panel_kernel(float2* __restrict__ A, int n, long long sA, int j0, int ib, int rows, int cc, float2* __restrict__ out,
                  const float* __restrict__ fro, float2* big) {
    constexpr int NB = kHb;
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int K = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int mat = blockIdx.x / K, top = j0 + 1, m = n - top;
    A += sA * mat;
    out += 4ll * n * NB * mat;
    extern __shared__ __align__(16) unsigned char hess_smem[];
    HessShared& S = *reinterpret_cast<HessShared*>(hess_smem);
    constexpr int ld = NB + 1, per_lane = NB / kHessSub;
    float2* const near = reinterpret_cast<float2*>(hess_smem + sizeof(HessShared));
    const long long per_cta = hess_cta_elems(rows, m);
    float2* V = big ? big + ((long long)mat * K + rank) * per_cta : near;    // [rows][ld]
    float2* Y = V + rows * ld;                                                // [rows][ld]
    float2* bv = Y + rows * ld;                                               // [2][m]: b, then v, by column parity
    float2* Ac = big ? near : bv + 2 * m;                                     // [rows][cc]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int r0 = rank * rows, nr = max(0, min(rows, m - r0)), cm = m - cc;  // columns top + cm .. are in Ac
    const float2* Ar = A + (long long)(top + r0) * n + top;                   // this CTA's rows, from column top on
    const float2 zero = make_float2(0.f, 0.f);
    for (int e = tid; e < rows * ld; e += kHessThreads) V[e] = Y[e] = zero;
    for (int e = tid; e < kHb * (kHb + 1); e += kHessThreads) (&S.T[0][0])[e] = zero;
    for (int e = tid; e < (kHb + 1) * (kHb + 1); e += kHessThreads) (&S.VP[0][0])[e] = zero;
    for (int e = tid; e < kHessMax * kHb; e += kHessThreads) (&S.w[0][0])[e] = (&S.u[0][0])[e] = zero;
    if (tid < kHessMax) S.nrm[tid] = 0.f;
    for (int r = warp; r < nr; r += kHessWarps)
#pragma unroll 8
        for (int c = lane; c < cc; c += 32) Ac[r * cc + c] = Ar[(long long)r * n + cm + c];
    const float neg2 = fro[mat] * CT<float2>::ulp * CT<float2>::ulp / (float)n;
    const int rl = warp * 8 + (lane & 7), sub = lane >> 3;                    // row loops: 8 rows x 4 lanes
    cluster.sync();                                  // every CTA runs before the first remote write
    for (int i = 0; i < ib; i++) {
        const int jl = i - 1, j = j0 + i;            // column j is top + jl
        // (another CTA may still read the values of the column before)
        float2* bs = bv + (i & 1) * m;
        // b = A(:, j) - Y V(j, :)^H; V(j, q) = VP[i - 1][q]; columns from i on are zero
        for (int rb = 0; rb < nr; rb += kHessWarps * 8) {
            const int r = rb + rl;
            float2 b = zero;
            if (r < nr) {
                if (sub == 0) b = jl >= cm ? Ac[r * cc + jl - cm] : Ar[(long long)r * n + jl];
                if (i > 0)
#pragma unroll
                    for (int t = 0; t < per_lane; t++) {
                        const int q = per_lane * sub + t;
                        b = csub(b, cmul(Y[r * ld + q], conjc(S.VP[i - 1][q])));
                    }
            }
            b.x += __shfl_xor_sync(0xffffffffu, b.x, 8);
            b.y += __shfl_xor_sync(0xffffffffu, b.y, 8);
            b.x += __shfl_xor_sync(0xffffffffu, b.x, 16);
            b.y += __shfl_xor_sync(0xffffffffu, b.y, 16);
            if (sub == 0 && r < nr) bs[r0 + r] = b;
        }
        __syncthreads();
        for (int q = warp; q < i; q += kHessWarps) {
            float2 s = zero;
            for (int r = lane; r < nr; r += 32) s = cfma(conjc(V[r * ld + q]), bs[r0 + r], s);
            s = wsum(s);
            if (lane < K) cluster.map_shared_rank(&S, lane)->w[rank][q] = s;
        }
        cluster.sync();
        // w2 = T^H w: 16 lanes per entry
        {
            const int q = tid >> 4, p = tid & 15;
            float2 w0 = zero, w1 = zero;
#pragma unroll
            for (int c = 0; c < kHessMax; c++) {         // zero from K on
                w0 = cadd(w0, S.w[c][p]);
                w1 = cadd(w1, S.w[c][p + 16]);
            }
            float2 s = cfma(conjc(S.T[p + 16][q]), w1, cmul(conjc(S.T[p][q]), w0));
            for (int o = 8; o > 0; o >>= 1) {
                s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
                s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
            }
            if (p == 0) S.w2[q] = s;
        }
        __syncthreads();
        // b -= V w2, to every CTA
        for (int rb = 0; rb < nr; rb += kHessWarps * 8) {
            const int r = rb + rl;
            float2 b = zero;
            if (r < nr) {
                if (sub == 0) b = bs[r0 + r];
#pragma unroll
                for (int t = 0; t < per_lane; t++) b = csub(b, cmul(V[r * ld + per_lane * sub + t], S.w2[per_lane * sub + t]));
            }
            b.x += __shfl_xor_sync(0xffffffffu, b.x, 8);
            b.y += __shfl_xor_sync(0xffffffffu, b.y, 8);
            b.x += __shfl_xor_sync(0xffffffffu, b.x, 16);
            b.y += __shfl_xor_sync(0xffffffffu, b.y, 16);
            if (r < nr) {
                if (sub == 0) bs[r0 + r] = b;
                for (int c = sub; c < K; c += kHessSub)
                    if (c != rank) (big ? bs + (c - rank) * per_cta : cluster.map_shared_rank(bs, c))[r0 + r] = b;
            }
        }
        __syncthreads();
        for (int q = warp; q <= i; q += kHessWarps) {       // q = i: the norm
            float2 s = zero;
            for (int r = max(0, jl + 2 - r0) + lane; r < nr; r += 32) {
                const float2 b = bs[r0 + r];
                if (q < i) s = cfma(conjc(V[r * ld + q]), b, s);
                else s.x += cabs2(b);
            }
            s = wsum(s);
            if (lane < K) {
                HessShared* d = cluster.map_shared_rank(&S, lane);
                if (q < i) d->u[rank][q] = s;
                else d->nrm[rank] = s.x;
            }
        }
        cluster.sync();
        // the reflector (zlarfg), the same in every CTA
        float x2 = 0.f;
#pragma unroll
        for (int c = 0; c < kHessMax; c++) x2 += S.nrm[c];
        const float2 alpha = bs[jl + 1];
        float2 tau = zero, scal = zero;
        float2 beta = alpha;
        const bool drop = x2 + cabs2(alpha) <= neg2;
        if (drop) {
            beta = zero;
        } else if (!(x2 == 0.f && alpha.y == 0.f)) {
            const float bt = -copysignf(sqrtf(alpha.x * alpha.x + alpha.y * alpha.y + x2), alpha.x);
            tau = make_float2((bt - alpha.x) / bt, -alpha.y / bt);
            beta = make_float2(bt, 0.f);
            scal = cdiv(make_float2(1.f, 0.f), csub(alpha, beta));     // (1 / |d|^2 would overflow below 5e-20)
        }
        const bool live = tau.x != 0.f || tau.y != 0.f;
        // column j of the Hessenberg form
        for (int r = tid; r < nr; r += kHessThreads) {
            const int g = r0 + r;
            A[(long long)(top + g) * n + j] = g <= jl ? bs[g] : g == jl + 1 ? beta : zero;
        }
        __syncthreads();                             // alpha and column j are read before v takes b's place
        if (live) {
            // v from row j + 1 on; V^H v = scal u + conj(V(j + 1, :))
            for (int r = jl + 1 + tid; r < m; r += kHessThreads) {
                const float2 v = r == jl + 1 ? make_float2(1.f, 0.f) : cmul(bs[r], scal);
                bs[r] = v;
                if (r <= kHb) S.VP[r][i] = v;
                if (r >= r0 && r < r0 + nr) V[(r - r0) * ld + i] = v;
            }
            if (warp == kHessWarps - 1) {
                float2 s = zero;
                if (lane < i) {
#pragma unroll
                    for (int c = 0; c < kHessMax; c++) s = cadd(s, S.u[c][lane]);
                    s = cadd(cmul(scal, s), conjc(S.VP[i][lane]));
                }
                S.vv[lane] = s;
            }
            __syncthreads();
            // y = tau (A v - Y V^H v)
            const int per_warp = (nr + kHessWarps - 1) / kHessWarps;
            if (per_warp <= 1) hess_rows<1>(Ar, n, Ac, cc, cm, bs, jl + 1, m, nr, Y, S.vv, tau, i);
            else if (per_warp <= 2) hess_rows<2>(Ar, n, Ac, cc, cm, bs, jl + 1, m, nr, Y, S.vv, tau, i);
            else if (per_warp <= 4) hess_rows<4>(Ar, n, Ac, cc, cm, bs, jl + 1, m, nr, Y, S.vv, tau, i);
            else hess_rows<6>(Ar, n, Ac, cc, cm, bs, jl + 1, m, nr, Y, S.vv, tau, i);
            // T(:, i) = -tau T V^H v: 16 lanes per entry
            {
                const int q = tid >> 4, p = tid & 15;
                float2 s = cfma(S.T[q][p + 16], S.vv[p + 16], cmul(S.T[q][p], S.vv[p]));
                for (int o = 8; o > 0; o >>= 1) {
                    s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
                    s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
                }
                __syncthreads();                     // T is read before its column i is written
                s = cmul(s, tau);
                if (p == 0 && q < i) S.T[q][i] = make_float2(-s.x, -s.y);
                if (p == 0 && q == i) S.T[i][i] = tau;
            }
        }
        __syncthreads();
    }
    // the factors of the trailing update
    for (int e = tid; e < nr * NB; e += kHessThreads) {
        const int r = e / NB, q = e % NB;
        float2 vt = zero, vth = zero;
        if (q < ib) {
            for (int p = 0; p <= q; p++) vt = cfma(V[r * ld + p], S.T[p][q], vt);
            for (int p = q; p < ib; p++) vth = cfma(V[r * ld + p], conjc(S.T[q][p]), vth);
        }
        const long long o = (long long)(top + r0 + r) * NB + q, per = (long long)n * NB;
        out[o] = V[r * ld + q];
        out[per + o] = Y[r * ld + q];
        out[2 * per + o] = vt;
        out[3 * per + o] = vth;
    }
    cluster.sync();                                  // no CTA leaves while another may write to it
}

// The panel's columns j0 + 1 .. j0 + ib - 1 of the rows 0 .. j0: A -= Y V^H, a warp per row, lane q: column j0 + q.
__global__ void __launch_bounds__(256)
hess_above_kernel(float2* __restrict__ A, int n, long long sA, int j0, int ib, int nb, const float2* __restrict__ pan) {
    A += sA * blockIdx.y;
    pan += 4ll * n * nb * blockIdx.y;
    const float2 *V = pan + (long long)(j0 + 1) * nb, *Y = pan + (long long)n * nb;
    const int r = blockIdx.x * 8 + (threadIdx.x >> 5), q = threadIdx.x & 31;
    if (r > j0 || q < 1 || q >= ib) return;
    float2 a = A[(long long)r * n + j0 + q];
    for (int p = 0; p < q; p++) a = csub(a, cmul(Y[(long long)r * nb + p], conjc(V[(long long)(q - 1) * nb + p])));
    A[(long long)r * n + j0 + q] = a;
}

}  // namespace z

// panels, W, and (for large n) V, Y and b of up to kHessMax CTAs
size_t hess32_ws_elems(int n) {
    const size_t far = (size_t)z::kHessMax * (size_t)z::hess_cta_elems((n + z::kHessMax - 1) / z::kHessMax, n);
    return (size_t)n * (5 * z::kHb) + 1 + (n > 2400 ? far : 0);
}

scw_status hess32(cudaStream_t st, float2* A, float2* Q, int n, int batch, float2* work, int share) {
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
    // in each; more where V, Y and b would not fit, and from 2475 rows on they are kept in global memory
    constexpr size_t kLimit = 220 * 1024;
    auto smem_of = [&](int k, int m) {               // without the rows of A
        return sizeof(z::HessShared) + sizeof(float2) * (size_t)z::hess_cta_elems((m + k - 1) / k, m);
    };
    int k = std::max(1, std::min({z::kHessMax, sms / (batch * std::max(1, share)), (n + 31) / 32}));
    while (k < z::kHessMax && smem_of(k, n) > kLimit) k++;
    constexpr int nb = z::kHb;
    SCW_CUDA_TRY(cudaFuncSetAttribute(z::hess_panel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLimit));
    auto config = [&](int ctas, size_t smem, cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at) {
        cfg = {};
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)ctas;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3((unsigned)(ctas * batch));
        cfg.blockDim = dim3(z::kHessThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cfg.attrs = at;
        cfg.numAttrs = 1;
    };
    // a cluster's CTAs share a GPC, so fewer clusters fit than the SMs would hold (16 of 7 CTAs on 152 SMs)
    for (; k > 1 && smem_of(k - 1, n) <= kLimit; k--) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at[1];
        config(k, kLimit, cfg, at);
        int fit = 0;
        SCW_CUDA_TRY(cudaOccupancyMaxActiveClusters(&fit, z::hess_panel_kernel, &cfg));
        if (fit >= batch * std::max(1, share)) break;
    }
    const long long per = (long long)n * nb, sp = 4 * per, sw = (long long)nb * n;
    float2 *V = pan, *Y = pan + per, *VT = pan + 2 * per, *VTH = pan + 3 * per, *W = pan + sp * batch, *big = W + sw * batch;
    for (int j0 = 0; j0 + 2 < n; j0 += nb) {
        const int ib = std::min(nb, n - 2 - j0), c = j0 + ib, rem = n - c, top = j0 + 1, m = n - top;
        const int rows = (m + k - 1) / k;
        const bool far = smem_of(k, m) > kLimit;
        const size_t fixed = far ? sizeof(z::HessShared) : smem_of(k, m);
        const int cc = (int)std::min<size_t>(m, (kLimit - fixed) / (sizeof(float2) * rows));
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at[1];
        config(k, fixed + sizeof(float2) * (size_t)rows * cc, cfg, at);
        SCW_CUDA_TRY(cudaLaunchKernelEx(&cfg, z::hess_panel_kernel, A, n, nn, j0, ib, rows, cc, pan, (const float*)fro,
                                        far ? big : (float2*)nullptr));
        // V and its products are zero above row top: from there on only.  Y(0 .. j0, :) = A V T
        const long long o = (long long)top * nb;
        scw_status s = cgemm(st, top, ib, m, 1.f, A + top, n, nn, kOpN, VT + o, nb, sp, kOpN, false, Y, nb, sp, batch);
        if (s != SCW_OK) return s;
        if (ib > 1) {
            z::hess_above_kernel<<<dim3((top + 7) / 8, batch), 256, 0, st>>>(A, n, nn, j0, ib, nb, pan);
            SCW_CUDA_TRY(cudaGetLastError());
        }
        // A(:, c..) -= Y V(c.., :)^H, then A(:, c..) -= V T^H (V^H A(:, c..)); Q -= (Q V T) V^H
        s = cgemm(st, n, rem, ib, -1.f, Y, nb, sp, kOpN, V + (long long)c * nb, nb, sp, kOpC, true, A + c, n, nn, batch);
        float2* At = A + (long long)top * n + c;
        if (s == SCW_OK) s = cgemm(st, ib, rem, m, 1.f, V + o, nb, sp, kOpC, At, n, nn, kOpN, false, W, n, sw, batch);
        if (s == SCW_OK) s = cgemm(st, m, rem, ib, -1.f, VTH + o, nb, sp, kOpN, W, n, sw, kOpN, true, At, n, nn, batch);
        if (s == SCW_OK) s = cgemm(st, n, ib, m, 1.f, Q + top, n, nn, kOpN, VT + o, nb, sp, kOpN, false, W, nb, sw, batch);
        if (s == SCW_OK) s = cgemm(st, n, m, ib, -1.f, W, nb, sw, kOpN, V + o, nb, sp, kOpC, true, Q + top, n, nn, batch);
        if (s != SCW_OK) return s;
    }
    return SCW_OK;
}

}  // namespace scw
