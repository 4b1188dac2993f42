// FP64 complex dense linear algebra on the GPU, written for the per-layer coupled-wave solve:
// batched GEMM, blocked LU with partial pivoting and solves, and the non-Hermitian eigenvalue
// problem (Householder Hessenberg reduction, single-shift complex QR with Schur vectors,
// triangular eigenvectors, back-transformation).  They replace the MKL LAPACKE_zgeev,
// LAPACKE_zgesv and cblas_zgemm calls of the reference (third_Lapack.h:38-87).
//
// Conventions: row-major storage, element (i, j) of a matrix with leading dimension ld at
// A[i * ld + j]; complex numbers are double2 (re, im); "batched" kernels take a batch stride in
// elements and run one matrix per blockIdx.z (GEMM) or per CTA (factorisations).
//
// The GB300 FP64 rate is low (about 8 GFLOP/s per SM), so the O(n^3) parts are products where the
// algorithm allows it (the trailing updates of LU), and those run on the tensor cores; the inherently
// sequential ones (Hessenberg reduction, QR sweeps) run one CTA per matrix and are batched over
// the slices of a sample.
#include <algorithm>
#include <atomic>
#include <type_traits>
#include <cmath>
#include <vector>

#include <cooperative_groups.h>

#include "scw_dense.h"
#include "scw_launch.h"
#include "scw_complex.cuh"

namespace scw {
namespace z {

// ------------------------------------------------------------------------------------
// GEMM on the FP32 / FP64 pipes: C = alpha A B + beta C or alpha A B^T + beta C.  64 x 64 tiles,
// 256 threads, each thread a 4 x 4 complex block; K staged 16 at a time through shared memory.
// FP64 products run on the tensor cores (gemm_tc.cu, 20 to 35 times faster) and come here only
// without a workspace: while the stream of scw_zgemm is being captured, or where memory is short.
// ------------------------------------------------------------------------------------
constexpr int kGT = 64, kGK = 16;

template <typename C>
__global__ void __launch_bounds__(256)
gemm_kernel(int M, int N, int K, C alpha, const C* __restrict__ A, int lda, long long sA, const C* __restrict__ B,
            int ldb, long long sB, int tb, C beta, C* __restrict__ Cm, int ldc, long long sC, const int* __restrict__ skip) {
    if (skipped(skip, blockIdx.z)) return;
    __shared__ C As[kGK][kGT + 1];
    __shared__ C Bs[kGK][kGT + 1];
    A += sA * blockIdx.z;
    B += sB * blockIdx.z;
    Cm += sC * blockIdx.z;
    const int i0 = blockIdx.y * kGT, j0 = blockIdx.x * kGT;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    const C zero = CT<C>::mk(0, 0);
    C acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 4; b++) acc[a][b] = zero;
    for (int k0 = 0; k0 < K; k0 += kGK) {
        for (int e = threadIdx.x; e < kGK * kGT; e += 256) {
            const int r = e / kGK, kk = e % kGK;         // A tile: rows i0 + r, cols k0 + kk
            const int gi = i0 + r, gk = k0 + kk;
            As[kk][r] = (gi < M && gk < K) ? A[(long long)gi * lda + gk] : zero;
            const int kk2 = tb ? e % kGK : e / kGT, c = tb ? e / kGK : e % kGT;         // B tile: rows k0 + kk2, cols j0 + c
            const int gk2 = k0 + kk2, gj = j0 + c;
            Bs[kk2][c] = (gk2 < K && gj < N) ? B[tb ? (long long)gj * ldb + gk2 : (long long)gk2 * ldb + gj] : zero;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < kGK; kk++) {
            C a[4], b[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                a[q] = As[kk][ty + 16 * q];
                b[q] = Bs[kk][tx + 16 * q];
            }
#pragma unroll
            for (int p = 0; p < 4; p++)
#pragma unroll
                for (int q = 0; q < 4; q++) acc[p][q] = cfma(a[p], b[q], acc[p][q]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int p = 0; p < 4; p++) {
        const int gi = i0 + ty + 16 * p;
        if (gi >= M) continue;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int gj = j0 + tx + 16 * q;
            if (gj >= N) continue;
            C* c = Cm + (long long)gi * ldc + gj;
            C v = cmul(alpha, acc[p][q]);
            if (beta.x != 0 || beta.y != 0) v = cfma(beta, *c, v);
            *c = v;
        }
    }
}

// ------------------------------------------------------------------------------------
// FP64 LU with partial pivoting, blocked, batched.  piv[k] = row swapped with row k at step k
// (LAPACK convention, 0-based).  info[b] = first zero pivot + 1 (0: nonsingular).
//
// The panel is what is serial: per column a pivot search, a swap and a rank-1 update.  A
// thread-block cluster of 8 CTAs holds the panel in shared memory, a slice of its rows in each.
// Per column every CTA sends its best candidate with that row's values and the candidate's inverse (and the
// owner of row k that row) to all eight, so one cluster barrier per column decides the pivot and brings
// everything the update needs; the candidate buffers alternate, so the next column's sends
// cannot reach a CTA that still reads.  FP64 instructions are the scarce thing (75 clocks a warp): the search
// compares integers, one lane per CTA divides, while the other warps bring the columns after the next one up to
// date.  A panel of 32 columns: 260 us when every thread compared and divided in FP64, now 94 us with 648
// rows and 63 with 50, where the barrier, the division and the sends are left; 1.05 ms on one CTA with the panel in
// global memory.
// ------------------------------------------------------------------------------------
constexpr int kNB = 32;
constexpr int kLuCtas = 8, kLuThreads = 256;

struct LuSlot {
    double2 inv;                       // of the candidate
    int hi;                            // |a| of the candidate: the double's upper and lower half; hi < 0: none
    unsigned lo;
    int row, pad;
    double2 v[kNB];
};

// 1 / p with one division: conj(p) / |p|^2 with p scaled by a power of two (Smith's form has two divisions in a row)
__device__ __forceinline__ double2 lu_inverse(double2 p) {
    const int be = max(__double2hiint(p.x) & 0x7ff00000, __double2hiint(p.y) & 0x7ff00000) >> 20;
    if (be == 2047) return cdiv(make_double2(1.0, 0.0), p);
    const double s = __hiloint2double((2046 - min(be, 2045)) << 20, 0);
    const double x = p.x * s, y = p.y * s, r = s / fma(x, x, y * y);
    return make_double2(x * r, -y * r);
}

// Pivot candidates are compared as integers (non-negative doubles order as their bits): an FP64 comparison by
// all threads costs as much as 75 clocks a warp.  Larger value first, then the smaller row; NaN: none.
struct LuKey {
    int hi, row;
    unsigned lo;
};
__device__ __forceinline__ LuKey lu_key(double2 v, int row) {
    const double a = cabs1(v);
    const long long bits = __double_as_longlong(a);
    const int hi = (int)(bits >> 32);
    const bool nan = (hi & 0x7fffffff) > 0x7ff00000 || ((hi & 0x7fffffff) == 0x7ff00000 && (unsigned)bits != 0u);
    return LuKey{nan ? -1 : hi, row, (unsigned)bits};
}
__device__ __forceinline__ LuKey lu_best(LuKey k) {      // over a warp
    const int hi = __reduce_max_sync(0xffffffffu, k.hi);
    const unsigned lo = __reduce_max_sync(0xffffffffu, k.hi == hi ? k.lo : 0u);
    const int row = __reduce_min_sync(0xffffffffu, k.hi == hi && k.lo == lo ? k.row : 0x7fffffff);
    return LuKey{hi, row, lo};
}
__device__ __forceinline__ double2 lu_sub(double2 x, double2 l, double2 p) {     // x - l p
    return make_double2(fma(-l.x, p.x, fma(l.y, p.y, x.x)), fma(-l.x, p.y, fma(-l.y, p.x, x.y)));
}

// kFar: where a CTA's rows do not fit into shared memory the panel stays in A
template <bool kFar>
__global__ void __cluster_dims__(kLuCtas, 1, 1) __launch_bounds__(kLuThreads)
lu_panel_kernel(double2* __restrict__ A, int n, int lda, long long sA, int k0, int nb, int rows, int* __restrict__ piv,
                long long sP, int* __restrict__ info, const int* __restrict__ skip) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), b = blockIdx.x / kLuCtas;
    if (skipped(skip, b)) return;                        // the whole cluster, before any barrier
    A += sA * b;
    piv += sP * b;
    extern __shared__ __align__(16) unsigned char lu_smem[];
    LuSlot* slot = reinterpret_cast<LuSlot*>(lu_smem);   // [2][kLuCtas]: candidates of column parity
    LuSlot* krow = slot + 2 * kLuCtas;                   // [2]: row k
    const int g0 = k0 + rank * rows;                     // this CTA's rows g0 .. g0 + nr - 1
    const int nr = max(0, min(rows, n - g0));
    double2* const P = kFar ? A + (long long)g0 * lda + k0 : reinterpret_cast<double2*>(krow + 2);   // [rows][ld]
    const std::conditional_t<kFar, long long, int> ld = kFar ? lda : nb + 1;
    constexpr int kWarps = kLuThreads / 32;
    __shared__ LuKey red[kWarps], mine;
    __shared__ double2 mine_inv;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (!kFar)
        for (int e = tid; e < nr * nb; e += kLuThreads) {
            const int r = e / nb, c = e - r * nb;
            P[r * ld + c] = A[(long long)(g0 + r) * lda + k0 + c];
        }
    __syncthreads();
    const LuKey nothing{-1, 0x7fffffff, 0u};
    auto better = [](const LuKey& x, const LuKey& y) {
        return x.hi > y.hi || (x.hi == y.hi && (x.lo > y.lo || (x.lo == y.lo && x.row < y.row)));
    };
    LuKey best = nothing;
    for (int r = tid; r < nr; r += kLuThreads) {
        const LuKey k = lu_key(P[r * ld], g0 + r);
        if (k.hi >= 0 && better(k, best)) best = k;
    }
    best = lu_best(best);
    if (lane == 0) red[warp] = best;
    cluster.sync();                                      // every CTA runs before the first remote write
    const double2* prow = nullptr;                       // the pivot row of the column before
    for (int j = 0; j < nb; j++) {
        const int k = k0 + j, par = j & 1;
        if (warp == 0) {
            // this CTA's candidate and its inverse
            best = lu_best(lane < kWarps ? red[lane] : nothing);
            if (lane == 0) {
                mine = best;
                const double2 d = best.hi >= 0 ? P[(best.row - g0) * ld + j] : make_double2(0.0, 0.0);
                mine_inv = best.hi >= 0 && (best.hi | (int)best.lo) != 0 ? lu_inverse(d) : make_double2(0.0, 0.0);
            }
        } else if (j > 0) {
            // meanwhile the others bring the columns from j + 1 on up to date, every lane with an entry
            const int w = nb - 1 - j, f = max(0, k - g0), cnt = (nr - f) * w, step = kLuThreads - 32;
            if (w > 0 && cnt > 0) {
                int e = tid - 32, r = e / w, c = e - r * w;
                const int dr = step / w, dc = step - dr * w;
                for (; e < cnt; e += step) {
                    double2* row = P + (f + r) * ld;
                    row[j + 1 + c] = lu_sub(row[j + 1 + c], row[j - 1], prow[j + 1 + c]);
                    r += dr;
                    c += dc;
                    if (c >= w) {
                        c -= w;
                        r++;
                    }
                }
            }
        }
        __syncthreads();
        // warp w sends to CTA w: the candidate with its row, and row k from its owner
        {
            LuSlot* dst = cluster.map_shared_rank(slot, warp) + par * kLuCtas + rank;
            const LuKey m = mine;
            if (m.hi >= 0 && lane < nb) dst->v[lane] = P[(m.row - g0) * ld + lane];
            if (lane == 0) {
                dst->hi = m.hi;
                dst->lo = m.lo;
                dst->row = m.row;
                dst->inv = mine_inv;
            }
            if (k >= g0 && k < g0 + nr) {
                LuSlot* dk = cluster.map_shared_rank(krow, warp) + par;
                if (lane < nb) dk->v[lane] = P[(k - g0) * ld + lane];
            }
        }
        cluster.sync();
        const LuSlot* cand = slot + par * kLuCtas;
        const LuKey got = lane < kLuCtas ? LuKey{cand[lane].hi, cand[lane].row, cand[lane].lo} : nothing;
        best = lu_best(got);
        const bool none = best.hi < 0;                   // no comparable value (all NaN): row k stays
        const unsigned who = __ballot_sync(0xffffffffu, got.hi == best.hi && got.lo == best.lo && got.row == best.row);
        const int pr = __ffs(who) - 1, p = none ? k : best.row;
        prow = none ? krow[par].v : cand[pr].v;
        const bool zero = best.hi == 0 && best.lo == 0u;
        const double2 inv = none ? make_double2(nan(""), nan("")) : cand[pr].inv;
        if (rank == 0 && tid == 0) {
            piv[k] = p;
            if (zero && info[b] == 0) info[b] = k + 1;
        }
        if (warp == 0 && p != k) {
            if (p >= g0 && p < g0 + nr && lane < nb) P[(p - g0) * ld + lane] = krow[par].v[lane];
            if (k >= g0 && k < g0 + nr && lane < nb) P[(k - g0) * ld + lane] = prow[lane];
        }
        __syncthreads();
        // scale the column below the pivot, the next column, and its candidate
        best = nothing;
        for (int r = max(0, k + 1 - g0) + tid; r < nr; r += kLuThreads) {
            double2* row = P + r * ld;
            const double2 l = cmul(row[j], inv);
            row[j] = l;
            if (j + 1 < nb) {
                const double2 v = lu_sub(row[j + 1], l, prow[j + 1]);
                row[j + 1] = v;
                const LuKey q = lu_key(v, g0 + r);
                if (q.hi >= 0 && better(q, best)) best = q;
            }
        }
        best = lu_best(best);
        if (lane == 0) red[warp] = best;
        __syncthreads();
    }
    if (!kFar)
        for (int e = tid; e < nr * nb; e += kLuThreads) {
            const int r = e / nb, c = e - r * nb;
            A[(long long)(g0 + r) * lda + k0 + c] = P[r * ld + c];
        }
}

// The panel's row interchanges on the columns outside it, then L11 U12 = A12 on the columns right of
// it, 32 columns per CTA.  The interchanges touch at most 64 rows: warp 0 follows them to the rows'
// sources (lane i: the source of row k0 + i, and a row below the panel that was exchanged with
// one of the panel), so that all rows are read at once and then written.
template <int C>
__global__ void __launch_bounds__(256)
lu_apply_kernel(double2* __restrict__ A, int ncols, int lda, long long sA, int k0, int nb, const int* __restrict__ piv,
                long long sP, const int* __restrict__ skip) {
    chain_wait();
    if (skipped(skip, blockIdx.y)) return;
    A += sA * blockIdx.y;
    piv += sP * blockIdx.y;
    __shared__ double2 X[kNB][C + 1], L[kNB][33];
    __shared__ int s_top[kNB], s_row[kNB], s_src[kNB];
    constexpr int G = 256 / C, Q = kNB / G;             // row groups, rows per thread
    const int tid = threadIdx.x, lane = tid & 31, c = tid % C, j = blockIdx.x * C + c;
    if (tid < 32) {
        int top = k0 + lane, orow = -1, osrc = -1;
        const int mine = lane < nb ? piv[k0 + lane] : 0;
        for (int i = 0; i < nb; i++) {
            const int p = __shfl_sync(0xffffffffu, mine, i), a = __shfl_sync(0xffffffffu, top, i);
            const unsigned hit = __ballot_sync(0xffffffffu, orow == p);
            const int t = p < k0 + nb ? p - k0 : 0, bt = __shfl_sync(0xffffffffu, top, t);
            const int q = hit ? __ffs(hit) - 1 : i, cur = __shfl_sync(0xffffffffu, osrc, q);
            if (p < k0 + nb) {
                if (lane == i) top = bt;
                else if (lane == t) top = a;
            } else {
                if (lane == i) top = hit ? cur : p;
                if (lane == q) {
                    orow = p;
                    osrc = a;
                }
            }
        }
        s_top[lane] = top;
        s_row[lane] = orow;
        s_src[lane] = osrc;
    }
    const bool live = j < ncols && !(j >= k0 && j < k0 + nb), right = live && j >= k0 + nb;
    __syncthreads();
    for (int e = tid; e < nb * nb; e += 256) {
        const int r = e / nb, q = e - r * nb;
        L[r][q] = A[(long long)(k0 + r) * lda + k0 + q];
    }
    double2 o[Q];
#pragma unroll
    for (int q = 0; q < Q; q++) {
        const int r = tid / C + G * q;
        o[q] = make_double2(0.0, 0.0);
        if (live && r < nb) {
            X[r][c] = A[(long long)s_top[r] * lda + j];
            if (s_row[r] >= 0) o[q] = A[(long long)s_src[r] * lda + j];
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < Q; q++) {
        const int r = tid / C + G * q;
        if (live && r < nb && s_row[r] >= 0) A[(long long)s_row[r] * lda + j] = o[q];
    }
    const int steps = blockIdx.x * C + C - 1 >= k0 + nb ? nb - 1 : 0;      // left of the panel: interchanges only
    for (int m = 0; m < steps; m++) {
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const int r = tid / C + G * q;
            if (right && r > m && r < nb) X[r][c] = lu_sub(X[r][c], L[r][m], X[m][c]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int q = 0; q < Q; q++) {
        const int r = tid / C + G * q;
        if (live && r < nb) A[(long long)(k0 + r) * lda + j] = X[r][c];
    }
}

// Row interchanges of B from getrf's pivots (LAPACK laswp order), one thread per column.
__global__ void __launch_bounds__(256)
laswp_kernel(const int* __restrict__ piv, long long sP, double2* __restrict__ B, int ldb, long long sB, int n, int nrhs,
             const int* __restrict__ skip) {
    if (skipped(skip, blockIdx.y)) return;
    piv += sP * blockIdx.y;
    B += sB * blockIdx.y;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= nrhs) return;
    for (int k = 0; k < n; k++) {
        const int p = piv[k];
        if (p != k) {
            const double2 t = B[(long long)k * ldb + j];
            B[(long long)k * ldb + j] = B[(long long)p * ldb + j];
            B[(long long)p * ldb + j] = t;
        }
    }
}

// q = x (1 / d) brought to the accuracy of a division; as it is where the correction is not finite (d
// infinite), and a division where 1 / d is not (d zero or below the range of its inverse)
__device__ __forceinline__ double2 z_div_fix(double2 x, double2 q, double2 d, double2 id) {
    if (!isfinite(id.x) || !isfinite(id.y)) return cdiv(x, d);
    const double2 r = lu_sub(x, q, d);
    const double2 f = make_double2(fma(r.x, id.x, fma(-r.y, id.y, q.x)), fma(r.x, id.y, fma(r.y, id.x, q.y)));
    return isfinite(f.x) && isfinite(f.y) ? f : q;
}

// Triangular solve restricted to the diagonal block rows [k0, k0 + nb) of the LU factors, 32
// right-hand-side columns per CTA in shared memory: unit lower L (upper == 0) or U (upper == 1).
// Rows outside the block were already folded in by the GEMM updates of the blocked solve.
template <int C>
__global__ void __launch_bounds__(256)
trsm_block_kernel(const double2* __restrict__ LU, int lda, long long sA, int k0, int nb, double2* __restrict__ B, int ldb,
                  long long sB, int nrhs, int upper, const int* __restrict__ skip) {
    chain_wait();
    if (skipped(skip, blockIdx.y)) return;
    LU += sA * blockIdx.y;
    B += sB * blockIdx.y;
    constexpr int G = 256 / C, Q = kNB / G;             // row groups, rows per thread
    __shared__ double2 X[kNB][C + 1], L[kNB][33], D[kNB];
    const int tid = threadIdx.x, c = tid % C, w = tid / C, j = blockIdx.x * C + c;
    const bool live = j < nrhs;
#pragma unroll
    for (int q = 0; q < Q; q++) {
        const int r = w + G * q;
        if (r < nb && live) X[r][c] = B[(long long)(k0 + r) * ldb + j];
    }
    for (int e = tid; e < nb * nb; e += 256) {
        const int r = e / nb, q = e - r * nb;
        const double2 v = LU[(long long)(k0 + r) * lda + k0 + q];
        L[r][q] = v;
        if (upper && r == q) D[r] = lu_inverse(v);
    }
    __syncthreads();
    for (int s = 0; s < nb; s++) {
        const int m = upper ? nb - 1 - s : s;
        if (upper) {
            // x / d as x (1 / d) and one correction by the residual x - (x / d) d
            if (w == 0 && live) {
                const double2 x = X[m][c], q = cmul(x, D[m]);
                X[m][c] = z_div_fix(x, q, L[m][m], D[m]);
            }
            __syncthreads();
        }
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const int r = w + G * q;
            if (live && r < nb && (upper ? r < m : r > m)) X[r][c] = lu_sub(X[r][c], L[r][m], X[m][c]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int q = 0; q < Q; q++) {
        const int r = w + G * q;
        if (r < nb && live) B[(long long)(k0 + r) * ldb + j] = X[r][c];
    }
}

// ------------------------------------------------------------------------------------
// Hessenberg reduction A -> Q^H A Q (zgehd2 semantics: H(k) = I - tau v v^H, v(k+1) = 1),
// one CTA per matrix, with the explicit unitary Q accumulated (Q := Q H(k)).
// ------------------------------------------------------------------------------------
__device__ double block_sum(double v, double* sh) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) sh[w] = v;
    __syncthreads();
    double s = 0;
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) s += sh[i];
    return s;
}

// y[i] = tau * sum_{j >= j0} M[i][j] v[j] for every row i: a warp per row, lanes along the row
// (coalesced), then a butterfly sum
__device__ __forceinline__ void row_products(const double2* __restrict__ M, const double2* __restrict__ v, double2* __restrict__ y, int n,
                                             int j0, double2 tau) {
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int i = threadIdx.x >> 5; i < n; i += nw) {
        const double2* row = M + (long long)i * n;
        double2 s = CT<double2>::mk(0, 0);
#pragma unroll 4
        for (int j = j0 + lane; j < n; j += 32) s = cfma(row[j], v[j], s);
        for (int o = 16; o > 0; o >>= 1) {
            s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
            s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
        }
        if (lane == 0) y[i] = cmul(tau, s);
    }
}

// col[i * ld] += u[i] * alpha for i in [i0, i1): kStripe rows at a time, loads before the
// updates, so that a thread has kStripe independent loads in flight instead of one
// load-update-store chain per row
__device__ __forceinline__ void column_axpy(double2* __restrict__ col, long long ld, int i0, int i1, const double2* __restrict__ u,
                                            double2 alpha) {
    constexpr int kStripe = 4;
    for (int b = i0; b < i1; b += kStripe) {
        double2 a[kStripe];
#pragma unroll
        for (int q = 0; q < kStripe; q++)
            if (b + q < i1) a[q] = col[(long long)(b + q) * ld];
#pragma unroll
        for (int q = 0; q < kStripe; q++)
            if (b + q < i1) col[(long long)(b + q) * ld] = cfma(u[b + q], alpha, a[q]);
    }
}

__global__ void __launch_bounds__(1024)
hessenberg_kernel(double2* __restrict__ A, double2* __restrict__ Q, int n, long long sA, double2* __restrict__ work,
                  const int* __restrict__ skip) {
    if (skipped(skip, blockIdx.x)) return;
    A += sA * blockIdx.x;
    Q += sA * blockIdx.x;
    double2* v = work + (long long)blockIdx.x * 3 * n;      // Householder vector (rows k+1..n-1)
    double2* y = v + 2 * n;                                   // tau A v / tau Q v (the work keeps 3 n per matrix)
    __shared__ double sh[32];
    __shared__ double2 s_tau, s_beta;
    constexpr int kStripe = 4;
    for (int i = threadIdx.x; i < n * n; i += blockDim.x) Q[i] = CT<double2>::mk((i / n) == (i % n) ? 1 : 0, 0);
    __syncthreads();
    for (int k = 0; k + 2 < n; k++) {
        // Householder for x = A[k+1:n, k] (zlarfg)
        double xn2 = 0;
        for (int i = k + 2 + threadIdx.x; i < n; i += blockDim.x) xn2 += cabs2(A[(long long)i * n + k]);
        xn2 = block_sum(xn2, sh);
        const double2 alpha = A[(long long)(k + 1) * n + k];
        if (threadIdx.x == 0) {
            if (xn2 == 0 && alpha.y == 0) {
                s_tau = CT<double2>::mk(0, 0);
                s_beta = alpha;
            } else {
                const double beta = -r_copysign(r_sqrt(alpha.x * alpha.x + alpha.y * alpha.y + xn2), alpha.x);
                s_tau = CT<double2>::mk((beta - alpha.x) / beta, -alpha.y / beta);
                s_beta = CT<double2>::mk(beta, 0);
            }
        }
        __syncthreads();
        const double2 tau = s_tau;
        if (tau.x == 0 && tau.y == 0) {
            __syncthreads();
            continue;
        }
        const double2 scal = cdiv(CT<double2>::mk(1, 0), csub(alpha, s_beta));
        for (int i = k + 1 + threadIdx.x; i < n; i += blockDim.x)
            v[i] = (i == k + 1) ? CT<double2>::mk(1, 0) : cmul(A[(long long)i * n + k], scal);
        __syncthreads();
        // right: A[:, k+1:] -= tau (A[:, k+1:] v) v^H   (all rows; a warp per row for the products)
        row_products(A, v, y, n, k + 1, tau);
        __syncthreads();
        // then left: A[k+1:, k+1:] -= conj(tau) v (v^H A[k+1:, k+1:]).  Both act on one column
        // at a time, so each thread owns its columns: right update (all rows) while summing
        // v^H of the updated column, then the left update of that column.
        for (int j = k + 1 + threadIdx.x; j < n; j += blockDim.x) {
            const double2 vc = CT<double2>::mk(v[j].x, -v[j].y);
            double2 s = CT<double2>::mk(0, 0);
            double2* col = A + j;
            // kStripe rows at a time: loads first, then the updates (see column_axpy)
            for (int i0 = 0; i0 < n; i0 += kStripe) {
                double2 a[kStripe];
#pragma unroll
                for (int q = 0; q < kStripe; q++)
                    if (i0 + q < n) a[q] = col[(long long)(i0 + q) * n];
#pragma unroll
                for (int q = 0; q < kStripe; q++) {
                    const int i = i0 + q;
                    if (i < n) {
                        a[q] = csub(a[q], cmul(y[i], vc));
                        col[(long long)i * n] = a[q];
                        if (i > k) s = cfma(CT<double2>::mk(v[i].x, -v[i].y), a[q], s);
                    }
                }
            }
            const double2 wj = cmul(CT<double2>::mk(tau.x, -tau.y), s);
            column_axpy(col, n, k + 1, n, v, CT<double2>::mk(-wj.x, -wj.y));
        }
        // column k below the subdiagonal
        for (int i = k + 1 + threadIdx.x; i < n; i += blockDim.x)
            A[(long long)i * n + k] = (i == k + 1) ? s_beta : CT<double2>::mk(0, 0);
        // Q[:, k+1:] -= (Q[:, k+1:] v) tau v^H
        __syncthreads();
        row_products(Q, v, y, n, k + 1, tau);
        __syncthreads();
        for (int j = k + 1 + threadIdx.x; j < n; j += blockDim.x)
            column_axpy(Q + j, n, 0, n, y, CT<double2>::mk(-v[j].x, v[j].y));
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------
// The same reduction spread over the whole GPU: per column k three short launches for the
// batch -- the Householder vector (one CTA per matrix), the products y = tau A[:, k+1:] v and
// z = tau Q[:, k+1:] v (a warp per row, rows of every matrix over all SMs), and the updates of
// the columns k+1.. of A (right then left, one thread per column) and of Q.  Every element sees
// the operations of hessenberg_kernel in the same order; the kernel boundaries replace its
// block barriers, so the O(n^2) work of a column runs on every SM instead of one per matrix.
// Per matrix the 3n work entries hold v (slot 0: tau), y and z.
// ------------------------------------------------------------------------------------
constexpr int kHwRows = 8;        // rows (warps) per CTA of the product kernel
constexpr int kHwCols = 128;      // columns (threads) per CTA of the update kernel

__global__ void __launch_bounds__(256) hw_init_kernel(double2* __restrict__ Q, int n, long long sA, const int* __restrict__ skip) {
    if (skipped(skip, blockIdx.y)) return;
    Q += sA * blockIdx.y;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < (long long)n * n;
         i += (long long)gridDim.x * blockDim.x)
        Q[i] = CT<double2>::mk((i / n) == (i % n) ? 1 : 0, 0);
}

__global__ void __launch_bounds__(256) hw_vec_kernel(double2* __restrict__ A, int n, long long sA, double2* __restrict__ work, int k,
                                                     const int* __restrict__ skip) {
    if (skipped(skip, blockIdx.x)) return;
    A += sA * blockIdx.x;
    double2* v = work + (long long)blockIdx.x * 3 * n;
    __shared__ double sh[32];
    __shared__ double2 s_beta;
    __shared__ int s_skip;
    double xn2 = 0;
    for (int i = k + 2 + threadIdx.x; i < n; i += blockDim.x) xn2 += cabs2(A[(long long)i * n + k]);
    xn2 = block_sum(xn2, sh);
    const double2 alpha = A[(long long)(k + 1) * n + k];
    if (threadIdx.x == 0) {
        s_skip = 0;
        if (xn2 == 0 && alpha.y == 0) {
            s_skip = 1;                       // already reduced
        } else {
            const double beta = -r_copysign(r_sqrt(alpha.x * alpha.x + alpha.y * alpha.y + xn2), alpha.x);
            v[0] = CT<double2>::mk((beta - alpha.x) / beta, -alpha.y / beta);      // tau
            s_beta = CT<double2>::mk(beta, 0);
        }
        if (s_skip) v[0] = CT<double2>::mk(0, 0);
    }
    __syncthreads();
    if (s_skip) return;
    const double2 scal = cdiv(CT<double2>::mk(1, 0), csub(alpha, s_beta));
    for (int i = k + 1 + threadIdx.x; i < n; i += blockDim.x) {
        v[i] = (i == k + 1) ? CT<double2>::mk(1, 0) : cmul(A[(long long)i * n + k], scal);
        A[(long long)i * n + k] = (i == k + 1) ? s_beta : CT<double2>::mk(0, 0);
    }
}

// rows 0..n-1: y[i] = tau sum_{j > k} A[i][j] v[j]; rows n..2n-1: z[i] = tau sum_{j > k} Q[i][j] v[j]
__global__ void __launch_bounds__(kHwRows * 32) hw_prod_kernel(const double2* __restrict__ A, const double2* __restrict__ Q, int n,
                                                               long long sA, double2* __restrict__ work, int k,
                                                               const int* __restrict__ skip) {
    if (skipped(skip, blockIdx.y)) return;
    double2* v = work + (long long)blockIdx.y * 3 * n;
    const double2 tau = v[0];
    if (tau.x == 0 && tau.y == 0) return;
    const int lane = threadIdx.x & 31;
    const int r = blockIdx.x * kHwRows + (threadIdx.x >> 5);
    if (r >= 2 * n) return;
    const double2* row = (r < n ? A + (long long)r * n : Q + (long long)(r - n) * n) + sA * blockIdx.y;
    double2 acc = CT<double2>::mk(0, 0);
#pragma unroll 4
    for (int j = k + 1 + lane; j < n; j += 32) acc = cfma(row[j], v[j], acc);
    for (int o = 16; o > 0; o >>= 1) {
        acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
        acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
    }
    if (lane == 0) v[n + r] = cmul(tau, acc);          // y = v + n, z = v + 2n
}

// columns j > k of A: right update (all rows) while summing v^H of the updated column, then the
// left update; columns j > k of Q (blocks past the A blocks): Q[:, j] -= z conj(v_j)
__global__ void __launch_bounds__(kHwCols) hw_update_kernel(double2* __restrict__ A, double2* __restrict__ Q, int n, long long sA,
                                                            const double2* __restrict__ work, int k, int nblk_a,
                                                            const int* __restrict__ skip) {
    if (skipped(skip, blockIdx.y)) return;
    const double2* v = work + (long long)blockIdx.y * 3 * n;
    const double2 tau = v[0];
    if (tau.x == 0 && tau.y == 0) return;
    constexpr int kStripe = 4;
    const bool isA = (int)blockIdx.x < nblk_a;
    const int j = k + 1 + (isA ? (int)blockIdx.x : (int)blockIdx.x - nblk_a) * kHwCols + threadIdx.x;
    if (j >= n) return;
    if (isA) {
        const double2* y = v + n;
        const double2 vc = CT<double2>::mk(v[j].x, -v[j].y);
        double2* col = A + sA * blockIdx.y + j;
        double2 s = CT<double2>::mk(0, 0);
        for (int i0 = 0; i0 < n; i0 += kStripe) {
            double2 a[kStripe];
#pragma unroll
            for (int q = 0; q < kStripe; q++)
                if (i0 + q < n) a[q] = col[(long long)(i0 + q) * n];
#pragma unroll
            for (int q = 0; q < kStripe; q++) {
                const int i = i0 + q;
                if (i < n) {
                    a[q] = csub(a[q], cmul(y[i], vc));
                    col[(long long)i * n] = a[q];
                    if (i > k) s = cfma(CT<double2>::mk(v[i].x, -v[i].y), a[q], s);
                }
            }
        }
        const double2 wj = cmul(CT<double2>::mk(tau.x, -tau.y), s);
        column_axpy(col, n, k + 1, n, v, CT<double2>::mk(-wj.x, -wj.y));
    } else {
        column_axpy(Q + sA * blockIdx.y + j, n, 0, n, v + 2 * n, CT<double2>::mk(-v[j].x, v[j].y));
    }
}

// ------------------------------------------------------------------------------------
// Single-shift complex QR (zlahqr semantics: wantt, wantz) on the upper Hessenberg H with
// Schur vectors accumulated into Z (Z := Z G^H).  One CTA per matrix.  status[b]: 0 ok,
// 1 no convergence within 30 n iterations.
// ------------------------------------------------------------------------------------
// G [x; y] (rows) and [x, y] G^H (columns) for G = [c, s; -conj(s), c]
__device__ __forceinline__ void rot_rows(double c, double2 s, double2& x, double2& y) {
    const double2 nx = CT<double2>::mk(c * x.x + (s.x * y.x - s.y * y.y), c * x.y + (s.x * y.y + s.y * y.x));
    const double2 ny = CT<double2>::mk(c * y.x - (s.x * x.x + s.y * x.y), c * y.y - (s.x * x.y - s.y * x.x));
    x = nx;
    y = ny;
}
__device__ __forceinline__ void rot_cols(double c, double2 s, double2& x, double2& y) {
    const double2 nx = CT<double2>::mk(c * x.x + (y.x * s.x + y.y * s.y), c * x.y + (y.y * s.x - y.x * s.y));
    const double2 ny = CT<double2>::mk(c * y.x - (x.x * s.x - x.y * s.y), c * y.y - (x.x * s.y + x.y * s.x));
    x = nx;
    y = ny;
}

// Rotations k0 .. k1-1 of a single-shift sweep over the active block [l, ihi].  Rotation k
// touches rows / columns k, k+1 only, so the chase needs just the window rows k0..k1+1,
// columns k0-1..k1: warp 0 runs it in shared memory (one rotation after another, no block
// barrier) and records the rotations.  Then the whole CTA applies them, in order, to what lies
// outside the window: rows k0..k1 right of column k1, columns k0..k1 above row k0, and the
// Schur vectors Z[:, k0..k1], each thread streaming one column or row with two values live.
// Every element sees the same operations in the same order as rotation-by-rotation.
constexpr int kHqrW = 64;

// Givens generator of the chase, from two reciprocal square roots (c = |f| / d,
// s = conj(g) f / (|f| d), r = f d / |f| with d = sqrt(|f|^2 + |g|^2)), which keeps the rotation
// unitary to a few ulp.  In FP64 this replaces zlartg's two square roots and five divisions:
// the chase is one warp working through each rotation's dependent chain, and GB300 issues FP64
// at about 2 operations per clock per SM, so that chain sets the FP64 sweep's time.

__device__ __forceinline__ void givens_chase(double2 f, double2 g, double& c, double2& s, double2& r) {
    const double gf = cabs2(g), ff = cabs2(f);
    if (gf == 0.0) {
        c = 1.0;
        s = CT<double2>::mk(0.0, 0.0);
        r = f;
        return;
    }
    if (ff == 0.0) {
        const double ig = rsqrt(gf);
        c = 0.0;
        s = CT<double2>::mk(g.x * ig, -g.y * ig);
        r = CT<double2>::mk(gf * ig, 0.0);
        return;
    }
    const double iaf = rsqrt(ff), id = rsqrt(ff + gf);
    c = ff * iaf * id;
    const double2 fs = CT<double2>::mk(f.x * iaf, f.y * iaf);
    const double2 t = cmulc(g, fs);
    s = CT<double2>::mk(t.x * id, t.y * id);
    const double d = (ff + gf) * id;
    r = CT<double2>::mk(fs.x * d, fs.y * d);
}

// The chase of rotations k0 .. k1-1 inside the shared-memory window (loaded from H, a block
// barrier, the chase by warp 0, a block barrier, stored back), the rotations recorded in hc / hs.
template <bool kCg>
__device__ void hqr_chase(double2* __restrict__ H, int n, int l, int ihi, int k0, int k1, double2 shift, double2* hw,
                          double* hc, double2* hs) {
    constexpr int ldw = kHqrW + 2;
    const int r1 = min(k1 + 1, ihi);
    const int c0 = (k0 > l) ? k0 - 1 : k0;
    const int nr = r1 - k0 + 1, nc = k1 - c0 + 1;
    for (int e = threadIdx.x; e < nr * nc; e += blockDim.x) {
        const int i = e / nc, j = e % nc;
        hw[i * ldw + j] = hld<kCg>(H + (long long)(k0 + i) * n + c0 + j);
    }
    __syncthreads();
#define HW(i, j) hw[((i) - k0) * ldw + ((j) - c0)]
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        for (int k = k0; k < k1; k++) {
            // every lane generates the rotation (no broadcast needed); lane 0 records it
            double2 f, g, r, s;
            double c;
            if (k == l) {
                f = csub(HW(l, l), shift);
                g = HW(l + 1, l);
            } else {
                f = HW(k, k - 1);
                g = HW(k + 1, k - 1);
            }
            givens_chase(f, g, c, s, r);
            __syncwarp();
            if (lane == 0) {
                if (k > l) {
                    HW(k, k - 1) = r;
                    HW(k + 1, k - 1) = CT<double2>::mk(0, 0);
                }
                hc[k - k0] = c;
                hs[k - k0] = s;
            }
            for (int j = k + lane; j <= k1; j += 32) rot_rows(c, s, HW(k, j), HW(k + 1, j));
            __syncwarp();
            const int rmax = min(k + 2, ihi);
            for (int i = k0 + lane; i <= rmax; i += 32) rot_cols(c, s, HW(i, k), HW(i, k + 1));
            __syncwarp();
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nr * nc; e += blockDim.x) {
        const int i = e / nc, j = e % nc;
        H[(long long)(k0 + i) * n + c0 + j] = hw[i * ldw + j];
    }
#undef HW
}

// The recorded rotations applied, in order, to what lies outside the window: tasks t0, t0 + dt,
// ... of the stripes (columns right of the window, rows above it, Schur-vector rows).  Each task
// streams one stripe of k1 - k0 + 1 values.  The values are loaded kStripe at a time into
// registers before the rotations run through them: a load-rotate-store chain per element would
// wait a full memory latency per element (the compiler cannot move a load of the stripe above the
// store to the element before it).
template <bool kCg>
__device__ void hqr_apply(double2* __restrict__ H, double2* __restrict__ Z, int n, int k0, int k1, const double* hc,
                          const double2* hs, int t0, int dt) {
    constexpr int kStripe = 4;
    const int nright = n - 1 - k1, nabove = k0;
    for (int t = t0; t < nright + nabove + n; t += dt) {
        const bool right = t < nright;              // column j (rows k0..k1), else a row (columns k0..k1)
        double2* base;
        long long step;
        if (right) {
            base = H + k1 + 1 + t;
            step = n;
        } else {
            base = (t < nright + nabove) ? H + (long long)(t - nright) * n : Z + (long long)(t - nright - nabove) * n;
            step = 1;
        }
        double2 x = hld<kCg>(base + (long long)k0 * step);
        for (int kb = k0; kb < k1; kb += kStripe) {
            const int m = min(kStripe, k1 - kb);
            double2 y[kStripe];
#pragma unroll
            for (int q = 0; q < kStripe; q++)
                if (q < m) y[q] = hld<kCg>(base + (long long)(kb + q + 1) * step);
#pragma unroll
            for (int q = 0; q < kStripe; q++) {
                if (q < m) {
                    if (right)
                        rot_rows(hc[kb + q - k0], hs[kb + q - k0], x, y[q]);
                    else
                        rot_cols(hc[kb + q - k0], hs[kb + q - k0], x, y[q]);
                    base[(long long)(kb + q) * step] = x;
                    x = y[q];
                }
            }
        }
        base[(long long)k1 * step] = x;
    }
}

__device__ void hqr_chunk(double2* __restrict__ H, double2* __restrict__ Z, int n, int l, int ihi, int k0, int k1, double2 shift,
                          double2* hw, double* hc, double2* hs) {
    hqr_chase<false>(H, n, l, ihi, k0, k1, shift, hw, hc, hs);
    hqr_apply<false>(H, Z, n, k0, k1, hc, hs, threadIdx.x, blockDim.x);
    __syncthreads();
}

// Shift of the next sweep over [l, ihi]: Wilkinson's from the trailing 2 x 2 block, and
// exceptional shifts every 10 iterations without a deflation (zlahqr's KEXSH rule).
template <bool kCg>
__device__ double2 hqr_shift(const double2* __restrict__ H, int n, int l, int ihi, int its) {
    const double2 hii = hld<kCg>(H + (long long)ihi * n + ihi);
    if (its % 20 == 0) return CT<double2>::mk(0.75 * r_abs(hld<kCg>(H + (long long)ihi * n + ihi - 1).x) + hii.x, hii.y);
    if (its % 10 == 0) {
        const double2 hll = hld<kCg>(H + (long long)l * n + l);
        return CT<double2>::mk(0.75 * r_abs(hld<kCg>(H + (long long)(l + 1) * n + l).x) + hll.x, hll.y);
    }
    const double2 a = hld<kCg>(H + (long long)(ihi - 1) * n + ihi - 1);
    const double2 b = hld<kCg>(H + (long long)(ihi - 1) * n + ihi);
    const double2 c = hld<kCg>(H + (long long)ihi * n + ihi - 1);
    const double2 d = hii;
    const double2 half = CT<double2>::mk(0.5 * (a.x - d.x), 0.5 * (a.y - d.y));
    const double2 bc = cmul(b, c);
    const double2 disc = cfma(half, half, bc);
    const double2 sq = zsqrt(disc);
    // choose the root that makes the shift closer to d
    double2 e1 = cadd(half, sq), e2 = csub(half, sq);
    const double2 den = cabs2(e1) >= cabs2(e2) ? e1 : e2;
    return (cabs2(den) == 0) ? d : csub(d, cdiv(bc, den));
}

constexpr size_t hqr_smem_bytes() {
    return sizeof(double2) * ((kHqrW + 2) * (kHqrW + 2) + kHqrW) + sizeof(double) * kHqrW;
}

__global__ void __launch_bounds__(1024)
hqr_kernel(double2* __restrict__ H, double2* __restrict__ Z, int n, long long sA, double2* __restrict__ eig, int* __restrict__ status,
           const int* __restrict__ skip) {
    if (skipped(skip, blockIdx.x)) return;
    H += sA * blockIdx.x;
    Z += sA * blockIdx.x;
    eig += (long long)n * blockIdx.x;
    __shared__ double2 s_s;
    __shared__ int s_red[32];
    extern __shared__ __align__(16) unsigned char hqr_smem[];
    double2* hw = reinterpret_cast<double2*>(hqr_smem);                         // (kHqrW + 2)^2 window
    double2* hs = hw + (kHqrW + 2) * (kHqrW + 2);                         // kHqrW rotation sines
    double* hc = reinterpret_cast<double*>(hs + kHqrW);                       // kHqrW rotation cosines
    int ihi = n - 1;
    int its = 0;
    const int itmax = 30 * max(10, n);
    int total = 0;
    while (ihi >= 0) {
        // the largest k in [1, ihi] whose subdiagonal entry may be set to zero (0: none);
        // each thread scans its ks downwards, then a block maximum
        int lk = 0;
        for (int k = ihi - (int)threadIdx.x; k > 0; k -= blockDim.x)
            if (hqr_deflates(H, n, k, ihi)) {
                lk = k;
                break;
            }
        lk = __reduce_max_sync(0xffffffffu, lk);
        if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = lk;
        __syncthreads();
        int l = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) l = max(l, s_red[w]);
        __syncthreads();
        if (l > 0) {
            if (threadIdx.x == 0) H[(long long)l * n + l - 1] = CT<double2>::mk(0, 0);
        }
        if (l >= ihi) {                                   // 1x1 block: eigenvalue converged
            if (threadIdx.x == 0) eig[ihi] = H[(long long)ihi * n + ihi];
            __syncthreads();
            ihi = l - 1;
            its = 0;
            continue;
        }
        if (total > itmax) {
            if (threadIdx.x == 0) status[blockIdx.x] = 1;
            return;
        }
        its++;
        total++;
        // shift; exceptional shifts every 10 iterations without a deflation (zlahqr's KEXSH rule)
        if (threadIdx.x == 0) s_s = hqr_shift<false>(H, n, l, ihi, its);
        __syncthreads();
        const double2 shift = s_s;
        __syncthreads();
        // implicit single-shift QR sweep over the active block [l, ihi], kHqrW rotations at a time
        for (int k0 = l; k0 < ihi; k0 += kHqrW) {
            const int k1 = min(k0 + kHqrW, ihi);
            hqr_chunk(H, Z, n, l, ihi, k0, k1, shift, hw, hc, hs);
        }
    }
}

// ------------------------------------------------------------------------------------
// The same QR with each matrix on a thread-block cluster of K CTAs (K = the cluster size, 2..8):
// rank 0 makes every decision (deflations, shift, end) and chases each window as hqr_kernel does;
// after a cluster barrier every CTA copies the window's rotations from rank 0's shared memory and
// applies them to its share of the stripes (task t to CTA t / blockDim mod K), then a second
// barrier.  The CTAs follow the decisions rank 0 leaves in its shared memory before a barrier,
// so all of them pass the same sequence of barriers and leave together.  H and Z are read through
// L2 only (other CTAs of the cluster write them) and every thread fences its writes before a
// barrier.  Each element sees the same rotations in the same order as in hqr_kernel; the two
// kernels are compiled apart and may fuse multiply-adds differently, so the results agree to
// rounding (measured: they differ in the last bits even where the second CTA has no stripe to
// update).  The deferred updates, 72-80 % of a sweep on one CTA (and nearly all of it in FP64,
// whose rate per SM is low), are spread over K SMs.
// ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(1024)
hqr_cluster_kernel(double2* __restrict__ H, double2* __restrict__ Z, int n, long long sA, double2* __restrict__ eig,
                   int* __restrict__ status, const int* __restrict__ skip) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int K = (int)cluster.num_blocks();
    const int rank = (int)cluster.block_rank();
    const int b = blockIdx.x / K;
    if (skipped(skip, b)) return;                       // the whole cluster, before any barrier
    H += sA * b;
    Z += sA * b;
    eig += (long long)n * b;
    __shared__ double2 s_shift;
    __shared__ int s_red[32];
    __shared__ int s_cmd[3];                            // rank 0: operation (0 sweep, 1 end), l, ihi
    extern __shared__ __align__(16) unsigned char hqr_smem[];
    double2* hw = reinterpret_cast<double2*>(hqr_smem);
    double2* hs = hw + (kHqrW + 2) * (kHqrW + 2);
    double* hc = reinterpret_cast<double*>(hs + kHqrW);
    const int* cmd0 = cluster.map_shared_rank(s_cmd, 0);
    const double2* hs0 = cluster.map_shared_rank(hs, 0);
    const double* hc0 = cluster.map_shared_rank(hc, 0);
    int ihi = n - 1;                                    // rank 0's state
    int its = 0;
    const int itmax = 30 * max(10, n);
    int total = 0;
    while (true) {
        if (rank == 0) {
            // deflations until a sweep is due, the matrix is done or the iteration limit is hit
            int op = 0, l = 0;
            while (true) {
                if (ihi < 0) {
                    op = 1;
                    break;
                }
                int lk = 0;
                for (int k = ihi - (int)threadIdx.x; k > 0; k -= blockDim.x)
                    if (hqr_deflates<double2, true>(H, n, k, ihi)) {
                        lk = k;
                        break;
                    }
                lk = __reduce_max_sync(0xffffffffu, lk);
                if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = lk;
                __syncthreads();
                l = 0;
                for (int w = 0; w < (int)(blockDim.x >> 5); w++) l = max(l, s_red[w]);
                __syncthreads();
                if (l > 0 && threadIdx.x == 0) H[(long long)l * n + l - 1] = CT<double2>::mk(0, 0);
                if (l >= ihi) {                           // 1x1 block: eigenvalue converged
                    if (threadIdx.x == 0) eig[ihi] = hld<true>(H + (long long)ihi * n + ihi);
                    __syncthreads();
                    ihi = l - 1;
                    its = 0;
                    continue;
                }
                if (total > itmax) {
                    if (threadIdx.x == 0) status[b] = 1;
                    op = 1;
                    break;
                }
                its++;
                total++;
                if (threadIdx.x == 0) s_shift = hqr_shift<true>(H, n, l, ihi, its);
                break;
            }
            if (threadIdx.x == 0) {
                s_cmd[0] = op;
                s_cmd[1] = l;
                s_cmd[2] = ihi;
            }
        }
        __threadfence();
        cluster.sync();
        const int op = cmd0[0], l = cmd0[1], hi = cmd0[2];
        if (op != 0) {
            cluster.sync();                              // rank 0's shared memory stays until all have read
            return;
        }
        // implicit single-shift QR sweep over [l, hi], kHqrW rotations at a time (l < hi)
        for (int k0 = l; k0 < hi; k0 += kHqrW) {
            const int k1 = min(k0 + kHqrW, hi);
            if (rank == 0) hqr_chase<true>(H, n, l, hi, k0, k1, s_shift, hw, hc, hs);
            __threadfence();
            cluster.sync();
            if (rank != 0) {
                for (int i = threadIdx.x; i < k1 - k0; i += blockDim.x) {
                    hc[i] = hc0[i];
                    hs[i] = hs0[i];
                }
                __syncthreads();
            }
            hqr_apply<true>(H, Z, n, k0, k1, hc, hs, rank * (int)blockDim.x + (int)threadIdx.x,
                               K * (int)blockDim.x);
            __threadfence();
            cluster.sync();
        }
    }
}

// ------------------------------------------------------------------------------------
// Eigenvectors of the upper triangular Schur factor T (ztrevc semantics, right vectors): vector k
// solves (T - T_kk I) x = 0 with x_k = 1, x_i = 0 for i > k.  One warp per vector.
// Vector k is written as row k of X (contiguous for the warp that builds it; the product with the
// Schur vectors reads X transposed).
// FP64: a denominator T_ii - T_kk below smin is replaced by smin, as ztrevc does.  FP32 (the
// first stage of the mixed solver): where both the denominator and the coupling sum
// sum_j T_ij x_j are within 16 ulp of max |T_jj|, the pair counts as one degenerate eigenvalue and
// x_i = 0, so each keeps its own Schur vector.  (Dividing rounding noise by rounding noise gives
// numerically parallel vectors for the exactly degenerate eigenvalues of homogeneous layers; the
// refinement resolves such clusters in FP64.)  A close pair with a real coupling is divided as in
// FP64: zeroing it would leave the coupling as residual, which the refinement of dense spectra
// (n = 3200 layers) could not remove.
// ------------------------------------------------------------------------------------
template <typename C>
__device__ __forceinline__ C warp_sum(C s) {
    for (int o = 16; o > 0; o >>= 1) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
        s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
    }
    return s;
}

template <typename C>
__global__ void __launch_bounds__(256)
trevc_kernel(const C* __restrict__ T, C* __restrict__ X, int n, long long sA, const int* __restrict__ skip) {
    using R = typename CT<C>::R;
    constexpr bool kDegenerateSkip = sizeof(R) == sizeof(float);
    if (skipped(skip, blockIdx.y)) return;
    T += sA * blockIdx.y;
    X += sA * blockIdx.y;
    // the longest vectors first: the last warps of the grid are short
    const int k = n - 1 - (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (k < 0) return;
    C* x = X + (long long)k * n;
    const R ulp = CT<C>::ulp;
    const C lam = T[(long long)k * n + k];
    const R smin = r_max(ulp * cabs1(lam), CT<C>::safmin * ((R)n / ulp));
    R deg = 0;
    if (kDegenerateSkip) {
        for (int i = lane; i < n; i += 32) deg = r_max(deg, cabs1(T[(long long)i * n + i]));
        for (int o = 16; o > 0; o >>= 1) deg = r_max(deg, __shfl_xor_sync(0xffffffffu, deg, o));
        deg *= R(16) * ulp;
    }
    // x_k = 1, x_{k+1..} = 0
    for (int i = lane; i < n; i += 32) x[i] = CT<C>::mk(i == k ? 1 : 0, 0);
    __syncwarp();
    for (int i = k - 1; i >= 0; i--) {
        // x_i = -(sum_{j=i+1..k} T_ij x_j) / (T_ii - lam)
        const C* row = T + (long long)i * n;
        C s = CT<C>::mk(0, 0);
#pragma unroll 4
        for (int j = i + 1 + lane; j <= k; j += 32) s = cfma(row[j], x[j], s);
        s = warp_sum(s);
        if (lane == 0) {
            C d = csub(row[i], lam);
            if (kDegenerateSkip && cabs1(d) <= deg && cabs1(s) <= deg) {
                x[i] = CT<C>::mk(0, 0);
            } else {
                if (cabs1(d) < smin) d = CT<C>::mk(smin, 0);
                x[i] = cdiv(CT<C>::mk(-s.x, -s.y), d);
            }
        }
        __syncwarp();
    }
}

// copy of the batch entries that are not skipped
__global__ void __launch_bounds__(256)
copy_kernel(const double2* __restrict__ src, double2* __restrict__ dst, long long count, const int* __restrict__ skip) {
    if (skipped(skip, blockIdx.y)) return;
    src += count * blockIdx.y;
    dst += count * blockIdx.y;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count; i += (long long)gridDim.x * blockDim.x)
        dst[i] = src[i];
}

// Inverse Z of a unit upper triangular matrix given by its columns (column j = row j of X): row r of
// Z X = I is z_r = 1, z_j = -sum_{i=r..j-1} z_i X_ij.  One warp per row.
template <typename C>
__global__ void __launch_bounds__(256)
trtri_kernel(const C* __restrict__ X, C* __restrict__ Z, int n, long long sA) {
    X += sA * blockIdx.y;
    Z += sA * blockIdx.y;
    const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (r >= n) return;
    C* z = Z + (long long)r * n;
    for (int j = lane; j <= r; j += 32) z[j] = CT<C>::mk(j == r ? 1 : 0, 0);
    __syncwarp();
    for (int j = r + 1; j < n; j++) {
        const C* col = X + (long long)j * n;
        C s = CT<C>::mk(0, 0);
#pragma unroll 4
        for (int i = r + lane; i < j; i += 32) s = cfma(z[i], col[i], s);
        s = warp_sum(s);
        if (lane == 0) z[j] = CT<C>::mk(-s.x, -s.y);
        __syncwarp();
    }
}

}  // namespace z

// ------------------------------------------------------------------------------------
// Host wrappers
// ------------------------------------------------------------------------------------
template <typename C>
scw_status gemm(cudaStream_t st, int M, int N, int K, C alpha, const C* A, int lda, long long sA, const C* B, int ldb,
                long long sB, C beta, C* Cm, int ldc, long long sC, int batch, const int* skip, int opB) {
    if (M <= 0 || N <= 0 || batch <= 0) return SCW_OK;
    dim3 grid((N + z::kGT - 1) / z::kGT, (M + z::kGT - 1) / z::kGT, batch);
    z::gemm_kernel<C><<<grid, 256, 0, st>>>(M, N, K, alpha, A, lda, sA, B, ldb, sB, opB == kOpT, beta, Cm, ldc, sC, skip);
    SCW_CUDA_TRY(cudaGetLastError());
    return SCW_OK;
}

// Columns per CTA of the triangular kernels: 32 reuse the block of L or U for more columns, but their FP64
// work (16 000 operations per column of 32 rows) then takes 20 us on one SM; 8 where 32 would leave SMs idle.
static bool few_columns(int cols, int batch) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return false;
    return (long long)((cols + 31) / 32) * batch < sms;
}

static cudaError_t trsm_block(cudaStream_t st, const double2* LU, int lda, long long sA, int k0, int nb, double2* B, int ldb, long long sB,
                       int nrhs, int upper, int batch, const int* skip) {
    if (few_columns(nrhs, batch))
        return launch_chained(true, st, dim3((nrhs + 7) / 8, batch), 256, 0, z::trsm_block_kernel<8>, LU, lda, sA, k0, nb, B, ldb,
                              sB, nrhs, upper, skip);
    return launch_chained(true, st, dim3((nrhs + 31) / 32, batch), 256, 0, z::trsm_block_kernel<32>, LU, lda, sA, k0, nb, B, ldb,
                          sB, nrhs, upper, skip);
}

scw_status zgetrf(cudaStream_t st, double2* A, int n, int ncols, int lda, long long sA, int* piv, long long sP, int* info,
                  int batch, const GemmWs& ws, const int* skip) {
    if (n <= 0 || batch <= 0) return SCW_OK;
    SCW_CUDA_TRY(cudaMemsetAsync(info, 0, sizeof(int) * batch, st));
    // the panel in the cluster's shared memory where 32 columns of it fit (up to 3264 rows), else in A, by way of L2.  (Narrower panels
    // in shared memory end at 53 872 rows and are no faster before: order 4096 78 ms with 16 columns, 80 here; 6400 375 with 8, 230 here.)
    constexpr size_t kLimit = 220 * 1024, kSlots = sizeof(z::LuSlot) * (2 * z::kLuCtas + 2);
    auto smem_of = [](int rows, int nb) { return kSlots + sizeof(double2) * (size_t)rows * (nb + 1); };
    SCW_CUDA_TRY(cudaFuncSetAttribute(z::lu_panel_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLimit));
    const double2 one = {1, 0}, minus = {-1, 0};
    constexpr int width = z::kNB;
    for (int k0 = 0; k0 < n; k0 += width) {
        const int nb = std::min(width, n - k0), rows = (n - k0 + z::kLuCtas - 1) / z::kLuCtas;
        if (smem_of(rows, nb) <= kLimit)
            z::lu_panel_kernel<false><<<z::kLuCtas * batch, z::kLuThreads, smem_of(rows, nb), st>>>(A, n, lda, sA, k0, nb, rows, piv,
                                                                                                 sP, info, skip);
        else
            z::lu_panel_kernel<true><<<z::kLuCtas * batch, z::kLuThreads, kSlots, st>>>(A, n, lda, sA, k0, nb, rows, piv, sP, info, skip);
        SCW_CUDA_TRY(cudaGetLastError());
        if (ncols > nb) {
            if (few_columns(ncols, batch))
                SCW_CUDA_TRY(launch_chained(true, st, dim3((ncols + 7) / 8, batch), 256, 0, z::lu_apply_kernel<8>, A, ncols, lda, sA,
                                            k0, nb, piv, sP, skip));
            else
                SCW_CUDA_TRY(launch_chained(true, st, dim3((ncols + 31) / 32, batch), 256, 0, z::lu_apply_kernel<32>, A, ncols, lda,
                                            sA, k0, nb, piv, sP, skip));
        }
        const int rem = n - k0 - nb;
        if (rem > 0) {
            // A22 -= L21 U12
            scw_status s = zgemm(st, rem, ncols - k0 - nb, nb, minus, A + (long long)(k0 + nb) * lda + k0, lda, sA,
                                 A + (long long)k0 * lda + k0 + nb, lda, sA, one,
                                 A + (long long)(k0 + nb) * lda + k0 + nb, lda, sA, batch, ws, skip);
            if (s != SCW_OK) return s;
        }
    }
    return SCW_OK;
}

scw_status ztrsm_upper(cudaStream_t st, const double2* LU, int n, int lda, long long sA, double2* B, int nrhs, int ldb,
                       long long sB, int batch, const GemmWs& ws, const int* skip) {
    // blocked: per diagonal block a small triangular solve, the rest of the rows updated by GEMM
    if (n <= 0 || nrhs <= 0 || batch <= 0) return SCW_OK;
    constexpr int kTB = z::kNB;
    const double2 one = {1, 0}, minus = {-1, 0};
    for (int k0 = ((n - 1) / kTB) * kTB; k0 >= 0; k0 -= kTB) {
        const int nb = std::min(kTB, n - k0);
        SCW_CUDA_TRY(trsm_block(st, LU, lda, sA, k0, nb, B, ldb, sB, nrhs, 1, batch, skip));
        if (k0 > 0) {
            scw_status s = zgemm(st, k0, nrhs, nb, minus, LU + k0, lda, sA, B + (long long)k0 * ldb, ldb, sB, one, B, ldb,
                                 sB, batch, ws, skip);
            if (s != SCW_OK) return s;
        }
    }
    return SCW_OK;
}

scw_status zgetrs(cudaStream_t st, const double2* LU, int n, long long sA, const int* piv, long long sP, double2* B,
                  int nrhs, long long sB, int batch, const GemmWs& ws, const int* skip) {
    if (n <= 0 || nrhs <= 0 || batch <= 0) return SCW_OK;
    constexpr int kTB = z::kNB;
    const double2 one = {1, 0}, minus = {-1, 0};
    z::laswp_kernel<<<dim3((nrhs + 255) / 256, batch), 256, 0, st>>>(piv, sP, B, nrhs, sB, n, nrhs, skip);
    SCW_CUDA_TRY(cudaGetLastError());
    for (int k0 = 0; k0 < n; k0 += kTB) {
        const int nb = std::min(kTB, n - k0);
        SCW_CUDA_TRY(trsm_block(st, LU, n, sA, k0, nb, B, nrhs, sB, nrhs, 0, batch, skip));
        const int rem = n - k0 - nb;
        if (rem > 0) {
            scw_status s = zgemm(st, rem, nrhs, nb, minus, LU + (long long)(k0 + nb) * n + k0, n, sA,
                                 B + (long long)k0 * nrhs, nrhs, sB, one, B + (long long)(k0 + nb) * nrhs, nrhs, sB,
                                 batch, ws, skip);
            if (s != SCW_OK) return s;
        }
    }
    return ztrsm_upper(st, LU, n, n, sA, B, nrhs, nrhs, sB, batch, ws, skip);
}

scw_status zgehrd(cudaStream_t st, double2* A, double2* Q, int n, int batch, double2* work) {
    if (n <= 0 || batch <= 0) return SCW_OK;
    z::hessenberg_kernel<<<batch, 1024, 0, st>>>(A, Q, n, (long long)n * n, work, nullptr);
    SCW_CUDA_TRY(cudaGetLastError());
    return SCW_OK;
}

// Hessenberg reduction with Schur-vector accumulation, spread over the GPU (3 launches per column)
static scw_status gehrd_wide(cudaStream_t st, double2* A, double2* Q, int n, int batch, double2* hw, const int* skip) {
    const long long nn = (long long)n * n;
    const unsigned gi = (unsigned)std::min<long long>((nn + 255) / 256, 1024);
    z::hw_init_kernel<<<dim3(gi, batch), 256, 0, st>>>(Q, n, nn, skip);
    SCW_CUDA_TRY(cudaGetLastError());
    for (int k = 0; k + 2 < n; k++) {
        z::hw_vec_kernel<<<batch, 256, 0, st>>>(A, n, nn, hw, k, skip);
        z::hw_prod_kernel<<<dim3((2 * n + z::kHwRows - 1) / z::kHwRows, batch), z::kHwRows * 32, 0, st>>>(
            A, Q, n, nn, hw, k, skip);
        const int nblk = (n - k - 1 + z::kHwCols - 1) / z::kHwCols;
        z::hw_update_kernel<<<dim3(2 * nblk, batch), z::kHwCols, 0, st>>>(A, Q, n, nn, hw, k, nblk, skip);
    }
    SCW_CUDA_TRY(cudaGetLastError());
    return SCW_OK;
}

// CTAs per matrix of the QR sweeps: 0 = chosen per call, 1 = one CTA (hqr_kernel), 2..8 = a
// cluster of that size (scw_set_qr_cluster)
static std::atomic<int> g_qr_cluster{0};

// The QR sweeps of `batch` matrices, `active` of them not skipped.  Single solves (wide) put each
// matrix on a cluster of K CTAs: the largest K <= 8 for which all active matrices' clusters are
// resident at once (cudaOccupancyMaxActiveClusters; the updates are bound by the FP64 rate of each
// SM and gain from more SMs down to few tasks per CTA).  Otherwise one CTA per matrix.
static scw_status hqr_launch(cudaStream_t st, double2* A, double2* Q, int n, long long nn, double2* W, int* status, const int* skip,
                             int batch, int active, bool wide) {
    const size_t smem = z::hqr_smem_bytes();
    const int force = g_qr_cluster.load();
    if (wide && force != 1 && active > 0) {
        int dev = 0, sms = 0;
        SCW_CUDA_TRY(cudaGetDevice(&dev));
        SCW_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        SCW_CUDA_TRY(cudaFuncSetAttribute(z::hqr_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)smem));
        int kmax = force > 1 ? std::min(force, 8) : std::min(8, sms / active);
        for (int k = kmax; k >= 2; k--) {
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = (unsigned)k;
            at[0].val.clusterDim.y = 1;
            at[0].val.clusterDim.z = 1;
            cfg.gridDim = dim3((unsigned)(k * batch));
            cfg.blockDim = dim3(1024);
            cfg.dynamicSmemBytes = smem;
            cfg.stream = st;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            int resident = 0;
            if (cudaOccupancyMaxActiveClusters(&resident, z::hqr_cluster_kernel, &cfg) != cudaSuccess) {
                cudaGetLastError();
                continue;
            }
            if (resident >= (force > 1 ? 1 : active)) {
                SCW_CUDA_TRY(cudaLaunchKernelEx(&cfg, z::hqr_cluster_kernel, A, Q, n, nn, W, status, skip));
                return SCW_OK;
            }
        }
    }
    SCW_CUDA_TRY(cudaFuncSetAttribute(z::hqr_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    z::hqr_kernel<<<batch, 1024, smem, st>>>(A, Q, n, nn, W, status, skip);
    SCW_CUDA_TRY(cudaGetLastError());
    return SCW_OK;
}

template <typename C>
scw_status trevc(cudaStream_t st, const C* T, C* X, int n, int batch, const int* skip) {
    z::trevc_kernel<C><<<dim3((n * 32 + 255) / 256, batch), 256, 0, st>>>(T, X, n, (long long)n * n, skip);
    SCW_CUDA_TRY(cudaGetLastError());
    return SCW_OK;
}

scw_status trtri_rows(cudaStream_t st, const float2* X, float2* Z, int n, int batch) {
    z::trtri_kernel<float2><<<dim3((n * 32 + 255) / 256, batch), 256, 0, st>>>(X, Z, n, (long long)n * n);
    SCW_CUDA_TRY(cudaGetLastError());
    return SCW_OK;
}

scw_status zgeev(cudaStream_t st, double2* A, double2* W, double2* V, int n, int batch, double2* work, int* status,
                 const int* skip, bool wide, const GemmWs& ws) {
    if (n <= 0 || batch <= 0) return SCW_OK;
    const long long nn = (long long)n * n;
    double2* Q = work;                       // batch * n * n: Schur vectors
    double2* hw = work + nn * batch;         // batch * 3n
    SCW_CUDA_TRY(cudaMemsetAsync(status, 0, sizeof(int) * batch, st));
    // single solves outside a stream capture count the matrices the skip mask leaves (and do
    // nothing when it leaves none)
    int active = batch;
    if (wide && skip) {
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        SCW_CUDA_TRY(cudaStreamIsCapturing(st, &cap));
        if (cap == cudaStreamCaptureStatusNone) {
            std::vector<int> sk(batch);
            SCW_CUDA_TRY(cudaMemcpyAsync(sk.data(), skip, sizeof(int) * batch, cudaMemcpyDeviceToHost, st));
            SCW_CUDA_TRY(cudaStreamSynchronize(st));
            active = (int)std::count(sk.begin(), sk.end(), 0);
            if (active == 0) return SCW_OK;
        }
    }
    if (wide && n >= kWideMinN) {
        scw_status s = gehrd_wide(st, A, Q, n, batch, hw, skip);
        if (s != SCW_OK) return s;
    } else {
        z::hessenberg_kernel<<<batch, 1024, 0, st>>>(A, Q, n, nn, hw, skip);
        SCW_CUDA_TRY(cudaGetLastError());
    }
    scw_status s = hqr_launch(st, A, Q, n, nn, W, status, skip, batch, active, wide);
    // triangular eigenvectors as the rows of V, then Q V^T over A, copied to V
    if (s == SCW_OK) s = trevc<double2>(st, A, V, n, batch, skip);
    GemmWs wp = ws;
    wp.parts = true;
    if (s == SCW_OK)
        s = zgemm(st, n, n, n, make_double2(1, 0), Q, n, nn, V, n, nn, make_double2(0, 0), A, n, nn, batch, wp, skip, 0.0, kOpT);
    if (s != SCW_OK) return s;
    z::copy_kernel<<<dim3((unsigned)std::min<long long>((nn + 255) / 256, 4096), batch), 256, 0, st>>>(A, V, nn, skip);
    SCW_CUDA_TRY(cudaGetLastError());
    return SCW_OK;
}

scw_status schur32(cudaStream_t st, float2* A, float2* Q, float2* W, int n, int batch, float2* work, int* status, int share) {
    scw_status s = hess32(st, A, Q, n, batch, work, share);
    if (s == SCW_OK) s = hqr32(st, A, Q, n, W, status, batch, g_qr_cluster.load(), share);
    return s;
}

// The product of Schur vectors and triangular eigenvectors on the CUDA cores: digit products of 30 bits would lose the
// vectors' small entries (n = 300: 13.0 ms either way).
scw_status cgeev(cudaStream_t st, float2* A, float2* W, float2* V, int n, int batch, float2* work, int* status, int share) {
    const long long nn = (long long)n * n;
    float2* Q = work;                        // batch * n * n: Schur vectors
    scw_status s = schur32(st, A, Q, W, n, batch, work + nn * batch, status, share);
    if (s == SCW_OK) s = trevc32(st, A, V, n, batch);
    if (s == SCW_OK) s = cgemm(st, n, n, n, 1.f, Q, n, nn, kOpN, V, n, nn, kOpT, false, A, n, nn, batch);
    if (s != SCW_OK) return s;
    SCW_CUDA_TRY(cudaMemcpyAsync(V, A, sizeof(float2) * nn * batch, cudaMemcpyDeviceToDevice, st));
    return SCW_OK;
}

template scw_status gemm<double2>(cudaStream_t, int, int, int, double2, const double2*, int, long long, const double2*, int,
                                  long long, double2, double2*, int, long long, int, const int*, int);
template scw_status trevc<float2>(cudaStream_t, const float2*, float2*, int, int, const int*);

}  // namespace scw

// ------------------------------------------------------------------------------------
// C ABI: GPU replacements of the reference's LAPACK wrappers (third_Lapack.h:38-87), on
// device buffers, batched.
// ------------------------------------------------------------------------------------
using scw::fail;

extern "C" {

scw_status scw_zgemm(scw_ctx ctx, int M, int N, int K, const double* alpha, const void* A, const void* B,
                     const double* beta, void* C, int batch) {
    if (!ctx || !A || !B || !C || !alpha || !beta || M < 0 || N < 0 || K < 0 || batch < 1)
        return fail(SCW_ERR_ARG, "scw_zgemm: bad arguments");
    SCW_ON_DEVICE(ctx->device);
    // the workspace and the launches that use it go together: calls of several threads on one context
    // must not interleave
    std::lock_guard<std::mutex> lock(ctx->dense_mu);
    ctx->launches += 4;
    scw::GemmWs ws;
    scw_status st = scw::ctx_gemm_ws(ctx, scw::zgemm_ws_bytes(M, N, K, 1), scw::zgemm_ws_bytes(M, N, K, batch), ws);
    if (st == SCW_ERR_NOMEM) ws = scw::GemmWs{};          // no room for the digits: on the FP64 pipes
    else if (st != SCW_OK) return st;
    ws.parts = true;
    return scw::zgemm(ctx->stream, M, N, K, make_double2(alpha[0], alpha[1]), (const double2*)A, K, (long long)M * K,
                      (const double2*)B, N, (long long)K * N, make_double2(beta[0], beta[1]), (double2*)C, N,
                      (long long)M * N, batch, ws);
}

scw_status scw_zgesv(scw_ctx ctx, int n, int nrhs, void* A, void* B, int batch, int* info_host) {
    if (!ctx || !A || !B || n < 1 || nrhs < 1 || batch < 1) return fail(SCW_ERR_ARG, "scw_zgesv: bad arguments");
    SCW_ON_DEVICE(ctx->device);
    int* dpiv = nullptr;
    int* dinfo = nullptr;
    if (cudaMalloc(&dpiv, sizeof(int) * (size_t)n * batch) != cudaSuccess ||
        cudaMalloc(&dinfo, sizeof(int) * (size_t)batch) != cudaSuccess) {
        cudaFree(dpiv);
        return fail(SCW_ERR_NOMEM, "scw_zgesv: pivots");
    }
    const long long nn = (long long)n * n;
    scw::DevBuf wbuf;
    scw::GemmWs ws;
    scw_status st = scw::reserve_gemm_ws(
        ctx, wbuf, std::max(scw::zgemm_ws_bytes(n, n, 32, 1), scw::zgemm_ws_bytes(n, nrhs, 32, 1)), batch, ws);
    if (st == SCW_ERR_NOMEM) st = SCW_OK;    // no room for the digits: on the FP64 pipes
    ws.parts = true;
    if (st == SCW_OK) st = scw::zgetrf(ctx->stream, (double2*)A, n, n, n, nn, dpiv, n, dinfo, batch, ws, nullptr);
    if (st == SCW_OK)
        st = scw::zgetrs(ctx->stream, (const double2*)A, n, nn, dpiv, n, (double2*)B, nrhs, (long long)n * nrhs, batch,
                         ws, nullptr);
    ctx->launches += 3;
    std::vector<int> info(batch, 0);
    if (st == SCW_OK) {
        cudaError_t e = cudaMemcpyAsync(info.data(), dinfo, sizeof(int) * batch, cudaMemcpyDeviceToHost, ctx->stream);
        if (e != cudaSuccess) st = fail(SCW_ERR_CUDA, cudaGetErrorString(e));
        else st = scw_ctx_synchronize(ctx);
    }
    cudaFree(dpiv);
    cudaFree(dinfo);
    if (st != SCW_OK) return st;
    int bad = 0;
    for (int b = 0; b < batch; b++) {
        if (info_host) info_host[b] = info[b];
        if (info[b]) bad = 1;
    }
    return bad ? fail(SCW_ERR_NUMERIC, "scw_zgesv: singular matrix") : SCW_OK;
}

scw_status scw_zgeev(scw_ctx ctx, int n, void* A, void* W, void* V, int batch, int* status_host) {
    if (!ctx || !A || !W || !V || n < 1 || batch < 1) return fail(SCW_ERR_ARG, "scw_zgeev: bad arguments");
    SCW_ON_DEVICE(ctx->device);
    double2* work = nullptr;
    int* dst = nullptr;
    const size_t wbytes = sizeof(double2) * ((size_t)n * n + 3 * (size_t)n) * batch;
    if (cudaMalloc(&work, wbytes) != cudaSuccess || cudaMalloc(&dst, sizeof(int) * batch) != cudaSuccess) {
        cudaFree(work);
        return fail(SCW_ERR_NOMEM, "scw_zgeev: workspace");
    }
    scw::DevBuf wbuf;
    scw::GemmWs ws;
    scw_status st = scw::reserve_gemm_ws(ctx, wbuf, scw::zgemm_ws_bytes(n, n, n, 1), batch, ws);
    if (st == SCW_ERR_NOMEM) st = SCW_OK;    // no room for the digits: on the FP64 pipes
    if (st == SCW_OK)
        st = scw::zgeev(ctx->stream, (double2*)A, (double2*)W, (double2*)V, n, batch, work, dst, nullptr, true, ws);
    ctx->launches += 4;
    std::vector<int> status(batch, 0);
    if (st == SCW_OK) {
        cudaError_t e = cudaMemcpyAsync(status.data(), dst, sizeof(int) * batch, cudaMemcpyDeviceToHost, ctx->stream);
        if (e != cudaSuccess) st = fail(SCW_ERR_CUDA, cudaGetErrorString(e));
        else st = scw_ctx_synchronize(ctx);
    }
    cudaFree(work);
    cudaFree(dst);
    if (st != SCW_OK) return st;
    int bad = 0;
    for (int b = 0; b < batch; b++) {
        if (status_host) status_host[b] = status[b];
        if (status[b]) bad = 1;
    }
    return bad ? fail(SCW_ERR_NUMERIC, "scw_zgeev: QR iteration did not converge") : SCW_OK;
}

scw_status scw_cgeev(scw_ctx ctx, int n, void* A, void* W, void* V, int batch, int* status_host) {
    if (!ctx || !A || !W || !V || n < 1 || batch < 1) return fail(SCW_ERR_ARG, "scw_cgeev: bad arguments");
    SCW_ON_DEVICE(ctx->device);
    float2* work = nullptr;
    int* dst = nullptr;
    const size_t wbytes = sizeof(float2) * ((size_t)n * n + scw::hess32_ws_elems(n)) * batch;
    if (cudaMalloc(&work, wbytes) != cudaSuccess || cudaMalloc(&dst, sizeof(int) * batch) != cudaSuccess) {
        cudaGetLastError();
        cudaFree(work);
        return fail(SCW_ERR_NOMEM, "scw_cgeev: workspace");
    }
    scw_status st = scw::cgeev(ctx->stream, (float2*)A, (float2*)W, (float2*)V, n, batch, work, dst, 1);
    ctx->launches += 5;
    std::vector<int> status(batch, 0);
    if (st == SCW_OK) {
        cudaError_t e = cudaMemcpyAsync(status.data(), dst, sizeof(int) * batch, cudaMemcpyDeviceToHost, ctx->stream);
        if (e != cudaSuccess) st = fail(SCW_ERR_CUDA, cudaGetErrorString(e));
        else st = scw_ctx_synchronize(ctx);
    }
    cudaFree(work);
    cudaFree(dst);
    if (st != SCW_OK) return st;
    int bad = 0;
    for (int b = 0; b < batch; b++) {
        if (status_host) status_host[b] = status[b];
        if (status[b]) bad = 1;
    }
    return bad ? fail(SCW_ERR_NUMERIC, "scw_cgeev: QR iteration did not converge") : SCW_OK;
}

scw_status scw_set_qr_cluster(int ctas) {
    if (ctas < 0 || ctas > 8) return fail(SCW_ERR_ARG, "scw_set_qr_cluster: 0 (per call), 1 or 2..8 CTAs");
    scw::g_qr_cluster.store(ctas);
    return SCW_OK;
}

}  // extern "C"
