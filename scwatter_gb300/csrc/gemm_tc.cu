// FP64 complex GEMM on the tensor cores (tcgen05, sm_103a): C = alpha A B + beta C, batched.
//
// GB300 issues about 1.7 FP64 FMA per SM and clock, against 4096 bf16 multiply-adds on the tensor
// core, so an FP64 product is far cheaper as a sum of exact integer products (the error-free
// splitting of Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59 (2012)):
//   * the inner index is rescaled by powers of two, A'(i,k) = A(i,k) 2^f_k and B'(k,j) = B(k,j)
//     2^-f_k with 2^f_k above row k of B, so that operands graded along it (the cascade's E^-1 rows) lose
//     nothing against a plain sum; then row i of A' gets the exponent e_i, column j of B' g_j;
//   * every value becomes a 62-bit integer in units of 2^(e_i - 62) (2^(g_j - 62)), cut into kS = 8
//     balanced base-256 digits, each in [-128, 128] and therefore exact in bf16;
//   * digit products of equal weight are summed on the tensor core in FP32.  A sum over K = 128
//     of the d + 1 <= 8 products of diagonal d, for both products of a complex part, is an integer
//     below 2^24 for d <= 3 (exact); the later diagonals weigh 2^-32 and less and could round only if
//     every digit were extreme at once.  After 128 terms the diagonals are drained into 64-bit
//     integers, and the final sum is rounded to FP64 once.
// Diagonals d >= 8 are dropped: at most 2^-57 of the largest product per term.  Measured against
// extended precision at n = 18 .. 1200 (random, constant, log-normal, diagonally dominant matrices,
// eigenvectors): error against the largest |a'| |b'| of the row and column 2e-17 .. 6.8e-16, where
// a sequential FP64 sum has 9e-17 .. 1.7e-15.  An entry more than 2^9 below its row's largest keeps fewer bits than
// FP64: oz_parts_kernel is for callers to whom that matters.  With 7 digits (55 bits) the diagonally dominant and
// eigenvector products came out 20 times less exact than an FP64 sum, so 8 it is (36 digit products
// instead of 28).
//
// Work per 128 x 32 tile and 16 inner indices: digit i of A (real or imaginary part, 128 x 16)
// multiplies digits 0 .. 7 - i of B side by side (N = 32 (8 - i) columns) and lands at column 32 i
// of the accumulator, so that digit i of A and j of B meet in diagonal i + j.  32 MMAs of N = 32 ..
// 256 use all 512 TMEM columns (real and imaginary diagonals).
//
// Measured (38.6 at n = 3200 and 26 TFLOP/s for 20 matrices of n = 648, counted as FP64 operations;
// the FP64 pipes give 1.05-1.25): 1.66 ms instead of 38 ms for the latter, of which 0.3 ms prepare
// the operands.  Measured parts of the latter: without copies 1.64 ms, without drains 1.42; an MMA takes
// N / 2 clocks but at least 57 (N = 32 .. 96), so a stage's 32 MMAs take 2660 clocks where the tensor core's rate alone
// would allow 2300; the drains add 400.  The drain runs on 16 warps with the next TMEM load on its way: against 8 warps
// and loads waited for one by one 67 instead of 79 us for 10 matrices of n = 216, 145 instead of 164 for one of
// n = 648 (where few tiles leave nothing else to hide it).  Neither a ring of single digits nor CTA pairs with
// multicast copies of A gained anything (1.87 and 1.76 ms): the copies are not what bounds it.
//
// The same kernel with 4 digits (30 bits) and 64 columns per tile serves the corrections of the
// eigen-solver and of the inverses, which need FP32 accuracy: 10 digit products instead of 36.
//
// Two launches prepare the operands (oz_inner_kernel: f_k; oz_split_kernel: e_i, g_j and the digits in
// the order the MMA reads them, so that a pipeline stage is two contiguous bulk copies), one runs
// the product: persistent CTAs, one thread copying, one issuing MMAs, 16 warps draining.
// Non-finite values: a row of A or a column of B with one gives NaN in its whole row / column.
#include <algorithm>
#include <cstdint>

#include "scw_complex.cuh"
#include "scw_dense.h"
#include "scw_launch.h"
#include "scw_tc.cuh"

namespace scw {
namespace oz {

constexpr int kTM = 128, kTK = 16;           // tile rows, inner indices per stage
constexpr int kDrainWarps = 16;
constexpr int kLd = 8;                       // columns per TMEM load
constexpr int kStageRow = 80;                // bytes of an output staging row: 64 and padding
template <int S>                             // S base-256 digits per value
struct Cfg {
    static constexpr int kBits = 8 * S - 2;      // integer bits before the cut
    static constexpr int kTN = 256 / S;          // tile columns: S diagonals x 2 parts fill the TMEM
    static constexpr int kABlk = 2 * S * kTM * kTK * 2;   // bytes of A per stage: re, im x digits x 128 x 16 bf16
    static constexpr int kBBlk = 2 * S * kTN * kTK * 2;
    static constexpr int kStages = S == 8 ? 2 : 3;
    static constexpr int kStageOff = kStages * (kABlk + kBBlk);      // output staging after the operands
    static constexpr int kBarOff = kStageOff + kDrainWarps * 32 * kStageRow;
    static constexpr size_t kSmem = (size_t)kBarOff + (2 * kStages + 4) * sizeof(uint64_t);
};
constexpr int kChunk = 8;                    // stages per drain (K = 128)
constexpr int kThreads = (kDrainWarps + 2) * 32;
constexpr int kSpecial = 1 << 20;            // exponent of a row or column with a non-finite value
constexpr int kNone = -100000;               // exponent of a zero row or column

// e with |v| < 2^e for the larger of the two parts; kNone for zero, kSpecial if not finite
__device__ __forceinline__ int cexpo(double2 v) {
    const unsigned a = (unsigned)__double2hiint(v.x) & 0x7fffffffu, b = (unsigned)__double2hiint(v.y) & 0x7fffffffu;
    const unsigned m = max(a, b) >> 20;
    if (m == 0x7ff) return kSpecial;
    if (m == 0 && v.x == 0.0 && v.y == 0.0) return kNone;
    return (int)max(m, 1u) - 1022;
}
__device__ __forceinline__ int cexpo(float2 v) {
    const unsigned m = max(__float_as_uint(v.x) & 0x7fffffffu, __float_as_uint(v.y) & 0x7fffffffu);
    if (m >= 0x7f800000u) return kSpecial;
    if (m == 0u) return kNone;
    return (int)max(m >> 23, 1u) - 126;
}

// round(v 2^s) for |v 2^s| < 2^62 (ties away from zero); v = +-m 2^(ex - 1075)
__device__ __forceinline__ long long fixed_point(bool neg, int ex, long long m, int s) {
    const int sh = ex - 1075 + s;
    if (sh >= 0) m <<= min(sh, 10);
    else m = sh < -55 ? 0 : (m + (1ll << (-sh - 1))) >> -sh;
    return neg ? -m : m;
}
__device__ __forceinline__ long long fixed_point(double v, int s) {
    const long long bits = __double_as_longlong(v);
    const int ex = (int)((bits >> 52) & 0x7ff);
    return fixed_point(bits < 0, max(ex, 1), (bits & 0xfffffffffffffll) | (ex ? 1ll << 52 : 0ll), s);
}
__device__ __forceinline__ long long fixed_point(float v, int s) {
    const unsigned bits = __float_as_uint(v);
    const int ex = (int)((bits >> 23) & 0xff);
    return fixed_point((int)bits < 0, max(ex, 1) - 127 + 1023, (long long)((bits & 0x7fffffu) | (ex ? 1u << 23 : 0u)) << 29, s);
}

// f[b][k] with |B(k, :)| < 2^f: a warp per inner index k; element (k, j) of B at k ks + j js
template <typename T>
__global__ void __launch_bounds__(256)
oz_inner_kernel(const T* __restrict__ B, long long ks, long long js, long long sB, int K, int N, int* __restrict__ f,
                const int* __restrict__ skip) {
    chain_wait();
    chain_trigger();
    if (z::skipped(skip, blockIdx.y)) return;
    B += sB * blockIdx.y;
    f += (long long)blockIdx.y * K;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (js == 1) {
        const int k = blockIdx.x * 8 + warp;
        if (k >= K) return;
        const T* row = B + k * ks;
        int e = kNone;
#pragma unroll 4
        for (int j = lane; j < N; j += 32) {
            const int x = cexpo(row[j]);
            if (x != kSpecial) e = max(e, x);
        }
        e = __reduce_max_sync(0xffffffffu, e);
        if (lane == 0) f[k] = e;
    } else {
        // inner index contiguous: 8 of them per block, threads 8 (k) x 32 (j)
        __shared__ int se[8][33];
        const int k = blockIdx.x * 8 + (threadIdx.x & 7), j0 = threadIdx.x >> 3;
        int e = kNone;
        if (k < K) {
#pragma unroll 4
            for (int j = j0; j < N; j += 32) {
                const int x = cexpo(B[k * ks + j * js]);
                if (x != kSpecial) e = max(e, x);
            }
        }
        se[threadIdx.x & 7][j0] = e;
        __syncthreads();
        const int r = __reduce_max_sync(0xffffffffu, se[warp][lane]);
        if (lane == 0 && blockIdx.x * 8 + warp < K) f[blockIdx.x * 8 + warp] = r;
    }
}

// the digits of 8 consecutive inner indices of one row (or column), real or imaginary part: one
// 16-byte store per digit, dst + digit * stride
template <int S>
__device__ __forceinline__ void store_digits(const long long (&q)[8], unsigned char* dst, int stride) {
    unsigned lo[8], hi[8];
#pragma unroll
    for (int t = 0; t < 8; t++) {       // + 128 in every digit below the top: bytes are digit + 128
        const unsigned long long b = (unsigned long long)(q[t] + (S == 8 ? 0x80808080808080ll : 0x808080ll));
        lo[t] = (unsigned)b;
        hi[t] = (unsigned)(b >> 32);
    }
#pragma unroll
    for (int s = 0; s < S; s++) {
        float v[8];
#pragma unroll
        for (int t = 0; t < 8; t++) {
            // integer to float through the low mantissa bits of 2^23
            if (s == 0) {
                v[t] = __uint_as_float(0x4b000000u + 256u + (unsigned)((int)(S == 8 ? hi[t] : lo[t]) >> 24)) -
                       (8388608.0f + 256.0f);
            } else {
                const int sh = 8 * (S - 1 - s);
                const unsigned byte = ((sh >= 32 ? hi[t] >> (sh - 32) : lo[t] >> sh) & 0xffu);
                v[t] = __uint_as_float(0x4b000000u | byte) - (8388608.0f + 128.0f);
            }
        }
        uint4 w;
        w.x = __byte_perm(__float_as_uint(v[0]), __float_as_uint(v[1]), 0x7632);
        w.y = __byte_perm(__float_as_uint(v[2]), __float_as_uint(v[3]), 0x7632);
        w.z = __byte_perm(__float_as_uint(v[4]), __float_as_uint(v[5]), 0x7632);
        w.w = __byte_perm(__float_as_uint(v[6]), __float_as_uint(v[7]), 0x7632);
        *reinterpret_cast<uint4*>(dst + s * stride) = w;
    }
}

// 512 threads: bound by the latency of its loads (operands of two products of n = 648: 50 us with 256, 35 with 512 and with
// 1024; of 20, with more blocks than SMs, 253, 234 and 245)
constexpr int kSplitThreads = 512, kSplitK = kSplitThreads / 16;

struct SplitArgs {
    const void *A, *B;
    long long rsA, ksA, rsB, ksB;      // element (row of A or column of B, inner index k) at row rs + k ks
    long long sA, sB;
    int conjB;                         // 1: the conjugate
    int M, N, K, nk, mt, nt;           // nk stages, mt x nt tiles
    int gA, gB, nA;                    // 16-row groups of A, 16-column groups of B per matrix; A blocks in all
    const int* f;
    int *eA, *gN;                      // e_i [b][16 gA], g_j [b][16 gB]
    unsigned char *dA, *dB;
    int fstep;                         // f stride per A matrix: 0 when all matrices share one B
};

// Exponents and digits of 16 rows of A or 16 columns of B: first the largest exponent of each over
// the inner index, then the digits, a warp per stage of 16 inner indices (lane = 8 rows x 2 halves of
// the stage x 2 row groups, so a warp stores 512 contiguous bytes per digit).
template <int S, bool kA, typename T>
__device__ __forceinline__ void split_group(const SplitArgs& p, int b, int g, int (*se)[kSplitK + 1]) {
    using C = Cfg<S>;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int per = kA ? p.gA : p.gB, r0 = g * 16, R = kA ? p.M : p.N;
    const T* src = (kA ? (const T*)p.A + p.sA * b : (const T*)p.B + p.sB * b);
    const long long rs = kA ? p.rsA : p.rsB, ks = kA ? p.ksA : p.ksB;
    const int* f = p.f + (long long)(kA ? b * p.fstep : b) * p.K;
    {
        // 16 x kSplitK threads, the faster ones along the contiguous index
        const bool kfast = ks == 1;
        const int r = kfast ? t / kSplitK : t & 15, kr = kfast ? t % kSplitK : t >> 4;
        int e = kNone;
        if (r0 + r < R) {
#pragma unroll 4
            for (int k = kr; k < p.K; k += kSplitK) {
                const int x = cexpo(src[(r0 + r) * rs + k * ks]);
                if (x == kSpecial) e = kSpecial;
                else if (x != kNone) e = max(e, kA ? x + f[k] : x - f[k]);
            }
        }
        se[r][kr] = e;
    }
    __syncthreads();
    if (t < 16) {
        int e = kNone;
        for (int q = 0; q < kSplitK; q++) e = max(e, se[t][q]);
        se[t][kSplitK] = e;
        (kA ? p.eA : p.gN)[(long long)b * per * 16 + r0 + t] = e;
    }
    __syncthreads();
    const int rl = (lane & 7) + 8 * (lane >> 4), kh = (lane >> 3) & 1;
    const int r = r0 + rl, e = se[rl][kSplitK];
    const bool live = r < R && e > kNone / 2 && e < kSpecial;
    constexpr int TR = kA ? kTM : C::kTN, blkb = kA ? C::kABlk : C::kBBlk, dig = TR * kTK * 2;
    unsigned char* dst = (kA ? p.dA + (long long)b * p.mt * p.nk * C::kABlk : p.dB + (long long)b * p.nt * p.nk * C::kBBlk) +
                         (long long)(r0 / TR) * p.nk * blkb + (r0 % TR) * 32 + (lane >> 4) * 256 + kh * 128 + (lane & 7) * 16;
    for (int st = warp; st < p.nk; st += kSplitThreads / 32) {
        const int k0 = st * kTK + kh * 8;
        long long qr[8], qi[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            qr[j] = qi[j] = 0;
            const int k = k0 + j;
            if (live && k < p.K) {
                const T v = src[r * rs + k * ks];
                const int s = (kA ? f[k] : -f[k]) - e + C::kBits;
                qr[j] = fixed_point(v.x, s);
                qi[j] = fixed_point(v.y, s);
                if (!kA && p.conjB) qi[j] = -qi[j];
            }
        }
        unsigned char* o = dst + (long long)st * blkb;
        store_digits<S>(qr, o, dig);
        store_digits<S>(qi, o + S * dig, dig);
    }
}

template <int S, typename TA, typename TB>
__global__ void __launch_bounds__(kSplitThreads) oz_split_kernel(SplitArgs p, const int* __restrict__ skip) {
    chain_wait();
    chain_trigger();
    __shared__ int se[16][kSplitK + 1];
    const bool isA = (int)blockIdx.x < p.nA;
    const int blk = isA ? blockIdx.x : blockIdx.x - p.nA;
    const int per = isA ? p.gA : p.gB;
    const int b = blk / per, g = blk - b * per;
    if (z::skipped(skip, b)) return;
    if (isA) split_group<S, true, TA>(p, b, g, se);
    else split_group<S, false, TB>(p, b, g, se);
}

// (hi 2^32 + lo) 2^e rounded once to FP64, with integer operations (FP64 ones cost 60 times more)
__device__ __forceinline__ double fx_to_double(long long hi, long long lo, int e) {
    hi += lo >> 32;
    unsigned L = (unsigned)lo;
    const bool neg = hi < 0;
    unsigned long long H = (unsigned long long)hi;
    if (neg) {
        L = 0u - L;
        H = ~H + (L == 0u ? 1ull : 0ull);
    }
    if (H == 0ull) {
        H = L;
        L = 0u;
        e -= 32;
        if (H == 0ull) return 0.0;
    }
    const int lz = __clzll((long long)H);            // >= 1: |hi| < 2^62
    const unsigned long long L64 = (unsigned long long)L << 32;
    const unsigned long long m = (H << lz) | (L64 >> (64 - lz));
    const bool sticky = (L64 << lz) != 0ull;
    unsigned long long r = m >> 11;
    const unsigned rem = (unsigned)m & 0x7ffu;
    r += (rem > 0x400u || (rem == 0x400u && (sticky || (r & 1ull)))) ? 1ull : 0ull;
    const int ex = 63 + 32 + e - lz + 1023;          // biased exponent of the value
    const unsigned long long sign = neg ? 1ull << 63 : 0ull;
    if (ex >= 1 && ex <= 2046) return __longlong_as_double((long long)(sign + ((unsigned long long)(ex - 1) << 52) + r));
    return scalbn(__longlong_as_double((long long)(sign + (1022ull << 52) + r)), max(-5000, min(5000, ex - 1023)));
}

// w 2^e in FP32 for |w| < 2^56: the two 24-bit and 32-bit parts are converted exactly but for the upper
// one's rounding
__device__ __forceinline__ float fx_to_float(long long w, int e) {
    const float f = fmaf((float)(int)(w >> 24), 16777216.f, (float)(int)((unsigned)w & 0xffffffu));
    e = max(-250, min(250, e));
    const int h = e >> 1;
    return f * __int_as_float((h + 127) << 23) * __int_as_float((e - h + 127) << 23);
}

struct GemmArgs {
    const unsigned char *dA, *dB;
    const int *eA, *gN;
    int M, N, nk, mt, nt, gA, gB;
    int a_shared, b_shared;            // all matrices use the digits of matrix 0
    double2 alpha, beta;
    double diag;                       // added on the diagonal of alpha A B
    void* C;
    int ldc;
    long long sC;
    int tiles;
    int* err;
    const unsigned* mask;              // a bit per element that oz_parts_kernel has written; null: none
};

__device__ __forceinline__ bool masked(const unsigned* mask, int M, int N, int b, int i, int j) {
    return mask[((long long)b * M + i) * ((N + 31) / 32) + (j >> 5)] >> (j & 31) & 1u;
}

__device__ __forceinline__ double2 to_d(double2 v) { return v; }
__device__ __forceinline__ double2 to_d(float2 v) { return make_double2(v.x, v.y); }
__device__ __forceinline__ void put(double2* p, double2 v) { *p = v; }
__device__ __forceinline__ void put(float2* p, double2 v) { *p = make_float2((float)v.x, (float)v.y); }
__device__ __forceinline__ void put(double2* p, float x, float y) { *p = make_double2(x, y); }
__device__ __forceinline__ void put(float2* p, float x, float y) { *p = make_float2(x, y); }

// The digits' error is at most 2 K 2^-59 R_i S_j per part (R, S: the row's and the column's powers of two), wherever the
// sum of the |products| that make up the part lies.  So that sum is formed here, in FP32 and within 1e-5, and parts
// where it is below R S max(2^-5, sqrt(K) 2^-7) are computed by FP64 operations: from 2^-6 on the digits' bound is
// below that of an FP64 sum, (2 K + 1) 2^-53 of the sum; sqrt(K) 2^-7 is where their typical errors meet (digits 2^-62 a
// product, a sequential sum K 2^-55 of the mean product).  A sum of zero is exact.  Rows of 10^10 and 1/3 times the identity had 1/3 to 9 digits.
// Ordinary sums are large enough after one or two steps of 16 inner indices, where the tile is left: products of order 648 take
// 132 us in place of 122, 20 of them 1680 in place of 1612, of order 3200 6.87 ms in place of 6.73.
constexpr int kPT = 64, kPK = 16;                // as gemm_kernel: 64 x 64 tiles, 4 x 4 per thread, 16 inner indices at a time

// |v| 2^s < 1 in FP32, rounded down to 21 bits; what is not zero at least 2^-60
__device__ __forceinline__ float scaled_abs(double v, int s) {
    const unsigned hi = (unsigned)__double2hiint(v) & 0x7fffffffu;
    int ex = (int)(hi >> 20);
    unsigned m = (hi & 0xfffffu) << 3;
    if (ex == 0) {
        if (v == 0.0) return 0.f;
        const unsigned long long q = (unsigned long long)__double_as_longlong(v) << 12;       // subnormal: normalised
        const int lz = __clzll((long long)q);
        ex = -lz;
        m = (unsigned)(q << lz << 1 >> 41);
    }
    ex += s - 1023;
    if (ex < -60) return 0x1p-60f;
    return __uint_as_float(((unsigned)(min(ex, 0) + 127) << 23) | m);
}

__global__ void __launch_bounds__(256)
oz_parts_kernel(SplitArgs p, int a_shared, int b_shared, double2 alpha, double2 beta, double2* __restrict__ C, int ldc, long long sC,
                unsigned* __restrict__ mask, const int* __restrict__ skip) {
    using z::cfma;
    chain_wait();
    const int b = blockIdx.z;
    if (z::skipped(skip, b)) return;
    const double2* A = (const double2*)p.A + p.sA * b;
    const double2* B = (const double2*)p.B + p.sB * b;
    const int ba = a_shared ? 0 : b, bb = b_shared ? 0 : b;
    const int *eA = p.eA + (long long)ba * p.gA * 16, *gN = p.gN + (long long)bb * p.gB * 16;
    const int *fA = p.f + (long long)(ba * p.fstep) * p.K, *fB = p.f + (long long)bb * p.K;
    const int i0 = blockIdx.y * kPT, j0 = blockIdx.x * kPT, tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    __shared__ __align__(16) double2 buf[2][kPK][kPT + 1];
    __shared__ unsigned bits[kPT][2];
    float2 (*As)[kPT + 1] = reinterpret_cast<float2(*)[kPT + 1]>(&buf[0][0][0]);
    float2 (*Bs)[kPT + 1] = reinterpret_cast<float2(*)[kPT + 1]>(&buf[1][0][0]);
    if (tid < 2 * kPT) bits[tid >> 1][tid & 1] = 0u;
    float re[4][4] = {}, im[4][4] = {};
    const float least = fmaxf(0x1p-5f, sqrtf((float)p.K) * 0x1p-7f);
    auto inside = [&](int r, int q) { return i0 + ty + 16 * r < p.M && j0 + tx + 16 * q < p.N; };
    const bool kfastA = p.ksA == 1, kfastB = p.ksB == 1;
    for (int k0 = 0; k0 < p.K; k0 += kPK) {
        for (int e = tid; e < kPK * kPT; e += 256) {
            const int ra = kfastA ? e / kPK : e % kPT, ka = kfastA ? e % kPK : e / kPT;
            const int rb = kfastB ? e / kPK : e % kPT, kb = kfastB ? e % kPK : e / kPT;
            float2 a = make_float2(0.f, 0.f), c = a;
            if (i0 + ra < p.M && k0 + ka < p.K) {
                const int ex = eA[i0 + ra], s = fA[k0 + ka] - ex;
                const double2 v = A[(i0 + ra) * p.rsA + (k0 + ka) * p.ksA];
                if (ex > kNone / 2 && ex < kSpecial) a = make_float2(scaled_abs(v.x, s), scaled_abs(v.y, s));
            }
            if (j0 + rb < p.N && k0 + kb < p.K) {
                const int ex = gN[j0 + rb], s = -fB[k0 + kb] - ex;
                const double2 v = B[(j0 + rb) * p.rsB + (k0 + kb) * p.ksB];
                if (ex > kNone / 2 && ex < kSpecial) c = make_float2(scaled_abs(v.x, s), scaled_abs(v.y, s));
            }
            As[ka][ra] = a;
            Bs[kb][rb] = c;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < kPK; kk++) {
            float2 a[4], c[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                a[q] = As[kk][ty + 16 * q];
                c[q] = Bs[kk][tx + 16 * q];
            }
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    re[r][q] = fmaf(a[r].x, c[q].x, fmaf(a[r].y, c[q].y, re[r][q]));
                    im[r][q] = fmaf(a[r].x, c[q].y, fmaf(a[r].y, c[q].x, im[r][q]));
                }
        }
        // no term is negative: enough is enough
        float low = least;
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int q = 0; q < 4; q++) low = fminf(low, inside(r, q) ? fminf(re[r][q], im[r][q]) : least);
        if (__syncthreads_and(low >= least)) break;
    }
    unsigned weak = 0u;
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int q = 0; q < 4; q++)
            if ((re[r][q] > 0.f && re[r][q] < least) || (im[r][q] > 0.f && im[r][q] < least)) {
                weak |= 1u << (4 * r + q);
                const int c = tx + 16 * q;
                atomicOr(&bits[ty + 16 * r][c >> 5], 1u << (c & 31));
            }
    const int any = __syncthreads_or((int)weak);
    if (tid < 2 * kPT && i0 + (tid >> 1) < p.M && j0 + 32 * (tid & 1) < p.N)
        mask[((long long)b * p.M + i0 + (tid >> 1)) * ((p.N + 31) / 32) + j0 / 32 + (tid & 1)] = bits[tid >> 1][tid & 1];
    if (!any) return;
    double2 acc[4][4];
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int q = 0; q < 4; q++) acc[r][q] = make_double2(0.0, 0.0);
    for (int k0 = 0; k0 < p.K; k0 += kPK) {
        for (int e = tid; e < kPK * kPT; e += 256) {
            const int ra = kfastA ? e / kPK : e % kPT, ka = kfastA ? e % kPK : e / kPT;
            const int rb = kfastB ? e / kPK : e % kPT, kb = kfastB ? e % kPK : e / kPT;
            const double2 zero = make_double2(0.0, 0.0);
            buf[0][ka][ra] = i0 + ra < p.M && k0 + ka < p.K ? A[(i0 + ra) * p.rsA + (k0 + ka) * p.ksA] : zero;
            double2 v = j0 + rb < p.N && k0 + kb < p.K ? B[(j0 + rb) * p.rsB + (k0 + kb) * p.ksB] : zero;
            if (p.conjB) v.y = -v.y;
            buf[1][kb][rb] = v;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < kPK; kk++) {
            double2 a[4], c[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                a[q] = buf[0][kk][ty + 16 * q];
                c[q] = buf[1][kk][tx + 16 * q];
            }
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int q = 0; q < 4; q++) acc[r][q] = cfma(a[r], c[q], acc[r][q]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (!(weak >> (4 * r + q) & 1u)) continue;
            double2* c = C + sC * b + (long long)(i0 + ty + 16 * r) * ldc + j0 + tx + 16 * q;
            double2 v = z::cmul(alpha, acc[r][q]);
            if (beta.x != 0.0 || beta.y != 0.0) v = cfma(beta, *c, v);
            *c = v;
        }
}

// kMask: elements whose bit p.mask has set are left as they are
template <int S, typename TC, bool kMask>
__global__ void __launch_bounds__(kThreads, 1)
oz_gemm_kernel(GemmArgs p, const int* __restrict__ skip) {
    using namespace tc;
    constexpr int kS = S, kTN = Cfg<S>::kTN, kABlk = Cfg<S>::kABlk, kBBlk = Cfg<S>::kBBlk, kStages = Cfg<S>::kStages;
    constexpr int kCols = kTN * 4 / kDrainWarps;  // columns of a drain warp
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* sA = smem;
    unsigned char* sB = smem + kStages * kABlk;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + Cfg<S>::kBarOff);
    uint64_t* full = bar;                         // [kStages] copies -> MMA
    uint64_t* empty = bar + kStages;              // [kStages] MMA -> copies
    uint64_t* acc_full = bar + 2 * kStages;       // MMA -> drain
    uint64_t* acc_empty = acc_full + 1;           // drain -> MMA
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(acc_full + 3);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int i = 0; i < kStages; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        mbar_init(acc_full, 1);
        mbar_init(acc_empty, kDrainWarps * 32);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        tmem_alloc(tmem_slot, kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const int per = p.mt * p.nt;
    chain_wait();

    if (warp == kDrainWarps) {
        // ---------------- copies ----------------
        if (lane == 0) {
            int it = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x) {
                const int b = tile / per, q = tile - b * per, m = q / p.nt, n = q - m * p.nt;
                if (z::skipped(skip, b)) continue;
                const unsigned char* ga = p.dA + ((long long)(p.a_shared ? 0 : b) * p.mt + m) * p.nk * kABlk;
                const unsigned char* gb = p.dB + ((long long)(p.b_shared ? 0 : b) * p.nt + n) * p.nk * kBBlk;
                for (int k = 0; k < p.nk; k++, it++) {
                    const int s = it % kStages;
                    if (*abort_flag || (it >= kStages && !mbar_wait(&empty[s], (uint32_t)((it / kStages - 1) & 1)))) {
                        *abort_flag = 1;
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(&full[s], kABlk + kBBlk);
                    bulk_load(sA + s * kABlk, ga + (long long)k * kABlk, kABlk, &full[s]);
                    bulk_load(sB + s * kBBlk, gb + (long long)k * kBBlk, kBBlk, &full[s]);
                }
            }
            // no copy into shared memory outlives the kernel (after an abort the MMA thread may not
            // have waited for the last ones)
            for (int i = max(0, it - kStages); i < it; i++) mbar_wait(&full[i % kStages], (uint32_t)((i / kStages) & 1));
        }
        __syncwarp();
    } else if (warp == kDrainWarps + 1) {
        // ---------------- MMA issue ----------------
        if (lane == 0) {
            constexpr uint32_t base = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kTM >> 4) << 24);
            constexpr uint32_t negA = 1u << 13;
            constexpr uint32_t im = kS * kTN;       // first column of the imaginary diagonals
            int it = 0, chunk = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x) {
                if (z::skipped(skip, tile / per)) continue;
                for (int k = 0; k < p.nk; k++, it++) {
                    const int s = it % kStages;
                    const bool first = k % kChunk == 0;
                    if (first && chunk > 0 && !mbar_wait(acc_empty, (uint32_t)((chunk - 1) & 1))) ok = false;
                    if (!ok || *abort_flag || !mbar_wait(&full[s], (uint32_t)((it / kStages) & 1))) {
                        *abort_flag = 1;
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a = smem_u32(sA + s * kABlk), bb = smem_u32(sB + s * kBBlk);
                    const uint64_t dbr = make_desc(bb, 128, 256), dbi = make_desc(bb + kS * kTN * kTK * 2, 128, 256);
#pragma unroll
                    for (int i = 0; i < kS; i++) {
                        const uint32_t id = base | ((uint32_t)((kS - i) * kTN >> 3) << 17);
                        const uint64_t dar = make_desc(a + i * kTM * kTK * 2, 128, 256);
                        const uint64_t dai = make_desc(a + (kS + i) * kTM * kTK * 2, 128, 256);
                        const uint32_t col = tmem + (uint32_t)(i * kTN);
                        const uint32_t acc = !(first && i == 0);
                        umma<1>(col, dar, dbr, id, acc);
                        umma<1>(col + im, dar, dbi, id, acc);
                        umma<1>(col, dai, dbi, id | negA, 1);
                        umma<1>(col + im, dai, dbr, id, 1);
                    }
                    umma_commit(&empty[s]);
                    if (k % kChunk == kChunk - 1 || k == p.nk - 1) {
                        umma_commit(acc_full);
                        chunk++;
                    }
                }
            }
            // the accumulators must be idle before TMEM is freed
            for (int i = max(0, it - kStages); i < it; i++) mbar_wait(&empty[i % kStages], (uint32_t)((i / kStages) & 1));
        }
        __syncwarp();
    } else {
        // -------- drain: warp w reads TMEM lanes 32 (w % 4) .., part w / 4 of each diagonal's columns --------
        const int quarter = warp & 3, part4 = warp >> 2;
        const uint32_t tb = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(part4 * kCols);
        constexpr int kW = S == 8 ? 2 : 1;       // 64-bit words per value: diagonals 0 .. 3 (and 4 .. 7)
        int chunk = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x) {
            const int b = tile / per, q = tile - b * per, m = q / p.nt, n = q - m * p.nt;
            if (z::skipped(skip, b)) continue;
            long long w[kW][2][kCols];
#pragma unroll
            for (int c = 0; c < kCols; c++)
#pragma unroll
                for (int h = 0; h < kW; h++) w[h][0][c] = w[h][1][c] = 0;
            for (int k = 0; k < p.nk; k += kChunk, chunk++) {
                int stop = *abort_flag;
                if (!stop && !mbar_wait(acc_full, (uint32_t)(chunk & 1))) stop = 1;
                if (__any_sync(0xffffffffu, stop)) {
                    *abort_flag = 1;
                    ok = false;
                    break;
                }
                tc_fence_after();
                // kLd columns at a time, the next ones on their way while these are added up
                uint32_t v[2][kLd];
                auto fetch = [&](int q) {
                    const int part = q / (kS * (kCols / kLd)), d = q / (kCols / kLd) % kS, c0 = q % (kCols / kLd) * kLd;
                    tmem_ld8(tb + (uint32_t)(part * kS * kTN + d * kTN + c0), v[q & 1]);
                };
                constexpr int kN = 2 * kS * (kCols / kLd);
                fetch(0);
#pragma unroll
                for (int q = 0; q < kN; q++) {
                    tmem_ld_wait8(v[q & 1]);
                    if (q + 1 < kN) fetch(q + 1);
                    const int part = q / (kS * (kCols / kLd)), d = q / (kCols / kLd) % kS, c0 = q % (kCols / kLd) * kLd;
#pragma unroll
                    for (int c = 0; c < kLd; c++) {
                        long long& acc = w[d >> 2][part][c0 + c];
                        asm("mad.wide.s32 %0, %1, %2, %0;"
                            : "+l"(acc)
                            : "r"(__float2int_rn(__uint_as_float(v[q & 1][c]))), "r"(1 << (8 * (3 - (d & 3)))));
                    }
                }
                tc_fence_before();
                mbar_arrive(acc_empty);
            }
            if (!ok) break;
            // kSeg columns at a time: every lane converts its row's values into the warp's staging rows
            // (80 bytes apart: no bank conflicts), then the warp reads and writes C in segments of
            // 64 contiguous bytes per row
            constexpr int kSeg = 64 / (int)sizeof(TC);
            unsigned char* stg = smem + Cfg<S>::kStageOff + warp * 32 * kStageRow;
            const int row0 = m * kTM + quarter * 32, row = row0 + lane, col0 = n * kTN + part4 * kCols;
            const int eA = row < p.M ? p.eA[(long long)(p.a_shared ? 0 : b) * p.gA * 16 + row] : kNone;
            const int* gN = p.gN + (long long)(p.b_shared ? 0 : b) * p.gB * 16 + col0;
            TC* out = (TC*)p.C + p.sC * b + (long long)row0 * p.ldc + col0;
            const bool unit = p.alpha.y == 0.0 && (p.alpha.x == 1.0 || p.alpha.x == -1.0);
            const bool add = p.beta.x != 0.0 || p.beta.y != 0.0;
            const bool add1 = p.beta.x == 1.0 && p.beta.y == 0.0;
            // an FP32 result without a diagonal needs no FP64 on the way
            const bool narrow = sizeof(TC) == sizeof(float2) && unit && p.diag == 0.0;
#pragma unroll
            for (int c0 = 0; c0 < kCols; c0 += kSeg) {
                if (row0 >= p.M || col0 + c0 >= p.N) break;      // uniform
                __syncwarp();
#pragma unroll
                for (int cc = 0; cc < kSeg; cc++) {
                    const int c = c0 + cc;
                    TC* dst = reinterpret_cast<TC*>(stg + lane * kStageRow) + cc;
                    const int g = col0 + c < p.N ? gN[c] : kNone;
                    // the last diagonal weighs 2^(8 (S - 1)); units 2^(eA - kBits) 2^(g - kBits)
                    const int e = eA + g + 8 * (kS - 1) - 2 * Cfg<S>::kBits;
                    if (narrow && eA < kSpecial && g < kSpecial) {
                        const float sg = p.alpha.x < 0.0 ? -1.f : 1.f;
                        put(dst, sg * fx_to_float(w[0][0][c], e), sg * fx_to_float(w[0][1][c], e));
                        continue;
                    }
                    double2 v;
                    if (eA >= kSpecial || g >= kSpecial) {
                        v.x = v.y = __longlong_as_double(0x7ff8000000000000ll);
                    } else if (kW == 2) {
                        v.x = fx_to_double(w[0][0][c], w[kW - 1][0][c], e);
                        v.y = fx_to_double(w[0][1][c], w[kW - 1][1][c], e);
                    } else {
                        v.x = fx_to_double(0, w[0][0][c], e);
                        v.y = fx_to_double(0, w[0][1][c], e);
                    }
                    if (unit) {
                        if (p.alpha.x < 0.0) v = make_double2(-v.x, -v.y);
                    } else {
                        v = z::cmul(p.alpha, v);
                    }
                    if (p.diag != 0.0 && row == col0 + c) v.x += p.diag;
                    put(dst, v);
                }
                __syncwarp();
#pragma unroll 4
                for (int q = lane; q < 32 * kSeg; q += 32) {
                    const int r = q / kSeg, cc = q % kSeg;
                    if (row0 + r >= p.M || col0 + c0 + cc >= p.N) continue;
                    if (kMask && masked(p.mask, p.M, p.N, b, row0 + r, col0 + c0 + cc)) continue;
                    TC v = reinterpret_cast<const TC*>(stg + r * kStageRow)[cc];
                    TC* o = out + (long long)r * p.ldc + c0 + cc;
                    if (add1) {
                        const TC x = *o;
                        v.x += x.x;
                        v.y += x.y;
                    } else if (add) {
                        put(&v, z::cfma(p.beta, to_d(*o), to_d(v)));
                    }
                    *o = v;
                }
            }
        }
    }
    __syncthreads();
    if (tid == 0 && *abort_flag) atomicExch(p.err, 1);
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
}

// y = alpha A x + beta y, a warp per row (the one-column products of the beta recursion)
__global__ void __launch_bounds__(256)
zgemv_kernel(int M, int K, double2 alpha, const double2* __restrict__ A, int lda, long long sA,
             const double2* __restrict__ x, int ldx, long long sX, double2 beta, double2* __restrict__ y, int ldy,
             long long sY, const int* __restrict__ skip) {
    chain_wait();
    if (z::skipped(skip, blockIdx.y)) return;
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i >= M) return;
    const double2* row = A + sA * blockIdx.y + (long long)i * lda;
    x += sX * blockIdx.y;
    double2 s = make_double2(0.0, 0.0);
#pragma unroll 4
    for (int k = lane; k < K; k += 32) s = z::cfma(row[k], x[(long long)k * ldx], s);
    for (int o = 16; o > 0; o >>= 1) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
        s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
    }
    if (lane == 0) {
        double2* o = y + sY * blockIdx.y + (long long)i * ldy;
        double2 v = z::cmul(alpha, s);
        if (beta.x != 0.0 || beta.y != 0.0) v = z::cfma(beta, *o, v);
        *o = v;
    }
}

static size_t al256(size_t x) { return (x + 255) / 256 * 256; }

struct Shape {
    int nk, mt, nt, gA, gB;
    size_t a, b, small_a, small_b, m;  // bytes per matrix: digits of A, of B, exponents, a bit per element of C
    Shape(int S, int M, int N, int K) {
        const int tn = 256 / S;
        nk = (K + kTK - 1) / kTK;
        mt = (M + kTM - 1) / kTM;
        nt = (N + tn - 1) / tn;
        gA = (M + 15) / 16;
        gB = (N + 15) / 16;
        a = (size_t)mt * nk * (2 * S * kTM * kTK * 2);
        b = (size_t)nt * nk * (2 * S * tn * kTK * 2);
        small_a = (size_t)gA * 16 * sizeof(int);
        small_b = ((size_t)gB * 16 + K) * sizeof(int);
        m = (size_t)M * ((N + 31) / 32) * sizeof(unsigned);
    }
    // for na A, nb B and (nc > 0) the mask of nc C
    size_t bytes(int na, int nb, int nc) const {
        return al256(na * small_a) + al256(nb * small_b) + al256(nc * m) + na * a + nb * b;
    }
};

// One product with S digits; element types double2 or float2 by operand.
template <int S, typename TA, typename TB, typename TC>
static scw_status run(cudaStream_t st, int M, int N, int K, double2 alpha, const TA* A, int lda, long long sA,
                      const TB* B, int ldb, long long sB, int opB, double2 beta, double diag, TC* C, int ldc, long long sC, int batch,
                      const GemmWs& ws, const int* skip) {
    if (M <= 0 || N <= 0 || batch <= 0) return SCW_OK;
    int sms = 0, dev = 0;
    SCW_CUDA_TRY(cudaGetDevice(&dev));
    SCW_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    constexpr size_t smem = Cfg<S>::kSmem;
    const Shape sh(S, M, N, K);
    const bool a1 = sA == 0 && !skip, b1 = sB == 0 && !skip;     // one operand for the whole batch
    // element (i, k) of op(A) at i rsA + k ksA, (k, j) of op(B) at k ksB + j rsB
    const long long rsA = lda, ksA = 1;
    const long long ksB = opB == kOpN ? ldb : 1, rsB = opB == kOpN ? 1 : ldb;
    // as many matrices at a time as the workspace holds
    int step = batch;
    const bool parts = ws.parts && S == 8;
    auto need = [&](int n) { return sh.bytes(a1 ? 1 : n, b1 ? 1 : n, parts ? n : 0); };
    while (step > 1 && need(step) > ws.bytes) step = (step + 1) / 2;
    if (need(1) > ws.bytes) return fail(SCW_ERR_NOMEM, "zgemm: workspace too small");
    for (int b0 = 0; b0 < batch; b0 += step) {
        const int nb = std::min(step, batch - b0);
        const int na_ = a1 ? 1 : nb, nb_ = b1 ? 1 : nb;
        char* cur = ws.base;
        int* eA = reinterpret_cast<int*>(cur);
        cur += al256(na_ * sh.small_a);
        int* gN = reinterpret_cast<int*>(cur);
        int* f = gN + (size_t)nb_ * sh.gB * 16;
        cur += al256(nb_ * sh.small_b);
        unsigned* mask = parts ? reinterpret_cast<unsigned*>(cur) : nullptr;
        if (parts) cur += al256(nb * sh.m);
        unsigned char* dA = reinterpret_cast<unsigned char*>(cur);
        unsigned char* dB = dA + na_ * sh.a;
        const TA* Ab = A + sA * b0;
        const TB* Bb = B + sB * b0;
        const int* sk = skip ? skip + b0 : nullptr;
        // with one A for several B the inner scaling would differ per matrix: none then
        const bool scale = !(a1 && !b1 && batch > 1);
        if (K > 0) {
            if (scale) {
                SCW_CUDA_TRY(launch_chained(true, st, dim3((K + 7) / 8, nb_), 256, 0, oz_inner_kernel<TB>, Bb, ksB, rsB, sB, K, N,
                                            f, sk));
            } else {
                SCW_CUDA_TRY(cudaMemsetAsync(f, 0, sizeof(int) * (size_t)K * nb_, st));
            }
        }
        SplitArgs sp{Ab, Bb, rsA, ksA, rsB, ksB, sA, sB, opB == kOpC, M, N, K, sh.nk, sh.mt, sh.nt, sh.gA, sh.gB,
                     na_ * sh.gA, f, eA, gN, dA, dB, b1 ? 0 : 1};
        SCW_CUDA_TRY(launch_chained(true, st, dim3(na_ * sh.gA + nb_ * sh.gB), kSplitThreads, 0, oz_split_kernel<S, TA, TB>, sp, sk));
        if constexpr (S == 8) {
            if (parts && K > 0)
                SCW_CUDA_TRY(launch_chained(true, st, dim3((N + kPT - 1) / kPT, (M + kPT - 1) / kPT, nb), 256, 0, oz_parts_kernel, sp,
                                            (int)a1, (int)b1, alpha, beta, C + sC * b0, ldc, sC, mask, sk));
            else if (parts)
                mask = nullptr;
        }
        const long long tiles = (long long)sh.mt * sh.nt * nb;
        if (tiles > (1ll << 30)) return fail(SCW_ERR_ARG, "zgemm: too many tiles");
        GemmArgs g{dA, dB, eA, gN, M, N, sh.nk, sh.mt, sh.nt, sh.gA, sh.gB, a1, b1, alpha, beta, diag,
                   (void*)(C + sC * b0), ldc, sC, (int)tiles, ws.err, mask};
        auto product = [&](auto kernel) -> scw_status {
            SCW_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            SCW_CUDA_TRY(launch_chained(true, st, dim3((unsigned)std::min<long long>(tiles, sms)), kThreads, smem, kernel, g, sk));
            return SCW_OK;
        };
        scw_status ps;
        if constexpr (S == 8) ps = mask ? product(oz_gemm_kernel<S, TC, true>) : product(oz_gemm_kernel<S, TC, false>);
        else ps = product(oz_gemm_kernel<S, TC, false>);
        if (ps != SCW_OK) return ps;
    }
    return SCW_OK;
}

}  // namespace oz

scw_status ctx_tc_flag(scw_ctx ctx) {
    // cleared once per synchronisation, when no kernel that may raise it is under way: a flag raised by an
    // earlier launch stays raised
    if (!ctx->tc_pending_check) *(volatile int*)ctx->tc_host = 0;
    ctx->tc_pending_check = true;
    return SCW_OK;
}

scw_status ctx_gemm_ws(scw_ctx ctx, size_t one, size_t all, GemmWs& ws) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    SCW_CUDA_TRY(cudaStreamIsCapturing(ctx->stream, &cap));
    ws = GemmWs{};
    if (cap != cudaStreamCaptureStatusNone) return SCW_OK;
    scw_status st = ctx->dense_ws.reserve(std::max(one, std::min(all, kGemmWsCap)));
    if (st == SCW_OK) st = ctx_tc_flag(ctx);
    ws = GemmWs{(char*)ctx->dense_ws.ptr, ctx->dense_ws.bytes, ctx->tc_err};
    return st;
}

scw_status reserve_gemm_ws(scw_ctx ctx, DevBuf& buf, size_t one, int batch, GemmWs& ws) {
    scw_status st = buf.reserve(std::max(one, std::min(one * batch, kGemmWsCap)));
    if (st == SCW_ERR_NOMEM && batch > 1) st = buf.reserve(one);
    if (st == SCW_OK) st = ctx_tc_flag(ctx);
    ws = st == SCW_OK ? GemmWs{(char*)buf.ptr, buf.bytes, ctx->tc_err} : GemmWs{};
    return st;
}

size_t zgemm_ws_bytes(int M, int N, int K, int batch) { return oz::Shape(8, M, N, K).bytes(batch, batch, batch); }

scw_status zgemm(cudaStream_t st, int M, int N, int K, double2 alpha, const double2* A, int lda, long long sA,
                 const double2* B, int ldb, long long sB, double2 beta, double2* C, int ldc, long long sC, int batch,
                 const GemmWs& ws, const int* skip, double diag, int opB) {
    if (M <= 0 || N <= 0 || batch <= 0) return SCW_OK;
    if (N == 1 && diag == 0.0 && opB == kOpN) {
        SCW_CUDA_TRY(launch_chained(true, st, dim3((M + 7) / 8, batch), 256, 0, oz::zgemv_kernel, M, K, alpha, A, lda, sA, B,
                                    ldb, sB, beta, C, ldc, sC, skip));
        return SCW_OK;
    }
    if (!ws.base && (diag != 0.0 || opB == kOpC)) return fail(SCW_ERR_ARG, "zgemm: this product needs a workspace");
    if (!ws.base) return gemm<double2>(st, M, N, K, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch, skip, opB);
    return oz::run<8>(st, M, N, K, alpha, A, lda, sA, B, ldb, sB, opB, beta, diag, C, ldc, sC, batch, ws, skip);
}

template <typename TA, typename TB, typename TC>
scw_status gemm32(cudaStream_t st, int n, double alpha, const TA* A, const TB* B, int opB, double beta, double diag, TC* C,
                  int batch, const GemmWs& ws, const int* skip) {
    const long long nn = (long long)n * n;
    return oz::run<4>(st, n, n, n, make_double2(alpha, 0.0), A, n, nn, B, n, nn, opB, make_double2(beta, 0.0), diag, C, n,
                      nn, batch, ws, skip);
}

#define SCW_GEMM32(TA, TB, TC)                                                                                        \
    template scw_status gemm32<TA, TB, TC>(cudaStream_t, int, double, const TA*, const TB*, int, double, double, TC*, \
                                           int, const GemmWs&, const int*);
SCW_GEMM32(float2, float2, float2)
SCW_GEMM32(float2, float2, double2)
SCW_GEMM32(double2, float2, double2)
SCW_GEMM32(double2, float2, float2)
SCW_GEMM32(double2, double2, double2)
#undef SCW_GEMM32

}  // namespace scw
