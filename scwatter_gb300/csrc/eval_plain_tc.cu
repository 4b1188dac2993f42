// Plain plane-wave summation as a matrix product on the tensor cores (tcgen05, sm_103a).
//
// On a plane's grid the phase of every wave separates: with the tile centre (a_c, b_c),
//   E_c(i, j) = sum_w [A'_wc e^{i kA_w (a_i - a_c)}] e^{i kB_w (b_j - b_c)} = sum_w L(40 c + i, w) R(w, j),
// whatever the waves are (k complex, no common grid).  So a tile of 40 columns x 64 rows of points and
// a run of waves is a complex product of a 120 x K by a K x 64 matrix, and a point and wave cost 36 tensor
// multiply-adds and the tile's share of the operands, where the summation of eval_plain.cu spends a sine, a
// cosine and 14 instructions on each.  (The separable evaluator gains far more where the waves share kx
// and ky; this one asks nothing of them.)
//
// Operands are built in shared memory, 32 waves (a chunk) at a time:
//   * warps 20-22 take a wave per lane, every third chunk each: base phase at the tile centre reduced
//     in FP64, amplitudes A' with that phase, scaled by the chunk's power of two for each component (one for all three cut a
//     component 2^-24 of the others to four digits), k in turns as two floats;
//   * warps 8-19 build L and R, a wave per lane and eight columns (or rows) of points per warp: sine and cosine of
//     the phase at columns 2 and 6 and of one step, phases in turns with both factors as two floats (an FP32
//     product would lose 1e-6 at 30 radians), from the Taylor series on [-pi/4, pi/4]; the columns between are one
//     or two steps away, times 1 + i k delta for delta, the rounding of that grid coordinate.  Values are split into
//     fp16 hi + lo (22 bits, 23 in R; L is scaled to 2^12 and R to 2^10, which leaves room for growth inside a tile
//     and keeps lo far above fp16's smallest values even for waves 2^-12 below the chunk's largest) and stored
//     as 16 bytes of eight points of one wave, the MN-major core-matrix row: lanes store side by side, where
//     rows of eight waves (K-major) had four lanes on the same banks;
//   * warp 23 issues the MMAs lo hi + hi lo + hi hi, the small products first, so that the
//     accumulator's rounding acts on the few last steps only.  R is kept as -im | re | im, so that re L x (re | im)
//     and im L x (-im | re) are each one MMA of twice the columns: it reads L half as often, and the MMAs
//     are bound by what they read from shared memory;
//   * warps 0-7 add each chunk's sum, 2^e scaled, to FP32 registers, every kRun chunks those to sums of two floats in
//     the other half of tensor memory, and every kMaxRun waves these to FP64 partial sums, which meet in the reduce
//     kernel, in a fixed order.  32 additions to a growing sum, not 1024: a run of 1024 waves loses less to rounding than the
//     summation kernel's 256 additions (45 against 64 roundings of a sum of 256 waves, over 4096 waves that all add up).
//     One FP32 sum of 4096 waves lost 1.5 times as much as that kernel.
// 409 600 waves x 3 planes of 200 x 200 points: 19.4 ms by the summation kernel, 4.47 ms here; 20 736 waves a layer on a
// 101 x 77 x 50 volume: 5.10 -> 1.39 ms (4.30 and 1.30 with one FP32 sum per 4096 waves:
// tensor memory answers late, and sums that are late hold up the MMAs).  A chunk takes about 1600 clocks: 700 of them are MMA reads of shared memory and
// 450 the stores of the operands, and the warps that build these issue half of the time.  Measured in the
// second case on the way: K-major operands with a sine and cosine for every point and wave 2.9 ms, this
// layout 1.55, operands in FP32 pairs with 9 and 12 warps 1.47 and 1.37 (7 warps 1.64).
#include <cuda_fp16.h>
#include <cstdint>

#include "plain_tc.h"
#include "scw_dense.h"
#include "scw_tc.cuh"

namespace scw {
namespace ptc {

constexpr int kChunk = 32;                    // waves per chunk
constexpr int kPartA = 128 * kChunk * 2;      // bytes of one part of L: 128 rows x 32 waves, fp16
constexpr int kPartB = 3 * kTileJ * kChunk * 2;       // hi or lo of R: -im, re, im
constexpr int kBufBytes = 4 * kPartA + 2 * kPartB;
constexpr int kBufs = 3;
constexpr uint32_t kGroup = kChunk * 16;              // bytes of a group of 8 points: 32 waves of 16 bytes
constexpr int kDrain = 8, kProd = 12, kStage = 3;      // warps
constexpr int kWarps = kDrain + kProd + kStage + 1, kThreads = kWarps * 32;
constexpr int kWaveSlots = 6;                 // staged chunks of waves
constexpr int kRun = 32;                      // chunks (1024 waves) added up in FP32
constexpr uint32_t kCols = 512;               // TMEM: two accumulators of re | im, up to 64 columns each, and the runs' sums
constexpr uint32_t kSumCol = 256, kSumLow = 128;      // their first column (re | im of all columns), and their low words
constexpr int kGroupsA = kTileI / 8, kGroupsB = kTileJ / 8;

// two floats per register pair: one issue slot for two results
struct F2 {
    unsigned long long v;
    __device__ __forceinline__ float x() const { return __uint_as_float((unsigned)v); }
    __device__ __forceinline__ float y() const { return __uint_as_float((unsigned)(v >> 32)); }
};
__device__ __forceinline__ F2 pack(float x, float y) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ F2 both(float x) { return pack(x, x); }
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ F2 neg2(F2 a) { return F2{a.v ^ 0x8000000080000000ull}; }
// hi + x, its rounding error added to lo (Knuth's two-sum; what lo holds where hi is not finite means nothing)
__device__ __forceinline__ void add_exact2(F2& hi, F2& lo, F2 x) {
    const F2 m = both(-1.f), s = add2(hi, x), b = fma2(hi, m, s), t = fma2(b, m, s);
    lo = add2(lo, add2(fma2(t, m, hi), fma2(b, m, x)));
    hi = s;
}
__device__ __forceinline__ float low_word(float hi, float lo) { return isfinite(hi) ? lo : 0.f; }

struct Wave {                                 // one staged wave
    float4 a;                                 // A'x re, im, A'y re, im (scaled)
    float4 b;                                 // A'z re, im, -Im kA log2e, -Im kB log2e
    float4 k;                                 // kA hi, lo, kB hi, lo (turns per unit length)
};

struct Smem {
    Wave wave[kWaveSlots][kChunk];
    float scale[kWaveSlots][3];               // 2^e of the chunk's result, per component
    int cplx[kWaveSlots];
    F2 grid[kGroupsA + kGroupsB][5];          // per group of eight points, L's first: see eight()
    uint64_t wave_full[kWaveSlots], wave_empty[kWaveSlots], full[kBufs], empty[kBufs], acc_full[2], acc_empty[2];
    int task[kGroupsA + kGroupsB];            // of a chunk, in order: group of L, or 64 + group of R
    Item item;                                // for the drain, which has no registers to spare for them
    Plane plane;
    uint32_t tmem;
    volatile int abort;
};

__device__ __forceinline__ float coord(float s, float d, int i) { return __fadd_rn(s, __fmul_rn(d, (float)i)); }

// sine and cosine of t turns, |t| < 2^20: nearest quarter turn, Taylor series to x^9 and x^8
__device__ __forceinline__ void sincos_turns(float t, float& s, float& c) {
    const float q = fmaf(t, 4.f, 12582912.f);             // rint(4 t) in the low bits
    const float x = fmaf(q - 12582912.f, -0.25f, t) * 6.2831853071795865f;
    const float y = x * x;
    const float sp = fmaf(y, fmaf(y, fmaf(y, fmaf(y, 1.f / 362880.f, -1.f / 5040.f), 1.f / 120.f), -1.f / 6.f), 1.f);
    const float cp = fmaf(y, fmaf(y, fmaf(y, fmaf(y, 1.f / 40320.f, -1.f / 720.f), 1.f / 24.f), -0.5f), 1.f);
    const float s0 = x * sp;
    const unsigned iq = __float_as_uint(q);
    const float a = (iq & 1u) ? cp : s0, b = (iq & 1u) ? s0 : cp;
    s = __uint_as_float(__float_as_uint(a) ^ ((iq & 2u) << 30));
    c = __uint_as_float(__float_as_uint(b) ^ (((iq + 1u) & 2u) << 30));
}

// sine and cosine of (kh + kl)(dh + dl) turns
__device__ __forceinline__ void phase(float kh, float kl, float2 d, float& s, float& c) {
    const float p = kh * d.x;
    float e = fmaf(kh, d.x, -p);
    e = fmaf(kh, d.y, e);
    e = fmaf(kl, d.x, e);
    const float r = (p + 12582912.f) - 12582912.f;
    sincos_turns((p - r) + e, s, c);
}

// phase() of two offsets (d: hi pair, lo pair)
__device__ __forceinline__ void phase2(float kh, float kl, F2 dh, F2 dl, F2& s, F2& c) {
    const F2 kk = both(kh), magic = both(12582912.f), nmagic = both(-12582912.f);
    const F2 p = mul2(kk, dh);
    F2 e = fma2(kk, dh, neg2(p));
    e = fma2(kk, dl, e);
    e = fma2(both(kl), dh, e);
    const F2 r = add2(add2(p, magic), nmagic);
    const F2 t = add2(add2(p, neg2(r)), e);
    const F2 q = fma2(t, both(4.f), magic);
    const F2 x = mul2(fma2(add2(q, nmagic), both(-0.25f), t), both(6.2831853071795865f));
    const F2 y = mul2(x, x);
    F2 sp = fma2(y, both(1.f / 362880.f), both(-1.f / 5040.f)), cp = fma2(y, both(1.f / 40320.f), both(-1.f / 720.f));
    sp = fma2(y, sp, both(1.f / 120.f));
    cp = fma2(y, cp, both(1.f / 24.f));
    sp = fma2(y, sp, both(-1.f / 6.f));
    cp = fma2(y, cp, both(-0.5f));
    sp = fma2(y, sp, both(1.f));
    cp = fma2(y, cp, both(1.f));
    sp = mul2(x, sp);
    float sv[2], cv[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const unsigned iq = h ? (unsigned)(q.v >> 32) : (unsigned)q.v;
        const float s0 = h ? sp.y() : sp.x(), c0 = h ? cp.y() : cp.x();
        const float a = (iq & 1u) ? c0 : s0, b = (iq & 1u) ? s0 : c0;
        sv[h] = __uint_as_float(__float_as_uint(a) ^ ((iq & 2u) << 30));
        cv[h] = __uint_as_float(__float_as_uint(b) ^ (((iq + 1u) & 2u) << 30));
    }
    s = pack(sv[0], sv[1]);
    c = pack(cv[0], cv[1]);
}

// e^{i k (offset)} x scale of eight points of a grid, columns u and u + 4 paired: two anchors (columns 2 and 6:
// offsets hi, lo) and one or two steps from them.  dev: what the offsets of columns 0, 1, 3 and 4, 5, 7 deviate from
// whole steps, x 2 pi.  G: the wave's growth per unit length (base 2), used where lossy.
__device__ __forceinline__ void eight(float kh, float kl, float G, bool lossy, const F2* grid, float d, float scale, F2 (&re)[4],
                                      F2 (&im)[4]) {
    float qs, qc;
    phase(kh, kl, make_float2(d, 0.f), qs, qc);
    const F2 anc = grid[0];
    phase2(kh, kl, anc, grid[1], im[2], re[2]);
    F2 m = both(scale);
    float pc = qc, ps = -qs;                  // one step back
    if (lossy) {
        const float up = exp2f(G * d), dn = exp2f(-G * d);
        qc *= up;
        qs *= up;
        pc *= dn;
        ps *= dn;
        m = mul2(m, pack(exp2f(G * anc.x()), exp2f(G * anc.y())));
    }
    re[2] = mul2(re[2], m);
    im[2] = mul2(im[2], m);
    const F2 x = re[2], y = im[2];
    auto turn = [&](int u, float c, float s) {
        re[u] = fma2(x, both(c), mul2(y, both(-s)));
        im[u] = fma2(x, both(s), mul2(y, both(c)));
    };
    turn(0, pc * pc - ps * ps, 2.f * pc * ps);
    turn(1, pc, ps);
    turn(3, qc, qs);
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const int u = i < 2 ? i : 3;
        const F2 dv = grid[2 + i], e = mul2(both(kh), dv), a = re[u], b = im[u];
        re[u] = fma2(neg2(e), b, a);
        im[u] = fma2(e, a, b);
        if (lossy) {
            const F2 f = mul2(both(G * 0.110317801f), dv);     // ln 2 / 2 pi
            re[u] = fma2(f, a, re[u]);
            im[u] = fma2(f, b, im[u]);
        }
    }
}

// Eight values as fp16 hi and lo (the rest, rounded).  kNear: hi is the nearest value of 11 bits, so that lo has either
// sign and half the size; else the upper 11 bits.  Nothing adds the product of two lo, and of two cut ones it leans one way:
// with both operands cut, sums of 600 random waves on grids of a hundredth of a wavelength were 2.9e-7 to 3.1e-7 off, where
// the summation kernel has 2.3e-7 to 3.1e-7; with R nearest they are 1.5e-7 to 2.1e-7 off on grids of every extent.  409 600
// waves on three 200 x 200 planes: 4.45 ms both cut, 4.47 R nearest, 4.73 L nearest, 4.73 both (1.2e-7 to 1.9e-7).
template <bool kNear>
__device__ __forceinline__ void split8(const F2 (&v)[4], uint4& h, uint4& l) {
    F2 hi[4], lo[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
        if (kNear) {
            const F2 m = both(-1.f), t = mul2(v[u], both(8193.f));
            hi[u] = fma2(fma2(v[u], m, t), m, t);
            lo[u] = fma2(hi[u], m, v[u]);
        } else {
            hi[u].v = v[u].v & 0xffffe000ffffe000ull;
            lo[u] = add2(v[u], neg2(hi[u]));
        }
    }
    auto half2 = [](float x, float y) {
        const __half2 q = __floats2half2_rn(x, y);
        return *reinterpret_cast<const uint32_t*>(&q);
    };
    h = make_uint4(half2(hi[0].x(), hi[1].x()), half2(hi[2].x(), hi[3].x()), half2(hi[0].y(), hi[1].y()), half2(hi[2].y(), hi[3].y()));
    l = make_uint4(half2(lo[0].x(), lo[1].x()), half2(lo[2].x(), lo[3].x()), half2(lo[0].y(), lo[1].y()), half2(lo[2].y(), lo[3].y()));
}

// kLong: items of more than kRun chunks among them
template <bool kLong>
__global__ void __launch_bounds__(kThreads, 1)
plain_tc_kernel(const Plane* __restrict__ planes, const Item* __restrict__ items, Waves W, double2* __restrict__ partials,
                int* __restrict__ err) {
    using namespace tc;
    extern __shared__ __align__(1024) unsigned char smem[];
    Smem& S = *reinterpret_cast<Smem*>(smem + kBufs * kBufBytes);
    const Item it = items[blockIdx.x];
    const Plane g = planes[it.plane];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nrow = it.jr1 - it.jr0, ncol = min(kTileI, g.Ni - it.i0);
    const int nchunk = (int)((it.w1 - it.w0 + kChunk - 1) / kChunk);
    const int nA = (ncol + 7) / 8, nB = (nrow + 7) / 8, T = nA + nB;      // groups of eight points
    const int N = nB * 8;                             // columns of re, and of im
    const float ac = coord(g.a0, g.da, it.i0 + kTileI / 2), bc = coord(g.b0, g.db, it.jr0 + N / 2);

    // rows past the tile stay zero
    for (uint32_t o = tid * 16; o < kBufs * kBufBytes; o += kThreads * 16)
        *reinterpret_cast<uint4*>(smem + o) = make_uint4(0, 0, 0, 0);
    for (int h = tid; h < 2 * (kGroupsA + kGroupsB); h += kThreads) {
        const bool A = h < 2 * kGroupsA;
        const int i = (A ? it.i0 + 4 * h : it.jr0 + 4 * (h - 2 * kGroupsA)) + 2;
        const float x0 = A ? g.a0 : g.b0, d = A ? g.da : g.db;
        const double x = (double)coord(x0, d, i), off = x - (double)(A ? ac : bc);
        float dev[4];
        for (int u = 0; u < 4; u++)
            dev[u] = (float)(6.283185307179586 * ((double)coord(x0, d, i - 2 + u) - x - (u - 2) * (double)d));
        float* o = reinterpret_cast<float*>(S.grid[h >> 1]) + (h & 1);
        o[0] = (float)off;
        o[2] = (float)(off - (double)(float)off);
        o[4] = dev[0];
        o[6] = dev[1];
        o[8] = dev[3];
    }
    if (tid < T) S.task[tid] = (tid + 1) * nA / T > tid * nA / T ? tid * nA / T : 64 + tid - tid * nA / T;
    if (tid == 0) {
        for (int i = 0; i < kWaveSlots; i++) {
            mbar_init(&S.wave_full[i], 32);
            mbar_init(&S.wave_empty[i], T + kDrain);
        }
        for (int i = 0; i < kBufs; i++) {
            mbar_init(&S.full[i], T);
            mbar_init(&S.empty[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&S.acc_full[i], 1);
            mbar_init(&S.acc_empty[i], kDrain);
        }
        S.abort = 0;
        S.item = it;
        S.plane = g;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        tmem_alloc(&S.tmem, kLong ? kCols : kSumCol);
        tmem_relinquish();
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = S.tmem;

    if (warp >= kDrain + kProd && warp < kDrain + kProd + kStage) {
        // ---------------- waves: one per lane, re-based to the tile centre ----------------
        const double inv_two_pi = 0.15915494309189533577;
        const double log2e = 1.4426950408889634074;
        const double xc = g.mode == 1 ? (double)g.c : (double)ac;
        const double yc = g.mode == 0 ? (double)bc : g.mode == 1 ? (double)ac : (double)g.c;
        const double zc = g.mode == 0 ? (double)g.c : (double)bc;
        const int cA = g.mode == 1 ? 1 : 0, cB = g.mode == 0 ? 1 : 2;
        const long long n = W.n;
        double kr[3], ki[3], zr = 0.0;
        float2 am[3];
        // a chunk's waves are loaded while the one before is worked on
        auto load = [&](int ch) {
            const long long w = it.w0 + (long long)ch * kChunk + lane;
            const bool in = ch < nchunk && w < it.w1;
#pragma unroll
            for (int q = 0; q < 3; q++) {
                kr[q] = in ? W.kre[q * n + w] : 0.0;
                ki[q] = in ? W.kim[q * n + w] : 0.0;
                am[q] = in ? W.amp[q * n + w] : make_float2(0.f, 0.f);
            }
            zr = in ? W.zref[w] : 0.0;
        };
        load(warp - kDrain - kProd);
        for (int ch = warp - kDrain - kProd; ch < nchunk; ch += kStage) {
            const int s = ch % kWaveSlots;
            const double rz = zc - zr;
            double t = fma(kr[2], rz, fma(kr[1], yc, kr[0] * xc)) * inv_two_pi;
            t -= rint(t);
            // (compared as integers: FP64 instructions are what this warp waits for)
            const bool lossy = ((__double_as_longlong(ki[0]) | __double_as_longlong(ki[1]) | __double_as_longlong(ki[2])) << 1) != 0;
            float m = 1.f;
            if (lossy) m = exp2f((float)(-fma(ki[2], rz, fma(ki[1], yc, ki[0] * xc)) * log2e));
            float sn, cs;
            sincos_turns((float)t, sn, cs);
            sn *= m;
            cs *= m;
            Wave v;
            v.a = make_float4(am[0].x * cs - am[0].y * sn, am[0].x * sn + am[0].y * cs, am[1].x * cs - am[1].y * sn,
                              am[1].x * sn + am[1].y * cs);
            const double kA = (cA == 0 ? kr[0] : kr[1]) * inv_two_pi, kB = (cB == 1 ? kr[1] : kr[2]) * inv_two_pi;
            const double kiA = cA == 0 ? ki[0] : ki[1], kiB = cB == 1 ? ki[1] : ki[2];
            v.b = make_float4(am[2].x * cs - am[2].y * sn, am[2].x * sn + am[2].y * cs, 0.f, 0.f);
            if (lossy) {
                v.b.z = (float)(-kiA * log2e);
                v.b.w = (float)(-kiB * log2e);
            }
            v.k = make_float4((float)kA, (float)(kA - (double)(float)kA), (float)kB, (float)(kB - (double)(float)kB));
            int cplx = (v.b.z != 0.f ? 1 : 0) | (v.b.w != 0.f ? 2 : 0);
            load(ch + kStage);
            // the chunk's largest finite part below 2^e, component by component: a weak one is not measured by the others
            auto part = [](float x) { return fabsf(x) <= 3.4e38f ? fabsf(x) : 0.f; };
            int e[3];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                float& re = c == 0 ? v.a.x : c == 1 ? v.a.z : v.b.x;
                float& im = c == 0 ? v.a.y : c == 1 ? v.a.w : v.b.y;
                const unsigned top = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(part(re), part(im))));
                e[c] = max(-100, min(128, (int)(top >> 23) - 126));
                const float up = __int_as_float((12 - e[c] + 127) << 23);
                re *= up;
                im *= up;
            }
            cplx = (int)__reduce_or_sync(0xffffffffu, (unsigned)cplx);
            int stop = S.abort;
            if (!stop && ch >= kWaveSlots && !mbar_wait(&S.wave_empty[s], (uint32_t)((ch / kWaveSlots - 1) & 1))) stop = 1;
            if (__any_sync(0xffffffffu, stop)) {
                S.abort = 1;
                break;
            }
            S.wave[s][lane] = v;
            if (lane == 0) {
#pragma unroll
                for (int c = 0; c < 3; c++) S.scale[s][c] = __int_as_float((e[c] - 22 + 127) << 23);
                S.cplx[s] = cplx;
            }
            mbar_arrive(&S.wave_full[s]);
        }
        __syncwarp();
    } else if (warp >= kDrain && warp < kDrain + kProd) {
        // ---------------- operands ----------------
        // the chunks' tasks are dealt round, shifted unevenly from chunk to chunk, so that every warp gets both
        // kinds whatever T
        for (int t = warp - kDrain;; t += kProd) {
            const int ch = t / T;
            if (ch >= nchunk) break;
            const int task = S.task[((unsigned)(t - ch * T) + (unsigned)ch * (unsigned)(ch + 1) / 2u) % (unsigned)T];
            const int s = ch % kWaveSlots, buf = ch % kBufs;
            int stop = S.abort;
            if (!stop && !mbar_wait(&S.wave_full[s], (uint32_t)((ch / kWaveSlots) & 1))) stop = 1;
            if (!stop && ch >= kBufs && !mbar_wait(&S.empty[buf], (uint32_t)((ch / kBufs - 1) & 1))) stop = 1;
            if (__any_sync(0xffffffffu, stop)) {
                S.abort = 1;
                break;
            }
            unsigned char* p = smem + buf * kBufBytes + lane * 16;
            const Wave& wv = S.wave[s][lane];
            const int cplx = S.cplx[s];
            const float4 k = wv.k, b = wv.b;
            F2 re[4], im[4];
            uint4 h, l;
            if (task < 64) {
                eight(k.x, k.y, b.z, cplx & 1, S.grid[task], g.da, 1.f, re, im);
                const float4 a = wv.a;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const float ar = c == 0 ? a.x : c == 1 ? a.z : b.x, ai = c == 0 ? a.y : c == 1 ? a.w : b.y;
                    unsigned char* pc = p + (kGroupsA * c + task) * kGroup;
                    F2 v[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) v[u] = fma2(both(ar), re[u], mul2(both(-ai), im[u]));
                    split8<false>(v, h, l);
                    *reinterpret_cast<uint4*>(pc) = h;
                    *reinterpret_cast<uint4*>(pc + kPartA) = l;
#pragma unroll
                    for (int u = 0; u < 4; u++) v[u] = fma2(both(ar), im[u], mul2(both(ai), re[u]));
                    split8<false>(v, h, l);
                    *reinterpret_cast<uint4*>(pc + 2 * kPartA) = h;
                    *reinterpret_cast<uint4*>(pc + 3 * kPartA) = l;
                }
            } else {
                const int gr = task - 64;
                eight(k.z, k.w, b.w, cplx & 2, S.grid[kGroupsA + gr], g.db, 1024.f, re, im);
                unsigned char* pb = p + 4 * kPartA + gr * kGroup;
                split8<true>(re, h, l);
                *reinterpret_cast<uint4*>(pb + nB * kGroup) = h;
                *reinterpret_cast<uint4*>(pb + nB * kGroup + kPartB) = l;
                split8<true>(im, h, l);
                *reinterpret_cast<uint4*>(pb + 2 * nB * kGroup) = h;
                *reinterpret_cast<uint4*>(pb + 2 * nB * kGroup + kPartB) = l;
                constexpr uint32_t neg = 0x80008000u;
                *reinterpret_cast<uint4*>(pb) = make_uint4(h.x ^ neg, h.y ^ neg, h.z ^ neg, h.w ^ neg);
                *reinterpret_cast<uint4*>(pb + kPartB) = make_uint4(l.x ^ neg, l.y ^ neg, l.z ^ neg, l.w ^ neg);
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&S.wave_empty[s]);
                mbar_arrive(&S.full[buf]);
            }
        }
        __syncwarp();
    } else if (warp == kDrain + kProd + kStage) {
        // ---------------- MMA issue ----------------
        if (lane == 0) {
            // f16 operands (format 0), both MN-major, f32 accumulator
            const uint32_t id = (1u << 4) | (3u << 15) | ((uint32_t)(2 * N >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
            int ch = 0;
            for (; ch < nchunk; ch++) {
                const int buf = ch % kBufs, acc = ch & 1;
                bool ok = !S.abort && mbar_wait(&S.full[buf], (uint32_t)((ch / kBufs) & 1));
                if (ok && ch >= 2) ok = mbar_wait(&S.acc_empty[acc], (uint32_t)((ch / 2 - 1) & 1));
                if (!ok) {
                    S.abort = 1;
                    break;
                }
                tc_fence_after();
                const uint32_t a = smem_u32(smem + buf * kBufBytes), bim = a + 4 * kPartA, bre = bim + nB * kGroup;
                const uint32_t d = tmem + (uint32_t)acc * 128u;
                // parts of L: 0 re hi, 1 re lo, 2 im hi, 3 im lo; 16 waves are two core matrices
                auto mul = [&](int pa, uint32_t b, uint32_t more) {
#pragma unroll
                    for (int ks = 0; ks < kChunk / 16; ks++)
                        umma<1>(d, make_desc(a + pa * kPartA + ks * 256, 128, kGroup), make_desc(b + ks * 256, 128, kGroup), id,
                                more | (uint32_t)(ks > 0));
                };
                mul(1, bre, 0u);
                mul(0, bre + kPartB, 1u);
                mul(3, bim, 1u);
                mul(2, bim + kPartB, 1u);
                mul(0, bre, 1u);
                mul(2, bim, 1u);
                umma_commit(&S.empty[buf]);
                umma_commit(&S.acc_full[acc]);
            }
            // the accumulators must be idle before TMEM is freed
            for (int i = max(0, ch - 2); i < ch; i++) mbar_wait(&S.acc_full[i & 1], (uint32_t)((i / 2) & 1));
        }
        __syncwarp();
    } else {
        // -------- drain: warp w reads TMEM lanes 32 (w % 4) .., rows j 32 (w / 4) .. + 31 --------
        const int quarter = warp & 3, half = warp >> 2;
        const uint32_t tb = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * 32);
        const bool busy = half * 32 < N;
        const int r = quarter * 32 + lane, comp = r / kTileI;
        F2 re[16], im[16];                    // columns 2 c and 2 c + 1
#pragma unroll
        for (int c = 0; c < 16; c++) re[c].v = im[c].v = 0;
        for (int ch = 0; ch < nchunk; ch++) {
            const int buf = ch & 1, s = ch % kWaveSlots;
            int stop = S.abort;
            if (!stop && !(mbar_wait(&S.wave_full[s], (uint32_t)((ch / kWaveSlots) & 1)) &&
                           mbar_wait(&S.acc_full[buf], (uint32_t)((ch / 2) & 1))))
                stop = 1;
            if (__any_sync(0xffffffffu, stop)) {
                S.abort = 1;
                break;
            }
            tc_fence_after();
            const F2 sc = both(S.scale[s][min(comp, 2)]);
            if (busy) {
#pragma unroll
                for (int c8 = 0; c8 < 32; c8 += 8) {
                    if (half * 32 + c8 < N) {
                        uint32_t v[8];
                        tmem_ld8(tb + (uint32_t)buf * 128u + c8, v);
                        tmem_ld_wait8(v);
#pragma unroll
                        for (int c = 0; c < 4; c++)
                            re[c8 / 2 + c] = fma2(pack(__uint_as_float(v[2 * c]), __uint_as_float(v[2 * c + 1])), sc, re[c8 / 2 + c]);
                        tmem_ld8(tb + (uint32_t)buf * 128u + (uint32_t)(N + c8), v);
                        tmem_ld_wait8(v);
#pragma unroll
                        for (int c = 0; c < 4; c++)
                            im[c8 / 2 + c] = fma2(pack(__uint_as_float(v[2 * c]), __uint_as_float(v[2 * c + 1])), sc, im[c8 / 2 + c]);
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&S.acc_empty[buf]);
                mbar_arrive(&S.wave_empty[s]);
            }
            if (!kLong) continue;
            // the end of a run: into the sums in tensor memory, and these at the end (and every kMaxRun waves) into
            // the item's FP64 partial sums, each element always by this thread
            const bool due = (ch + 1) % (kMaxRun / kChunk) == 0, end = ch + 1 == nchunk;
            if (busy && (end || (ch + 1) % kRun == 0)) {
                const bool first = ch % (kMaxRun / kChunk) < kRun;          // nothing in the sums yet
                const uint32_t sum = tb + kSumCol;
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    // columns c8 .. c8 + 7 of re (even q) or im
                    const int c8 = q / 2 * 8, p = q & 1;
                    if (half * 32 + c8 < N) {
                        const uint32_t at = sum + (uint32_t)(c8 + 64 * p);
                        uint32_t hv[8], lv[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                        if (!first) {
                            tmem_ld8(at, hv);
                            tmem_ld8(at + kSumLow, lv);
                            tmem_ld_wait8(hv);
                            tmem_ld_wait8(lv);
                        }
#pragma unroll
                        for (int u = 0; u < 4; u++) {
                            F2& x = p ? im[c8 / 2 + u] : re[c8 / 2 + u];
                            F2 hi = x;
                            if (!first) {
                                hi = pack(__uint_as_float(hv[2 * u]), __uint_as_float(hv[2 * u + 1]));
                                F2 lo = pack(__uint_as_float(lv[2 * u]), __uint_as_float(lv[2 * u + 1]));
                                add_exact2(hi, lo, x);
                                lv[2 * u] = __float_as_uint(lo.x());
                                lv[2 * u + 1] = __float_as_uint(lo.y());
                            }
                            hv[2 * u] = __float_as_uint(hi.x());
                            hv[2 * u + 1] = __float_as_uint(hi.y());
                            x.v = 0;
                        }
                        tmem_st8(at, hv);
                        tmem_st8(at + kSumLow, lv);
                    }
                }
                tmem_st_wait();
                if (end || (due && S.item.slot >= 0)) {
                    const bool add = ch >= kMaxRun / kChunk;
                    const int slot = S.item.slot, jr0 = S.item.jr0, i0 = S.item.i0, rows = min(32, S.item.jr1 - jr0 - half * 32);
                    const int Ni = S.plane.Ni;
                    const int i = r - comp * kTileI;
                    const bool out = comp < 3 && i < min(kTileI, Ni - i0);
                    float2* E = reinterpret_cast<float2*>(S.plane.out) + ((long long)(jr0 + half * 32) * Ni + i0 + i) * 3 + comp;
                    double2* o = partials + ((long long)slot * kTileJ + half * 32) * (3 * kTileI) + r;
#pragma unroll 1
                    for (int c4 = 0; c4 < rows; c4 += 4, E += 12 * Ni, o += 4 * 3 * kTileI) {
                        uint32_t xh[4], xl[4], yh[4], yl[4];
                        tmem_ld4(sum + c4, xh);
                        tmem_ld4(sum + c4 + kSumLow, xl);
                        tmem_ld4(sum + c4 + 64, yh);
                        tmem_ld4(sum + c4 + 64 + kSumLow, yl);
                        tmem_ld_wait4(xh);
                        tmem_ld_wait4(xl);
                        tmem_ld_wait4(yh);
                        tmem_ld_wait4(yl);
#pragma unroll
                        for (int u = 0; u < 4; u++) {
                            if (c4 + u >= rows || !out) continue;
                            const float ah = __uint_as_float(xh[u]), al = low_word(ah, __uint_as_float(xl[u]));
                            const float bh = __uint_as_float(yh[u]), bl = low_word(bh, __uint_as_float(yl[u]));
                            if (slot < 0) {
                                E[(long long)u * 3 * Ni] = make_float2(ah + al, bh + bl);
                            } else {
                                double2* q = o + u * 3 * kTileI;
                                double2 v = make_double2((double)ah, (double)bh);
                                if (!first) v = make_double2(v.x + (double)al, v.y + (double)bl);
                                if (add) v = make_double2(q->x + v.x, q->y + v.y);
                                *q = v;
                            }
                        }
                    }
                }
            }
        }
        const int i = r - comp * kTileI;
        if ((!kLong || nchunk == 0) && comp < 3 && i < ncol && !S.abort) {
            // one run (or no wave at all): from the registers
#pragma unroll
            for (int c = 0; c < 32; c++) {
                const int j = half * 32 + c;
                if (j < nrow) {
                    const float x = c & 1 ? re[c / 2].y() : re[c / 2].x(), y = c & 1 ? im[c / 2].y() : im[c / 2].x();
                    if (it.slot >= 0)
                        partials[((long long)it.slot * kTileJ + j) * (3 * kTileI) + r] = make_double2((double)x, (double)y);
                    else
                        reinterpret_cast<float2*>(g.out)[((long long)(it.jr0 + j) * g.Ni + it.i0 + i) * 3 + comp] = make_float2(x, y);
                }
            }
        }
    }
    __syncthreads();
    if (tid == 0 && S.abort) atomicExch(err, 1);
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, kLong ? kCols : kSumCol);
    }
}

__global__ void __launch_bounds__(128)
plain_tc_reduce_kernel(const Plane* __restrict__ planes, const Tile* __restrict__ tiles, const double2* __restrict__ partials) {
    const Tile t = tiles[blockIdx.x];
    const Plane g = planes[t.plane];
    const int r = threadIdx.x, j = blockIdx.y;
    const int comp = r / kTileI, i = r - comp * kTileI;
    if (j >= t.jr1 - t.jr0 || comp >= 3 || i >= g.Ni - t.i0) return;
    double x = 0.0, y = 0.0;
    const double2* p = partials + ((long long)t.slot0 * kTileJ + j) * (3 * kTileI) + r;
#pragma unroll 4
    for (int k = 0; k < t.nslots; k++) {
        const double2 v = p[(long long)k * kTileJ * 3 * kTileI];
        x += v.x;
        y += v.y;
    }
    reinterpret_cast<float2*>(g.out)[((long long)(t.jr0 + j) * g.Ni + t.i0 + i) * 3 + comp] = make_float2((float)x, (float)y);
}

scw_status launch(scw_ctx ctx, const Plane* planes, const Item* items, int nitems, const Tile* tiles, int ntiles, int max_rows,
                  long long longest, const Waves& W, double2* partials) {
    constexpr size_t smem = kBufs * kBufBytes + sizeof(Smem);
    static_assert(smem <= 227 * 1024, "shared memory of the plain evaluator");
    // items of one run each, as small evaluations have, go from registers to memory: 9604 waves on 30 x 60 x 10 points, 750 items,
    // take 94 us, by the kernel for long ones 121
    auto kernel = longest > kRun * kChunk ? plain_tc_kernel<true> : plain_tc_kernel<false>;
    SCW_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    scw_status st = ctx_tc_flag(ctx);
    if (st != SCW_OK) return st;
    {
        LaunchTimer lt(ctx, "plain_tc_kernel");
        kernel<<<nitems, kThreads, smem, ctx->stream>>>(planes, items, W, partials, ctx->tc_err);
    }
    SCW_CUDA_TRY(cudaGetLastError());
    ctx->launches++;
    if (ntiles) {
        LaunchTimer lt(ctx, "plain_tc_reduce_kernel");
        plain_tc_reduce_kernel<<<dim3(ntiles, max_rows), 128, 0, ctx->stream>>>(planes, tiles, partials);
        SCW_CUDA_TRY(cudaGetLastError());
        ctx->launches++;
    }
    return SCW_OK;
}

}  // namespace ptc
}  // namespace scw
