// FP32 Schur form of complex Hessenberg matrices: the QR stage of the mixed-precision eigen-solver.
//
// Small-bulge multishift QR with aggressive early deflation (Braman, Byers and Mathias, SIAM J. Matrix
// Anal. Appl. 23 (2002) 929-973, parts I and II), arranged for one thread-block cluster per matrix:
//   * Rank 0 (the leader) takes the trailing kNW x kNW window of the active block into shared memory,
//     brings it to Schur form there, and deflates every eigenvalue whose spike entry is negligible
//     (moved to the bottom by swaps; the others serve as shifts).  Blocks of at most kNW are
//     finished this way.
//   * A sweep chases a chain of kM single-shift bulges, two rows apart: rotation k of bulge b runs at
//     step t = k - l + 2 b, so the rotations of one step act on disjoint row and column pairs.  A
//     window of kStep steps touches kW = 64 consecutive rows; the leader runs it in shared memory,
//     a warp per bulge, two barriers per step.
//   * The kM x kStep rotations of a window are then applied to everything outside it (columns to the
//     right, rows above, Schur vectors), a thread per vector of 64 values staged in shared memory, four
//     bulges per pass over the vector.  The leader applies them to the columns that the next
//     window needs and goes on chasing; the other CTAs of the cluster do the rest meanwhile.
// What bounds it: at n = 648 half of the time is the serial QR of the deflation windows (44 of them, 0.18 ms
// each) and a third the leader's chase (290 windows of 512 rotations, 18 us each).  Measured: 18.2 ms for
// 20 matrices of n = 648 on clusters of 6 CTAs, 3.76 ms for 10 of n = 216, 0.58 ms for 4 of n = 50; with the deflation
// window's column operations after each sweep 2.2, 0.7 and 0.14 more; a chase of one bulge at a time (800 clocks per
// rotation, no deflation windows) took 316 and 23.6 ms.
// H and Z are read through L2 (ld.global.cg): other CTAs of the cluster write them between barriers.
#include <algorithm>
#include <atomic>
#include <cmath>

#include <cooperative_groups.h>

#include "scw_complex.cuh"
#include "scw_dense.h"

namespace scw {
namespace z {

constexpr int kM = 16;            // bulges per sweep (warps of the CTA)
constexpr int kStep = 32;         // steps per window
constexpr int kW = 64;            // rows of a window: 2 (kM - 1) + kStep + 2
constexpr int kLd = kW + 1;       // odd: row and column walks without bank conflicts
constexpr int kNW = 32;           // deflation window
constexpr int kLdn = kNW + 1;
constexpr int kQrThreads = kM * 32;
constexpr int kVec = 320;         // vectors staged per pass of the update
static_assert(2 * (kM - 1) + kStep + 2 == kW, "window geometry");

struct QrRot {                    // rotations of one step for four bulges
    float c[4];
    float2 s[4];
};

struct QrSmem {
    float2 T[kW * kLd];                       // chase window (column u at u + 1), or the deflation window
    float2 V[kNW * kLdn];                     // its Schur vectors
    QrRot rot[2][kStep][kM / 4];
    float2 vec[kVec * kLd];                   // staged vectors of the updates
    float2 shift[kNW], refl[kNW];
    float4 lr[2][kNW];                        // rotations c, s of the deflation window's sweeps (two in flight)
    int ll[2], ln[2], wl, wh, wbuf;           // sweeps for warp 1, the current one for warp 2
    int cmd[8];                               // op, l, hi, shifts | op, kw, nw
    int red[kM];
    float2 spike;
    int ns, fail;
};

enum : int { kOpEnd = 0, kOpDeflate = 1, kOpSweep = 2 };

__device__ __forceinline__ void rot32_rows(float c, float2 s, float2& x, float2& y) {
    const float2 nx = make_float2(c * x.x + (s.x * y.x - s.y * y.y), c * x.y + (s.x * y.y + s.y * y.x));
    const float2 ny = make_float2(c * y.x - (s.x * x.x + s.y * x.y), c * y.y - (s.x * x.y - s.y * x.x));
    x = nx;
    y = ny;
}
__device__ __forceinline__ float2 conjf2(float2 s) { return make_float2(s.x, -s.y); }

// The power of two that brings a largest value `big` to [1, 2), and its inverse (within what a float can be scaled by).
__device__ __forceinline__ void unit_scale(float big, float& up, float& back) {
    const int e = min(max((int)(__float_as_uint(big) >> 23), 1), 253);
    up = __uint_as_float((unsigned)(254 - e) << 23);
    back = __uint_as_float((unsigned)e << 23);
}

// rotation (c, s) with [c, s; -conj(s), c] [f; g] = [r; 0], from two reciprocal square roots of scaled values: the squares
// of values near the ends of the range would leave it, or lose the digits that make the rotation unitary
__device__ __forceinline__ void givens32(float2 f, float2 g, float& c, float2& s, float2& r) {
    float up, back;
    unit_scale(fmaxf(fmaxf(fabsf(f.x), fabsf(f.y)), fmaxf(fabsf(g.x), fabsf(g.y))), up, back);
    const float2 fu = make_float2(f.x * up, f.y * up), gu = make_float2(g.x * up, g.y * up);
    const float gf = cabs2(gu), ff = cabs2(fu);
    if (gf < 1e-30f) {                        // |g| < 1e-15 |f|, or both zero
        c = 1.f;
        s = make_float2(0.f, 0.f);
        r = f;
        return;
    }
    if (ff < 1e-30f) {
        const float ig = rsqrtf(gf);
        c = 0.f;
        s = make_float2(gu.x * ig, -gu.y * ig);
        r = make_float2(gf * ig * back, 0.f);
        return;
    }
    const float iaf = rsqrtf(ff), id = rsqrtf(ff + gf);
    c = ff * iaf * id;
    const float2 fs = make_float2(fu.x * iaf, fu.y * iaf);
    const float2 t = cmulc(gu, fs);
    s = make_float2(t.x * id, t.y * id);
    const float d = (ff + gf) * id * back;
    r = make_float2(fs.x * d, fs.y * d);
}

// The same where no branch is needed but for values near the ends of the range.
__device__ __forceinline__ float rsqrt_fast(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ void givens32_fast(float2 f, float2 g, float& c, float2& s, float2& r) {
    const float gf = cabs2(g), ff = cabs2(f), sum = ff + gf;
    if (fminf(gf, ff) < 1e-30f || sum > 1e36f) {
        givens32(f, g, c, s, r);
        return;
    }
    const float iaf = rsqrt_fast(ff), id = rsqrt_fast(sum);
    const float2 fs = make_float2(f.x * iaf, f.y * iaf);
    const float2 t = cmulc(g, fs);
    c = ff * iaf * id;
    s = make_float2(t.x * id, t.y * id);
    const float d = sum * id;
    r = make_float2(fs.x * d, fs.y * d);
}

// Wilkinson's shift of the trailing 2 x 2 block; exceptional ones every 10 iterations (zlahqr's rule).
// Approximate square root and division: a shift need not be exact.
__device__ __forceinline__ float2 shift32(const float2* T, int ld, int l, int ihi, int its) {
    const float2 d = T[ihi * ld + ihi];
    if (its % 20 == 0) return make_float2(0.75f * fabsf(T[ihi * ld + ihi - 1].x) + d.x, d.y);
    if (its % 10 == 0) {
        const float2 a = T[l * ld + l];
        return make_float2(0.75f * fabsf(T[(l + 1) * ld + l].x) + a.x, a.y);
    }
    const float2 a = T[(ihi - 1) * ld + ihi - 1], b = T[(ihi - 1) * ld + ihi], c = T[ihi * ld + ihi - 1];
    // scaled by a power of two to about 1: the root is of the entries' fourth powers
    const float2 h0 = make_float2(0.5f * (a.x - d.x), 0.5f * (a.y - d.y));
    const float big = fmaxf(fmaxf(fmaxf(fabsf(h0.x), fabsf(h0.y)), fmaxf(fabsf(b.x), fabsf(b.y))), fmaxf(fabsf(c.x), fabsf(c.y)));
    float up, back;
    unit_scale(big, up, back);
    auto scaled = [&](float2 v) { return make_float2(v.x * up, v.y * up); };
    const float2 half = scaled(h0);
    const float2 bc = cmul(scaled(b), scaled(c));
    const float2 q = cfma(half, half, bc);
    const float m2 = cabs2(q);
    float2 sq = make_float2(0.f, 0.f);
    if (m2 > 0.f) {                                     // principal root: the larger part first
        const float t2 = 0.5f * (fabsf(q.x) + m2 * rsqrtf(m2)), it = rsqrtf(t2), t = t2 * it, o = 0.5f * q.y * it;
        sq = q.x >= 0.f ? make_float2(t, o) : make_float2(fabsf(o), copysignf(t, q.y));
    }
    const float2 e1 = cadd(half, sq), e2 = csub(half, sq);
    const float2 den = cabs2(e1) >= cabs2(e2) ? e1 : e2;
    const float dd = cabs2(den);
    if (dd == 0.f) return d;
    const float2 x = cmulc(den, bc);                    // bc / den
    return make_float2(fmaf(-back, __fdividef(x.x, dd), d.x), fmaf(-back, __fdividef(x.y, dd), d.y));
}

// hqr_deflates of the window's entry (k, k - 1), all entries loaded at once and without exact divisions
__device__ __forceinline__ bool window_deflates(const float2* T, int k, int ihi) {
    const float2 a = T[k * kLdn + k - 1], d = T[k * kLdn + k], p = T[(k - 1) * kLdn + k - 1], u = T[(k - 1) * kLdn + k];
    const float ulp = CT<float2>::ulp, small = CT<float2>::safmin * ((float)kLdn / ulp);
    const float a1 = cabs1(a), u1 = cabs1(u), d1 = cabs1(d), dd = cabs1(csub(p, d)), tst = cabs1(p) + d1;
    if (tst == 0.f) return hqr_deflates<float2, false>(T, kLdn, k, ihi);
    const float ab = fmaxf(a1, u1), ba = fminf(a1, u1), aa = fmaxf(d1, dd), bb = fminf(d1, dd), is = __fdividef(1.f, aa + ab);
    const bool far = ba * (ab * is) <= fmaxf(small, ulp * (bb * (aa * is))) || ba * ab <= (ulp * d1) * (ulp * d1);
    return a1 <= small || (a1 <= ulp * tst && far);
}

// The rotations of a sweep over columns l .. l + cnt - 1, in order, on row `row` of X from column ks on: a
// lane per row, the running value in a register, the values four columns ahead already loaded.
__device__ __forceinline__ void sweep_columns(float2* X, int row, bool live, int ks, int l, int cnt, const float4* rot) {
    float2* p = X + row * kLdn;
    const int k1 = l + cnt;
    float2 x = live && ks < k1 ? p[ks] : make_float2(0.f, 0.f);
    for (int k = l; k < k1; k += 4) {
        float2 y[4];
#pragma unroll
        for (int i = 0; i < 4; i++) y[i] = live && k + i >= ks && k + i < k1 ? p[k + i + 1] : make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (k + i < k1) {
                const float4 g = rot[k + i - l];
                const float cc = g.x;
                const float2 ss = make_float2(g.y, -g.z);
                if (live && k + i >= ks) {
                    rot32_rows(cc, ss, x, y[i]);
                    p[k + i] = x;
                    x = y[i];
                }
            }
        }
    }
    if (live && ks < k1) p[k1] = x;
}

// Householder vector of x (x_0 in lane 0 .., zero from lane cnt on): returns tau, beta in lane 0's terms; x
// becomes w with w_0 = 1.  (I - tau w w^H)^H x = beta e_0.
__device__ __forceinline__ void reflector32(float2& x, int lane, int cnt, float2& tau, float& beta, bool& none) {
    float up, back;                            // (scaled, as in givens32)
    unit_scale(__uint_as_float(__reduce_max_sync(0xffffffffu, lane < cnt ? __float_as_uint(fmaxf(fabsf(x.x), fabsf(x.y))) : 0u)), up, back);
    x = make_float2(x.x * up, x.y * up);
    float n2 = (lane >= 1 && lane < cnt) ? cabs2(x) : 0.f;
    for (int o = 16; o > 0; o >>= 1) n2 += __shfl_xor_sync(0xffffffffu, n2, o);
    const float ax = __shfl_sync(0xffffffffu, x.x, 0), ay = __shfl_sync(0xffffffffu, x.y, 0);
    none = n2 == 0.f && ay == 0.f;
    if (none) {
        tau = make_float2(0.f, 0.f);
        beta = ax * back;
        return;
    }
    beta = -copysignf(sqrtf(ax * ax + ay * ay + n2), ax);
    tau = make_float2((beta - ax) / beta, -ay / beta);
    const float2 scal = cdiv(make_float2(1.f, 0.f), make_float2(ax - beta, ay));
    x = lane == 0 ? make_float2(1.f, 0.f) : lane < cnt ? cmul(x, scal) : make_float2(0.f, 0.f);
    beta *= back;
}

__device__ __forceinline__ void pair_sync() { asm volatile("bar.sync 1, 64;" ::: "memory"); }
// warp 0 announces, warp 2 waits; the barriers 2 .. 12 are used once per sweep each
constexpr int kColGroup = 3, kColDone = 14;
static_assert(2 + (kNW - 2) / kColGroup < kColDone, "named barriers");
__device__ __forceinline__ void bar_arrive(int id) { asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory"); }
__device__ __forceinline__ void bar_wait(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }

// Schur form of the nw x nw Hessenberg window T with vectors V (warps 0 .. 2), then deflation against the
// spike s, the Hessenberg form of what is left (warp 0).  Sets S.ns (undeflated, at the top), S.shift (their
// eigenvalues) and S.fail.
//
// A sweep is one chain of rotations, so its latency per rotation is what counts.  Lane j carries column
// j of the row that the chase is at: row operations need no shared-memory round trip.  What the next
// rotation is made of (columns k, k + 1 of the rows k .. k + 2) every lane computes for itself, from the
// diagonal and subdiagonal entries, loaded ahead, and one value of row k, whose shuffle overlaps the
// rotation's square roots.  Warp 2 applies the column operations to the rows above, a lane per row, three
// rotations behind, and warp 1 those of the sweep before to V.  A rotation takes 305 clocks (106 the
// rotation itself, 60 what the next is made of, 120 the rows and their stores); with those columns from shuffles in the
// chain and the column operations after the sweep 317 + 143, through shared memory 550.
__device__ void deflation_window(QrSmem& S, int nw) {
    const int lane = threadIdx.x & 31;
    float2 *T = S.T, *V = S.V;
    if (threadIdx.x >= 64) {
        while (true) {
            bar_wait(2);
            const int l = S.wl, hi = S.wh;
            if (hi < 0) return;
            const float4* rot = S.lr[S.wbuf];
            float2 x = make_float2(0.f, 0.f);
            float2* row = T + lane * kLdn;
            for (int q = 0, k = l;; q++) {
                if (q > 0) bar_wait(2 + q);
                // rows up to k + i are complete, each takes part from its own column on
                float2 y[kColGroup], d[kColGroup];
                float4 g[kColGroup];
#pragma unroll
                for (int i = 0; i < kColGroup; i++) {
                    const int kk = min(k + i, hi - 1);
                    y[i] = lane <= kk ? row[kk + 1] : make_float2(0.f, 0.f);
                    d[i] = lane <= kk ? row[kk] : make_float2(0.f, 0.f);
                    g[i] = rot[kk - l];
                }
#pragma unroll
                for (int i = 0; i < kColGroup; i++) {
                    if (k + i < hi && lane <= k + i) {
                        if (lane == k + i || k + i == l) x = d[i];
                        rot32_rows(g[i].x, make_float2(g[i].y, -g[i].z), x, y[i]);
                        row[k + i] = x;
                        x = y[i];
                    }
                }
                k += kColGroup;
                if (k >= hi) break;
            }
            if (lane < hi) row[hi] = x;
            __syncwarp();
            bar_wait(kColDone);
        }
    }
    if (threadIdx.x >= 32) {
        for (int i = 0; i < nw; i++) V[i * kLdn + lane] = make_float2(i == lane ? 1.f : 0.f, 0.f);
        __syncwarp();
        for (int q = 0;; q ^= 1) {
            pair_sync();
            const int cnt = S.ln[q], l = S.ll[q];
            if (cnt < 0) return;
            sweep_columns(V, lane, lane < nw, l, l, cnt, S.lr[q]);
            __syncwarp();
        }
    }
    // single-shift QR
    int ihi = nw - 1, its = 0, total = 0, buf = 0;
    bool fail = false;
    while (ihi >= 0) {
        const bool d = lane >= 1 && lane <= ihi && window_deflates(T, lane, ihi);
        const unsigned mask = __ballot_sync(0xffffffffu, d);
        const int l = mask ? 31 - __clz(mask) : 0;
        if (l > 0 && lane == 0) T[l * kLdn + l - 1] = make_float2(0.f, 0.f);
        __syncwarp();
        if (l >= ihi) {
            ihi = l - 1;
            its = 0;
            continue;
        }
        if (total > 30 * kNW) {
            fail = true;
            break;
        }
        its++;
        total++;
        const float2 shift = shift32(T, kLdn, l, ihi, its);
        const float2 zero = make_float2(0.f, 0.f);
        if (lane == 0) {
            S.wl = l;
            S.wh = ihi;
            S.wbuf = buf;
        }
        // R: row k of column `lane` with the rotations so far, N, M: rows k + 1 and k + 2; (k, k), (k + 1, k) and
        // (k + 1, k + 1), (k + 2, k + 1) in every lane, the latter two without rotations.  What is read past row
        // ihi or column nw stays in T's storage and reaches nothing that is kept.
        const bool live = lane < nw;
        float2 R = T[l * kLdn + lane], N = T[(l + 1) * kLdn + lane], M = T[(l + 2) * kLdn + lane];
        float2 Rk = T[l * kLdn + l], Nk = T[(l + 1) * kLdn + l];
        float2 n1 = T[(l + 1) * kLdn + l + 1], m1 = T[(l + 2) * kLdn + l + 1];
        float2 f = csub(Rk, shift), g = Nk;
        __syncwarp();
        // rotation k on R, N; R then takes row k + 3.  true: the sweep's last
        auto step = [&](int k, float2& R, float2& N, float2& M) {
            const float2* next = T + (k + 2) * kLdn + k + 2;
            const float2 r1 = make_float2(__shfl_sync(0xffffffffu, R.x, k + 1), __shfl_sync(0xffffffffu, R.y, k + 1));
            const float2 n2 = next[0], m2 = next[kLdn];
            float2 s, r;
            float c;
            givens32_fast(f, g, c, s, r);
            // columns k, k + 1 of row k + 1 with this rotation from both sides, and of row k + 2 (zero, m1)
            float2 a = make_float2(c * Nk.x - (s.x * Rk.x + s.y * Rk.y), c * Nk.y - (s.x * Rk.y - s.y * Rk.x));
            float2 b = make_float2(c * n1.x - (s.x * r1.x + s.y * r1.y), c * n1.y - (s.x * r1.y - s.y * r1.x));
            rot32_rows(c, conjf2(s), a, b);
            f = a;
            g = cmulc(s, m1);
            Rk = b;
            Nk = make_float2(c * m1.x, c * m1.y);
            n1 = n2;
            m1 = m2;
            rot32_rows(c, s, R, N);                 // R: row k done, N: row k + 1
            if (live && lane >= max(k - 1, l)) T[k * kLdn + lane] = lane == k - 1 ? r : R;
            if (lane == 0) S.lr[buf][k - l] = make_float4(c, s.x, s.y, 0.f);
            R = T[(k + 3) * kLdn + lane];
            if (lane == k + 1) {
                N = b;
                M = make_float2(c * M.x, c * M.y);
            }
            if (k + 1 < ihi) return false;
            if (lane >= ihi && live) T[ihi * kLdn + lane] = N;
            if (lane == ihi - 1) T[ihi * kLdn + lane] = f;
            return true;
        };
        static_assert(kColGroup == 3, "a group is one turn of the three rows");
        for (int k = l, group = 2;; k += 3, group++) {
            const bool end = step(k, R, N, M) || step(k + 1, N, M, R) || step(k + 2, M, R, N);
            __syncwarp();
            bar_arrive(group);
            if (end) break;
        }
        if (lane == 0) {
            S.ll[buf] = l;
            S.ln[buf] = ihi - l;
        }
        __syncwarp();
        pair_sync();
        bar_wait(kColDone);
        buf ^= 1;
    }
    if (lane == 0) {
        S.ln[buf] = -1;
        S.wh = -1;
    }
    __syncwarp();
    bar_arrive(2);
    pair_sync();                                    // V is complete
    // From the bottom up: an eigenvalue with a negligible spike entry is moved down past those that stay
    // and deflated there.
    const float2 sp = S.spike;
    const float asp = cabs1(sp);
    int ns = nw;
    if (asp == 0.f) {
        ns = 0;
    } else {
        const float small = CT<float2>::safmin * ((float)nw / CT<float2>::ulp);
        auto negligible = [&](int i) {
            float foo = cabs1(T[i * kLdn + i]);
            if (foo == 0.f) foo = asp;
            return asp * cabs1(V[i]) <= fmaxf(small, CT<float2>::ulp * foo);
        };
        for (int i = nw - 1; i >= 0; i--) {
            if (!negligible(i)) continue;
            for (int k = i; k + 1 < ns; k++) {         // swap the eigenvalues k and k + 1
                const float2 t11 = T[k * kLdn + k], t12 = T[k * kLdn + k + 1], t22 = T[(k + 1) * kLdn + k + 1];
                // rows k, k + 1 right of them (lane: column), columns k, k + 1 above them (lane: row)
                const bool right = lane >= k + 2 && lane < nw, above = lane < k;
                float2 *px = right ? T + k * kLdn + lane : T + lane * kLdn + k;
                float2 *py = right ? px + kLdn : px + 1;
                float2 x = make_float2(0.f, 0.f), y = x, vx = x, vy = x;
                if (right || above) {
                    x = *px;
                    y = *py;
                }
                if (lane < nw) {
                    vx = V[lane * kLdn + k];
                    vy = V[lane * kLdn + k + 1];
                }
                float c;
                float2 s, r;
                givens32(t12, csub(t22, t11), c, s, r);
                __syncwarp();
                rot32_rows(c, right ? s : conjf2(s), x, y);
                rot32_rows(c, conjf2(s), vx, vy);
                if (right || above) {
                    *px = x;
                    *py = y;
                }
                if (lane == k) {
                    T[k * kLdn + k] = t22;
                    T[(k + 1) * kLdn + k + 1] = t11;
                }
                if (lane < nw) {
                    V[lane * kLdn + k] = vx;
                    V[lane * kLdn + k + 1] = vy;
                }
                __syncwarp();
            }
            if (negligible(ns - 1)) ns--;
        }
    }
    if (lane < ns) S.shift[lane] = T[lane * kLdn + lane];
    if (lane == 0) {
        S.ns = ns;
        S.fail = fail;
    }
    __syncwarp();
    if (ns == nw || ns <= 1 || fail) return;
    // the spike s conj(V(0, :)) of the undeflated part back to its first entry, then Hessenberg form:
    // reflectors of column p act on rows / columns p + 1 .. ns - 1 (p = -1: the spike, 0 .. ns - 1)
    for (int p = -1; p + 2 < ns; p++) {
        const int o = p + 1, cnt = ns - o;             // reflector entries i -> row o + i, lane i
        float2 w = make_float2(0.f, 0.f);
        if (lane < cnt) w = p < 0 ? conjf2(V[lane]) : T[(o + lane) * kLdn + p];
        float2 tau;
        float beta;
        bool none;
        reflector32(w, lane, cnt, tau, beta, none);
        if (none) continue;                            // uniform
        S.refl[lane] = w;
        __syncwarp();
        if (p >= 0 && lane < cnt) T[(o + lane) * kLdn + p] = lane == 0 ? make_float2(beta, 0.f) : make_float2(0.f, 0.f);
        // left, H^H T: lane = column (p + 1 .. nw - 1)
        if (lane >= max(o, 0) && lane < nw) {
            float2 d = make_float2(0.f, 0.f);
            for (int i = 0; i < cnt; i++) d = cfma(conjf2(S.refl[i]), T[(o + i) * kLdn + lane], d);
            d = cmul(conjf2(tau), d);
            for (int i = 0; i < cnt; i++) T[(o + i) * kLdn + lane] = csub(T[(o + i) * kLdn + lane], cmul(S.refl[i], d));
        }
        __syncwarp();
        // right, T H: lane = row (0 .. ns - 1); V H: all rows
        if (lane < ns) {
            float2 d = make_float2(0.f, 0.f);
            for (int i = 0; i < cnt; i++) d = cfma(T[lane * kLdn + o + i], S.refl[i], d);
            d = cmul(tau, d);
            for (int i = 0; i < cnt; i++)
                T[lane * kLdn + o + i] = csub(T[lane * kLdn + o + i], cmul(d, conjf2(S.refl[i])));
        }
        if (lane < nw) {
            float2 d = make_float2(0.f, 0.f);
            for (int i = 0; i < cnt; i++) d = cfma(V[lane * kLdn + o + i], S.refl[i], d);
            d = cmul(tau, d);
            for (int i = 0; i < cnt; i++)
                V[lane * kLdn + o + i] = csub(V[lane * kLdn + o + i], cmul(d, conjf2(S.refl[i])));
        }
        __syncwarp();
    }
}

// Steps t0 .. t0 + kStep - 1 of the chain in shared memory; rotations into rot, the window back to H.
__device__ void chase32(QrSmem& S, float2* __restrict__ H, int n, int l, int ihi, int t0, int ms, QrRot (*rot)[kM / 4]) {
    const int tid = threadIdx.x, b = tid >> 5, lane = tid & 31;
    const int vb = l + t0 - 2 * (kM - 1);
    const int lo = max(l, vb), hi = min(ihi, vb + kW - 1);
    const int c0 = lo > l ? lo - 1 : lo;              // with the column left of the window
    float2* T = S.T;
    const int nr = hi - lo + 1, nc = hi - c0 + 1;
    for (int e = tid; e < nr * nc; e += kQrThreads) {
        const int i = e / nc, j = e - i * nc;
        T[(lo - vb + i) * kLd + (c0 - vb + j) + 1] = __ldcg(H + (long long)(lo + i) * n + c0 + j);
    }
    const float2 sigma = b < ms ? S.shift[b] : make_float2(0.f, 0.f);
    const int uhi = hi - vb, ulo = lo - vb;
    __syncthreads();
#define TT(i, j) T[(i) * kLd + (j) + 1]
    for (int tt = 0; tt < kStep; tt++) {
        const int k = l + t0 + tt - 2 * b, u = tt + 2 * (kM - 1 - b);
        const bool act = b < ms && k >= l && k < ihi;
        float c = 1.f;
        float2 s = make_float2(0.f, 0.f);
        if (act) {
            float2 f, g, r;
            if (k == l) {
                f = csub(TT(u, u), sigma);
                g = TT(u + 1, u);
            } else {
                f = TT(u, u - 1);
                g = TT(u + 1, u - 1);
            }
            givens32_fast(f, g, c, s, r);
            __syncwarp();
            if (lane == 0 && k > l) {
                TT(u, u - 1) = r;
                TT(u + 1, u - 1) = make_float2(0.f, 0.f);
            }
            for (int j = u + lane; j <= uhi; j += 32) rot32_rows(c, s, TT(u, j), TT(u + 1, j));
        }
        if (lane == 0) {
            rot[tt][b >> 2].c[b & 3] = c;
            rot[tt][b >> 2].s[b & 3] = s;
        }
        __syncthreads();
        if (act) {
            const int umax = min(k + 2, ihi) - vb;
            for (int i = ulo + lane; i <= umax; i += 32) rot32_rows(c, conjf2(s), TT(i, u), TT(i, u + 1));
        }
        __syncthreads();
    }
#undef TT
    for (int e = tid; e < nr * nc; e += kQrThreads) {
        const int i = e / nc, j = e - i * nc;
        H[(long long)(lo + i) * n + c0 + j] = T[(lo - vb + i) * kLd + (c0 - vb + j) + 1];
    }
}

// A window's rotations on the columns j0 .. j1-1 (rows lo .. hi of H) and on the rows r0 .. r1-1 of the
// list "rows 0 .. lo-1 of H, then the rows of Z" (columns lo .. hi), kVec vectors at a time.
__device__ void apply32(QrSmem& S, float2* __restrict__ H, float2* __restrict__ Z, int n, int vb, int lo, int hi, int j0,
                        int j1, int r0, int r1, const QrRot (*rot)[kM / 4]) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ncol = max(0, j1 - j0), nv = ncol + max(0, r1 - r0);
    const int ulo = lo - vb, cnt = hi - lo + 1;
    for (int v0 = 0; v0 < nv; v0 += kVec) {
        const int m = min(kVec, nv - v0), mc = max(0, min(ncol - v0, m));     // the first mc of them are columns
        __syncthreads();
        for (int e = tid; e < mc * cnt; e += kQrThreads) {
            const int u = e / mc, v = e - u * mc;
            S.vec[v * kLd + ulo + u] = __ldcg(H + (long long)(lo + u) * n + j0 + v0 + v);
        }
        for (int v = mc + warp; v < m; v += kM) {
            const int r = r0 + v0 + v - ncol;
            const float2* src = (r < lo ? H + (long long)r * n : Z + (long long)(r - lo) * n) + lo;
            for (int u = lane; u < cnt; u += 32) S.vec[v * kLd + ulo + u] = __ldcg(src + u);
        }
        __syncthreads();
        if (tid < m) {
            float2* p = S.vec + tid * kLd;
            const float sg = tid < mc ? 1.f : -1.f;    // columns of H rotate by s, rows by conj(s)
#pragma unroll 1
            for (int g = 0; g < kM / 4; g++) {
                // bulges 4 g .. 4 g + 3 act on (w6, w7), (w4, w5), (w2, w3), (w0, w1) of the eight values
                // from e0 + step on; value e sits in register e & 7
                const int e0 = 2 * (kM - 1) - 6 - 8 * g;
                float2 w[8];
#pragma unroll
                for (int i = 0; i < 8; i++) w[i] = p[e0 + i];
#pragma unroll 1
                for (int t8 = 0; t8 < kStep; t8 += 8) {
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const QrRot& q = rot[t8 + i][g];
                        const float4 c4 = *reinterpret_cast<const float4*>(q.c);
                        const float4 s01 = *reinterpret_cast<const float4*>(&q.s[0]);
                        const float4 s23 = *reinterpret_cast<const float4*>(&q.s[2]);
                        rot32_rows(c4.x, make_float2(s01.x, sg * s01.y), w[(i + 6) & 7], w[(i + 7) & 7]);
                        rot32_rows(c4.y, make_float2(s01.z, sg * s01.w), w[(i + 4) & 7], w[(i + 5) & 7]);
                        rot32_rows(c4.z, make_float2(s23.x, sg * s23.y), w[(i + 2) & 7], w[(i + 3) & 7]);
                        rot32_rows(c4.w, make_float2(s23.z, sg * s23.w), w[i & 7], w[(i + 1) & 7]);
                        p[e0 + t8 + i] = w[i & 7];
                        w[i & 7] = p[min(e0 + t8 + i + 8, kW)];
                    }
                }
                // the last loads run past the values the group rotates; seven of them stay in registers
#pragma unroll
                for (int i = 0; i < 7; i++) p[e0 + kStep + i] = w[i];
            }
        }
        __syncthreads();
        for (int e = tid; e < mc * cnt; e += kQrThreads) {
            const int u = e / mc, v = e - u * mc;
            H[(long long)(lo + u) * n + j0 + v0 + v] = S.vec[v * kLd + ulo + u];
        }
        for (int v = mc + warp; v < m; v += kM) {
            const int r = r0 + v0 + v - ncol;
            float2* dst = (r < lo ? H + (long long)r * n : Z + (long long)(r - lo) * n) + lo;
            for (int u = lane; u < cnt; u += 32) dst[u] = S.vec[v * kLd + ulo + u];
        }
    }
}

// The deflation window's V on this CTA's share of what lies outside it: columns right of the window
// (V^H times them) and rows above it and of Z (times V).  V is in S.V.
__device__ void deflation_update(QrSmem& S, float2* __restrict__ H, float2* __restrict__ Z, int n, int kw, int nw, int rank,
                                 int K) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int right = n - (kw + nw), rows = kw + n;
    const int jc = (right + K - 1) / K, rc = (rows + K - 1) / K;
    const int j0 = kw + nw + min(right, rank * jc), j1 = kw + nw + min(right, (rank + 1) * jc);
    const int r0 = min(rows, rank * rc), r1 = min(rows, (rank + 1) * rc);
    const int ncol = j1 - j0, nv = ncol + r1 - r0;
    // entries past nw read as zeros in both V and the vectors
    for (int v0 = 0; v0 < nv; v0 += kVec) {
        const int m = min(kVec, nv - v0), mc = max(0, min(ncol - v0, m));
        __syncthreads();
        for (int e = tid; e < mc * nw; e += kQrThreads) {
            const int u = e / mc, v = e - u * mc;
            S.vec[v * kLd + u] = __ldcg(H + (long long)(kw + u) * n + j0 + v0 + v);
        }
        for (int v = mc + warp; v < m; v += kM) {
            const int r = r0 + v0 + v - ncol;
            const float2* src = (r < kw ? H + (long long)r * n : Z + (long long)(r - kw) * n) + kw;
            if (lane < nw) S.vec[v * kLd + lane] = __ldcg(src + lane);
        }
        __syncthreads();
        if (tid < m) {
            float2* p = S.vec + tid * kLd;
            const float sg = tid < mc ? -1.f : 1.f;    // columns: conj(V)
            float2 x[kNW];
#pragma unroll
            for (int i = 0; i < kNW; i++) x[i] = i < nw ? p[i] : make_float2(0.f, 0.f);
#pragma unroll 1
            for (int j = 0; j < nw; j++) {
                float2 a = make_float2(0.f, 0.f);
#pragma unroll
                for (int i = 0; i < kNW; i++) {
                    const float2 v = S.V[i * kLdn + j];
                    a = cfma(x[i], make_float2(v.x, sg * v.y), a);
                }
                p[j] = a;
            }
        }
        __syncthreads();
        for (int e = tid; e < mc * nw; e += kQrThreads) {
            const int u = e / mc, v = e - u * mc;
            H[(long long)(kw + u) * n + j0 + v0 + v] = S.vec[v * kLd + u];
        }
        for (int v = mc + warp; v < m; v += kM) {
            const int r = r0 + v0 + v - ncol;
            float2* dst = (r < kw ? H + (long long)r * n : Z + (long long)(r - kw) * n) + kw;
            if (lane < nw) dst[lane] = S.vec[v * kLd + lane];
        }
    }
}

__global__ void __launch_bounds__(kQrThreads, 1)
hqr32_kernel(float2* __restrict__ H, float2* __restrict__ Z, int n, long long sA, float2* __restrict__ eig,
             int* __restrict__ status) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int K = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int mat = blockIdx.x / K;
    H += sA * mat;
    Z += sA * mat;
    eig += (long long)n * mat;
    extern __shared__ __align__(16) unsigned char qr_smem[];
    QrSmem& S = *reinterpret_cast<QrSmem*>(qr_smem);
    QrSmem* S0 = cluster.map_shared_rank(&S, 0);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // values of a staged vector outside the window (identity rotations run over them)
    for (int e = tid; e < kVec * kLd; e += kQrThreads) S.vec[e] = make_float2(0.f, 0.f);
    int ihi = n - 1, idle = 0, rounds = 0;              // rank 0's state
    int sweep_l = 0, sweep_hi = -1, sweep_ms = 0;       // rank 0: a sweep is due
    const int limit = 30 * max(10, n);
    // larger windows deflate more at a time, but their QR grows with the square (measured with 16, 20, 24, 28, 32 on layers: n =
    // 216 4.08, 3.79, 3.72, 3.95, 3.99 ms; n = 648 21.3, 19.4, 18.4, 17.7, 17.8 ms; between them on graded random matrices, 24 and 32:
    // n = 100 1.9, 2.1; 216 5.1, 5.3; 288 7.1, 7.5; 350 9.4, 9.8; 450 13.5, 14.1; 576 19.9, 20.8; 648 24.2, 25.0 ms.  Up to 400 both
    // kinds want 24; beyond, layers, which gain from more shifts, decide.)
    const int window = n < 400 ? 24 : kNW;
    while (true) {
        if (rank == 0) {
            int op = kOpEnd, a1 = 0, a2 = 0, a3 = 0;
            if (sweep_ms > 0) {
                op = kOpSweep;
                a1 = sweep_l;
                a2 = sweep_hi;
                a3 = sweep_ms;
                sweep_ms = 0;
            } else {
                while (ihi >= 0) {
                    __syncthreads();
                    // the largest k in [1, ihi] whose subdiagonal entry may be set to zero (0: none)
                    int lk = 0;
                    for (int k = ihi - tid; k > 0; k -= kQrThreads)
                        if (hqr_deflates<float2, true>(H, n, k, ihi)) {
                            lk = k;
                            break;
                        }
                    lk = __reduce_max_sync(0xffffffffu, lk);
                    if (lane == 0) S.red[warp] = lk;
                    __syncthreads();
                    int l = 0;
#pragma unroll
                    for (int w = 0; w < kM; w++) l = max(l, S.red[w]);
                    if (++rounds > limit) {
                        if (tid == 0) status[mat] = 1;
                        ihi = -1;
                        break;
                    }
                    const int size = ihi - l + 1, nw = size <= kNW ? size : window, kw = ihi - nw + 1;
                    for (int e = tid; e < nw * nw; e += kQrThreads) {
                        const int i = e / nw, j = e - i * nw;
                        S.T[i * kLdn + j] = j + 1 < i ? make_float2(0.f, 0.f) : __ldcg(H + (long long)(kw + i) * n + kw + j);
                    }
                    if (tid == 0) {
                        S.spike = kw > l ? __ldcg(H + (long long)kw * n + kw - 1) : make_float2(0.f, 0.f);
                        if (l > 0) H[(long long)l * n + l - 1] = make_float2(0.f, 0.f);
                    }
                    __syncthreads();
                    if (warp < 3) deflation_window(S, nw);
                    __syncthreads();
                    if (S.fail) {
                        if (tid == 0) status[mat] = 1;
                        ihi = -1;
                        break;
                    }
                    const int ns = S.ns, nd = nw - ns, old = ihi;
                    // eigenvalues that are done, the shifts of the next sweep
                    if (tid < nw && tid >= ns) eig[kw + tid] = S.T[tid * kLdn + tid];
                    ihi -= nd;
                    idle = nd ? 0 : idle + 1;
                    // a sweep unless more than half of the window deflated (measured at 25, 50 and 75 %: 20.0,
                    // 17.5, 18.1 ms for 20 matrices of n = 648, 4.03, 3.67, 3.73 for 10 of n = 216)
                    if (ihi - l + 1 > kNW && 2 * nd <= nw) {
                        sweep_l = l;
                        sweep_hi = ihi;
                        sweep_ms = min(kM, ns);
                        __syncthreads();
                        float2 s = make_float2(0.f, 0.f);
                        if (tid < sweep_ms) {
                            s = S.shift[ns - sweep_ms + tid];
                            if (idle > 0 && idle % 6 == 0) {      // exceptional shifts
                                const int i = ihi - sweep_ms + 1 + tid;
                                const float2 d = __ldcg(H + (long long)i * n + i);
                                s = make_float2(d.x + 0.75f * cabs1(__ldcg(H + (long long)i * n + i - 1)), d.y);
                            }
                        }
                        __syncthreads();
                        if (tid < sweep_ms) S.shift[tid] = s;
                    }
                    if (nd > 0) {
                        // the window (Hessenberg at the top, triangular below) back to H
                        for (int e = tid; e < nw * nw; e += kQrThreads) {
                            const int i = e / nw, j = e - i * nw;
                            const bool keep = j >= i || (j + 1 == i && i < ns);
                            H[(long long)(kw + i) * n + kw + j] = keep ? S.T[i * kLdn + j] : make_float2(0.f, 0.f);
                        }
                        if (tid == 0 && kw > l)
                            H[(long long)kw * n + kw - 1] = ns > 0 ? cmul(S.spike, conjf2(S.V[0])) : make_float2(0.f, 0.f);
                        for (int e = tid; e < kNW * kNW; e += kQrThreads)
                            if (e / kNW >= nw || e % kNW >= nw) S.V[(e / kNW) * kLdn + e % kNW] = make_float2(0.f, 0.f);
                        op = kOpDeflate;
                        a1 = kw;
                        a2 = old - kw + 1;
                        break;
                    }
                    if (sweep_ms > 0) {
                        op = kOpSweep;
                        a1 = sweep_l;
                        a2 = sweep_hi;
                        a3 = sweep_ms;
                        sweep_ms = 0;
                        break;
                    }
                }
            }
            __syncthreads();
            if (tid == 0) {
                S.cmd[0] = op;
                S.cmd[1] = a1;
                S.cmd[2] = a2;
                S.cmd[3] = a3;
            }
        }
        __threadfence();
        cluster.sync();
        const int op = S0->cmd[0], a1 = S0->cmd[1], a2 = S0->cmd[2], a3 = S0->cmd[3];
        if (op == kOpEnd) {
            cluster.sync();                              // rank 0's shared memory stays until all have read
            return;
        }
        if (op == kOpDeflate) {
            if (rank != 0)
                for (int e = tid; e < kNW * kLdn; e += kQrThreads) S.V[e] = S0->V[e];
            __syncthreads();
            deflation_update(S, H, Z, n, a1, a2, rank, K);
            __threadfence();
            cluster.sync();
            continue;
        }
        const int l = a1, hi_ = a2, ms = a3;
        const int nsteps = (hi_ - l) + 2 * (ms - 1);
        const int nwin = (nsteps + kStep - 1) / kStep;
        if (rank == 0) chase32(S, H, n, l, hi_, 0, ms, S.rot[0]);
        for (int w = 0; w < nwin; w++) {
            const int t0 = w * kStep, vb = l + t0 - 2 * (kM - 1);
            const int lo = max(l, vb), hi = min(hi_, vb + kW - 1);
            // columns the next window needs: the leader's
            const int next = w + 1 < nwin ? min(hi_, vb + kStep + kW - 1) : hi;
            __threadfence();
            cluster.sync();
            if (K == 1) {
                apply32(S, H, Z, n, vb, lo, hi, hi + 1, n, 0, lo + n, S.rot[w & 1]);
                __syncthreads();
                if (w + 1 < nwin) chase32(S, H, n, l, hi_, t0 + kStep, ms, S.rot[(w + 1) & 1]);
            } else if (rank == 0) {
                apply32(S, H, Z, n, vb, lo, hi, hi + 1, next + 1, 0, 0, S.rot[w & 1]);
                __syncthreads();
                if (w + 1 < nwin) chase32(S, H, n, l, hi_, t0 + kStep, ms, S.rot[(w + 1) & 1]);
            } else {
                const int* src = reinterpret_cast<const int*>(S0->rot[w & 1]);
                int* dst = reinterpret_cast<int*>(S.rot[0]);
                for (int e = tid; e < (int)(sizeof(QrRot) * kStep * (kM / 4) / sizeof(int)); e += kQrThreads) dst[e] = src[e];
                __syncthreads();
                const int right = n - (next + 1), rows = lo + n, P = K - 1, q = rank - 1;
                const int jc = (right + P - 1) / P, rc = (rows + P - 1) / P;
                apply32(S, H, Z, n, vb, lo, hi, next + 1 + min(right, q * jc), next + 1 + min(right, (q + 1) * jc),
                        min(rows, q * rc), min(rows, (q + 1) * rc), S.rot[0]);
            }
        }
        __threadfence();
        cluster.sync();
    }
}

}  // namespace z

scw_status hqr32(cudaStream_t st, float2* H, float2* Z, int n, float2* W, int* status, int batch, int ctas, int share) {
    if (n <= 0 || batch <= 0) return SCW_OK;
    constexpr size_t smem = sizeof(z::QrSmem);
    static_assert(smem <= 227 * 1024, "shared memory of the QR kernel");
    SCW_CUDA_TRY(cudaFuncSetAttribute(z::hqr32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int dev = 0, sms = 0;
    SCW_CUDA_TRY(cudaGetDevice(&dev));
    SCW_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    SCW_CUDA_TRY(cudaMemsetAsync(status, 0, sizeof(int) * batch, st));
    // The largest cluster for which all matrices (of `share` such batches at a time) are resident at
    // once, at most 8 CTAs and no more than have a warp of vectors each beside the leader; 2 leave
    // the leader's helper alone with all of the update, which is no slower than one CTA doing both in turn.
    int k = ctas > 0 ? std::min(ctas, 8) : std::min({8, sms / (batch * std::max(1, share)), 1 + (2 * n + 31) / 32});
    const long long nn = (long long)n * n;
    for (; k >= 2; k--) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)k;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3((unsigned)(k * batch));
        cfg.blockDim = dim3(z::kQrThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int resident = 0;
        if (cudaOccupancyMaxActiveClusters(&resident, z::hqr32_kernel, &cfg) != cudaSuccess) {
            cudaGetLastError();
            continue;
        }
        if (resident >= (ctas > 0 ? 1 : batch)) {
            SCW_CUDA_TRY(cudaLaunchKernelEx(&cfg, z::hqr32_kernel, H, Z, n, nn, W, status));
            return SCW_OK;
        }
    }
    z::hqr32_kernel<<<batch, z::kQrThreads, smem, st>>>(H, Z, n, nn, W, status);
    SCW_CUDA_TRY(cudaGetLastError());
    return SCW_OK;
}

}  // namespace scw
