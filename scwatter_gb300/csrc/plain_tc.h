// Tensor-core form of the plain summation (eval_plain_tc.cu), planned and chosen by eval_plain.cu.
#pragma once

#include <cuda_runtime.h>

#include "scw_internal.h"

namespace scw {
namespace ptc {

constexpr int kTileI = 40;        // columns of a tile: 3 components of five groups of eight in an MMA's 128 rows
constexpr int kTileJ = 64;        // most rows
constexpr int kMaxRun = 4096;     // waves added up in two floats (1024 in one) before they go to FP64 partial sums

struct Plane {
    float a0, b0, c;   // start along i (a) and j (b), fixed coordinate c
    float da, db;      // spacings along i and j
    int Ni, Nj;
    int mode;          // 0: (a,b,c) = (x,y,z); 1: (y,z,x); 2: (x,z,y)
    int pad;
    float* out;        // [Nj][Ni][6] floats
};

struct Item {          // rows [jr0, jr1) of one region, columns i0 .., waves [w0, w1)
    int plane, i0, jr0, jr1;
    int slot;          // partial-sum slot, or -1 (at most kMaxRun waves): write the output directly
    int pad;
    long long w0, w1;
};

struct Tile {          // partial sums slot0 .. slot0 + nslots - 1 to the output
    int plane, i0, jr0, jr1, slot0, nslots;
};

struct Waves {
    const double* kre;
    const double* kim;
    const double* zref;
    const float2* amp;
    long long n;
};

// longest: the most waves of an item; partials: kTileJ x 3 kTileI double2 per slot
scw_status launch(scw_ctx ctx, const Plane* planes, const Item* items, int nitems, const Tile* tiles, int ntiles, int max_rows,
                  long long longest, const Waves& W, double2* partials);

}  // namespace ptc
}  // namespace scw
