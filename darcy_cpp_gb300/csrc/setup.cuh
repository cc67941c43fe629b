// Hierarchy construction on the device, in FP64 (the Galerkin sums and the
// reciprocal diagonal are the steps whose accuracy the cycle rests on; an FP32
// cycle takes its reciprocal diagonal from the FP32 copy of d instead).
#pragma once

#include <math.h>

#include "common.cuh"

namespace dgpu {

// FP64 level storage, plus the boundary west/south faces used only here.
struct Lvl64 {
    int n;
    double* e;
    double* nf;
    double* d;
    double* id;
    double* wb;  // west boundary face of row i (cell (i, 0))
    double* sb;  // south boundary face of column j (cell (0, j))
};

// include/darcy/level.hpp:57. 2*x*y is (2x)*y: exact scaling then one rounded
// product, so harmonic(x, y) == harmonic(y, x) bit for bit.
__device__ __forceinline__ double harmonic(double x, double y) { return 2.0 * x * y / (x + y); }

// level.hpp:79-97 plus validate_permeability (solver.hpp:68-77): the first
// offending flat index is folded into *bad with atomicMin. A CTA builds a tile
// of kFineX x kFineY cells: every thread its cell's east and north face, two
// warps the faces on the tile's west and south edge, then every thread sums
// its four (a neighbour's face has the same bits: harmonic is symmetric). Bound
// by the FP64 divisions, 3.25 a cell instead of the 5 of a cell on its own:
// 2048^2 396 -> 248 us, 1024^2 102 -> 63 (the pipe needs ~230 and 58).
constexpr int kFineX = 32, kFineY = 8;
__device__ __forceinline__ void build_fine(const double* __restrict__ a, const Lvl64& L, unsigned long long* bad) {
    __shared__ double se[kFineY][kFineX + 1], sn[kFineY + 1][kFineX];
    const int n = L.n, tx = threadIdx.x % kFineX, ty = threadIdx.x / kFineX;
    const int tiles = (n + kFineX - 1) / kFineX, i0 = blockIdx.x / tiles * kFineY, j0 = blockIdx.x % tiles * kFineX;
    const int i = i0 + ty, j = j0 + tx, k = i * n + j;  // n^2 < 2^31
    const bool inside = i < n && j < n;
    double e = 0.0, nn = 0.0;
    if (inside) {
        const double c = a[k];
        if (!(c > 0.0) || !isfinite(c)) atomicMin(bad, (unsigned long long)k);
        e = (j + 1 < n) ? harmonic(c, a[k + 1]) : c;
        nn = (i + 1 < n) ? harmonic(c, a[k + n]) : c;
        se[ty][tx + 1] = e;
        sn[ty + 1][tx] = nn;
    }
    if (ty == 0 && j < n) {  // (i0 < n)
        const int q = i0 * n + j;
        sn[0][tx] = (i0 > 0) ? harmonic(a[q], a[q - n]) : a[q];
    }
    if (ty == 1 && tx < kFineY && i0 + tx < n) {
        const int q = (i0 + tx) * n + j0;
        se[tx][0] = (j0 > 0) ? harmonic(a[q], a[q - 1]) : a[q];
    }
    __syncthreads();
    if (!inside) return;
    const double w = se[ty][tx], s = sn[ty][tx];
    const double dd = e + w + nn + s;
    L.e[k] = e;
    L.nf[k] = nn;
    L.d[k] = dd;
    L.id[k] = 1.0 / dd;
    if (j == 0) L.wb[i] = w;
    if (i == 0) L.sb[j] = s;
}

// Galerkin coarse operator P^T A P by face summation (level.hpp:171-211),
// including the width-one trailing aggregate of an odd grid. West/south fine
// faces come from the neighbour's east/north face (same bits) or, on the
// domain boundary, from wb/sb; summation order is the reference's.
template <class S>
__device__ __forceinline__ void coarsen(const Lvl64& F, const Lvl64& C) {
    const int n = F.n, nc = C.n, mc = nc * nc;  // n^2 < 2^31
    for (int K = (int)S::start(); K < mc; K += (int)S::stride()) {
        const int I = K / nc, J = K - I * nc;
        const int i0 = 2 * I, i1 = (2 * I + 1 < n) ? 2 * I + 1 : 2 * I;
        const int j0 = 2 * J, j1 = (2 * J + 1 < n) ? 2 * J + 1 : 2 * J;
        double ce = 0.0, cw = 0.0, cn = 0.0, cs = 0.0;
        for (int i = i0; i <= i1; ++i) {
            ce += F.e[i * n + j1];
            cw += (j0 > 0) ? F.e[i * n + j0 - 1] : F.wb[i];
        }
        for (int j = j0; j <= j1; ++j) {
            cn += F.nf[i1 * n + j];
            cs += (i0 > 0) ? F.nf[(i0 - 1) * n + j] : F.sb[j];
        }
        const double dd = ce + cw + cn + cs;
        C.e[K] = ce;
        C.nf[K] = cn;
        C.d[K] = dd;
        C.id[K] = 1.0 / dd;
        if (J == 0) C.wb[I] = cw;
        if (I == 0) C.sb[J] = cs;
    }
}

// FP32 copy of a level's coefficients for the mixed-precision cycle. When
// the lo pointers are given, also the rounding remainders of e, nf, d
// (c - (double)(float)c, rounded to FP32): hi + lo carries ~48 bits.
__device__ __forceinline__ void to_fp32(const Lvl64& L, float* e, float* nf, float* d, float* id, float* elo,
                                        float* nlo, float* dlo) {
    const int64_t m = (int64_t)L.n * L.n;
    for (int64_t k = GridScope::start(); k < m; k += GridScope::stride()) {
        float eh, el, nh, nl, dh, dl;  // split_f64: the conversions' bits without the FP64 pipe
        split_f64(L.e[k], eh, el);
        split_f64(L.nf[k], nh, nl);
        split_f64(L.d[k], dh, dl);
        e[k] = eh;
        nf[k] = nh;
        d[k] = dh;
        id[k] = round_f64(L.id[k]);
        if (elo) {
            elo[k] = el;
            nlo[k] = nl;
            dlo[k] = dl;
        }
    }
}

}  // namespace dgpu
