// Level operations of the block engine (one CTA, one problem) on a padded
// layout, two cells of a colour at a time.
//
// A level of side n is stored with side np = 2 nc, nc = (n + 1) / 2: an even
// pitch, so that rows and pairs are 8- / 16-byte aligned for every n, and
// whole 2 x 2 aggregates ("patches"), so that one index serves the four cells
// of a patch and its coarse cell. Cells outside the domain (the last row and
// column of an odd side) hold zero coefficients and stay zero. Once the next
// coarser level is built, the faces on the domain's east and north boundary
// are set to zero, and nf has np zeros and e two zeros before the array, x
// np zeros before and after it: a neighbour outside the domain then enters as
// 0 * (some finite number), which leaves the sum as the reference's skipped
// term does, and no pass tests for a boundary.
//
// Two things follow. The number has to be finite: arenas are cleared whenever
// it may not be (block_clear). And beyond the end of a row lies the next row's
// first cell, of the same colour as the last: a pass may read it while the
// thread that owns it writes it. Such a read races, and gets the old value or
// the new (the accesses are aligned scalars of 4 or 8 bytes); both are finite
// and both enter as zero, so the result does not depend on which.
//
// Why patches: the earlier passes walked the cells of one colour with an
// integer division, four boundary tests and ten scalar loads a cell; a
// 64 x 64 problem took ~120 thousand warp instructions an iteration and the
// scheduler had nothing to issue 58% (FP32 cycle) to 78% (FP64) of the time.
#pragma once

#include "common.cuh"

namespace dgpu {

template <class T>
struct PLvl {
    int n, nc, np;
    unsigned rcp;   // ceil(2^32 / nc) while the product below is exact, else 0
    unsigned rper;  // the same for nc^2 (levels with many right-hand sides)
    const T* e;
    const T* nf;
    const T* d;
    const T* id;
    T* x;
    T* b;
};

template <class T>
struct Pair;
template <>
struct Pair<float> {
    using type = float2;
};
template <>
struct Pair<double> {
    using type = double2;
};
template <class T>
using Pair_t = typename Pair<T>::type;

template <class T>
__device__ __forceinline__ Pair_t<T> load_pair(const T* p) {
    return *reinterpret_cast<const Pair_t<T>*>(p);
}

// q / nc for q < 2 nc^2 (pairs of a level) as the high half of a product:
// exact while 2 nc^3 < 2^32.
__host__ __device__ inline unsigned row_reciprocal(int nc) {
    return nc >= 2 && nc <= 1280 ? (unsigned)((0x100000000ull + (unsigned)nc - 1) / (unsigned)nc) : 0u;
}
__device__ __forceinline__ int patch_row(int q, int nc, unsigned rcp) {
    return rcp ? (int)__umulhi((unsigned)q, rcp) : q / nc;
}

// The passes below work on one patch whose first cell is k = 2 I np + 2 J.
// Colour 0 holds the cells (0, 0) and (1, 1) of a patch, colour 1 the cells
// (0, 1) and (1, 0). Terms in the order of include/darcy/level.hpp:105-161.

// Colour 0 from a zero iterate: x = b / d.
template <class T>
__device__ __forceinline__ void patch_red_zero(const PLvl<T>& L, T* x, const T* b, int k) {
    const int k1 = k + L.np + 1;
    const T v0 = b[k] * L.id[k], v1 = b[k1] * L.id[k1];
    x[k] = v0;
    x[k1] = v1;
}

template <class T>
__device__ __forceinline__ void patch_red(const PLvl<T>& L, const T* x, const T* b, int k, T& o0, T& o1) {
    const int np = L.np, k1 = k + np + 1;
    const T x01 = x[k + 1], x10 = x[k + np];
    const Pair_t<T> n0 = load_pair(L.nf + k), e1 = load_pair(L.e + k + np);
    T v0 = b[k], v1 = b[k1];
    v0 += L.e[k] * x01;
    v1 += e1.y * x[k1 + 1];
    v0 += L.e[k - 1] * x[k - 1];
    v1 += e1.x * x10;
    v0 += n0.x * x10;
    v1 += L.nf[k1] * x[k1 + np];
    v0 += L.nf[k - np] * x[k - np];
    v1 += n0.y * x01;
    o0 = v0 * L.id[k];
    o1 = v1 * L.id[k1];
}

template <class T>
__device__ __forceinline__ void patch_black(const PLvl<T>& L, const T* x, const T* b, int k, T& o0, T& o1) {
    const int np = L.np, kb = k + 1, kc = k + np;
    const T x00 = x[k], x11 = x[kc + 1];
    const Pair_t<T> n0 = load_pair(L.nf + k), e0 = load_pair(L.e + k);
    T v0 = b[kb], v1 = b[kc];
    v0 += e0.y * x[kb + 1];
    v1 += L.e[kc] * x11;
    v0 += e0.x * x00;
    v1 += L.e[kc - 1] * x[kc - 1];
    v0 += n0.y * x11;
    v1 += L.nf[kc] * x[kc + np];
    v0 += L.nf[kb - np] * x[kb - np];
    v1 += n0.x * x00;
    o0 = v0 * L.id[kb];
    o1 = v1 * L.id[kc];
}

// Colour 1 seeing colour 0 through the prolongation x + P xc. The colour-0
// pass that follows overwrites every colour-0 cell and colour 1 never reads
// its own value, so the corrected iterate is not stored (level.hpp:230-237
// followed by :145-161).
template <class T>
__device__ __forceinline__ void patch_black_prolong(const PLvl<T>& L, const T* x, const T* b, int k,
                                                    const T* xc, int K, int npc, T& o0, T& o1) {
    const int np = L.np, kb = k + 1, kc = k + np;
    const T c = xc[K];
    const T x00 = x[k] + c, x11 = x[kc + 1] + c;
    const Pair_t<T> n0 = load_pair(L.nf + k), e0 = load_pair(L.e + k);
    T v0 = b[kb], v1 = b[kc];
    v0 += e0.y * (x[kb + 1] + xc[K + 1]);
    v1 += L.e[kc] * x11;
    v0 += e0.x * x00;
    v1 += L.e[kc - 1] * (x[kc - 1] + xc[K - 1]);
    v0 += n0.y * x11;
    v1 += L.nf[kc] * (x[kc + np] + xc[K + npc]);
    v0 += L.nf[kb - np] * (x[kb - np] + xc[K - npc]);
    v1 += n0.x * x00;
    o0 = v0 * L.id[kb];
    o1 = v1 * L.id[kc];
}

// Sum of b - A x over the patch (level.hpp:122-137, :214-227) after a
// colour-1 pass. That pass has just solved the colour-1 cells' equations, so
// their residual is zero (up to the rounding of the very values it would be
// computed from) and only the two colour-0 cells contribute: half the
// arithmetic and none of the loads of colour 1's d and b.
//
// kFromZero: the colour-0 values come from the pass x = b / d on a zero
// iterate, so b - d x is zero too (again up to rounding) and what is left is
// the flow from the colour-1 neighbours. (FP64, where the pipe is 88% busy:
// 27 operations a patch become 9 or 13; 1024 x 64^2 8.25 -> 6.97 ms, 512 x
// 128^2 30.9 -> 26.8 ms. Mean iterations to 1e-10 with all four residuals ->
// with these, over 2048 fields of 64^2 and 600 of 97^2: FP64 25.46 -> 25.46 and
// 29.62 -> 29.62 at contrast 1e4, 28.35 -> 28.36 and 34.35 -> 34.02 at 1e6;
// FP32 28.13 -> 28.13 and 34.29 -> 34.26, 33.89 -> 33.73 and 43.78 -> 43.89.)
template <class T, bool kFromZero>
__device__ __forceinline__ T patch_residual(const PLvl<T>& L, const T* x, const T* b, int k) {
    const int np = L.np, k1 = k + np + 1;
    const T x01 = x[k + 1], x10 = x[k + np];
    const Pair_t<T> n0 = load_pair(L.nf + k), e1 = load_pair(L.e + k + np);
    T v0, v1;
    if (kFromZero) {
        v0 = L.e[k] * x01;
        v1 = e1.y * x[k1 + 1];
    } else {
        v0 = b[k] - L.d[k] * x[k];
        v1 = b[k1] - L.d[k1] * x[k1];
        v0 += L.e[k] * x01;
        v1 += e1.y * x[k1 + 1];
    }
    v0 += L.e[k - 1] * x[k - 1];
    v1 += e1.x * x10;
    v0 += n0.x * x10;
    v1 += L.nf[k1] * x[k1 + np];
    v0 += L.nf[k - np] * x[k - np];
    v1 += n0.y * x01;
    return v0 + v1;
}

// The same sum over all four cells, each residual rounded on its own, cells in
// row-major order and products in the order of cell_residual (the first two
// terms as e x_E subtracted from the rounded d x): the grid engine's rounding,
// which its tail operator keeps.
__device__ __forceinline__ double patch_residual_all(const PLvl<double>& L, const double* x, const double* b, int k) {
    const int np = L.np;
    double s = 0.0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int q = k + (c >> 1) * np + (c & 1);
        double v = fma(-L.e[q], x[q + 1], __dmul_rn(L.d[q], x[q]));
        v = fma(-L.e[q - 1], x[q - 1], v);
        v = fma(-L.nf[q], x[q + np], v);
        v = fma(-L.nf[q - np], x[q - np], v);
        s += b[q] - v;
    }
    return s;
}

// `calls` calls from zero of the side-2 level A, and of the 1 x 1 level below
// it (reciprocal diagonal idc), for one right-hand side, by one thread: the
// level has one patch, and its ~10 passes in one step save the CTA as many
// barrier-separated ones. Arithmetic and order as the passes with
// patch_residual_all; terms of absent neighbours (zero faces) left out.
__device__ __forceinline__ void solve_side2(const PLvl<double>& A, double idc, const double* b, double* x, int pre,
                                            int post, int calls) {
    const double e0 = A.e[0], e1 = A.e[2], n0 = A.nf[0], n1 = A.nf[1];
    const double b0 = b[0], b1 = b[1], b2 = b[2], b3 = b[3];
    const double i0 = A.id[0], i1 = A.id[1], i2 = A.id[2], i3 = A.id[3];
    // (products and sums that must round on their own are kept from contracting)
    double x0 = __dmul_rn(b0, i0), x1 = 0.0, x2 = 0.0, x3 = __dmul_rn(b3, i3);  // colour 0 from a zero iterate
    // cells 0, 3: colour 0; cells 1, 2: colour 1; terms east, west, north, south
    auto red = [&] {
        x0 = __dmul_rn(fma(n0, x2, fma(e0, x1, b0)), i0);
        x3 = __dmul_rn(fma(n1, x1, fma(e1, x2, b3)), i3);
    };
    auto black = [&](double c0, double c3) {
        x1 = __dmul_rn(fma(n1, c3, fma(e0, c0, b1)), i1);
        x2 = __dmul_rn(fma(n0, c0, fma(e1, c3, b2)), i2);
    };
    for (int call = 0; call < calls; ++call) {
        black(x0, x3);
        for (int s = 1; s < pre; ++s) {
            red();
            black(x0, x3);
        }
        double s = b0 - fma(-n0, x2, fma(-e0, x1, __dmul_rn(A.d[0], x0)));
        s += b1 - fma(-n1, x3, fma(-e0, x0, __dmul_rn(A.d[1], x1)));
        s += b2 - fma(-n0, x0, fma(-e1, x3, __dmul_rn(A.d[2], x2)));
        s += b3 - fma(-n1, x1, fma(-e1, x2, __dmul_rn(A.d[3], x3)));
        const double c = __dmul_rn(s, idc);  // the 1 x 1 level, exactly; prolonged to the patch
        black(__dadd_rn(x0, c), __dadd_rn(x3, c));
        for (int q = 1; q < post; ++q) {
            red();
            black(x0, x3);
        }
        red();
    }
    x[0] = x0;
    x[1] = x1;
    x[2] = x2;
    x[3] = x3;
}

// The same for the block engine's own residual (patch_residual: the colour-0
// cells, and only their flow after a first call's x = b / d). id64: see
// patch_cycle_m.
template <class T>
__device__ __forceinline__ void solve_side2_flow(const PLvl<T>& A, const PLvl<T>& B, const double* id64, const T* b,
                                                 T* x, int pre, int post, int calls) {
    const T e0 = A.e[0], e1 = A.e[2], n0 = A.nf[0], n1 = A.nf[1];
    const T b0 = b[0], b1 = b[1], b2 = b[2], b3 = b[3];
    const T i0 = A.id[0], i1 = A.id[1], i2 = A.id[2], i3 = A.id[3];
    T x0 = b0 * i0, x1 = T(0), x2 = T(0), x3 = b3 * i3;
    auto red = [&] {
        x0 = (b0 + e0 * x1 + n0 * x2) * i0;
        x3 = (b3 + e1 * x2 + n1 * x1) * i3;
    };
    auto black = [&](T c0, T c3) {
        x1 = (b1 + e0 * c0 + n1 * c3) * i1;
        x2 = (b2 + e1 * c3 + n0 * c0) * i2;
    };
    for (int call = 0; call < calls; ++call) {
        black(x0, x3);
        for (int s = 1; s < pre; ++s) {
            red();
            black(x0, x3);
        }
        T r0 = T(0), r3 = T(0);
        if (call > 0 || pre > 1) {
            r0 = b0 - A.d[0] * x0;
            r3 = b3 - A.d[3] * x3;
        }
        const T s = (r0 + e0 * x1 + n0 * x2) + (r3 + e1 * x2 + n1 * x1);
        const T c = id64 ? (T)((double)s * id64[0]) : s * B.id[0];
        black(x0 + c, x3 + c);
        for (int q = 1; q < post; ++q) {
            red();
            black(x0, x3);
        }
        red();
    }
    x[0] = x0;
    x[1] = x1;
    x[2] = x2;
    x[3] = x3;
}

// ------------------------------------------------------------ CTA passes
//
// (Two patches of a thread at once, all loads before the first store, measured
// slower: 4096 x 64^2 mixed 13.2 -> 13.8 ms at 256 threads and 32 KiB.)

template <class T>
__device__ __forceinline__ void pass_red_zero(const PLvl<T>& L) {
    const int nc = L.nc, cnt = nc * nc;
    for (int q = threadIdx.x; q < cnt; q += blockDim.x)
        patch_red_zero(L, L.x, L.b, 2 * q + 2 * patch_row(q, nc, L.rcp) * nc);
}

template <class T, int kColour>
__device__ __forceinline__ void pass_colour(const PLvl<T>& L) {
    const int nc = L.nc, cnt = nc * nc, np = L.np;
    for (int q = threadIdx.x; q < cnt; q += blockDim.x) {
        const int k = 2 * q + 2 * patch_row(q, nc, L.rcp) * nc;
        T o0, o1;
        if (kColour == 0)
            patch_red(L, L.x, L.b, k, o0, o1);
        else
            patch_black(L, L.x, L.b, k, o0, o1);
        L.x[k + (kColour == 0 ? 0 : 1)] = o0;
        L.x[k + (kColour == 0 ? np + 1 : np)] = o1;
    }
}

template <class T>
__device__ __forceinline__ void pass_black_prolong(const PLvl<T>& L, const PLvl<T>& C) {
    const int nc = L.nc, cnt = nc * nc, np = L.np, npc = C.np;
    for (int q = threadIdx.x; q < cnt; q += blockDim.x) {
        const int I = patch_row(q, nc, L.rcp), k = 2 * q + 2 * I * nc;
        T o0, o1;
        patch_black_prolong(L, L.x, L.b, k, C.x, q + I * (npc - nc), npc, o0, o1);
        L.x[k + 1] = o0;
        L.x[k + np] = o1;
    }
}

template <class T, bool kFromZero>
__device__ __forceinline__ void pass_residual_restrict(const PLvl<T>& L, const PLvl<T>& C) {
    const int nc = L.nc, cnt = nc * nc, npc = C.np;
    for (int q = threadIdx.x; q < cnt; q += blockDim.x) {
        const int I = patch_row(q, nc, L.rcp);
        C.b[q + I * (npc - nc)] = patch_residual<T, kFromZero>(L, L.x, L.b, 2 * q + 2 * I * nc);
    }
}

// x = Tt b for the dense tail operator (N x N, N the padded cells of the
// tail's first level, rows `pitch` apart): four lanes a row, each taking
// every fourth 16-byte vector of it. With rows 64 bytes past a multiple of
// 128 apart, the eight lanes of a quarter warp (two rows) read distinct banks.
// One warp a row, two elements a lane, spent its time in the five dependent
// shuffles of each row's sum.
template <class T>
__host__ __device__ inline int tail_pitch(int N) {
    const int bytes = N * (int)sizeof(T);
    return (int)(((bytes + 63) / 128 * 128 + 64) / sizeof(T));
}
template <class T>
__device__ __forceinline__ void block_matvec(const T* __restrict__ Tt, int N, int pitch, const T* b, T* x) {
    constexpr int kW = 16 / sizeof(T);
    const int lane4 = threadIdx.x & 3;
    for (int t = threadIdx.x; (t & ~31) < 4 * N; t += blockDim.x) {
        const int row = t >> 2;
        T acc = T(0);
        if (row < N) {
            const T* Tr = Tt + row * pitch;
#pragma unroll 4
            for (int c = lane4 * kW; c < N; c += 4 * kW) {
                if constexpr (sizeof(T) == 4) {
                    const float4 m = *reinterpret_cast<const float4*>(Tr + c), v = *reinterpret_cast<const float4*>(b + c);
                    acc += m.x * v.x;
                    acc += m.y * v.y;
                    acc += m.z * v.z;
                    acc += m.w * v.w;
                } else {
                    const double2 m = *reinterpret_cast<const double2*>(Tr + c),
                                  v = *reinterpret_cast<const double2*>(b + c);
                    acc += m.x * v.x;
                    acc += m.y * v.y;
                }
            }
        }
        acc += __shfl_down_sync(0xffffffffu, acc, 2, 4);
        acc += __shfl_down_sync(0xffffffffu, acc, 1, 4);
        if (row < N && lane4 == 0) x[row] = acc;
    }
}

// ------------------------------------------------------------ the cycle
//
// One cycle at level 0 (include/darcy/multigrid.hpp:88-127, the recursion
// unrolled into two bits of remaining calls a level) without its first
// colour-0 pass from zero and without its last colour-0 pass: the caller
// merges those into the loops that produce b and consume x. The levels from
// tl down are the dense operator Tt ("x = 0, then gamma cycles"); with Tt ==
// null they are visited down to the 1 x 1 level, solved exactly (with the
// FP64 reciprocal diagonal id64 in the FP32 cycle). At least two levels.
//
// A level's second call starts where its first ended: that call's last
// colour-0 pass reads the same colour-1 values as the second call's first
// would, so the latter is skipped (same bits).
template <class T>
__device__ void patch_cycle(const PLvl<T>* lv, int nlev, int pre, int post, int gamma, const double* id64,
                            const T* Tt, int tl) {
    unsigned long long calls = 1;  // remaining calls, two bits a level
    int l = 0;
    bool zero = true;              // the level's iterate is zero (its first call)
    const int last = Tt ? tl - 1 : nlev - 2;  // deepest level that is smoothed
    auto descend = [&](int lvl) {
        const PLvl<T>& A = lv[lvl];
        if (zero && lvl > 0) {
            pass_red_zero(A);
            __syncthreads();
        }
        pass_colour<T, 1>(A);
        __syncthreads();
        for (int s = 1; s < pre; ++s) {
            pass_colour<T, 0>(A);
            __syncthreads();
            pass_colour<T, 1>(A);
            __syncthreads();
        }
        if (zero && pre == 1)
            pass_residual_restrict<T, true>(A, lv[lvl + 1]);
        else
            pass_residual_restrict<T, false>(A, lv[lvl + 1]);
        __syncthreads();
    };
    auto ascend = [&](int lvl) {
        const PLvl<T>& A = lv[lvl];
        pass_black_prolong(A, lv[lvl + 1]);
        __syncthreads();
        for (int s = 1; s < post; ++s) {
            pass_colour<T, 0>(A);
            __syncthreads();
            pass_colour<T, 1>(A);
            __syncthreads();
        }
        if (lvl > 0) {
            pass_colour<T, 0>(A);
            __syncthreads();
        }
    };
    for (;;) {
        while (l < last) {
            descend(l);
            ++l;
            calls = (calls & ~(3ull << (2 * l))) | ((unsigned long long)gamma << (2 * l));
            zero = true;
        }
        descend(l);
        if (Tt) {
            const PLvl<T>& B = lv[tl];
            const int N = B.np * B.np;
            block_matvec<T>(Tt, N, tail_pitch<T>(N), B.b, B.x);
        } else if (threadIdx.x == 0) {  // the 1 x 1 level; a second call finds its exact solution again
            const PLvl<T>& B = lv[nlev - 1];
            B.x[0] = id64 ? (T)((double)B.b[0] * id64[0]) : B.b[0] * B.id[0];
        }
        __syncthreads();
        ascend(l);
        for (;;) {
            calls -= 1ull << (2 * l);
            if ((calls >> (2 * l)) & 3ull) break;  // run this level's cycle again
            if (l == 0) return;
            --l;
            ascend(l);
        }
        zero = false;
    }
}

// -------------------------------------------------- many right-hand sides
//
// `top` calls of level l0 from zero for `nrhs` right-hand sides at once, used
// to build a dense operator of the levels from l0 down. Right-hand side r of a
// level is at x + r * stride, b + r * stride, stride = np^2 + 2 np. id64: the
// FP64 reciprocal diagonal of the 1 x 1 level (FP32 cycle), or null. kAll (FP64):
// residuals by patch_residual_all. The side-2 level and what is below it is one
// thread's work for a right-hand side: 38 passes instead of 90 for the tail of
// an 8 x 8 level (a 64^2 problem at 256 threads: 188 -> 124 thousand cycles in
// FP32, 391 -> 313 in FP64, of ~4.5 and 7.8 million for the whole problem).

__host__ __device__ inline int rhs_stride(int np) { return np * np + 2 * np; }

template <class T, class F>
__device__ __forceinline__ void for_patches_m(const PLvl<T>& L, int nrhs, F&& f) {
    const int nc = L.nc, per = nc * nc, st = rhs_stride(L.np);
    for (int t = threadIdx.x; t < per * nrhs; t += blockDim.x) {
        const int r = patch_row(t, per, L.rper), q = t - r * per;
        const int I = patch_row(q, nc, L.rcp);
        f(L.x + r * st, L.b + r * st, r, 2 * q + 2 * I * nc, q, I);
    }
    __syncthreads();
}

template <class T, bool kAll = false>
__device__ void patch_cycle_m(const PLvl<T>* lv, int l0, int nlev, int pre, int post, int gamma, int top, int nrhs,
                              const double* id64) {
    const int lb = nlev - 2 >= l0 ? nlev - 2 : nlev - 1;  // the side-2 or the 1 x 1 level
    unsigned long long calls = (unsigned long long)top << (2 * l0);
    int l = l0;
    bool zero = true;
    auto red = [&](const PLvl<T>& A) {
        for_patches_m(A, nrhs, [&](T* x, const T* b, int, int k, int, int) {
            T o0, o1;
            patch_red(A, x, b, k, o0, o1);
            x[k] = o0;
            x[k + A.np + 1] = o1;
        });
    };
    auto black = [&](const PLvl<T>& A) {
        for_patches_m(A, nrhs, [&](T* x, const T* b, int, int k, int, int) {
            T o0, o1;
            patch_black(A, x, b, k, o0, o1);
            x[k + 1] = o0;
            x[k + A.np] = o1;
        });
    };
    for (;;) {
        while (l < lb) {
            const PLvl<T>& A = lv[l];
            const PLvl<T>& C = lv[l + 1];
            const int stc = rhs_stride(C.np), npc = C.np;
            if (zero)
                for_patches_m(A, nrhs, [&](T* x, const T* b, int, int k, int, int) { patch_red_zero(A, x, b, k); });
            for (int s = 1;; ++s) {
                black(A);
                if (s >= pre) break;
                red(A);
            }
            const bool from_zero = zero && pre == 1;
            for_patches_m(A, nrhs, [&](T* x, const T* b, int r, int k, int q, int I) {
                T s;
                if constexpr (kAll)
                    s = patch_residual_all(A, x, b, k);
                else
                    s = from_zero ? patch_residual<T, true>(A, x, b, k) : patch_residual<T, false>(A, x, b, k);
                C.b[r * stc + q + I * (npc - A.nc)] = s;
            });
            ++l;
            calls = (calls & ~(3ull << (2 * l))) | ((unsigned long long)gamma << (2 * l));
            zero = true;
        }
        {  // the bottom: level lb and what is below it
            const PLvl<T>& A = lv[l];
            const int st = rhs_stride(A.np);
            for (int r = threadIdx.x; r < nrhs; r += blockDim.x) {
                if (A.n == 2) {
                    const int todo = (int)((calls >> (2 * l)) & 3ull);
                    if constexpr (kAll)
                        solve_side2(A, lv[l + 1].id[0], A.b + r * st, A.x + r * st, pre, post, todo);
                    else
                        solve_side2_flow(A, lv[l + 1], id64, A.b + r * st, A.x + r * st, pre, post, todo);
                    continue;
                }
                A.x[r * st] = id64 ? (T)((double)A.b[r * st] * id64[0]) : A.b[r * st] * A.id[0];
            }
            __syncthreads();
            calls &= ~(3ull << (2 * l));  // done (further calls of the 1 x 1 level change nothing)
        }
        for (;;) {
            if (((calls >> (2 * l)) & 3ull) != 0) calls -= 1ull << (2 * l);
            if (l < lb && ((calls >> (2 * l)) & 3ull) != 0) break;
            if (l == l0) return;
            --l;
            const PLvl<T>& A = lv[l];
            const PLvl<T>& C = lv[l + 1];
            const int stc = rhs_stride(C.np), npc = C.np;
            for_patches_m(A, nrhs, [&](T* x, const T* b, int r, int k, int q, int I) {
                T o0, o1;
                patch_black_prolong(A, x, b, k, C.x + r * stc, q + I * (npc - A.nc), npc, o0, o1);
                x[k + 1] = o0;
                x[k + A.np] = o1;
            });
            for (int s = 1;; ++s) {
                red(A);
                if (s >= post) break;
                black(A);
            }
        }
        zero = false;
    }
}

}  // namespace dgpu
