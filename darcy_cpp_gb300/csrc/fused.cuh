// Fused level visits for the grid engine: one kernel for everything before
// the coarse-grid correction, one for everything after it.
//
//   k_visit_pre : red sweep, black sweep, residual and 2x2 restriction
//                 (multigrid.hpp:108-115 with pre_sweeps = 1)
//   k_visit_post: prolongation, black sweep, red sweep, and on level 0 the
//                 r . z reduction (multigrid.hpp:119-126, solver.hpp:167-171)
//
// Each CTA owns a TH x TW tile (even origin, so it holds whole aggregates)
// and stages a halo in shared memory: red-black updates only look one cell
// away, so a tile can finish k dependent colour passes on its own if it
// recomputes k rings of halo. Cells outside the domain are staged as zero
// (x = 0 and face = 0), which reproduces the reference's skipped boundary
// terms exactly: adding e * 0 leaves the running sum bit-identical.
//
// Coefficients do not change during a solve (they are written by the setup
// kernels, which complete before the solve's loop starts), so they are
// staged before the programmatic-launch wait and their load overlaps the
// previous kernel; everything the previous kernel produces is read after it.
//
// FP32 cycle (mixed form). Smoothing and transfers run in FP32. The residual
// that is restricted is formed in double-float arithmetic -- FP32 hi/lo
// coefficient pairs, error-free products (FMA) and compensated sums -- which
// is accurate to ~2^-48 of its largest term while using only the FP32 pipes:
// at high permeability contrast b - A x cancels far below the size of its
// terms, where a plain FP32 residual weakens the cycle and costs CG
// iterations, and GB300's FP64 (and FP64<->FP32 conversion) rate is ~1/60 of
// its FP32 rate.
//
// Both kernels read x from one buffer and write another (the halo of a
// neighbouring tile must see the values from before this pass), so the host
// alternates two iterate buffers per level. They do not look at the solve's
// `done` flag: after convergence the rest of that loop iteration only
// rewrites cycle scratch, which nothing reads.
#pragma once

#include "common.cuh"
#include "setup.cuh"

namespace dgpu {

template <int TH, int TW, int R>
struct Tile {
    static constexpr int SH = TH + 2 * R, SW = TW + 2 * R, S = SH * SW;
};

// Level data a fused visit reads. For T = double: the FP64 hierarchy, lo
// pointers null. For T = float: FP32 hi parts and the lo parts of e, nf, d
// (c = hi + lo to ~2^-48); blo is the lo part of b where it exists (level 0).
template <class T>
struct VisitLevel {
    int n;
    const T* e;
    const T* nf;
    const T* d;
    const T* id;
    const T* elo;
    const T* nlo;
    const T* dlo;
    const T* b;
    const T* blo;
};

// ---------------------------------------------------------- double-float
struct DF {
    float hi, lo;
};
// s + v, v = (vh, vl) with |vl| << |vh|: TwoSum on the hi parts.
__device__ __forceinline__ void df_add(DF& s, float vh, float vl) {
    const float t = s.hi + vh;
    const float bb = t - s.hi;
    const float err = (s.hi - (t - bb)) + (vh - bb);
    s.hi = t;
    s.lo += err + vl;
}
// s += sign * (ch + cl) * x, x exact in FP32: error-free hi product.
__device__ __forceinline__ void df_axpy(DF& s, float ch, float cl, float x, float sign) {
    const float p = ch * x;
    const float pe = fmaf(ch, x, -p);
    df_add(s, sign * p, sign * (pe + cl * x));
}

// -------------------------------------------------------------- staging
//
// A thread's cells are all loaded before any of them is stored to shared
// memory: a tile's halo has up to 384 cells for 256 threads, and one cell at a
// time (load, store, load, store) cost a second L2 round trip on the way from
// one visit to the next.

constexpr int kVisitThreads = 256;

template <class T, int TH, int TW, int R, bool WITH_D, bool WITH_LO>
__device__ __forceinline__ void stage_coeffs(const VisitLevel<T>& V, int ti0, int tj0, T* es, T* ns, T* ds, T* is,
                                             T* elo, T* nlo, T* dlo) {
    using G = Tile<TH, TW, R>;
    constexpr int kIter = (G::S + kVisitThreads - 1) / kVisitThreads;
    const int n = V.n;
    T ev[kIter], nv[kIter], dv[kIter], iv[kIter], el[kIter], nl[kIter], dl[kIter];
#pragma unroll
    for (int u = 0; u < kIter; ++u) {
        const int q = threadIdx.x + u * kVisitThreads;
        const int li = q / G::SW, lj = q - li * G::SW;
        const int gi = ti0 - R + li, gj = tj0 - R + lj;
        ev[u] = nv[u] = dv[u] = iv[u] = el[u] = nl[u] = dl[u] = T(0);
        if (q < G::S && gi >= 0 && gi < n && gj >= 0 && gj < n) {
            const int k = gi * n + gj;
            ev[u] = __ldg(V.e + k);
            nv[u] = __ldg(V.nf + k);
            if (WITH_D) dv[u] = __ldg(V.d + k);
            iv[u] = __ldg(V.id + k);
            if (WITH_LO) {
                el[u] = __ldg(V.elo + k);
                nl[u] = __ldg(V.nlo + k);
                if (WITH_D) dl[u] = __ldg(V.dlo + k);
            }
        }
    }
#pragma unroll
    for (int u = 0; u < kIter; ++u) {
        const int q = threadIdx.x + u * kVisitThreads;
        if (q >= G::S) break;
        es[q] = ev[u];
        ns[q] = nv[u];
        if (WITH_D) ds[q] = dv[u];
        is[q] = iv[u];
        if (WITH_LO) {
            elo[q] = el[u];
            nlo[q] = nl[u];
            if (WITH_D) dlo[q] = dl[u];
        }
    }
}

// x (+ the prolongation xc[aggregate] when xc != null), b and b's lo part.
template <class T, int TH, int TW, int R>
__device__ __forceinline__ void stage_vectors(const VisitLevel<T>& V, const T* __restrict__ xin,
                                              const T* __restrict__ xc, int ti0, int tj0, T* xs, T* bs, T* bls) {
    using G = Tile<TH, TW, R>;
    constexpr int kIter = (G::S + kVisitThreads - 1) / kVisitThreads;
    const int n = V.n, nc = (n + 1) >> 1;
    T xv[kIter], cv[kIter], bv[kIter], bl[kIter];
#pragma unroll
    for (int u = 0; u < kIter; ++u) {
        const int q = threadIdx.x + u * kVisitThreads;
        const int li = q / G::SW, lj = q - li * G::SW;
        const int gi = ti0 - R + li, gj = tj0 - R + lj;
        xv[u] = cv[u] = bv[u] = bl[u] = T(0);
        if (q < G::S && gi >= 0 && gi < n && gj >= 0 && gj < n) {
            const int k = gi * n + gj;
            if (xin) xv[u] = xin[k];
            if (xc) cv[u] = xc[(gi >> 1) * nc + (gj >> 1)];
            bv[u] = V.b[k];
            if (bls && V.blo) bl[u] = V.blo[k];
        }
    }
#pragma unroll
    for (int u = 0; u < kIter; ++u) {
        const int q = threadIdx.x + u * kVisitThreads;
        if (q >= G::S) break;
        xs[q] = xc ? xv[u] + cv[u] : xv[u];
        bs[q] = bv[u];
        if (bls) bls[q] = bl[u];
    }
}

// One colour pass over the in-domain cells of colour c inside local rows /
// cols [LO, S-LO): every row of the region holds exactly half its cells of
// each colour (the staged width is even), so cells are enumerated directly.
// `zero`: the iterate is zero, x = b / d (the same bits as adding e * 0).
template <class T, int TH, int TW, int R, int LO>
__device__ __forceinline__ void stage_gs(int n, int ti0, int tj0, int c, T* xs, const T* es, const T* ns,
                                         const T* is, const T* bs, bool zero = false) {
    using G = Tile<TH, TW, R>;
    constexpr int h = G::SH - 2 * LO, hw = (G::SW - 2 * LO) / 2;
    static_assert((G::SW - 2 * LO) % 2 == 0, "even staged width");
    for (int q = threadIdx.x; q < h * hw; q += blockDim.x) {
        const int r = q / hw, k = q - r * hw;
        const int li = LO + r;
        const int gi = ti0 - R + li;
        // first local column of colour c in this row
        const int par = (c - gi - (tj0 - R) - LO) & 1;
        const int lj = LO + par + 2 * k;
        const int gj = tj0 - R + lj;
        if (gi < 0 || gi >= n || gj < 0 || gj >= n) continue;
        const int s = li * G::SW + lj;
        T v = bs[s];
        if (!zero) {
            v += es[s] * xs[s + 1];
            v += es[s - 1] * xs[s - 1];
            v += ns[s] * xs[s + G::SW];
            v += ns[s - G::SW] * xs[s - G::SW];
        }
        xs[s] = v * is[s];
    }
}

// The restricted residual of the tile (level.hpp:122-137, :214-227), four
// threads an aggregate, one per cell: each forms its cell's terms, the sums run
// over the four in the order of one thread doing all of them (same bits; cells
// outside the domain contribute zero). One thread an aggregate left one warp
// of the CTA with all of this, at the end of the chain from visit to visit
// (with the staging above: 1024^2 mixed 232 -> 208 us an iteration, FP64 335 ->
// 293 us).
template <class T, int TH, int TW, int R>
__device__ __forceinline__ void stage_residual(int n, int ti0, int tj0, const T* xs, const T* es, const T* ns,
                                               const T* ds, const T* bs, const T* elo, const T* nlo, const T* dlo,
                                               const T* bls, T* bc) {
    using G = Tile<TH, TW, R>;
    const int nc = (n + 1) >> 1;
    static_assert((TH * TW) % 32 == 0, "whole warps");
#pragma unroll 1
    for (int t = threadIdx.x; t < TH * TW; t += kVisitThreads) {
        const int agg = t >> 2, cell = t & 3, ai = agg / (TW / 2), aj = agg - ai * (TW / 2);
        const int I = (ti0 >> 1) + ai, J = (tj0 >> 1) + aj;
        const int s = (R + 2 * ai + (cell >> 1)) * G::SW + (R + 2 * aj + (cell & 1));
        const bool inside = 2 * I + (cell >> 1) < n && 2 * J + (cell & 1) < n;
        if constexpr (sizeof(T) == 8) {
            T v = fma(ds[s], xs[s], -__dmul_rn(es[s], xs[s + 1]));  // which product rounds alone is fixed here
            v = fma(-es[s - 1], xs[s - 1], v);
            v = fma(-ns[s], xs[s + G::SW], v);
            v = fma(-ns[s - G::SW], xs[s - G::SW], v);
            const T r = inside ? bs[s] - v : T(0);
            T acc = __shfl_sync(0xffffffffu, r, 0, 4);
            acc += __shfl_sync(0xffffffffu, r, 1, 4);
            acc += __shfl_sync(0xffffffffu, r, 2, 4);
            acc += __shfl_sync(0xffffffffu, r, 3, 4);
            if (cell == 0 && I < nc && J < nc) bc[I * nc + J] = acc;
        } else {
            // r = b - d x + e xE + w xW + n xN + s xS as (hi, lo) terms
            float vh[6], vl[6];
            auto term = [&](int k, float ch, float cl, float x, float sign) {
                const float p = ch * x;
                const float pe = fmaf(ch, x, -p);
                vh[k] = inside ? sign * p : 0.f;
                vl[k] = inside ? sign * (pe + cl * x) : 0.f;
            };
            vh[0] = inside ? bs[s] : 0.f;
            vl[0] = inside ? bls[s] : 0.f;
            term(1, ds[s], dlo[s], xs[s], -1.f);
            term(2, es[s], elo[s], xs[s + 1], 1.f);
            term(3, es[s - 1], elo[s - 1], xs[s - 1], 1.f);
            term(4, ns[s], nlo[s], xs[s + G::SW], 1.f);
            term(5, ns[s - G::SW], nlo[s - G::SW], xs[s - G::SW], 1.f);
            DF acc{0.f, 0.f};
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
                for (int k = 0; k < 6; ++k)
                    df_add(acc, __shfl_sync(0xffffffffu, vh[k], c, 4), __shfl_sync(0xffffffffu, vl[k], c, 4));
            if (cell == 0 && I < nc && J < nc) bc[I * nc + J] = acc.hi + acc.lo;
        }
    }
}

template <class T, int TH, int TW>
struct VisitSmem {
    // FP64: e, nf, d, id, x, b. FP32: + e_lo, nf_lo, d_lo, b_lo.
    static constexpr int arrays = sizeof(T) == 8 ? 6 : 10;
    static constexpr size_t bytes = sizeof(T) * arrays * Tile<TH, TW, 3>::S;
};
template <class T, int TH, int TW>
struct PostSmem {
    static constexpr size_t bytes = sizeof(T) * 5 * Tile<TH, TW, 2>::S;
};

// Pre-smoothing (1 sweep: red then black), residual, restriction. xin == null
// means the iterate is known to be zero (first call from the parent).
template <class T, int TH, int TW>
__global__ void __launch_bounds__(kVisitThreads) k_visit_pre(VisitLevel<T> V, const T* __restrict__ xin, T* __restrict__ xout,
                                                   T* __restrict__ bc) {
    constexpr int R = 3;
    constexpr bool LO = sizeof(T) == 4;
    using G = Tile<TH, TW, R>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* es = reinterpret_cast<T*>(smem_raw);
    T* ns = es + G::S;
    T* ds = ns + G::S;
    T* is = ds + G::S;
    T* xs = is + G::S;
    T* bs = xs + G::S;
    T* elo = LO ? bs + G::S : nullptr;
    T* nlo = LO ? elo + G::S : nullptr;
    T* dlo = LO ? nlo + G::S : nullptr;
    T* bls = LO ? dlo + G::S : nullptr;
    const int n = V.n;
    const int tiles_x = (n + TW - 1) / TW, tiles = tiles_x * ((n + TH - 1) / TH);
    bool waited = false;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int ti0 = (tile / tiles_x) * TH, tj0 = (tile % tiles_x) * TW;
        stage_coeffs<T, TH, TW, R, true, LO>(V, ti0, tj0, es, ns, ds, is, elo, nlo, dlo);
        if (!waited) {
            pdl_enter();
            waited = true;
        }
        stage_vectors<T, TH, TW, R>(V, xin, nullptr, ti0, tj0, xs, bs, bls);
        __syncthreads();
        stage_gs<T, TH, TW, R, 1>(n, ti0, tj0, 0, xs, es, ns, is, bs, !xin);  // red, rings <= 2
        __syncthreads();
        stage_gs<T, TH, TW, R, 2>(n, ti0, tj0, 1, xs, es, ns, is, bs);  // black, rings <= 1
        __syncthreads();
        stage_residual<T, TH, TW, R>(n, ti0, tj0, xs, es, ns, ds, bs, elo, nlo, dlo, bls, bc);
        // the smoothed iterate of the tile
        for (int q = threadIdx.x; q < TH * TW; q += blockDim.x) {
            const int li = q / TW, lj = q - li * TW;
            const int gi = ti0 + li, gj = tj0 + lj;
            if (gi < n && gj < n) xout[gi * n + gj] = xs[(R + li) * G::SW + (R + lj)];
        }
        __syncthreads();
    }
    if (!waited) pdl_enter();
}

// The W-cycle's second call of a level follows the first call's
// post-smoothing directly: post (prolongation, black, red) then pre (red,
// black, residual, restriction). The two red passes in the middle read the
// same black values and produce the same result, so one is kept: prolongation
// + black + red + black + residual/restriction in one kernel, halo 4.
template <class T, int TH, int TW>
struct MidSmem {
    static constexpr int arrays = sizeof(T) == 8 ? 6 : 10;
    static constexpr size_t bytes = sizeof(T) * arrays * Tile<TH, TW, 4>::S;
};

template <class T, int TH, int TW>
__global__ void __launch_bounds__(kVisitThreads) k_visit_mid(VisitLevel<T> V, const T* __restrict__ xin,
                                                   const T* __restrict__ xc, T* __restrict__ xout,
                                                   T* __restrict__ bc) {
    constexpr int R = 4;
    constexpr bool LO = sizeof(T) == 4;
    using G = Tile<TH, TW, R>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* es = reinterpret_cast<T*>(smem_raw);
    T* ns = es + G::S;
    T* ds = ns + G::S;
    T* is = ds + G::S;
    T* xs = is + G::S;
    T* bs = xs + G::S;
    T* elo = LO ? bs + G::S : nullptr;
    T* nlo = LO ? elo + G::S : nullptr;
    T* dlo = LO ? nlo + G::S : nullptr;
    T* bls = LO ? dlo + G::S : nullptr;
    const int n = V.n;
    const int tiles_x = (n + TW - 1) / TW, tiles = tiles_x * ((n + TH - 1) / TH);
    bool waited = false;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int ti0 = (tile / tiles_x) * TH, tj0 = (tile % tiles_x) * TW;
        stage_coeffs<T, TH, TW, R, true, LO>(V, ti0, tj0, es, ns, ds, is, elo, nlo, dlo);
        if (!waited) {
            pdl_enter();
            waited = true;
        }
        stage_vectors<T, TH, TW, R>(V, xin, xc, ti0, tj0, xs, bs, bls);  // x + prolongation
        __syncthreads();
        stage_gs<T, TH, TW, R, 1>(n, ti0, tj0, 1, xs, es, ns, is, bs);  // post black, rings <= 3
        __syncthreads();
        stage_gs<T, TH, TW, R, 2>(n, ti0, tj0, 0, xs, es, ns, is, bs);  // red (post and pre), rings <= 2
        __syncthreads();
        stage_gs<T, TH, TW, R, 3>(n, ti0, tj0, 1, xs, es, ns, is, bs);  // pre black, rings <= 1
        __syncthreads();
        stage_residual<T, TH, TW, R>(n, ti0, tj0, xs, es, ns, ds, bs, elo, nlo, dlo, bls, bc);
        for (int q = threadIdx.x; q < TH * TW; q += blockDim.x) {
            const int li = q / TW, lj = q - li * TW;
            const int gi = ti0 + li, gj = tj0 + lj;
            if (gi < n && gj < n) xout[gi * n + gj] = xs[(R + li) * G::SW + (R + lj)];
        }
        __syncthreads();
    }
    if (!waited) pdl_enter();
}

// Prolongation + post-smoothing (1 sweep: black then red). On level 0 (r
// given) also r . z and beta, like k_gs0_dot.
template <class T, int TH, int TW>
__global__ void __launch_bounds__(kVisitThreads) k_visit_post(VisitLevel<T> V, const T* __restrict__ xin,
                                                    const T* __restrict__ xc, T* __restrict__ xout,
                                                    const double* __restrict__ r, CgState* st, double* partials) {
    constexpr int R = 2;
    using G = Tile<TH, TW, R>;
    __shared__ double red[256];  // block_sum_wide: one double per thread
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* es = reinterpret_cast<T*>(smem_raw);
    T* ns = es + G::S;
    T* is = ns + G::S;
    T* xs = is + G::S;
    T* bs = xs + G::S;
    const int n = V.n;
    const int tiles_x = (n + TW - 1) / TW, tiles = tiles_x * ((n + TH - 1) / TH);
    double acc = 0.0;
    bool waited = false;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int ti0 = (tile / tiles_x) * TH, tj0 = (tile % tiles_x) * TW;
        stage_coeffs<T, TH, TW, R, false, false>(V, ti0, tj0, es, ns, nullptr, is, nullptr, nullptr, nullptr);
        if (!waited) {
            pdl_enter();
            waited = true;
        }
        stage_vectors<T, TH, TW, R>(V, xin, xc, ti0, tj0, xs, bs, nullptr);
        __syncthreads();
        stage_gs<T, TH, TW, R, 1>(n, ti0, tj0, 1, xs, es, ns, is, bs);  // black, rings <= 1
        __syncthreads();
        stage_gs<T, TH, TW, R, 2>(n, ti0, tj0, 0, xs, es, ns, is, bs);  // red, ring 0
        __syncthreads();
        for (int q = threadIdx.x; q < TH * TW; q += blockDim.x) {
            const int li = q / TW, lj = q - li * TW;
            const int gi = ti0 + li, gj = tj0 + lj;
            if (gi < n && gj < n) {
                const int k = gi * n + gj;
                const T v = xs[(R + li) * G::SW + (R + lj)];
                xout[k] = v;
                if (r) acc += r[k] * widen_f32(v);
            }
        }
        __syncthreads();
    }
    if (!waited) pdl_enter();
    if (!r) return;
    double tot;
    if (!grid_sum_last(acc, partials, &st->ticket[1], red, tot)) return;
    if (threadIdx.x == 0) {
        st->beta = st->it == 0 ? 0.0 : (tot - st->rzo) / st->rz;
        st->rz = tot;
    }
}

}  // namespace dgpu
