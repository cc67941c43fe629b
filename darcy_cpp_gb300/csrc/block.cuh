// Block-engine building blocks: one CTA owns one problem (layout of its
// scratch, hierarchy setup, operator application, one preconditioner cycle).
// Shared by the batched engine (kernels.cu) and the allocation-free
// preconditioner entry point (noalloc.cu).
#pragma once

#include <math.h>

#include "engine.h"
#include "patch.cuh"

namespace dgpu {

// y = A x at one cell, FP64 (level.hpp:105-119).
__device__ __forceinline__ double apply_cell(const Lvl64& L, const double* __restrict__ x, int i, int j) {
    const int n = L.n;
    const int64_t k = (int64_t)i * n + j;
    double v = L.d[k] * x[k];
    if (j + 1 < n) v -= L.e[k] * x[k + 1];
    if (j > 0) v -= L.e[k - 1] * x[k - 1];
    if (i + 1 < n) v -= L.nf[k] * x[k + n];
    if (i > 0) v -= L.nf[k - n] * x[k - n];
    return v;
}

// Per-CTA layout for one side-n problem, every level in the padded layout of
// patch.cuh. Global arena (L2-resident while the CTA works on the problem):
// the FP64 hierarchy (e, nf, d, id per level, wb/sb boundary vectors), the
// FP64 CG vectors r, p, Ap and u, the cycle's arrays that are not in shared
// memory, and the scratch used once per problem to build the dense tail. The
// level-0 vectors of an FP64 cycle are CG's own: r (right-hand side) and z
// (iterate).
//
// Shared memory, up to `sbudget` bytes: the dense tail operator, then the
// cycle's arrays level by level from the coarsest (a visit of level l moves
// ~4^-l of level 0's bytes and happens 2^l times per W-cycle, so a byte of a
// coarse level is read more often), in a level the arrays most read first.
//
// Dense tail: the levels from tl (the first level of side <= kBlockTailSide,
// when that is not level 0) down implement the fixed map "x = 0, then gamma
// cycles"; it is built once per problem as an N x N matrix (N = side_tl^2,
// one column per unit right-hand side, all columns at once) and the cycle
// applies it with one product per visit of level tl - 1 instead of visiting
// 2^k levels below. Same operator as the recursion, to rounding.
// Shared by host sizing and device carving (gbase/sbase == null: size only);
// returns the arena's bytes.
constexpr int kBlockTailSide = 8;
constexpr int kBlockLevels = 20;  // sides below 2^17: more than the int cell index allows

template <class T>
struct BlockViews {
    Lvl64 h[kBlockLevels];      // FP64 hierarchy; .n is the side, arrays padded
    PLvl<T> lv[kBlockLevels];   // the cycle's levels
    PLvl<T> lm[kBlockLevels];   // tail construction: the tail levels with N right-hand sides, in the
                                // cycle's precision (FP32 copies of the coefficients for the mixed form)
    double *r, *p, *ap, *u;     // CG vectors (padded)
    T* tail;                    // dense tail operator (ntail rows of tail_pitch), or null
    int nlev, tl, ntail;        // ntail: padded cells of level tl
};

template <class T>
__host__ __device__ size_t carve(int n, char* gbase, char* sbase, size_t sbudget, BlockViews<T>* v) {
    size_t goff = 0, soff = 0;
    // `lead` and `trail` bytes of guard around an array of `bytes` (multiples of 16)
    auto gtake = [&](size_t lead, size_t bytes, size_t trail) -> char* {
        char* ptr = gbase ? gbase + goff + ((lead + 255) & ~(size_t)255) : nullptr;
        goff += ((lead + 255) & ~(size_t)255) + ((bytes + trail + 255) & ~(size_t)255);
        return ptr;
    };
    auto take = [&](size_t lead, size_t bytes, size_t trail) -> char* {
        lead = (lead + 15) & ~(size_t)15;
        const size_t all = lead + ((bytes + trail + 15) & ~(size_t)15);
        if (soff + all <= sbudget) {
            char* ptr = sbase ? sbase + soff + lead : nullptr;
            soff += all;
            return ptr;
        }
        return gtake(lead, bytes, trail);
    };
    int sides[kBlockLevels];
    int nlev = 0;
    for (int s = n; nlev < kBlockLevels;) {
        sides[nlev++] = s;
        if (s <= 1) break;
        s = (s + 1) / 2;
    }
    int tl = 0;
    for (int l = 1; l < nlev; ++l)
        if (sides[l] <= kBlockTailSide) {
            tl = l;
            break;
        }
    const bool fp32 = sizeof(T) == 4;
    const size_t w = sizeof(T);
    auto padded = [&](int l) { return (size_t)(2 * ((sides[l] + 1) / 2)); };
    const int ntail = tl ? (int)(padded(tl) * padded(tl)) : 0;
    const int cyc_levels = tl ? tl : nlev;  // levels the cycle itself visits
    if (v) {
        v->nlev = nlev;
        v->tl = tl;
        v->ntail = ntail;
        v->tail = nullptr;
    }
    if (tl) {
        T* tp = (T*)take(0, w * (size_t)ntail * tail_pitch<T>(ntail), 0);
        if (v) v->tail = tp;
    }
    for (int l = 0; l < nlev; ++l) {
        const size_t np = padded(l), m = np * np;
        Lvl64 H;
        H.n = sides[l];
        H.e = (double*)gtake(16, 8 * m, 0);
        H.nf = (double*)gtake(8 * np, 8 * m, 0);
        H.d = (double*)gtake(0, 8 * m, 0);
        H.id = (double*)gtake(0, 8 * m, 0);
        H.wb = (double*)gtake(0, 8 * (size_t)sides[l], 0);
        H.sb = (double*)gtake(0, 8 * (size_t)sides[l], 0);
        if (v) v->h[l] = H;
    }
    const size_t np0 = padded(0), m0 = np0 * np0;
    {
        double* p = (double*)gtake(8 * np0, 8 * m0, 8 * np0);
        double* ap = (double*)gtake(0, 8 * m0, 0);
        double* u = (double*)gtake(8 * np0, 8 * m0, 8 * np0);
        double* r = fp32 ? (double*)gtake(0, 8 * m0, 0) : nullptr;
        if (v) {
            v->p = p;
            v->ap = ap;
            v->u = u;
            v->r = r;
        }
    }
    for (int l = nlev - 1; l >= 0; --l) {
        const size_t np = padded(l), m = np * np;
        PLvl<T> V{};
        V.n = sides[l];
        V.nc = (int)(np / 2);
        V.np = (int)np;
        V.rcp = row_reciprocal(V.nc);
        if (!tl || l <= tl) {
            // most read first: the iterate (every pass reads five values a
            // cell), the faces, 1/d and the right-hand side, d (residual only)
            V.x = (T*)take(w * np, w * m, w * np);
            if (l < cyc_levels) {
                // (FP64: the hierarchy itself where shared memory has no room)
                auto coeff = [&](size_t lead, const double* h) -> const T* {
                    const size_t ld = (lead + 15) & ~(size_t)15, all = ld + ((w * m + 15) & ~(size_t)15);
                    if (!fp32 && soff + all > sbudget) return (const T*)h;
                    return (const T*)take(lead, w * m, 0);
                };
                V.e = coeff(16, v ? v->h[l].e : nullptr);
                V.nf = coeff(w * np, v ? v->h[l].nf : nullptr);
                V.id = coeff(0, v ? v->h[l].id : nullptr);
                V.b = (T*)take(0, w * m, 0);
                V.d = coeff(0, v ? v->h[l].d : nullptr);
            } else {
                V.b = (T*)take(0, w * m, 0);  // the tail's input
            }
        }
        if (v) v->lv[l] = V;
    }
    if (v && !fp32) v->r = (double*)v->lv[0].b;
    if (tl) {  // tail construction scratch: every tail level with ntail right-hand sides
        for (int l = tl; l < nlev; ++l) {
            const size_t np = padded(l), m = np * np, st = (size_t)rhs_stride((int)np);
            PLvl<T> M{};
            M.n = sides[l];
            M.nc = (int)(np / 2);
            M.np = (int)np;
            M.rcp = row_reciprocal(M.nc);
            M.rper = row_reciprocal(M.nc * M.nc);
            M.x = (T*)gtake(w * np, w * st * ntail, 0);
            M.b = (T*)gtake(w * np, w * st * ntail, 0);
            if (fp32) {
                M.e = (const T*)gtake(16, w * m, 0);
                M.nf = (const T*)gtake(w * np, w * m, 0);
                M.d = (const T*)gtake(0, w * m, 0);
                M.id = (const T*)gtake(0, w * m, 0);
            } else if (v) {
                M.e = (const T*)v->h[l].e;
                M.nf = (const T*)v->h[l].nf;
                M.d = (const T*)v->h[l].d;
                M.id = (const T*)v->h[l].id;
            }
            if (v) v->lm[l] = M;
        }
    }
    return goff;
}

// Zeroes what the stencils may read before a pass has written it: the guards
// around the arrays, the iterates (at the end of a row a pass reads the next
// row's first cell, times a zero face, which must be finite), the padding of
// r, u and the coarse right-hand sides. Needed once per layout (no pass writes
// a guard, padding stays zero) and after a problem that left non-finite values.
template <class T>
__device__ void block_clear(const BlockViews<T>& V) {
    const int t0 = threadIdx.x, ts = blockDim.x;
    auto zero = [&](auto* ptr, int count) {
        for (int t = t0; t < count; t += ts) ptr[t] = 0;
    };
    for (int l = 0; l < V.nlev; ++l) {
        const Lvl64& H = V.h[l];
        const int np = 2 * ((H.n + 1) / 2), m = np * np;
        zero(H.e - 2, 2);
        zero(H.nf - np, np);
        const PLvl<T>& A = V.lv[l];
        if (A.x) {
            zero(A.x - np, m + 2 * np);
            zero(A.b, m);
        }
        if (A.e) {
            zero((T*)A.e - 2, 2);
            zero((T*)A.nf - np, np);
        }
        if (V.tl && l >= V.tl) {
            const PLvl<T>& M = V.lm[l];
            zero(M.x - np, rhs_stride(np) * V.ntail);
            zero(M.b - np, rhs_stride(np) * V.ntail);
            zero((T*)M.e - 2, 2);
            zero((T*)M.nf - np, np);
        }
    }
    const int np = V.lv[0].np, m = np * np;
    zero(V.p - np, np);
    zero(V.p + m, np);
    zero(V.u - np, m + 2 * np);
    zero(V.r, m);
    __syncthreads();
}

// Cell c of the cycle's copy of a level, in the cycle's precision (FP32 for
// the mixed form, shared-memory copies for FP64 arrays held on chip), written
// while the FP64 values are in registers: reading the level back for it took a
// fifth of the mixed form's setup. (ce, cn): the faces with those on the
// domain's boundary zero. The FP32 reciprocal diagonal is the correctly
// rounded reciprocal of the FP32 d (the FP64 id, one FP64 division per cell, is
// built for FP32 cycles on the coarsest level only); FP64 copies take id as built.
template <class T>
__device__ __forceinline__ void block_emit_cell(const Lvl64& H, const PLvl<T>& V, int c, double ce, double cn,
                                                double dd, double id) {
    if (!V.e) return;  // not visited
    if constexpr (sizeof(T) == 4) {
        ((T*)V.e)[c] = narrow_to<T>(ce);
        ((T*)V.nf)[c] = narrow_to<T>(cn);
        const T dk = narrow_to<T>(dd);
        ((T*)V.d)[c] = dk;
        // (FP64 zero, tested off the FP64 pipe: a cell outside the domain)
        ((T*)V.id)[c] = __double_as_longlong(dd) != 0 ? __frcp_rn(dk) : T(0);
    } else {
        if (V.e != H.e) ((T*)V.e)[c] = ce;
        if (V.nf != H.nf) ((T*)V.nf)[c] = cn;
        if (V.d != H.d) ((T*)V.d)[c] = dd;
        if (V.id != H.id) ((T*)V.id)[c] = id;
    }
}

// The fine level (level.hpp:79-97, validation solver.hpp:68-77) with every
// face computed once (one division per face instead of two; FP64 division is
// tens of instructions on the narrow FP64 pipe): the east/north faces and the
// boundary faces first, then the diagonal from the stored faces in
// build_fine's summation order. A cell's west/south face is its neighbour's
// east/north face, the same bits since harmonic() is symmetric, so the level
// equals build_fine's bit for bit. with_id false leaves id unwritten (the
// FP32 cycle computes its own reciprocal from the FP32 diagonal). `a` has
// pitch n, the level the padded pitch; rows by patch_row, an integer division
// being ~25 instructions a cell.
template <class T>
__device__ __forceinline__ void block_build_fine(const double* __restrict__ a, const Lvl64& L, const PLvl<T>& V,
                                                 unsigned long long* bad, bool with_id, bool emit) {
    const int n = L.n, nc = V.nc, np = V.np, m = np * np;
    const unsigned rcp = V.rcp;
    for (int c = threadIdx.x; c < m; c += blockDim.x) {
        const int i = patch_row(c >> 1, nc, rcp), j = c - i * np;
        double e = 0.0, nf = 0.0;
        if (i < n && j < n) {
            const int64_t k = (int64_t)i * n + j;
            const double ac = a[k];
            if (!(ac > 0.0) || !isfinite(ac)) atomicMin(bad, (unsigned long long)k);
            e = (j + 1 < n) ? harmonic(ac, a[k + 1]) : ac;
            nf = (i + 1 < n) ? harmonic(ac, a[k + n]) : ac;
            if (j == 0) L.wb[i] = ac;
            if (i == 0) L.sb[j] = ac;
        }
        L.e[c] = e;
        L.nf[c] = nf;
    }
    __syncthreads();
    for (int c = threadIdx.x; c < m; c += blockDim.x) {
        const int i = patch_row(c >> 1, nc, rcp), j = c - i * np;
        double dd = 0.0, id = 0.0, e = 0.0, nf = 0.0;
        if (i < n && j < n) {
            const double w = (j > 0) ? L.e[c - 1] : L.wb[i];
            const double s = (i > 0) ? L.nf[c - np] : L.sb[j];
            e = L.e[c];
            nf = L.nf[c];
            dd = e + w + nf + s;
            if (with_id) id = 1.0 / dd;
        }
        L.d[c] = dd;
        if (with_id) L.id[c] = id;
        if (emit) block_emit_cell<T>(L, V, c, j + 1 < n ? e : 0.0, i + 1 < n ? nf : 0.0, dd, id);
    }
    __syncthreads();
}

// Galerkin coarse operator (coarsen in setup.cuh) between padded levels.
template <class T>
__device__ __forceinline__ void block_coarsen(const Lvl64& F, const Lvl64& C, const PLvl<T>& V, bool with_id,
                                              bool emit) {
    const int n = F.n, np = 2 * ((n + 1) / 2), nc = C.n, npc = V.np, mc = npc * npc;
    for (int c = threadIdx.x; c < mc; c += blockDim.x) {
        const int I = patch_row(c >> 1, V.nc, V.rcp), J = c - I * npc;
        double ce = 0.0, cw = 0.0, cn = 0.0, cs = 0.0, dd = 0.0, id = 0.0;
        if (I < nc && J < nc) {
            const int i0 = 2 * I, i1 = (2 * I + 1 < n) ? 2 * I + 1 : 2 * I;
            const int j0 = 2 * J, j1 = (2 * J + 1 < n) ? 2 * J + 1 : 2 * J;
            for (int i = i0; i <= i1; ++i) {
                ce += F.e[i * np + j1];
                cw += (j0 > 0) ? F.e[i * np + j0 - 1] : F.wb[i];
            }
            for (int j = j0; j <= j1; ++j) {
                cn += F.nf[i1 * np + j];
                cs += (i0 > 0) ? F.nf[(i0 - 1) * np + j] : F.sb[j];
            }
            dd = ce + cw + cn + cs;
            if (with_id) id = 1.0 / dd;
            if (J == 0) C.wb[I] = cw;
            if (I == 0) C.sb[J] = cs;
        }
        C.e[c] = ce;
        C.nf[c] = cn;
        C.d[c] = dd;
        if (with_id) C.id[c] = id;
        if (emit) block_emit_cell<T>(C, V, c, J + 1 < nc ? ce : 0.0, I + 1 < nc ? cn : 0.0, dd, id);
    }
}

// The faces on the domain's east and north boundary enter d and the coarser
// levels' faces only; zero, they drop out of every stencil (patch.cuh).
__device__ __forceinline__ void block_drop_boundary(const Lvl64& L) {
    const int n = L.n, np = 2 * ((n + 1) / 2);
    for (int t = threadIdx.x; t < n; t += blockDim.x) {
        L.e[t * np + n - 1] = 0.0;
        L.nf[(n - 1) * np + t] = 0.0;
    }
}

// y = A x of two horizontally adjacent cells (pair q of a padded level of
// pitch 2 * n2), terms in apply_cell's order.
__device__ __forceinline__ double2 pair_apply(const Lvl64& L, const double* __restrict__ x, int q, int n2,
                                              double2 xc) {
    const double2* x2 = reinterpret_cast<const double2*>(x);
    const double2* nf2 = reinterpret_cast<const double2*>(L.nf);
    const double2 dd = reinterpret_cast<const double2*>(L.d)[q], ee = reinterpret_cast<const double2*>(L.e)[q];
    const double2 nn = nf2[q], ns = nf2[q - n2], xn = x2[q + n2], xs = x2[q - n2];
    double v0 = dd.x * xc.x, v1 = dd.y * xc.y;
    v0 -= ee.x * xc.y;
    v1 -= ee.y * x[2 * q + 2];
    v0 -= L.e[2 * q - 1] * x[2 * q - 1];
    v1 -= ee.x * xc.x;
    v0 -= nn.x * xn.x;
    v1 -= nn.y * xn.y;
    v0 -= ns.x * xs.x;
    v1 -= ns.y * xs.y;
    return make_double2(v0, v1);
}

// y = A x over a block, FP64, returning then(sum x . y).
//
// kAhead: ask for the next pair's lines one step ahead, as the mixed form's
// other FP64 passes do. Its problems together exceed L2 (4 CTAs an SM hold
// ~210 MB at 64^2), so a step otherwise starts with a DRAM round trip: 4096 x
// 64^2 12.9 -> 12.5 ms, 512 x 128^2 18.3 -> 17.6 ms. The FP64 form is bound by the FP64 pipe and
// measured level (64^2) to 2% slower (128^2): it does not.
template <bool kAhead, class F>
__device__ __forceinline__ double block_apply_dot(const Lvl64& L, const double* x, double* y, double* red,
                                                  F&& then) {
    const int n2 = (L.n + 1) / 2, m2 = 2 * n2 * n2;
    double acc = 0.0;
    for (int q = threadIdx.x; q < m2; q += blockDim.x) {
        if (const int z = q + blockDim.x; kAhead && z < m2) {
            prefetch_l2(x + 2 * (z + n2));
            prefetch_l2(L.e + 2 * z);
            prefetch_l2(L.nf + 2 * z);
            prefetch_l2(L.d + 2 * z);
        }
        const double2 xc = reinterpret_cast<const double2*>(x)[q];
        const double2 v = pair_apply(L, x, q, n2, xc);
        reinterpret_cast<double2*>(y)[q] = v;
        acc += xc.x * v.x;
        acc += xc.y * v.y;
    }
    return block_sum_then(acc, red, then);
}

// b = r in the cycle's precision and the cycle's first pass (colour 0 from a
// zero iterate) for pair q. The two cells of a pair are one of each colour.
template <class T>
__device__ __forceinline__ void pair_start_cycle(const PLvl<T>& L, int q, double2 rv) {
    const int odd = patch_row(q, L.nc, L.rcp) & 1;  // n2 = nc pairs a row: the row's parity
    const T b0 = narrow_to<T>(rv.x), b1 = narrow_to<T>(rv.y);
    if constexpr (sizeof(T) == 4) {  // (FP64: b is r itself)
        Pair_t<T> bb;
        bb.x = b0;
        bb.y = b1;
        reinterpret_cast<Pair_t<T>*>(L.b)[q] = bb;
    }
    L.x[2 * q + odd] = (odd ? b1 : b0) * L.id[2 * q + odd];
}

// z = M r for one problem, r already handed over by pair_start_cycle on every
// pair (multigrid) and the CTA synchronised since; returns then(r . z). The
// cycle's iterate lv[0].x is z, in the cycle's precision.
template <class T, class F>
__device__ double block_precondition(const BatchArgs& A, const BlockViews<T>& V, double* red, F&& then) {
    const PLvl<T>& L = V.lv[0];
    const double* r = V.r;
    double acc = 0.0;
    if (A.pc == kPcMultigrid) {
        const double* id64 = sizeof(T) == 4 ? V.h[V.nlev - 1].id : nullptr;  // FP64 exact coarsest solve
        if (V.nlev == 1) {  // one cell, solved exactly
            if (threadIdx.x == 0) {
                L.x[0] = id64 ? (T)((double)L.b[0] * id64[0]) : L.b[0] * L.id[0];
                acc = r[0] * widen_f32(L.x[0]);
            }
        } else {
            patch_cycle<T>(V.lv, V.nlev, A.pre, A.post, A.gamma, id64, V.tail, V.tl);
            // the last colour-0 pass and r . z
            const int nc = L.nc, cnt = nc * nc, np = L.np;
            for (int q = threadIdx.x; q < cnt; q += blockDim.x) {
                const int k = 2 * q + 2 * patch_row(q, nc, L.rcp) * nc;
                T o0, o1;
                if (const int z = q + blockDim.x; sizeof(T) == 4 && z < cnt) {
                    const int kz = 2 * z + 2 * patch_row(z, nc, L.rcp) * nc;
                    prefetch_l2(r + kz);
                    prefetch_l2(r + kz + np);
                }
                patch_red(L, L.x, L.b, k, o0, o1);
                L.x[k] = o0;
                L.x[k + np + 1] = o1;
                const double2 r0 = load_pair(r + k), r1 = load_pair(r + k + np);
                acc += r0.x * widen_f32(o0);
                acc += r0.y * widen_f32(L.x[k + 1]);
                acc += r1.x * widen_f32(L.x[k + np]);
                acc += r1.y * widen_f32(o1);
            }
        }
    } else {  // (FP64 only)
        const int m = L.np * L.np;
        for (int k = threadIdx.x; k < m; k += blockDim.x) {
            const double zk = A.pc == kPcJacobi ? r[k] * V.h[0].id[k] : r[k];
            L.x[k] = (T)zk;
            acc += r[k] * zk;
        }
    }
    return block_sum_then(acc, red, then);
}

// The dense tail of one problem: column j = the tail map applied to e_j, all
// columns at once, in the cycle's precision (the FP32 smoothing of the mixed
// form, with the exact 1 x 1 coarsest solve in FP64), stored row-major; rows
// and columns of padding cells are zero.
// Building it in FP64 cost the mixed form about a third of its FP64 work. Not
// inlined: called once a problem, and expanded in the solve it costs the
// loop there registers (4096 x 64^2 mixed 12.54 -> 12.36 ms).
template <class T>
__device__ __noinline__ void block_build_tail(const BatchArgs& A, const BlockViews<T>& V) {
    const int tl = V.tl, N = V.ntail, pitch = tail_pitch<T>(N);
    const PLvl<T>& L = V.lm[tl];
    const int st = rhs_stride(L.np);
    for (int t = threadIdx.x; t < N * N; t += blockDim.x) {
        const int j = t / N, k = t - j * N;  // right-hand side j, cell k
        L.b[j * st + k] = (k == j && j / L.np < L.n && j % L.np < L.n) ? T(1) : T(0);
    }
    __syncthreads();
    patch_cycle_m<T>(V.lm, tl, V.nlev, A.pre, A.post, A.gamma, A.gamma, N,
                     sizeof(T) == 4 ? V.h[V.nlev - 1].id : nullptr);
    for (int t = threadIdx.x; t < N * N; t += blockDim.x) {
        const int j = t / N, k = t - j * N;
        V.tail[k * pitch + j] = L.x[j * st + k];
    }
    __syncthreads();
}

// Build the hierarchy of one problem into the CTA's arena (and its dense
// tail). Returns the first invalid permeability index (~0 if valid).
template <class T>
__device__ unsigned long long block_setup(const BatchArgs& A, const double* a, const BlockViews<T>& V,
                                          unsigned long long* s_bad) {
    if (threadIdx.x == 0) *s_bad = ~0ull;
    __syncthreads();
    // FP64 reciprocal diagonals: every level for an FP64 cycle; level 0 for
    // the Jacobi preconditioner; otherwise the coarsest level's exact solve only.
    const bool fp64_id = sizeof(T) == 8 || A.pc != kPcMultigrid;
    const bool mg = A.pc == kPcMultigrid;
    block_build_fine<T>(a, V.h[0], V.lv[0], s_bad, fp64_id || V.nlev == 1, mg);
    for (int l = 1; l < V.nlev; ++l) {
        block_coarsen<T>(V.h[l - 1], V.h[l], V.lv[l], fp64_id || l == V.nlev - 1, mg);
        __syncthreads();
        block_drop_boundary(V.h[l - 1]);  // (read by the coarsening just done)
    }
    block_drop_boundary(V.h[V.nlev - 1]);
    __syncthreads();
    if (mg) {
        if constexpr (sizeof(T) == 4) {  // (FP64: the hierarchy itself)
            for (int l = V.tl ? V.tl : V.nlev; l < V.nlev; ++l) {
                const Lvl64& H = V.h[l];
                const int m = V.lm[l].np * V.lm[l].np;
                for (int c = threadIdx.x; c < m; c += blockDim.x)
                    block_emit_cell<T>(H, V.lm[l], c, H.e[c], H.nf[c], H.d[c], 0.0);
            }
        }
        __syncthreads();
        if (V.tl && *s_bad == ~0ull) block_build_tail<T>(A, V);
    }
    __syncthreads();
    return *s_bad;
}

}  // namespace dgpu
