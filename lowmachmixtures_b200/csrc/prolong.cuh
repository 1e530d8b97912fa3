// prolong.cuh - stag_prolongation (stag_mg_solver.f90:1424-1633) by pairs of
// fine faces of a row.
//
// The two fine cells 2h, 2h+1 of a row lie in one coarse cell and read the same
// coarse rows, so a thread that takes both reads 8 to 12 coarse values per
// component instead of 4 to 8 per face, forms the row offsets once, and reads
// and writes phi in pairs.  One face per thread was bound by its instructions
// (327 per cell, 60% of the issue slots at 128^3 FP32), not by memory.
// Same expressions as prolong_one: same bits.
#pragma once
#include "kernels.cuh"

namespace lmm {

// where a fine pair sits on the coarse grid: its cell, the cells left and
// right of it, and the coarse rows of its transverse and normal offsets
struct PairAt {
    int h, l, r;             // along x
    int y, yo, yn;           // row bases: the cell's, the nearer neighbour's (odd: +1, even: -1), +1
    int z, zo, zn;           // plane bases likewise
    int jodd, kodd;
};
template <int DM>
__device__ __forceinline__ PairAt pair_at(const Dims& Dc, int h, int j, int k) {
    PairAt p;
    p.h = h;
    p.l = h == 0 ? Dc.nx - 1 : h - 1;
    p.r = h == Dc.nx - 1 ? 0 : h + 1;
    p.jodd = j & 1;
    p.kodd = DM == 3 ? (k & 1) : 0;
    const int cy = j >> 1, yn = cy == Dc.ny - 1 ? 0 : cy + 1, ym = cy == 0 ? Dc.ny - 1 : cy - 1;
    p.y = cy * Dc.nx;
    p.yn = yn * Dc.nx;
    p.yo = p.jodd ? p.yn : ym * Dc.nx;
    p.z = p.zo = p.zn = 0;
    const int pl = Dc.nx * Dc.ny;
    if constexpr (DM == 3) {
        const int cz = k >> 1, zn = cz == Dc.nz - 1 ? 0 : cz + 1, zm = cz == 0 ? Dc.nz - 1 : cz - 1;
        p.z = cz * pl;
        p.zn = zn * pl;
        p.zo = p.kodd ? p.zn : zm * pl;
    } else {
        p.z = k * pl;   // the instance of a batch
    }
    return p;
}

// v0, v1 += the interpolated coarse correction of component COMP
template <class T, int DM, int COMP, bool W>
__device__ __forceinline__ void prolong_pair(const T* q, const PairAt& p, T& v0, T& v1) {
    auto Q = [&](int x, int y, int z) { return ld(q, x + y + z); };
    if constexpr (DM == 2) {
        if constexpr (COMP == 0) {
            const T a = Q(p.h, p.y, p.z), b = Q(p.h, p.yo, p.z), c = Q(p.r, p.y, p.z), d = Q(p.r, p.yo, p.z);
            v0 = madd<W>(T(0.25), b, madd<W>(T(0.75), a, v0));
            v1 = madd<W>(T(0.125), d, madd<W>(T(0.375), c, madd<W>(T(0.125), b, madd<W>(T(0.375), a, v1))));
        } else {
            const T a = Q(p.h, p.y, p.z), l = Q(p.l, p.y, p.z), r = Q(p.r, p.y, p.z);
            if (!p.jodd) {
                v0 = madd<W>(T(0.25), l, madd<W>(T(0.75), a, v0));
                v1 = madd<W>(T(0.25), r, madd<W>(T(0.75), a, v1));
            } else {
                const T A = Q(p.h, p.yn, p.z), Lc = Q(p.l, p.yn, p.z), R = Q(p.r, p.yn, p.z);
                v0 = madd<W>(T(0.125), Lc, madd<W>(T(0.375), A, madd<W>(T(0.125), l, madd<W>(T(0.375), a, v0))));
                v1 = madd<W>(T(0.125), R, madd<W>(T(0.375), A, madd<W>(T(0.125), r, madd<W>(T(0.375), a, v1))));
            }
        }
    } else {
        const T n16 = T(9.0 / 16.0), t16 = T(3.0 / 16.0), o16 = T(1.0 / 16.0);
        const T n32 = T(9.0 / 32.0), t32 = T(3.0 / 32.0), o32 = T(1.0 / 32.0);
        if constexpr (COMP == 0) {
            const T a = Q(p.h, p.y, p.z), b = Q(p.h, p.yo, p.z), c = Q(p.h, p.y, p.zo), d = Q(p.h, p.yo, p.zo);
            const T A = Q(p.r, p.y, p.z), B = Q(p.r, p.yo, p.z), C = Q(p.r, p.y, p.zo), E = Q(p.r, p.yo, p.zo);
            v0 = madd<W>(o16, d, madd<W>(t16, c, madd<W>(t16, b, madd<W>(n16, a, v0))));
            v1 = madd<W>(o32, E, madd<W>(t32, C, madd<W>(t32, B, madd<W>(n32, A, madd<W>(o32, d, madd<W>(t32, c, madd<W>(t32, b, madd<W>(n32, a, v1))))))));
        } else {
            // the row of the cell (f) and the one at its second transverse offset (g), at normal offset 0 and 1
            const int f = p.y + p.z, g = COMP == 1 ? p.y + p.zo : p.yo + p.z;
            const T a = Q(p.h, f, 0), l = Q(p.l, f, 0), r = Q(p.r, f, 0), c = Q(p.h, g, 0), cl = Q(p.l, g, 0), cr = Q(p.r, g, 0);
            if (!(COMP == 1 ? p.jodd : p.kodd)) {
                v0 = madd<W>(o16, cl, madd<W>(t16, c, madd<W>(t16, l, madd<W>(n16, a, v0))));
                v1 = madd<W>(o16, cr, madd<W>(t16, c, madd<W>(t16, r, madd<W>(n16, a, v1))));
            } else {
                const int F = COMP == 1 ? p.yn + p.z : p.y + p.zn, G = COMP == 1 ? p.yn + p.zo : p.yo + p.zn;
                const T A = Q(p.h, F, 0), Lc = Q(p.l, F, 0), R = Q(p.r, F, 0), C = Q(p.h, G, 0), CL = Q(p.l, G, 0), CR = Q(p.r, G, 0);
                v0 = madd<W>(o32, CL, madd<W>(t32, C, madd<W>(t32, Lc, madd<W>(n32, A, madd<W>(o32, cl, madd<W>(t32, c, madd<W>(t32, l, madd<W>(n32, a, v0))))))));
                v1 = madd<W>(o32, CR, madd<W>(t32, C, madd<W>(t32, R, madd<W>(n32, A, madd<W>(o32, cr, madd<W>(t32, c, madd<W>(t32, r, madd<W>(n32, a, v1))))))));
            }
        }
    }
}

// the faces of the fine cells (2h, j, k), (2h + 1, j, k): v[component][cell]
// plus the correction.  W: a pair whose coarse stencil stays inside the walls
// is a periodic one, the others take the wall rules face by face
template <class T, int DM, bool W>
__device__ __forceinline__ void prolong_cells(const Dims& Dc, const T* q0, const T* q1, const T* q2, int h, int j, int k, T (&v)[3][2]) {
    if constexpr (W) {
        auto edge = [&](int d, int c, int n) { return ((Dc.wall >> d) & 1) && (c == 0 || c >= n - 1); };
        if (edge(0, h, Dc.nx) || edge(1, j >> 1, Dc.ny) || (DM == 3 && edge(2, k >> 1, Dc.nz))) {
#pragma unroll 1
            for (int e = 0; e < 2; ++e) {
                const int i = 2 * h + e;
                T a = e ? v[0][1] : v[0][0], b = e ? v[1][1] : v[1][0];
                a = prolong_one<T, DM, 0, 0, true>(Dc, q0, a, i, j, k);
                b = prolong_one<T, DM, 1, 0, true>(Dc, q1, b, i, j, k);
                T c = T(0);
                if constexpr (DM == 3) {
                    c = e ? v[2][1] : v[2][0];
                    c = prolong_one<T, DM, 2, 0, true>(Dc, q2, c, i, j, k);
                }
                if (e) {
                    v[0][1] = a;
                    v[1][1] = b;
                    v[2][1] = c;
                } else {
                    v[0][0] = a;
                    v[1][0] = b;
                    v[2][0] = c;
                }
            }
            return;
        }
    }
    const PairAt p = pair_at<DM>(Dc, h, j, k);
    prolong_pair<T, DM, 0, W>(q0, p, v[0][0], v[0][1]);
    prolong_pair<T, DM, 1, W>(q1, p, v[1][0], v[1][1]);
    if constexpr (DM == 3) prolong_pair<T, DM, 2, W>(q2, p, v[2][0], v[2][1]);
}

template <class T, int DM, bool W>
__global__ void __launch_bounds__(kThreads) k_prolong_pairs(Dims F, Dims Dc, const T* __restrict__ q0, const T* __restrict__ q1,
                                                            const T* __restrict__ q2, T* __restrict__ f0, T* __restrict__ f1,
                                                            T* __restrict__ f2) {
    using V2 = typename Pair2<T>::type;
    pdl_enter();
    const Pos q = pos3(F.nx >> 1, F.ny);
    if (!q.ok) return;
    const int t = q.i + (F.nx >> 1) * (q.j + F.ny * q.k);
    T* f[3] = {f0, f1, f2};
    T v[3][2] = {};
#pragma unroll
    for (int d = 0; d < DM; ++d) {
        const V2 x = reinterpret_cast<const V2*>(f[d])[t];
        v[d][0] = x.x;
        v[d][1] = x.y;
    }
    prolong_cells<T, DM, W>(Dc, q0, q1, q2, q.i, q.j, q.k, v);
#pragma unroll
    for (int d = 0; d < DM; ++d) {
        V2 x;
        x.x = v[d][0];
        x.y = v[d][1];
        reinterpret_cast<V2*>(f[d])[t] = x;
    }
}

template <class T>
void launch_prolong_add(const LevelDev<T>& F, const LevelDev<T>& Cc, const T* const phi_c[3], T* const phi_f[3], cudaStream_t s) {
    // pairs: an even fine row (any level with a coarser one) and fields that start on a pair
    bool al = (F.D.nx & 1) == 0;
    for (int d = 0; d < F.D.dm; ++d) al = al && reinterpret_cast<uintptr_t>(phi_f[d]) % (2 * sizeof(T)) == 0;
    const G3 g = al ? (F.D.wall ? geom3(F.D.nx / 2, F.D.ny, F.D.nz)
                                : geom3_tuned(TK_PROLONG, sizeof(T), 0, F.D, F.D.nx / 2, F.D.ny, F.D.nz))
                    : geom3(F.D.nx, F.D.ny, F.D.nz);
#define PR(K_) launch_pdl(K_, g.grid, g.block, 0, s, F.D, Cc.D, phi_c[0], phi_c[1], phi_c[2], phi_f[0], phi_f[1], phi_f[2])
#define PRW(DM_)                                     \
    if (al && F.D.wall) PR((k_prolong_pairs<T, DM_, true>));  \
    else if (al) PR((k_prolong_pairs<T, DM_, false>));        \
    else if (F.D.wall) PR((k_prolong_add<T, DM_, true>));     \
    else PR((k_prolong_add<T, DM_, false>));
    if (F.D.dm == 2) {
        PRW(2)
    } else {
        PRW(3)
    }
#undef PRW
#undef PR
}

}  // namespace lmm
