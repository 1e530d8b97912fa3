// pair3.cuh - L phi of all faces of two neighbouring cells of a row (3D,
// periodic), for the residual and the coupled operator.
//
// One face per thread reads 22 to 26 operands and spends about 165 instructions,
// most of them on addresses; its issue slots bound it (128^3 FP32: 63% of them
// used at 38% of the DRAM rate).  The six faces of the cells (2h, j, k) and
// (2h + 1, j, k) share their operands: 30 phi and 13 coefficient loads, most of
// them pairs, and one set of row offsets for the six.
//
// A thread then holds 45 operands, so the registers set how many loads an SM has
// in flight: 128-thread blocks, five of them (92 registers) for the FP32 residual
// and four (up to 128) for FP64 arithmetic measured best; one block fewer or more
// costs 10 to 50%.  Live: FP32 residual 44.4 -> 22.7 us at 128^3, 6.5 -> 3.8 at
// 64^3; FP64 26.8 -> 19.4 at 96^3; operator on an FP32 vector 57.7 -> 40.7 at
// 128^3 (L2), 449 -> 309 at 256^3 (4.3 TB/s), on an FP64 one 53.3 -> 47.5 at 128^3.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "kernels.h"
#include "pdl.cuh"
#include "stencil.cuh"

namespace lmm {

constexpr int kPairThreads = 128;

// a block of pairs: the autotuner's shape for this grid where it found a better
// one, else rows of 32 pairs where they divide the row, else of 16 (96^3: 23.0 -> 19.4 us)
static inline dim3 pair_block(const Dims& D, int kernel, int wbytes, int visc) {
    const int half = D.nx / 2, bx = half % 32 == 0 ? 32 : (half >= 16 ? 16 : 8);
    Shape s = forced_shape();
    if (!s.bx) s = tuned_shape(kernel, wbytes, visc, D);
    if (s.bx && s.bx <= half && s.by <= D.ny && s.bx * s.by <= kPairThreads) return dim3(s.bx, s.by);
    return dim3(bx, kPairThreads / bx);
}
static inline dim3 pair_grid(const Dims& D, dim3 b) { return dim3((D.nx / 2 + b.x - 1) / b.x, (D.ny + b.y - 1) / b.y, D.nz); }
// the level takes the pair kernels: rows of pairs, variable coefficients (FP32:
// visc_type -2, whose contractions face_L3_sum_fused spells out); p, q: the other
// arrays, every one starting on a pair
template <class T, class P, class Q>
static bool pairs_supported(const Dims& D, const Coef<T>& C, int visc, const P* const* p, int np, const Q* const* q, int nq) {
    if (D.dm != 3 || D.wall || (D.nx & 1) || visc >= 0 || (sizeof(T) == 4 && visc != -2)) return false;
    auto al = [](const void* a, size_t e) { return reinterpret_cast<uintptr_t>(a) % (2 * e) == 0; };
    bool ok = al(C.beta, sizeof(T)) && al(C.gamma, sizeof(T));
    for (int d = 0; d < 3; ++d) ok = ok && al(C.bed[d], sizeof(T));
    for (int i = 0; i < np; ++i) ok = ok && al(p[i], sizeof(P));
    for (int i = 0; i < nq; ++i) ok = ok && al(q[i], sizeof(Q));
    return ok;
}

// two consecutive entries of a row, and those before and after them where a stencil reaches them
template <class T>
struct Row2 {
    T v[2], l, r;
    // entry n of the row, n in -1..2
    __device__ __forceinline__ T operator[](int n) const { return n < 0 ? l : (n > 1 ? r : v[n]); }
};
template <class TX>
struct PairVec;
template <>
struct PairVec<double> {
    using type = double2;
};
template <>
struct PairVec<float> {
    using type = float2;
};
struct PairRows {
    int x0, xl, xr;                       // first entry, the entries left and right of the pair
    int c, yp, ym, zp, zm, ypzm, ymzp;    // row bases
};
__device__ __forceinline__ PairRows pair_rows(const Dims& D, int h, int j, int k) {
    const int sz = D.nx * D.ny, jp = j == D.ny - 1 ? 0 : j + 1, jm = j == 0 ? D.ny - 1 : j - 1;
    const int kp = k == D.nz - 1 ? 0 : k + 1, km = k == 0 ? D.nz - 1 : k - 1;
    PairRows x;
    x.x0 = 2 * h;
    x.xl = h == 0 ? D.nx - 1 : 2 * h - 1;
    x.xr = 2 * h + 2 == D.nx ? 0 : 2 * h + 2;
    x.c = D.nx * j + sz * k;
    x.yp = D.nx * jp + sz * k;
    x.ym = D.nx * jm + sz * k;
    x.zp = D.nx * j + sz * kp;
    x.zm = D.nx * j + sz * km;
    x.ypzm = D.nx * jp + sz * km;
    x.ymzp = D.nx * jm + sz * kp;
    return x;
}
template <class T, bool L, bool R, class TX>
__device__ __forceinline__ Row2<T> row2(const TX* p, int at, const PairRows& x) {
    Row2<T> r;
    const typename PairVec<TX>::type a = ld2(reinterpret_cast<const typename PairVec<TX>::type*>(p + at + x.x0), 0);
    r.v[0] = (T)a.x;
    r.v[1] = (T)a.y;
    r.l = L ? (T)ld(p, at + x.xl) : T(0);
    r.r = R ? (T)ld(p, at + x.xr) : T(0);
    return r;
}

// face_L3_sum of visc_type -2 in FP32 with the contractions the compiler gives
// it in the kernels that evaluate one face (in a thread that evaluates several,
// products they share would not be contracted, and the bits would differ)
__device__ __forceinline__ float face_L3_sum_fused(float centre, float p0, const float (&nb)[6], int D, const float (&q1)[4],
                                                   const float (&q2)[4], float be, float bm, float E1, float E1p, float E2, float E2p,
                                                   float dxsqinv) {
    const int t1 = (D == 0) ? 1 : 0, t2 = (D == 2) ? 1 : 2;
    float s = fmaf(2.f * nb[2 * D], be, __fmul_rn(2.f * nb[2 * D + 1], bm));
    s = fmaf(nb[2 * t1], E1p, s);
    s = fmaf(nb[2 * t1 + 1], E1, s);
    s = fmaf(nb[2 * t2], E2p, s);
    s = fmaf(nb[2 * t2 + 1], E2, s);
    s = fmaf(q1[0], E1p, s);
    s = fmaf(-q1[1], E1, s);
    s = fmaf(-q1[2], E1p, s);
    s = fmaf(q1[3], E1, s);
    s = fmaf(q2[0], E2p, s);
    s = fmaf(-q2[1], E2, s);
    s = fmaf(-q2[2], E2p, s);
    s = fmaf(q2[3], E2, s);
    return fmaf(p0, centre, -__fmul_rn(s, dxsqinv));
}

// phi of the pair and its neighbours, and L phi of the six faces: L[component][cell]
template <class T>
struct PairFaces {
    Row2<T> P[3], Pyp1, Pzp2;   // own rows (with the entry right of the pair), y component at j + 1, z component at k + 1
    T L[3][2];
};
template <class T, int VISC, class TX>
__device__ __forceinline__ void pair_faces(const Dims& D, const PairRows& x, const Coef<T>& C, const TX* u0, const TX* u1, const TX* u2, T dxsqinv,
                                           PairFaces<T>& F) {
    static_assert(VISC < 0, "variable coefficients");
    constexpr bool GAM = VISC == -3;
    const Row2<T> X = row2<T, true, true>(u0, x.c, x), Xyp = row2<T, false, false>(u0, x.yp, x), Xym = row2<T, false, true>(u0, x.ym, x),
                  Xzp = row2<T, false, false>(u0, x.zp, x), Xzm = row2<T, false, true>(u0, x.zm, x);
    const Row2<T> Y = row2<T, true, true>(u1, x.c, x), Yyp = row2<T, true, false>(u1, x.yp, x), Yym = row2<T, false, false>(u1, x.ym, x),
                  Yzp = row2<T, false, false>(u1, x.zp, x), Yzm = row2<T, false, false>(u1, x.zm, x),
                  Yypzm = row2<T, false, false>(u1, x.ypzm, x);
    const Row2<T> Z = row2<T, true, true>(u2, x.c, x), Zyp = row2<T, false, false>(u2, x.yp, x), Zym = row2<T, false, false>(u2, x.ym, x),
                  Zzp = row2<T, true, false>(u2, x.zp, x), Zzm = row2<T, false, false>(u2, x.zm, x),
                  Zymzp = row2<T, false, false>(u2, x.ymzp, x);
    const Row2<T> B = row2<T, true, false>(C.beta, x.c, x), Bym = row2<T, false, false>(C.beta, x.ym, x),
                  Bzm = row2<T, false, false>(C.beta, x.zm, x);
    const Row2<T> XY = row2<T, false, true>(C.bed[0], x.c, x), XYyp = row2<T, false, false>(C.bed[0], x.yp, x);
    const Row2<T> XZ = row2<T, false, true>(C.bed[1], x.c, x), XZzp = row2<T, false, false>(C.bed[1], x.zp, x);
    const Row2<T> YZ = row2<T, false, false>(C.bed[2], x.c, x), YZzp = row2<T, false, false>(C.bed[2], x.zp, x),
                  YZyp = row2<T, false, false>(C.bed[2], x.yp, x);
    Row2<T> G{}, Gym{}, Gzm{};
    if (GAM) {
        G = row2<T, true, false>(C.gamma, x.c, x);
        Gym = row2<T, false, false>(C.gamma, x.ym, x);
        Gzm = row2<T, false, false>(C.gamma, x.zm, x);
    }
    auto face = [&](auto dir, int e, T p0, const T(&nb)[6], const T(&q1)[4], const T(&q2)[4], T be, T bm, T E1, T E1p, T E2, T E2p, T g, T gm) {
        constexpr int D_ = decltype(dir)::value;
        const T a = alpha_at(C, D_, x.c + x.x0 + e);
        const T diag = face_diag3_vals<T, VISC>(a, be, bm, E1, E1p, E2, E2p, g, gm, dxsqinv, T(0), T(0));
        const T centre = face_centre3_vals<T, VISC>(diag, a, dxsqinv, T(0), T(0));
        if constexpr (sizeof(T) == 4)
            F.L[D_][e] = face_L3_sum_fused(centre, p0, nb, D_, q1, q2, be, bm, E1, E1p, E2, E2p, dxsqinv);
        else
            F.L[D_][e] = face_L3_sum<T, VISC>(centre, p0, nb, D_, q1, q2, be, bm, E1, E1p, E2, E2p, g, gm, dxsqinv, T(0), T(0));
    };
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        {
            const T nb[6] = {X[e + 1], X[e - 1], Xyp[e], Xym[e], Xzp[e], Xzm[e]};
            const T q1[4] = {Yyp[e], Y[e], Yyp[e - 1], Y[e - 1]}, q2[4] = {Zzp[e], Z[e], Zzp[e - 1], Z[e - 1]};
            face(std::integral_constant<int, 0>{}, e, X[e], nb, q1, q2, B[e], B[e - 1], XY[e], XYyp[e], XZ[e], XZzp[e], G[e], G[e - 1]);
        }
        {
            const T nb[6] = {Y[e + 1], Y[e - 1], Yyp[e], Yym[e], Yzp[e], Yzm[e]};
            const T q1[4] = {X[e + 1], X[e], Xym[e + 1], Xym[e]}, q2[4] = {Zzp[e], Z[e], Zymzp[e], Zym[e]};
            face(std::integral_constant<int, 1>{}, e, Y[e], nb, q1, q2, B[e], Bym[e], XY[e], XY[e + 1], YZ[e], YZzp[e], G[e], Gym[e]);
        }
        {
            const T nb[6] = {Z[e + 1], Z[e - 1], Zyp[e], Zym[e], Zzp[e], Zzm[e]};
            const T q1[4] = {X[e + 1], X[e], Xzm[e + 1], Xzm[e]}, q2[4] = {Yyp[e], Y[e], Yypzm[e], Yzm[e]};
            face(std::integral_constant<int, 2>{}, e, Z[e], nb, q1, q2, B[e], Bzm[e], XZ[e], XZ[e + 1], YZ[e], YZyp[e], G[e], Gzm[e]);
        }
    }
    F.P[0] = X;
    F.P[1] = Y;
    F.P[2] = Z;
    F.Pyp1 = Yyp;
    F.Pzp2 = Zzp;
}

// r = (L phi - rhs) * -1 on every face of the pair
template <class T, int VISC>
__global__ void __launch_bounds__(kPairThreads, sizeof(T) == 4 ? 5 : 4) k_residual_pairs(Dims D, Coef<T> C, const T* __restrict__ r0, const T* __restrict__ r1,
                                                        const T* __restrict__ r2, const T* __restrict__ p0, const T* __restrict__ p1,
                                                        const T* __restrict__ p2, T* __restrict__ o0, T* __restrict__ o1,
                                                        T* __restrict__ o2, T dxsqinv) {
    using V = typename PairVec<T>::type;
    pdl_enter();
    const Pos q = pos3(D.nx >> 1, D.ny);
    if (!q.ok) return;
    const PairRows x = pair_rows(D, q.i, q.j, q.k);
    PairFaces<T> F;
    pair_faces<T, VISC>(D, x, C, p0, p1, p2, dxsqinv, F);
    const T* r[3] = {r0, r1, r2};
    T* o[3] = {o0, o1, o2};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const Row2<T> b = row2<T, false, false>(r[d], x.c, x);
        V v;
        v.x = (F.L[d][0] - b.v[0]) * T(-1);
        v.y = (F.L[d][1] - b.v[1]) * T(-1);
        *reinterpret_cast<V*>(o[d] + x.c + x.x0) = v;
    }
}

template <class T>
bool launch_residual_pairs(const LevelDev<T>& L, int visc, const T* const rhs[3], const T* const phi[3], T* const out[3], cudaStream_t s) {
    const T* in[6] = {rhs[0], rhs[1], rhs[2], phi[0], phi[1], phi[2]};
    if (!pairs_supported<T>(L.D, L.coef(), visc, in, 6, out, 3)) return false;
    const dim3 b = pair_block(L.D, TK_RESIDUAL, sizeof(T), visc), g = pair_grid(L.D, b);
    const T dxsqinv = T(1.0 / (L.dx * L.dx));
#define RP(V_) launch_pdl(k_residual_pairs<T, V_>, g, b, 0, s, L.D, L.coef(), rhs[0], rhs[1], rhs[2], phi[0], phi[1], phi[2], out[0], out[1], out[2], dxsqinv)
    if constexpr (sizeof(T) == 4) {
        RP(-2);
    } else {
        if (visc == -1) RP(-1); else if (visc == -2) RP(-2); else RP(-3);
    }
#undef RP
    return true;
}

// the coupled operator of the pair: {L u + grad p, -div u} (k_apply_matrix)
template <int VISC, class TX>
__global__ void __launch_bounds__(kPairThreads, 4) k_apply_matrix_pairs(Dims D, Coef<double> C, const TX* __restrict__ u0, const TX* __restrict__ u1,
                                                            const TX* __restrict__ u2, const TX* __restrict__ p, double* __restrict__ o0,
                                                            double* __restrict__ o1, double* __restrict__ o2, double* __restrict__ op,
                                                            double dxsqinv, double dxinv) {
    pdl_enter();
    const Pos q = pos3(D.nx >> 1, D.ny);
    if (!q.ok) return;
    const PairRows x = pair_rows(D, q.i, q.j, q.k);
    PairFaces<double> F;
    pair_faces<double, VISC>(D, x, C, u0, u1, u2, dxsqinv, F);
    const Row2<double> pc = row2<double, true, false>(p, x.c, x), pym = row2<double, false, false>(p, x.ym, x),
                       pzm = row2<double, false, false>(p, x.zm, x);
    double2 a[3], dv;
    double v[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        F.L[0][e] = F.L[0][e] + (pc[e] - pc[e - 1]) * dxinv;
        F.L[1][e] = F.L[1][e] + (pc[e] - pym[e]) * dxinv;
        F.L[2][e] = F.L[2][e] + (pc[e] - pzm[e]) * dxinv;
        v[e] = (F.P[0][e + 1] - F.P[0][e]) * dxinv + (F.Pyp1[e] - F.P[1][e]) * dxinv;
        v[e] = (v[e] + (F.Pzp2[e] - F.P[2][e]) * dxinv) * -1.0;
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) a[d] = make_double2(F.L[d][0], F.L[d][1]);
    dv = make_double2(v[0], v[1]);
    const int t = x.c + x.x0;
    *reinterpret_cast<double2*>(o0 + t) = a[0];
    *reinterpret_cast<double2*>(o1 + t) = a[1];
    *reinterpret_cast<double2*>(o2 + t) = a[2];
    *reinterpret_cast<double2*>(op + t) = dv;
}

}  // namespace lmm
