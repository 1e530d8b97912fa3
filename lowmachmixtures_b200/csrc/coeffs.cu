// coeffs.cu - the coefficient hierarchy of a solve (theta*alpha, beta,
// beta_ed, gamma and the pressure's 1/alpha on every level, in FP64 and, for
// the mixed method, FP32) and the copies of a solve's vectors.  Built with
// -fmad=false (reference rounding).
//
// Reference: the coefficient coarsening of stag_mg_solver.f90:200-230,
// 873-968, 1229-1244, 1326-1367, done once per coefficient load.
//
// What bounds it: one pass over the arrays on the finest level (each input
// read once, each output written once), and launches below.  One launch per
// level forms everything the level needs; separate scale, reciprocal, copy,
// coarsening, conversion and uniformity launches were about 15 a level (a 2D
// 64^2 solve spent 250 us of 1900 in them).
#include <algorithm>

#include "coeffs.cuh"
#include "pdl.cuh"

namespace lmm {
namespace {
constexpr int kT = 256;
inline int blocks(int64_t n) { return (int)std::max<int64_t>(1, (n + kT - 1) / kT); }

__device__ __forceinline__ bool differs(double a, double b) { return __double_as_longlong(a) != __double_as_longlong(b); }

// entry t of an array of the finest level, which may be the output array
// itself (a plain load); a field holds fewer than 2^31 entries
__device__ __forceinline__ double in(const double* p, int64_t t) { return ldp<1>(p, (int)t); }

// flags of a block: set where a thread saw a value that differs
__device__ __forceinline__ void raise(bool diff, int* flag) {
    if (__syncthreads_or(diff) && threadIdx.x == 0) *flag = 1;
}

// w: the value of `v` on the finest level or a coarse one, in FP64 and FP32
__device__ __forceinline__ void put(double* o, float* f, int64_t t, double v) {
    o[t] = v;
    if (f) f[t] = (float)v;
}

// Finest level: theta alpha, 1/alpha (the pressure's face coefficient, zero
// on wall faces: homogeneous Neumann pressure at walls), beta, edges, gamma.
template <int DM, bool W>
__global__ void __launch_bounds__(kT) k_coeffs_fine(CoefFine A) {
    pdl_enter();
    const int64_t t = blockIdx.x * (int64_t)kT + threadIdx.x;
    const int64_t n = (int64_t)A.D.nx * A.D.ny * A.D.nz;
    const double a0 = in(A.alpha[0], 0), s0 = a0 * A.theta, r0 = 1.0 / a0;
    bool ds = false, dr = false;
    if (t < n) {
        int x[3] = {1, 1, 1};
        if constexpr (W) {
            const int q = (int)(t / A.D.nx);
            x[0] = (int)(t - (int64_t)q * A.D.nx);
            x[2] = q / A.D.ny;
            x[1] = q - x[2] * A.D.ny;
        }
#pragma unroll
        for (int d = 0; d < DM; ++d) {
            const double a = in(A.alpha[d], t), s = a * A.theta, r = 1.0 / a;
            put(A.o_alpha[d], A.f_alpha[d], t, s);
            put(A.o_ainv[d], A.f_ainv[d], t, r);
            ds = ds || differs(s, s0);
            dr = dr || differs(r, r0);
            if constexpr (W)
                if (A.o_pa[d]) put(A.o_pa[d], A.f_pa[d], t, (((A.D.wall >> d) & 1) && x[d] == 0) ? 0.0 : r);
        }
        put(A.o_beta, A.f_beta, t, in(A.beta, t));
        put(A.o_gamma, A.f_gamma, t, A.gamma ? in(A.gamma, t) : 0.0);
    }
#pragma unroll
    for (int e = 0; e < (DM == 2 ? 1 : 3); ++e)
        if (t < A.ne[e]) put(A.o_bed[e], A.f_bed[e], t, in(A.bed[e], t));
    raise(ds, A.flag_a);
    raise(dr, A.flag_p);
    if (t == 0) {
        *A.val_a = s0;
        *A.val_p = r0;
    }
}

// the mean of the fine faces a coarse face of component d covers
template <int DM>
__device__ __forceinline__ double face_mean(const double* a, const Dims& F, int d, int I, int J, int K) {
    auto at = [&](int i, int j, int k) { return ld(a, i + F.nx * (j + F.ny * k)); };
    if constexpr (DM == 2)
        return d == 0 ? 0.5 * (at(I, J, K) + at(I, J + 1, K)) : 0.5 * (at(I, J, K) + at(I + 1, J, K));
    if (d == 0) return 0.25 * (at(I, J, K) + at(I, J + 1, K) + at(I, J, K + 1) + at(I, J + 1, K + 1));
    if (d == 1) return 0.25 * (at(I, J, K) + at(I + 1, J, K) + at(I, J, K + 1) + at(I + 1, J, K + 1));
    return 0.25 * (at(I, J, K) + at(I + 1, J, K) + at(I, J + 1, K) + at(I + 1, J + 1, K));
}
template <int DM>
__device__ __forceinline__ double cell_mean(const double* a, const Dims& F, int I, int J, int K) {
    auto at = [&](int i, int j, int k) { return ld(a, i + F.nx * (j + F.ny * k)); };
    if constexpr (DM == 2) return 0.25 * (at(I, J, K) + at(I + 1, J, K) + at(I, J + 1, K) + at(I + 1, J + 1, K));
    return 0.125 * (at(I, J, K) + at(I + 1, J, K) + at(I, J + 1, K) + at(I + 1, J + 1, K) + at(I, J, K + 1) + at(I + 1, J, K + 1) +
                    at(I, J + 1, K + 1) + at(I + 1, J + 1, K + 1));
}

// One coarse level from the level above it.  The launch covers the level's
// edge extents (n+1 along walls).
template <int DM>
__global__ void __launch_bounds__(kT) k_coeffs_coarse(CoefCoarse A) {
    pdl_enter();
    const Dims F = A.F, C = A.C;
    const int ex = C.nx + (C.wall & 1), ey = C.ny + ((C.wall >> 1) & 1);
    const int64_t w = blockIdx.x * (int64_t)kT + threadIdx.x;
    const int64_t r = w / ex;
    const int i = (int)(w - r * ex), k = (int)(r / ey), j = (int)(r - (int64_t)k * ey);
    const int kmax = C.nz + (DM == 3 ? (C.wall >> 2) & 1 : 0);
    const int I = 2 * i, J = 2 * j, K = DM == 3 ? 2 * k : k;
    bool da = false, dp = false;
    if (i < C.nx && j < C.ny && k < C.nz) {
        const int64_t t = i + (int64_t)C.nx * (j + (int64_t)C.ny * k);
        if (A.alpha[0]) {
            const double v0 = face_mean<DM>(A.alpha[0], F, 0, 0, 0, 0);
#pragma unroll
            for (int d = 0; d < DM; ++d) {
                const double v = face_mean<DM>(A.alpha[d], F, d, I, J, K);
                put(A.o_alpha[d], A.f_alpha[d], t, v);
                da = da || differs(v, v0);
            }
            put(A.o_beta, A.f_beta, t, cell_mean<DM>(A.beta, F, I, J, K));
            put(A.o_gamma, A.f_gamma, t, cell_mean<DM>(A.gamma, F, I, J, K));
            if (t == 0) *A.val_a = v0;
        }
        if (A.pa[0]) {
            const double v0 = face_mean<DM>(A.pa[0], F, 0, 0, 0, 0);
#pragma unroll
            for (int d = 0; d < DM; ++d) {
                const double v = face_mean<DM>(A.pa[d], F, d, I, J, K);
                put(A.o_pa[d], A.f_pa[d], t, v);
                dp = dp || differs(v, v0);
            }
            if (t == 0) *A.val_p = v0;
        }
    }
    if (A.alpha[0] && k < kmax) {
        // nodal injection in 2D (nodal_restriction), two-point average along
        // the edge in 3D (edge_restriction)
#pragma unroll
        for (int e = 0; e < (DM == 2 ? 1 : 3); ++e) {
            const int cx = edge_ext(C, e, 0), cy = edge_ext(C, e, 1), cz = DM == 3 ? edge_ext(C, e, 2) : C.nz;
            if (i >= cx || j >= cy || k >= cz) continue;
            const int fx = edge_ext(F, e, 0), fy = edge_ext(F, e, 1);
            auto at = [&](int a, int b, int c) { return ld(A.bed[e], a + fx * (b + fy * c)); };
            double v;
            if (DM == 2)
                v = at(I, J, K);
            else if (e == 0)
                v = 0.5 * (at(I, J, K) + at(I, J, K + 1));
            else if (e == 1)
                v = 0.5 * (at(I, J, K) + at(I, J + 1, K));
            else
                v = 0.5 * (at(I, J, K) + at(I + 1, J, K));
            put(A.o_bed[e], A.f_bed[e], i + (int64_t)cx * (j + (int64_t)cy * k), v);
        }
    }
    raise(da, A.flag_a);
    raise(dp, A.flag_p);
}

__global__ void __launch_bounds__(kT) k_copy_fields(CopyFields A) {
    pdl_enter();
    const double* s = A.src[blockIdx.y];
    double* d = A.dst[blockIdx.y];
    const int64_t stride = (int64_t)gridDim.x * kT, t0 = blockIdx.x * (int64_t)kT + threadIdx.x;
    if ((((uintptr_t)s | (uintptr_t)d) & 15) == 0) {
        const int64_t n2 = A.n >> 1;
        for (int64_t t = t0; t < n2; t += stride) reinterpret_cast<double2*>(d)[t] = __ldg(reinterpret_cast<const double2*>(s) + t);
        if ((A.n & 1) && t0 == 0) d[A.n - 1] = s[A.n - 1];
    } else {
        for (int64_t t = t0; t < A.n; t += stride) d[t] = __ldg(s + t);
    }
}
}  // namespace

void launch_coeffs_fine(const CoefFine& A, cudaStream_t s) {
    int64_t m = (int64_t)A.D.nx * A.D.ny * A.D.nz;
    for (int e = 0; e < (A.D.dm == 2 ? 1 : 3); ++e) m = std::max(m, A.ne[e]);
    if (A.D.dm == 2) {
        if (A.D.wall)
            launch_pdl(k_coeffs_fine<2, true>, blocks(m), kT, 0, s, A);
        else
            launch_pdl(k_coeffs_fine<2, false>, blocks(m), kT, 0, s, A);
    } else {
        if (A.D.wall)
            launch_pdl(k_coeffs_fine<3, true>, blocks(m), kT, 0, s, A);
        else
            launch_pdl(k_coeffs_fine<3, false>, blocks(m), kT, 0, s, A);
    }
}

void launch_coeffs_coarse(const CoefCoarse& A, cudaStream_t s) {
    const Dims& C = A.C;
    const int64_t m = (int64_t)(C.nx + (C.wall & 1)) * (C.ny + ((C.wall >> 1) & 1)) * (C.nz + (C.dm == 3 ? (C.wall >> 2) & 1 : 0));
    if (C.dm == 2)
        launch_pdl(k_coeffs_coarse<2>, blocks(m), kT, 0, s, A);
    else
        launch_pdl(k_coeffs_coarse<3>, blocks(m), kT, 0, s, A);
}

void launch_copy_fields(const CopyFields& A, int count, cudaStream_t s) {
    const int64_t b = std::min<int64_t>(blocks((A.n + 1) / 2), 1184);
    launch_pdl(k_copy_fields, dim3((unsigned)b, count), kT, 0, s, A);
}

}  // namespace lmm

// the bounds-check table and record of this translation unit (empty
// unless built with -DLMM_BOUNDS_CHECK)
LMM_BC_UNIT(coeffs)
