// tail.cuh - the coarse end of the V-cycles in one thread block.
//
// Every multigrid level below a size threshold (its smooths, residual
// restrictions, bottom smooths and prolongations: stag_mg_solver.f90:338-760
// for the velocity, and this library's cell-centred pressure V-cycle) runs
// inside ONE kernel of a single thread block.  phi and rhs of all those
// levels live in shared memory for the whole tail; steps are separated by
// block barriers instead of kernel boundaries, so the ~30 launches per coarse
// level collapse into one.  Only the first tail level's phi goes back to
// global memory.  Every face and cell goes through the value functions of the
// per-level kernels, so results are bit-identical.
//
// What bounds it: the serial chain of one colour after another (100 of them
// on 8^3 cells), each a few hundred cycles long, not memory.  So a thread
// owns the same cells of a level through all its sweeps (two neighbours of a
// row, one of each colour; one cell on a level with odd counts) and keeps
// their neighbour offsets, coefficients and diagonals in registers: a colour
// is then its phi loads from shared memory, the face arithmetic, one division
// and a barrier among the warps that own cells of the level (a __syncwarp
// where one warp owns them all).  The coefficients are touched before the wait
// for the previous kernel, so the loads of a level hit L1.
//
// 2D batches (Dims::nz instances stacked along the third index): one block
// per instance, blockIdx.x = the instance; its views see one instance
// (nz = 1, every array offset by instance x nx*ny of that level).
#pragma once
#include <cstring>

#include "kernels.cuh"

namespace lmm {

constexpr int kTailThreads = 512;
constexpr int kMaxTail = 12;

template <class T>
struct TailLevel {
    Dims D;
    T dxsqinv;
    Coef<T> C;
    const T* pa[3];
    int pa_uniform;    // every face coefficient of pa is pa_value
    T pa_value;
    int off;           // the level's first element in shared memory
};

template <class T>
struct TailArgs {
    int nl;
    int nu1, nu2, nub, smoother;
    int tmp;           // first element of the scratch arrays in shared memory
    int zero;          // the first level's phi is zero (not read from global memory)
    T omega;
    T* g_phi[3];       // first tail level, global memory (in/out)
    const T* g_rhs[3]; // first tail level, global memory (in)
    T* g_pphi;         // pressure: first level phi (in/out)
    const T* g_prhs;   // pressure: first level rhs (in)
    TailLevel<T> L[kMaxTail];
};

__host__ __device__ __forceinline__ int ncells(const Dims& D) { return D.nx * D.ny * D.nz; }

__device__ __forceinline__ void unflat3d(const Dims& D, int w, int& i, int& j, int& k) {
    i = w % D.nx;
    int r = w / D.nx;
    j = r % D.ny;
    k = r / D.ny;
}

// this block's offset into a level's arrays: 2D, instance blockIdx.x of
// the batch; 3D, none
template <int DM>
__device__ __forceinline__ int64_t inst_offset(const Dims& D) {
    return DM == 2 ? (int64_t)blockIdx.x * D.nx * D.ny : 0;
}
template <class T>
__device__ __forceinline__ const T* shift(const T* p, int64_t o) {
    return p ? p + o : p;
}

// one level as the block sees it: its dimensions and coefficients (of this
// block's instance), phi and rhs in shared memory; tmp is shared by all levels
template <class T>
struct TailView {
    Dims D;
    T dxsqinv;
    Coef<T> C;
    T* phi[3];
    T* rhs[3];
    T* tmp[3];
};
template <class T, int DM>
__device__ __forceinline__ TailView<T> tail_view(const TailArgs<T>& A, T* sm, int l) {
    TailView<T> v;
    v.D = A.L[l].D;
    v.dxsqinv = A.L[l].dxsqinv;
    v.C = A.L[l].C;
    if constexpr (DM == 2) {
        const int64_t io = inst_offset<DM>(v.D);
        // an instance's edge array: n+1 nodes along a nodal wall-bounded direction
        const int64_t ie = (int64_t)blockIdx.x * edge_ext(v.D, 0, 0) * edge_ext(v.D, 0, 1);
        v.D.nz = 1;
#pragma unroll
        for (int d = 0; d < 2; ++d) v.C.alpha[d] = shift(v.C.alpha[d], io);
        v.C.bed[0] = shift(v.C.bed[0], ie);
        v.C.beta = shift(v.C.beta, io);
        v.C.gamma = shift(v.C.gamma, io);
    }
    const int n = ncells(v.D);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        v.phi[d] = sm + A.L[l].off + (d < DM ? d : 0) * n;
        v.rhs[d] = sm + A.L[l].off + (DM + (d < DM ? d : 0)) * n;
        v.tmp[d] = sm + A.tmp + (d < DM ? d : 0) * n;
    }
    return v;
}

// touch an array of the coarse coefficients, one load per 32-byte sector:
// they are written once per coefficient load, never by the kernel before
// this one, so this runs ahead of the wait for it
template <class T>
__device__ __forceinline__ void touch(const T* p, int n) {
    constexpr int step = 32 / sizeof(T);
    for (int t = threadIdx.x * step; t < n; t += blockDim.x * step) {
        const T v = ld(p, t);
        if constexpr (sizeof(T) == 8)
            asm volatile("" ::"d"(v));
        else
            asm volatile("" ::"f"(v));
    }
}

// barrier among the first `warps` warps of the block
__device__ __forceinline__ void warps_sync(int warps) {
    if (warps == 1)
        __syncwarp();
    else
        asm volatile("bar.sync 1, %0;" ::"r"(warps * 32) : "memory");
}

// ------------------------------------------------------------------ owned cells
// A cell a thread owns on a level: neighbour offsets, the coefficients of its
// DM faces (beta at the cell and at -e_d; every edge array at the cell and
// one step along each of its two nodal directions) and their diagonals.
template <class T, int DM, int VISC, bool W>
struct Owned {
    static constexpr int NE = DM == 3 ? 3 : 1;
    bool on;
    int s, op[3], om[3];
    int lo, hi, nlo, nhi;   // W: wall bits of the cell; nlo / nhi: no-slip walls
    T be[DM + 1], g[DM + 1], e[NE][3], diag[DM], cen[DM];

    // the coefficients of face D, with its direction order (Perm3)
    template <int D>
    __device__ __forceinline__ void edges(T& E1, T& E1p, T& E2, T& E2p) const {
        if constexpr (DM == 2) {
            E1 = e[0][0];
            E1p = e[0][D == 0 ? 2 : 1];
            E2 = E2p = T(0);
        } else {
            constexpr int e1 = Perm3<D>::e1, e2 = Perm3<D>::e2;
            E1 = e[e1][0];
            E1p = e[e1][D == 0 ? 2 : 1];              // t1: +y (xy) for x faces, +x (xy, xz) for y and z faces
            E2 = e[e2][0];
            E2p = e[e2][D == 2 ? 1 : 2];              // t2: +z (xz, yz) for x and y faces, +y (yz) for z faces
        }
    }
    template <int D>
    __device__ __forceinline__ void set_diag(const TailView<T>& L, T b, T c) {
        const T a = alpha_at(L.C, D, s);
        T E1, E1p, E2, E2p;
        edges<D>(E1, E1p, E2, E2p);
        if constexpr (DM == 2) {
            const FaceCoef2<T> k{a, be[0], be[1 + D], E1, E1p, g[0], g[1 + D]};
            diag[D] = face_diag2_vals<T, VISC>(k, L.dxsqinv, b, c);
            cen[D] = face_centre2_vals<T, VISC>(k, L.dxsqinv, b, c);
        } else {
            diag[D] = face_diag3_vals<T, VISC>(a, be[0], be[1 + D], E1, E1p, E2, E2p, g[0], g[1 + D], L.dxsqinv, b, c);
            cen[D] = face_centre3_vals<T, VISC>(diag[D], a, L.dxsqinv, b, c);
        }
    }
    __device__ __forceinline__ void load(const TailView<T>& L, int i, int j, int k, T b, T c) {
        const Nb n = W ? make_nbw(L.D, i, j, k) : make_nb(L.D, i, j, k);
        s = n.s;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            op[d] = n.op[d];
            om[d] = n.om[d];
        }
        lo = hi = nlo = nhi = 0;
        if constexpr (W) {
            lo = n.lo;
            hi = n.hi;
            nlo = n.lo & ~n.D.slip_lo;
            nhi = n.hi & ~n.D.slip_hi;
        }
#pragma unroll
        for (int d = 0; d <= DM; ++d) be[d] = g[d] = T(0);
        if constexpr (VISC < 0) {
            be[0] = ld(L.C.beta, s);
#pragma unroll
            for (int d = 0; d < DM; ++d) be[1 + d] = ld(L.C.beta, s + om[d]);
#pragma unroll
            for (int q = 0; q < NE; ++q) {
                const int ta = DM == 2 ? 0 : (q == 2 ? 1 : 0), tb = DM == 2 ? 1 : (q == 0 ? 1 : 2);
                e[q][0] = ld(L.C.bed[q], W ? edge_at(n, q, -1) : s);
                e[q][1] = ld(L.C.bed[q], W ? edge_at(n, q, ta) : s + op[ta]);
                e[q][2] = ld(L.C.bed[q], W ? edge_at(n, q, tb) : s + op[tb]);
            }
        } else {
#pragma unroll
            for (int q = 0; q < NE; ++q) e[q][0] = e[q][1] = e[q][2] = T(0);
        }
        if constexpr (VISC == -3) {
            g[0] = ld(L.C.gamma, s);
#pragma unroll
            for (int d = 0; d < DM; ++d) g[1 + d] = ld(L.C.gamma, s + om[d]);
        }
        set_diag<0>(L, b, c);
        set_diag<1>(L, b, c);
        if constexpr (DM == 3) set_diag<2>(L, b, c);
    }
    // phi at the +1 / -1 neighbour in direction d for face component D
    template <int D>
    __device__ __forceinline__ T up(const T* p, int d) const {
        const T v = ldp<1>(p, s + op[d]);
        if constexpr (W) {
            if (d == D) return ((hi >> d) & 1) ? T(0) : v;
            return ((nhi >> d) & 1) ? -v : v;
        }
        return v;
    }
    template <int D>
    __device__ __forceinline__ T down(const T* p, int d) const {
        const T v = ldp<1>(p, s + om[d]);
        if constexpr (W) {
            if (d != D) return ((nlo >> d) & 1) ? -v : v;
        }
        return v;
    }
    // cross terms of component t for face component D
    template <int D>
    __device__ __forceinline__ void cross(const T* q, int t, T (&x)[4]) const {
        if constexpr (VISC == 1 || VISC == -1) {
            x[0] = x[1] = x[2] = x[3] = T(0);
            return;
        }
        x[0] = ldp<1>(q, s + op[t]);
        x[1] = ldp<1>(q, s);
        x[2] = ldp<1>(q, s + om[D] + op[t]);
        x[3] = ldp<1>(q, s + om[D]);
        if constexpr (W) {
            if ((hi >> t) & 1) x[0] = x[2] = T(0);
        }
    }
    template <int D>
    __device__ __forceinline__ bool face() const {   // a face that is updated (not a wall face)
        return on && !(W && ((lo >> D) & 1));
    }
    template <int D>
    __device__ __forceinline__ T apply(const TailView<T>& L, T p0, T b, T c) const {
        T E1, E1p, E2, E2p;
        edges<D>(E1, E1p, E2, E2p);
        const T* p = L.phi[D];
        if constexpr (DM == 2) {
            constexpr int t = 1 - D;
            T x[4];
            cross<D>(L.phi[t], t, x);
            const FaceCoef2<T> k{T(0), be[0], be[1 + D], E1, E1p, g[0], g[1 + D]};
            return face_L2_sum<T, VISC>(cen[D], p0, up<D>(p, D), down<D>(p, D), up<D>(p, t), down<D>(p, t), x, k, L.dxsqinv, b, c);
        } else {
            constexpr int t1 = Perm3<D>::t1, t2 = Perm3<D>::t2;
            T q1[4], q2[4], nb[6];
            cross<D>(L.phi[t1], t1, q1);
            cross<D>(L.phi[t2], t2, q2);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                nb[2 * d] = up<D>(p, d);
                nb[2 * d + 1] = down<D>(p, d);
            }
            return face_L3_sum<T, VISC>(cen[D], p0, nb, D, q1, q2, be[0], be[1 + D], E1, E1p, E2, E2p, g[0], g[1 + D], L.dxsqinv, b, c);
        }
    }
};

// one colour of component D on the owned cells (o.on: the cell is this
// colour's).  odd: cells of one colour can be neighbours, so every new value
// is formed before any is stored (as k_colour_update)
template <int D, class T, int DM, int VISC, bool W>
__device__ __forceinline__ void owned_colour(const TailView<T>& L, const Owned<T, DM, VISC, W>& o, T omega, T b, T c, bool odd, int warps) {
    T v = T(0);
    const bool act = o.template face<D>();
    if (act) {
        const T p0 = ldp<1>(L.phi[D], o.s);
        v = gs_update(p0, omega, ldp<1>(L.rhs[D], o.s), o.template apply<D>(L, p0, b, c), o.diag[D]);
    }
    if (odd) warps_sync(warps);
    if (act) L.phi[D][o.s] = v;
    warps_sync(warps);
}
// residual (L phi - rhs) * -1 of the owned cell's faces (zero on wall faces)
template <int D, class T, int DM, int VISC, bool W>
__device__ __forceinline__ void owned_residual(const TailView<T>& L, const Owned<T, DM, VISC, W>& o, T b, T c) {
    if (!o.on) return;
    T v = T(0);
    if (o.template face<D>()) v = (o.template apply<D>(L, ldp<1>(L.phi[D], o.s), b, c) - ldp<1>(L.rhs[D], o.s)) * T(-1);
    L.tmp[D][o.s] = v;
}

// nsm Gauss-Seidel sweeps of one level by the threads that own its cells,
// then (resid) the residual of every face into tmp; false: the level has more
// cells than the block can own, nothing done.  Ends with a block barrier.
template <class T, int DM, int VISC, bool W>
__device__ __forceinline__ bool owned_level(const TailView<T>& L, int nsm, T omega, bool resid) {
    const bool odd = odd_level(L.D);
    const int n = ncells(L.D), count = odd ? n : n >> 1;
    if (count > (int)blockDim.x) return false;
    const int warps = (count + 31) >> 5, t = threadIdx.x;
    if (t < warps * 32) {
        const T b = ld(L.C.beta, 0), c = ld(L.C.gamma, 0);
        Owned<T, DM, VISC, W> A, B;   // the cells of even and of odd i + j + k
        int i, j, k;
        if (odd) {
            unflat3d(L.D, t, i, j, k);
            const int par = (i + j + k) & 1;
            A.on = t < count && par == 0;
            B.on = t < count && par == 1;
            if (A.on) A.load(L, i, j, k, b, c);
            if (B.on) B.load(L, i, j, k, b, c);
        } else {
            const int half = L.D.nx >> 1;
            i = 2 * (t % half);
            j = t / half;
            k = j / L.D.ny;
            j -= k * L.D.ny;
            A.on = B.on = t < count;
            const int p = (j + k) & 1;
            if (A.on) {
                A.load(L, i + p, j, k, b, c);
                B.load(L, i + 1 - p, j, k, b, c);
            }
        }
        for (int s = 0; s < nsm; ++s) {
            owned_colour<0>(L, A, omega, b, c, odd, warps);
            owned_colour<0>(L, B, omega, b, c, odd, warps);
            owned_colour<1>(L, A, omega, b, c, odd, warps);
            owned_colour<1>(L, B, omega, b, c, odd, warps);
            if constexpr (DM == 3) {
                owned_colour<2>(L, A, omega, b, c, odd, warps);
                owned_colour<2>(L, B, omega, b, c, odd, warps);
            }
        }
        if (resid) {
            owned_residual<0>(L, A, b, c);
            owned_residual<0>(L, B, b, c);
            owned_residual<1>(L, A, b, c);
            owned_residual<1>(L, B, b, c);
            if constexpr (DM == 3) {
                owned_residual<2>(L, A, b, c);
                owned_residual<2>(L, B, b, c);
            }
        }
    }
    __syncthreads();
    return true;
}

// ------------------------------------------------------------------ larger levels, Jacobi
// one colour of component COMP with the faces strided over the block
template <class T, int DM, int VISC, int COMP, bool W>
__device__ __forceinline__ void tail_colour(const TailView<T>& L, int parity, T omega, bool odd) {
    const T b = ld(L.C.beta, 0), c = ld(L.C.gamma, 0);
    const T* phi[3] = {L.phi[0], L.phi[1], L.phi[2]};
    T* p = L.phi[COMP];
    if (odd) {
        // every new value from the values before the colour's pass, staged in tmp
        const int n = ncells(L.D);
        for (int pass = 0; pass < 2; ++pass) {
            for (int w = threadIdx.x; w < n; w += blockDim.x) {
                int i, j, k;
                unflat3d(L.D, w, i, j, k);
                if (((i + j + k) & 1) != parity) continue;
                if (pass == 1) {
                    p[w] = L.tmp[COMP][w];
                    continue;
                }
                Nb nb = W ? make_nbw(L.D, i, j, k) : make_nb(L.D, i, j, k);
                L.tmp[COMP][w] = (W && wall_face(nb, COMP))
                                     ? p[w]
                                     : face_update<T, DM, VISC, COMP, 1, W>(phi, L.C, L.rhs[COMP], nb, L.dxsqinv, b, c, omega);
            }
            if (pass == 0) __syncthreads();
        }
        return;
    }
    const int half = L.D.nx >> 1;
    const int count = half * L.D.ny * L.D.nz;
    for (int w = threadIdx.x; w < count; w += blockDim.x) {
        const int ih = w % half;
        const int q = w / half;
        const int j = q % L.D.ny, k = q / L.D.ny;
        const int i = 2 * ih + ((j + k + parity) & 1);
        Nb nb = W ? make_nbw(L.D, i, j, k) : make_nb(L.D, i, j, k);
        if (W && wall_face(nb, COMP)) continue;
        p[nb.s] = face_update<T, DM, VISC, COMP, 1, W>(phi, L.C, L.rhs[COMP], nb, L.dxsqinv, b, c, omega);
    }
}

// every face of component COMP at cell (i, j, k): its Jacobi update
// (resid = false) or residual, into tmp
template <class T, int DM, int VISC, int COMP, bool W>
__device__ __forceinline__ void tail_face_to_tmp(const TailView<T>& L, const Nb& nb, T omega, T b, T c, bool resid) {
    const T* phi[3] = {L.phi[0], L.phi[1], L.phi[2]};
    T v = T(0);
    if (!(W && wall_face(nb, COMP))) {
        const T Lp = face_L<T, DM, VISC, COMP, 1, T, W>(phi, L.C, nb, L.dxsqinv, b, c);
        const T r = ldp<1>(L.rhs[COMP], nb.s);
        v = resid ? (Lp - r) * T(-1)
                  : gs_update(ldp<1>(phi[COMP], nb.s), omega, r, Lp, face_diag<T, DM, VISC, COMP, W>(L.C, nb, L.dxsqinv, b, c));
    }
    L.tmp[COMP][nb.s] = v;
}
template <class T, int DM, int VISC, bool W>
__device__ __forceinline__ void tail_all_to_tmp(const TailView<T>& L, T omega, bool resid) {
    const T b = ld(L.C.beta, 0), c = ld(L.C.gamma, 0);
    const int n = ncells(L.D);
    for (int w = threadIdx.x; w < n; w += blockDim.x) {
        int i, j, k;
        unflat3d(L.D, w, i, j, k);
        const Nb nb = W ? make_nbw(L.D, i, j, k) : make_nb(L.D, i, j, k);
        tail_face_to_tmp<T, DM, VISC, 0, W>(L, nb, omega, b, c, resid);
        tail_face_to_tmp<T, DM, VISC, 1, W>(L, nb, omega, b, c, resid);
        if constexpr (DM == 3) tail_face_to_tmp<T, DM, VISC, 2, W>(L, nb, omega, b, c, resid);
    }
    __syncthreads();
}

// nsm sweeps of one level, then (resid) the residual into tmp
template <class T, int DM, int VISC, bool W>
__device__ __forceinline__ void tail_smooth(const TailView<T>& L, int nsm, int smoother, T omega, bool resid) {
    if (smoother != 0 && owned_level<T, DM, VISC, W>(L, nsm, omega, resid)) return;
    const int n = ncells(L.D);
    const bool odd = odd_level(L.D);
    for (int s = 0; s < nsm; ++s) {
        if (smoother == 0) {
            tail_all_to_tmp<T, DM, VISC, W>(L, omega, false);
            for (int w = threadIdx.x; w < n; w += blockDim.x)
#pragma unroll
                for (int d = 0; d < DM; ++d) L.phi[d][w] = L.tmp[d][w];
            __syncthreads();
        } else {
            for (int color = 1; color <= 2 * DM; ++color) {
                const int comp = (color - 1) / 2;
                const int parity = (color % 2 == 1) ? 0 : 1;
                if (comp == 0)
                    tail_colour<T, DM, VISC, 0, W>(L, parity, omega, odd);
                else if (comp == 1)
                    tail_colour<T, DM, VISC, 1, W>(L, parity, omega, odd);
                else if constexpr (DM == 3)
                    tail_colour<T, DM, VISC, 2, W>(L, parity, omega, odd);
                __syncthreads();
            }
        }
    }
    if (resid) tail_all_to_tmp<T, DM, VISC, W>(L, omega, true);
}

// The coarse end of a staggered V-cycle.  In: the first tail level's rhs and
// phi (global); out: its phi (global).  Levels below are zeroed in shared
// memory.
template <class T, int DM, int VISC, bool W = false>
__global__ void __launch_bounds__(kTailThreads, 1) k_vcycle_tail(const __grid_constant__ TailArgs<T> A) {
    extern __shared__ __align__(16) unsigned char tail_smem[];
    T* sm = reinterpret_cast<T*>(tail_smem);
    for (int l = 0; l < A.nl; ++l) {
        const TailView<T> v = tail_view<T, DM>(A, sm, l);
        const int n = ncells(v.D);
        if constexpr (VISC < 0) {
            touch(v.C.beta, n);
#pragma unroll
            for (int e = 0; e < (DM == 2 ? 1 : 3); ++e) touch(v.C.bed[e], edge_ext(v.D, e, 0) * edge_ext(v.D, e, 1) * (DM == 3 ? edge_ext(v.D, e, 2) : 1));
        }
        if (!v.C.alpha_uniform)
#pragma unroll
            for (int d = 0; d < DM; ++d) touch(v.C.alpha[d], n);
        if (l > 0)
            for (int w = threadIdx.x; w < DM * n; w += blockDim.x) v.phi[0][w] = T(0);
    }
    pdl_enter();
    const int64_t g0 = inst_offset<DM>(A.L[0].D);
    const TailView<T> V0 = tail_view<T, DM>(A, sm, 0);
    const int n0 = ncells(V0.D);
#pragma unroll
    for (int d = 0; d < DM; ++d)
        for (int w = threadIdx.x; w < n0; w += blockDim.x) {
            V0.phi[d][w] = A.zero ? T(0) : A.g_phi[d][g0 + w];
            V0.rhs[d][w] = A.g_rhs[d][g0 + w];
        }
    __syncthreads();
    // down to the coarsest level and back up (one smoothing call in the code,
    // so it is inlined and its shared-memory accesses stay such)
    for (int st = 0; st < 2 * A.nl - 1; ++st) {
        const bool up = st >= A.nl, down = st < A.nl - 1;
        const int l = up ? 2 * A.nl - 2 - st : st;
        const TailView<T> F = tail_view<T, DM>(A, sm, l);
        if (up) {
            const TailView<T> Cc = tail_view<T, DM>(A, sm, l + 1);
            const int nf = ncells(F.D);
            for (int w = threadIdx.x; w < nf; w += blockDim.x) {
                int i, j, k;
                unflat3d(F.D, w, i, j, k);
                F.phi[0][w] = prolong_one<T, DM, 0, 1, W>(Cc.D, Cc.phi[0], F.phi[0][w], i, j, k);
                F.phi[1][w] = prolong_one<T, DM, 1, 1, W>(Cc.D, Cc.phi[1], F.phi[1][w], i, j, k);
                if constexpr (DM == 3) F.phi[2][w] = prolong_one<T, DM, 2, 1, W>(Cc.D, Cc.phi[2], F.phi[2][w], i, j, k);
            }
            __syncthreads();
        }
        tail_smooth<T, DM, VISC, W>(F, up ? A.nu2 : (down ? A.nu1 : A.nub), A.smoother, A.omega, down);
        if (down) {
            const TailView<T> Cc = tail_view<T, DM>(A, sm, l + 1);
            const int nc = ncells(Cc.D);
            for (int w2 = threadIdx.x; w2 < nc * DM; w2 += blockDim.x) {
                const int comp = w2 / nc, w = w2 - comp * nc;
                int i, j, k;
                unflat3d(Cc.D, w, i, j, k);
                if (comp == 0)
                    Cc.rhs[0][w] = restrict_one<T, DM, 0, W, 1>(F.D, F.tmp[0], Cc.D, i, j, k);
                else if (comp == 1)
                    Cc.rhs[1][w] = restrict_one<T, DM, 1, W, 1>(F.D, F.tmp[1], Cc.D, i, j, k);
                else if constexpr (DM == 3)
                    Cc.rhs[2][w] = restrict_one<T, DM, 2, W, 1>(F.D, F.tmp[2], Cc.D, i, j, k);
            }
            __syncthreads();
        }
    }
#pragma unroll
    for (int d = 0; d < DM; ++d)
        for (int w = threadIdx.x; w < n0; w += blockDim.x) A.g_phi[d][g0 + w] = V0.phi[d][w];
}

// ------------------------------------------------------------------ pressure
template <class T>
struct TailPView {
    Dims D;
    T dxsqinv;
    const T* pa[3];
    int u;        // every face coefficient is c
    T c;
    T* phi;
    T* rhs;
    T* tmp;
};
template <class T, int DM>
__device__ __forceinline__ TailPView<T> tail_pview(const TailArgs<T>& A, T* sm, int l) {
    TailPView<T> v;
    v.D = A.L[l].D;
    v.dxsqinv = A.L[l].dxsqinv;
    const int64_t io = inst_offset<DM>(v.D);
    if (DM == 2) v.D.nz = 1;
#pragma unroll
    for (int d = 0; d < 3; ++d) v.pa[d] = shift(A.L[l].pa[d], io);
    v.u = A.L[l].pa_uniform;
    v.c = A.L[l].pa_value;
    const int n = ncells(v.D);
    v.phi = sm + A.L[l].off;
    v.rhs = v.phi + n;
    v.tmp = sm + A.tmp;
    return v;
}

// a cell a thread owns: neighbour offsets, face coefficients, diagonal
template <class T, int DM, bool U>
struct OwnedCell {
    bool on;
    int s, op[3], om[3];
    T k[6], diag, rhs;
    __device__ __forceinline__ void load(const TailPView<T>& L, int i, int j, int kk) {
        const Nb n = make_nb(L.D, i, j, kk);
        s = n.s;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            op[d] = n.op[d];
            om[d] = n.om[d];
        }
        cc_coef<T, DM, U>(L.pa, L.c, n, k);
        diag = cc_diag_vals<T, DM>(k, L.dxsqinv);
        rhs = ldp<1>(L.rhs, s);
    }
};
template <class T, int DM, bool U>
__device__ __forceinline__ void owned_cc_colour(const TailPView<T>& L, const OwnedCell<T, DM, U>& o, bool odd, int warps) {
    T v = T(0);
    if (o.on) {
        T nb[6];
#pragma unroll
        for (int d = 0; d < DM; ++d) {
            nb[2 * d] = ldp<1>(L.phi, o.s + o.op[d]);
            nb[2 * d + 1] = ldp<1>(L.phi, o.s + o.om[d]);
        }
        const T p = ldp<1>(L.phi, o.s);
        const T res = o.rhs - cc_lap_vals<T, DM>(o.k, p, nb, L.dxsqinv);
        v = p + res / o.diag;
    }
    if (odd) warps_sync(warps);
    if (o.on) L.phi[o.s] = v;
    warps_sync(warps);
}

// nsweeps red/black sweeps of one pressure level; ends with a block barrier
template <class T, int DM, bool U>
__device__ __forceinline__ void tail_cc_sweeps(const TailPView<T>& L, int nsweeps) {
    const bool odd = odd_level(L.D);
    const int n = ncells(L.D), half = L.D.nx >> 1, count = odd ? n : n >> 1, t0 = threadIdx.x;
    if (count <= (int)blockDim.x) {
        const int warps = (count + 31) >> 5;
        if (t0 < warps * 32) {
            OwnedCell<T, DM, U> A, B;
            int i, j, k;
            if (odd) {
                unflat3d(L.D, t0, i, j, k);
                const int par = (i + j + k) & 1;
                A.on = t0 < count && par == 0;
                B.on = t0 < count && par == 1;
                if (A.on) A.load(L, i, j, k);
                if (B.on) B.load(L, i, j, k);
            } else {
                i = 2 * (t0 % half);
                j = t0 / half;
                k = j / L.D.ny;
                j -= k * L.D.ny;
                A.on = B.on = t0 < count;
                const int p = (j + k) & 1;
                if (A.on) {
                    A.load(L, i + p, j, k);
                    B.load(L, i + 1 - p, j, k);
                }
            }
            for (int s = 0; s < nsweeps; ++s) {
                owned_cc_colour(L, A, odd, warps);
                owned_cc_colour(L, B, odd, warps);
            }
        }
        __syncthreads();
        return;
    }
    if (odd) {
        // each colour from the values before its pass
        for (int s = 0; s < nsweeps; ++s)
            for (int q = 0; q < 4; ++q) {
                for (int w = t0; w < n; w += blockDim.x) {
                    int i, j, k;
                    unflat3d(L.D, w, i, j, k);
                    if (((i + j + k) & 1) != (q >> 1)) continue;
                    if (q & 1)
                        L.phi[w] = L.tmp[w];
                    else
                        L.tmp[w] = cc_update<T, DM, U, 1>(L.pa, L.c, L.phi, L.rhs, make_nb(L.D, i, j, k), L.dxsqinv);
                }
                __syncthreads();
            }
        return;
    }
    // the block's stride through (pair, row, plane), kept as three counters
    // instead of two divisions per cell
    const int dr = blockDim.x / half, di = blockDim.x - dr * half, dk = dr / L.D.ny, dj = dr - dk * L.D.ny;
    const int r0 = t0 / half, i0 = t0 - r0 * half, k0 = r0 / L.D.ny, j0 = r0 - k0 * L.D.ny;
    for (int s = 0; s < nsweeps; ++s)
        for (int parity = 0; parity < 2; ++parity) {
            int ih = i0, j = j0, k = k0;
            for (int w = t0; w < count; w += blockDim.x) {
                const Nb nb = make_nb(L.D, 2 * ih + ((j + k + parity) & 1), j, k);
                L.phi[nb.s] = cc_update<T, DM, U, 1>(L.pa, L.c, L.phi, L.rhs, nb, L.dxsqinv);
                ih += di;
                j += dj;
                k += dk;
                if (ih >= half) {
                    ih -= half;
                    ++j;
                }
                if (j >= L.D.ny) {
                    j -= L.D.ny;
                    ++k;
                }
            }
            __syncthreads();
        }
}
template <class T, int DM, bool U>
__device__ __forceinline__ void tail_cc_restrict(const TailPView<T>& F, const TailPView<T>& Cc) {
    const int nc = ncells(Cc.D);
    for (int w = threadIdx.x; w < nc; w += blockDim.x) {
        int i, j, k;
        unflat3d(Cc.D, w, i, j, k);
        auto R = [&](int a, int b, int c) {
            return cc_resid<T, DM, U, 1>(F.pa, F.c, F.phi, F.rhs, make_nb(F.D, 2 * i + a, 2 * j + b, 2 * k + c), F.dxsqinv);
        };
        if constexpr (DM == 2)
            Cc.rhs[w] = T(0.25) * (R(0, 0, 0) + R(1, 0, 0) + R(0, 1, 0) + R(1, 1, 0));
        else
            Cc.rhs[w] = T(0.125) * (R(0, 0, 0) + R(1, 0, 0) + R(0, 1, 0) + R(1, 1, 0) + R(0, 0, 1) + R(1, 0, 1) + R(0, 1, 1) + R(1, 1, 1));
    }
}

template <class T, int DM>
__global__ void __launch_bounds__(kTailThreads, 1) k_ccmg_tail(const __grid_constant__ TailArgs<T> A) {
    extern __shared__ __align__(16) unsigned char tail_smem[];
    T* sm = reinterpret_cast<T*>(tail_smem);
    for (int l = 0; l < A.nl; ++l) {
        const TailPView<T> v = tail_pview<T, DM>(A, sm, l);
        const int n = ncells(v.D);
        if (!v.u)
#pragma unroll
            for (int d = 0; d < DM; ++d) touch(v.pa[d], n);
        if (l > 0)
            for (int w = threadIdx.x; w < n; w += blockDim.x) v.phi[w] = T(0);
    }
    pdl_enter();
    const int64_t g0 = inst_offset<DM>(A.L[0].D);
    const TailPView<T> V0 = tail_pview<T, DM>(A, sm, 0);
    const int n0 = ncells(V0.D);
    for (int w = threadIdx.x; w < n0; w += blockDim.x) {
        V0.phi[w] = A.zero ? T(0) : A.g_pphi[g0 + w];
        V0.rhs[w] = A.g_prhs[g0 + w];
    }
    __syncthreads();
    for (int st = 0; st < 2 * A.nl - 1; ++st) {
        const bool up = st >= A.nl, down = st < A.nl - 1;
        const int l = up ? 2 * A.nl - 2 - st : st;
        const TailPView<T> F = tail_pview<T, DM>(A, sm, l);
        if (up) {
            const TailPView<T> Cc = tail_pview<T, DM>(A, sm, l + 1);
            const int nf = ncells(F.D);
            for (int w = threadIdx.x; w < nf; w += blockDim.x) {
                int i, j, k;
                unflat3d(F.D, w, i, j, k);
                F.phi[w] = F.phi[w] + Cc.phi[(i >> 1) + Cc.D.nx * ((j >> 1) + Cc.D.ny * (k >> 1))];
            }
            __syncthreads();
        }
        const int nsm = up ? A.nu2 : (down ? A.nu1 : A.nub);
        if (F.u)
            tail_cc_sweeps<T, DM, true>(F, nsm);
        else
            tail_cc_sweeps<T, DM, false>(F, nsm);
        if (down) {
            const TailPView<T> Cc = tail_pview<T, DM>(A, sm, l + 1);
            if (F.u)
                tail_cc_restrict<T, DM, true>(F, Cc);
            else
                tail_cc_restrict<T, DM, false>(F, Cc);
            __syncthreads();
        }
    }
    for (int w = threadIdx.x; w < n0; w += blockDim.x) A.g_pphi[g0 + w] = V0.phi[w];
}

// ------------------------------------------------------------------ launchers
// cells of one instance of a level
template <class T>
static int64_t inst_cells(const LevelDev<T>& L) {
    return L.n / (L.D.dm == 2 ? L.D.nz : 1);
}

template <class T>
static TailArgs<T> tail_args(const LevelDev<T>* L, int nl, int nu1, int nu2, int nub, int smoother, double omega, bool stag, bool zero) {
    TailArgs<T> a;
    memset(&a, 0, sizeof(a));
    a.nl = nl;
    a.nu1 = nu1;
    a.nu2 = nu2;
    a.nub = nub;
    a.smoother = smoother;
    a.omega = (T)omega;
    a.zero = zero ? 1 : 0;
    for (int d = 0; d < 3; ++d) {
        a.g_phi[d] = L[0].phi[d];
        a.g_rhs[d] = L[0].rhs[d];
    }
    a.g_pphi = L[0].pphi;
    a.g_prhs = L[0].prhs;
    int off = 0;
    for (int l = 0; l < nl; ++l) {
        TailLevel<T>& t = a.L[l];
        t.D = L[l].D;
        t.dxsqinv = (T)(1.0 / (L[l].dx * L[l].dx));
        t.C = L[l].coef();
        for (int d = 0; d < 3; ++d) t.pa[d] = L[l].pa[d];
        t.pa_uniform = L[l].pa_uniform;
        t.pa_value = L[l].pa_value;
        t.off = off;
        off += (int)inst_cells(L[l]) * (stag ? 2 * L[l].D.dm : 2);
    }
    a.tmp = off;
    return a;
}

// shared memory of a tail over levels L[0..nl-1]: phi and rhs of each, and
// one level's scratch (velocity: the residual, Jacobi's and an odd level's
// new values; pressure: an odd level's new values)
template <class T>
size_t tail_smem_bytes(const LevelDev<T>* L, int nl, bool stag) {
    size_t e = 0;
    for (int l = 0; l < nl; ++l) e += (size_t)inst_cells(L[l]) * (stag ? 2 * (size_t)L[l].D.dm : 2);
    if (stag)
        e += (size_t)inst_cells(L[0]) * (size_t)L[0].D.dm;
    else
        for (int l = 0; l < nl; ++l)
            if (odd_level(L[l].D)) {
                e += (size_t)inst_cells(L[l]);
                break;
            }
    return e * sizeof(T);
}

// threads of a tail block: one per owned pair of cells (an odd level: per
// cell) of the level that needs most, 128 to kTailThreads
template <class T>
static int tail_threads(const LevelDev<T>* L, int nl) {
    int64_t most = 128;
    for (int l = 0; l < nl; ++l) most = std::max<int64_t>(most, odd_level(L[l].D) ? inst_cells(L[l]) : inst_cells(L[l]) / 2);
    return (int)std::min<int64_t>((most + 31) / 32 * 32, kTailThreads);
}

// the dynamic shared-memory limit is raised once per kernel (never while a
// stream is being captured into a graph: the first call always runs eagerly)
template <class K, class A>
static cudaError_t launch_tail(K kernel, const A& args, int threads, size_t smem, cudaStream_t s) {
    cudaError_t e = raise_smem_limit((const void*)kernel, smem);
    if (e != cudaSuccess) return e;
    // one block per instance of a 2D batch (nz instances), else one block
    const int blocks = args.L[0].D.dm == 2 ? args.L[0].D.nz : 1;
    launch_pdl(kernel, dim3(blocks), dim3(threads), smem, s, args);
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_vcycle_tail(const LevelDev<T>* L, int nl, int visc, int nu1, int nu2, int nub, int smoother, double omega,
                               cudaStream_t s, bool zero) {
    if (nl < 1 || nl > kMaxTail) return cudaErrorInvalidValue;
    const TailArgs<T> a = tail_args<T>(L, nl, nu1, nu2, nub, smoother, omega, true, zero);
    const size_t smem = tail_smem_bytes<T>(L, nl, true);
    const int nt = tail_threads<T>(L, nl);
    cudaError_t e = cudaErrorInvalidValue;
    const bool wall = L[0].D.wall != 0;
    if (L[0].D.dm == 2) {
        if (wall) {
            LMM_VISC_DISPATCH(visc, (e = launch_tail(k_vcycle_tail<T, 2, V, true>, a, nt, smem, s)))
        } else {
            LMM_VISC_DISPATCH(visc, (e = launch_tail(k_vcycle_tail<T, 2, V>, a, nt, smem, s)))
        }
    } else {
        if (wall) {
            LMM_VISC_DISPATCH(visc, (e = launch_tail(k_vcycle_tail<T, 3, V, true>, a, nt, smem, s)))
        } else {
            LMM_VISC_DISPATCH(visc, (e = launch_tail(k_vcycle_tail<T, 3, V>, a, nt, smem, s)))
        }
    }
    return e;
}

template <class T>
cudaError_t launch_ccmg_tail(const LevelDev<T>* L, int nl, int nu1, int nu2, int nub, cudaStream_t s, bool zero) {
    if (nl < 1 || nl > kMaxTail) return cudaErrorInvalidValue;
    const TailArgs<T> a = tail_args<T>(L, nl, nu1, nu2, nub, 1, 1.0, false, zero);
    const size_t smem = tail_smem_bytes<T>(L, nl, false);
    const int nt = tail_threads<T>(L, nl);
    if (L[0].D.dm == 2) return launch_tail(k_ccmg_tail<T, 2>, a, nt, smem, s);
    return launch_tail(k_ccmg_tail<T, 3>, a, nt, smem, s);
}

#define LMM_INSTANTIATE_TAIL(T)                                                                                       \
    template cudaError_t launch_vcycle_tail<T>(const LevelDev<T>*, int, int, int, int, int, int, double, cudaStream_t, bool); \
    template cudaError_t launch_ccmg_tail<T>(const LevelDev<T>*, int, int, int, int, cudaStream_t, bool);             \
    template size_t tail_smem_bytes<T>(const LevelDev<T>*, int, bool);

}  // namespace lmm
