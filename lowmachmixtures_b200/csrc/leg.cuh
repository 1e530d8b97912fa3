// leg.cuh - one level's leg of a staggered V-cycle in one launch of a
// thread-block cluster: down = the smooths, the residual and its restriction
// (stag_mg_solver.f90:338-445); up = the prolongation and the smooths
// (:640-760).  For the levels between the single-block tail (tail.cuh) and
// those large enough to fill the chip.
//
// What bounds such a level: a colour is a few hundred cycles of work, but as a
// launch of its own it takes 1.4-1.7 us (index arithmetic, its loads' trip to
// L2, the stores' drain, the next launch).  Here the level is split in slabs
// of planes (3D: z, 2D: y), one per CTA; phi of the slab and of one plane on
// each side lives in shared memory, a thread keeps its cells' coefficients and
// diagonals in registers (Owned, tail.cuh), and a colour is shared-memory
// loads, the face arithmetic, one store (and one into the neighbour's halo
// plane for the cells next to it, by distributed shared memory) and a cluster
// barrier.  Every face goes through the value functions of the per-level
// kernels: same bits.
//
// Measured (live, a leg of two sweeps): FP32 16^3 8 us against 24 us of
// launches, 32^3 (16 CTAs, two pairs a thread) 17 against 24; 2D FP32 96 x 48
// with walls 7 against 15, 192 x 96 12 against 16.  A colour costs 0.4 us with
// one pair a thread and 0.9 with two, where the SM's issue slots bound it; more
// cells than that (leg_shape) keep their launches.
#pragma once
#include "pair3.cuh"
#include "prolong.cuh"
#include "tail.cuh"

namespace lmm {

constexpr int kLegThreads = 512;

template <class T>
struct LegArgs {
    Dims D, Dc;
    T dxsqinv, omega;
    Coef<T> C;
    int nsm, up, zero, nc;   // nc: CTAs of a cluster
    T* phi[3];
    const T* rhs[3];
    T* tmp[3];               // down: the residual on its way to the restriction
    const T* cphi[3];        // up: the coarse correction
    T* crhs[3];              // down: the coarse right-hand side
};

// A cell a thread owns.  phi of the slab is stored by parity of i + j + k, each
// half densely along pairs (2h, 2h + 1), so the lanes of a warp read and write
// consecutive words whichever colour they are on (interleaved, every access had
// a two-way bank conflict).  A step along one direction changes the parity, two
// steps don't; the position within a half moves by op / om, which add up.
// rdn / rup: where the cell lies in the halo planes of the CTAs below / above
// (component 0; 0: the cell is not next to that CTA).
template <class T, int DM, int VISC, bool W, int PAR>
struct LegCell {
    Owned<T, DM, VISC, W> o;   // o.s, o.op, o.om: positions in a half
    int r;                     // the cell's entry of rhs
    unsigned rdn, rup;

    // W: the ghost behind a wall mirrors the cell itself
    template <int D>
    __device__ __forceinline__ T up(const T* same, const T* opp, int d) const {
        if constexpr (W) {
            const T v = ldp<1>((o.hi >> d) & 1 ? same + o.s : opp + o.s + o.op[d], 0);
            if (d == D) return ((o.hi >> d) & 1) ? T(0) : v;
            return ((o.nhi >> d) & 1) ? -v : v;
        }
        return ldp<1>(opp, o.s + o.op[d]);
    }
    template <int D>
    __device__ __forceinline__ T down(const T* same, const T* opp, int d) const {
        if constexpr (W) {
            const T v = ldp<1>((o.lo >> d) & 1 ? same + o.s : opp + o.s + o.om[d], 0);
            if (d != D) return ((o.nlo >> d) & 1) ? -v : v;
            return v;
        }
        return ldp<1>(opp, o.s + o.om[d]);
    }
    template <int D>
    __device__ __forceinline__ void cross(const T* same, const T* opp, int t, T (&x)[4]) const {
        if constexpr (VISC == 1 || VISC == -1) {
            x[0] = x[1] = x[2] = x[3] = T(0);
            return;
        }
        x[0] = ldp<1>(opp, o.s + o.op[t]);
        x[1] = ldp<1>(same, o.s);
        x[2] = ldp<1>(same, o.s + o.om[D] + o.op[t]);
        x[3] = ldp<1>(opp, o.s + o.om[D]);
        if constexpr (W)
            if ((o.hi >> t) & 1) x[0] = x[2] = T(0);
    }
    // L phi of face D; p: phi in shared memory, pitch elements per component, hp per half
    template <int D>
    __device__ __forceinline__ T apply(const T* p, int pitch, int hp, T dxsqinv, T p0, T b, T c) const {
        T E1, E1p, E2, E2p;
        o.template edges<D>(E1, E1p, E2, E2p);
        const T* same = p + D * pitch + PAR * hp;
        const T* opp = p + D * pitch + (1 - PAR) * hp;
        if constexpr (DM == 2) {
            constexpr int t = 1 - D;
            T x[4];
            cross<D>(p + t * pitch + PAR * hp, p + t * pitch + (1 - PAR) * hp, t, x);
            const FaceCoef2<T> k{T(0), o.be[0], o.be[1 + D], E1, E1p, o.g[0], o.g[1 + D]};
            return face_L2_sum<T, VISC>(o.cen[D], p0, up<D>(same, opp, D), down<D>(same, opp, D), up<D>(same, opp, t), down<D>(same, opp, t), x, k,
                                        dxsqinv, b, c);
        } else {
            constexpr int t1 = Perm3<D>::t1, t2 = Perm3<D>::t2;
            T q1[4], q2[4], nb[6];
            cross<D>(p + t1 * pitch + PAR * hp, p + t1 * pitch + (1 - PAR) * hp, t1, q1);
            cross<D>(p + t2 * pitch + PAR * hp, p + t2 * pitch + (1 - PAR) * hp, t2, q2);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                nb[2 * d] = up<D>(same, opp, d);
                nb[2 * d + 1] = down<D>(same, opp, d);
            }
            return face_L3_sum<T, VISC>(o.cen[D], p0, nb, D, q1, q2, o.be[0], o.be[1 + D], E1, E1p, E2, E2p, o.g[0], o.g[1 + D], dxsqinv,
                                        b, c);
        }
    }
    // phi of component d, here and in the neighbours' halo planes
    __device__ __forceinline__ void put(T* p, int pitch, int hp, int d, T v) const {
        p[d * pitch + PAR * hp + o.s] = v;
        if (rdn) dsmem_store(rdn + (unsigned)(d * pitch * sizeof(T)), v);
        if (rup) dsmem_store(rup + (unsigned)(d * pitch * sizeof(T)), v);
    }
    template <int D>
    __device__ __forceinline__ void colour(T* p, const T* rhs, int pitch, int hp, int rp, T omega, T dxsqinv, T b, T c) const {
        if (o.template face<D>()) {
            const T p0 = ldp<1>(p, D * pitch + PAR * hp + o.s);
            put(p, pitch, hp, D, gs_update(p0, omega, ldp<1>(rhs, D * rp + r), apply<D>(p, pitch, hp, dxsqinv, p0, b, c), o.diag[D]));
        }
    }
    template <int D>
    __device__ __forceinline__ T resid(const T* p, const T* rhs, int pitch, int hp, int rp, T dxsqinv, T b, T c) const {
        if (!o.template face<D>()) return T(0);
        return (apply<D>(p, pitch, hp, dxsqinv, ldp<1>(p, D * pitch + PAR * hp + o.s), b, c) - ldp<1>(rhs, D * rp + r)) * T(-1);
    }
};

// PP: pairs of cells a thread owns
template <class T, int DM, int VISC, bool W, int PP>
__global__ void __launch_bounds__(kLegThreads, 1) k_level_leg(const __grid_constant__ LegArgs<T> A) {
    extern __shared__ __align__(16) unsigned char leg_smem[];
    T* sm = reinterpret_cast<T*>(leg_smem);
    constexpr int SD = DM - 1;
    const int NC = A.nc, rank = (int)cluster_rank();
    const int plane = DM == 3 ? A.D.nx * A.D.ny : A.D.nx, S = DM == 3 ? A.D.nz : A.D.ny;
    const int half = A.D.nx >> 1, hplane = plane >> 1;
    const int z0 = rank * S / NC, z1 = (rank + 1) * S / NC, t = z1 - z0;
    const int hp = ((S + NC - 1) / NC + 2) * hplane, pitch = 2 * hp;   // entries of a half, of one component
    const int rp = 2 * PP * blockDim.x;                                // entries of one component of rhs
    T* rhs = sm + DM * pitch;
    TailView<T> L;
    L.D = A.D;
    L.dxsqinv = A.dxsqinv;
    L.C = A.C;
    const Dims Dc = A.Dc;
    // the coefficients, ahead of the wait for the previous kernel: they are
    // written once per coefficient load, never by the launch before this one
    const T b = ld(L.C.beta, 0), c = ld(L.C.gamma, 0);
    LegCell<T, DM, VISC, W, 0> E[PP];   // the cells of even i + j + k
    LegCell<T, DM, VISC, W, 1> O[PP];   // and of odd
    int at[PP], jk[PP];                 // a pair's first cell: index in the level, j and k
    {
        const int pairs = t * hplane;
        const unsigned base = (unsigned)__cvta_generic_to_shared(sm);
        const int below = rank == 0 ? NC - 1 : rank - 1, above = rank == NC - 1 ? 0 : rank + 1;
        const int tb = (below + 1) * S / NC - below * S / NC;   // planes of the CTA below
#pragma unroll
        for (int u = 0; u < PP; ++u) {
            const int w = threadIdx.x + u * blockDim.x;
            E[u].o.on = O[u].o.on = w < pairs;
            E[u].rdn = E[u].rup = O[u].rdn = O[u].rup = 0;
            E[u].r = 2 * u * blockDim.x + threadIdx.x;
            O[u].r = E[u].r + blockDim.x;
            at[u] = jk[u] = 0;
            if (w < pairs) {
                const int h = w % half, r = w / half;
                const int j = DM == 3 ? r % A.D.ny : z0 + r, k = DM == 3 ? z0 + r / A.D.ny : 0, z = DM == 3 ? k : j;
                const int q = DM == 3 ? h + half * j : h;   // within a half plane
                at[u] = 2 * q + z * plane;
                jk[u] = j | (k << 16);
                auto take = [&](auto& x, int i, int par) {
                    x.o.load(L, i, j, k, b, c);
                    x.o.s = (z - z0 + 1) * hplane + q;
                    x.o.op[0] = (i & 1) ? (h == half - 1 ? 1 - half : 1) : 0;
                    x.o.om[0] = (i & 1) ? 0 : (h == 0 ? half - 1 : -1);
                    if constexpr (DM == 3) {
                        x.o.op[1] = j == A.D.ny - 1 ? -(A.D.ny - 1) * half : half;
                        x.o.om[1] = j == 0 ? (A.D.ny - 1) * half : -half;
                    }
                    x.o.op[SD] = hplane;
                    x.o.om[SD] = -hplane;
                    if (z == z0) x.rdn = dsmem_at(base + (unsigned)((par * hp + (tb + 1) * hplane + q) * sizeof(T)), below);
                    if (z == z1 - 1) x.rup = dsmem_at(base + (unsigned)((par * hp + q) * sizeof(T)), above);
                };
                const int p = (j + k) & 1;
                take(E[u], 2 * h + p, 0);
                take(O[u], 2 * h + 1 - p, 1);
            }
        }
    }
    const bool zero = !A.up && A.zero;
    if (zero)
        for (int w = threadIdx.x; w < DM * pitch; w += blockDim.x) sm[w] = T(0);
    pdl_enter();
    cluster_sync();   // every CTA of the cluster runs: its halo planes can be written
#pragma unroll
    for (int u = 0; u < PP; ++u) {
        if (!E[u].o.on) continue;
        const int j = jk[u] & 0xffff, k = jk[u] >> 16, p = (j + k) & 1, h = (at[u] % A.D.nx) >> 1;
        const int g = at[u];
#pragma unroll
        for (int d = 0; d < DM; ++d) {
            const T f0 = ldp<1>(A.rhs[d], g), f1 = ldp<1>(A.rhs[d], g + 1);
            rhs[d * rp + E[u].r] = p ? f1 : f0;
            rhs[d * rp + O[u].r] = p ? f0 : f1;
        }
        if (!zero) {
            T v[3][2] = {};
#pragma unroll
            for (int d = 0; d < DM; ++d) {
                v[d][0] = ldp<1>(A.phi[d], g);
                v[d][1] = ldp<1>(A.phi[d], g + 1);
            }
            if (A.up) prolong_cells<T, DM, W>(Dc, A.cphi[0], A.cphi[1], A.cphi[DM - 1], h, j, k, v);
#pragma unroll
            for (int d = 0; d < DM; ++d) {
                E[u].put(sm, pitch, hp, d, p ? v[d][1] : v[d][0]);
                O[u].put(sm, pitch, hp, d, p ? v[d][0] : v[d][1]);
            }
        }
    }
    if (!zero) cluster_sync();
    for (int s = 0; s < A.nsm; ++s) {
#define LMM_LEG_COLOUR(D_, X_)                                                                                                 \
    _Pragma("unroll") for (int u = 0; u < PP; ++u) X_[u].template colour<D_>(sm, rhs, pitch, hp, rp, A.omega, A.dxsqinv, b, c); \
    cluster_sync();
        LMM_LEG_COLOUR(0, E)
        LMM_LEG_COLOUR(0, O)
        LMM_LEG_COLOUR(1, E)
        LMM_LEG_COLOUR(1, O)
        if constexpr (DM == 3) {
            LMM_LEG_COLOUR(2, E)
            LMM_LEG_COLOUR(2, O)
        }
#undef LMM_LEG_COLOUR
    }
#pragma unroll
    for (int u = 0; u < PP; ++u) {
        if (!E[u].o.on) continue;
        const int p = ((jk[u] & 0xffff) + (jk[u] >> 16)) & 1;
        const int g = at[u];
#pragma unroll
        for (int d = 0; d < DM; ++d) {
            A.phi[d][g + p] = sm[d * pitch + E[u].o.s];
            A.phi[d][g + 1 - p] = sm[d * pitch + hp + O[u].o.s];
        }
        if (A.up) continue;
        A.tmp[0][g + p] = E[u].template resid<0>(sm, rhs, pitch, hp, rp, A.dxsqinv, b, c);
        A.tmp[0][g + 1 - p] = O[u].template resid<0>(sm, rhs, pitch, hp, rp, A.dxsqinv, b, c);
        A.tmp[1][g + p] = E[u].template resid<1>(sm, rhs, pitch, hp, rp, A.dxsqinv, b, c);
        A.tmp[1][g + 1 - p] = O[u].template resid<1>(sm, rhs, pitch, hp, rp, A.dxsqinv, b, c);
        if constexpr (DM == 3) {
            A.tmp[2][g + p] = E[u].template resid<2>(sm, rhs, pitch, hp, rp, A.dxsqinv, b, c);
            A.tmp[2][g + 1 - p] = O[u].template resid<2>(sm, rhs, pitch, hp, rp, A.dxsqinv, b, c);
        }
    }
    if (A.up) return;
    cluster_sync();   // the residual is in L2 for every CTA of the cluster
    const int nc = Dc.nx * Dc.ny * Dc.nz;
    for (int w2 = rank * blockDim.x + threadIdx.x; w2 < nc * DM; w2 += NC * blockDim.x) {
        const int comp = w2 / nc, w = w2 - comp * nc;
        int i, j, k;
        unflat3d(Dc, w, i, j, k);
        if (comp == 0)
            A.crhs[0][w] = restrict_one<T, DM, 0, W, 2>(L.D, A.tmp[0], Dc, i, j, k);
        else if (comp == 1)
            A.crhs[1][w] = restrict_one<T, DM, 1, W, 2>(L.D, A.tmp[1], Dc, i, j, k);
        else if constexpr (DM == 3)
            A.crhs[2][w] = restrict_one<T, DM, 2, W, 2>(L.D, A.tmp[2], Dc, i, j, k);
    }
}

// how a level is split: nc CTAs, pp pairs per thread; nc = 0: not taken
struct LegShape {
    int nc = 0, pp = 0, threads = 0;
    size_t smem = 0;
};
template <class T>
LegShape leg_shape(const LevelDev<T>& L, int visc) {
    LegShape r;
    if (visc >= 0 || odd_level(L.D) || (L.D.dm == 2 && L.D.nz != 1)) return r;   // (a batch stacks nz instances)
    const int dm = L.D.dm, plane = dm == 3 ? L.D.nx * L.D.ny : L.D.nx, S = dm == 3 ? L.D.nz : L.D.ny;
    for (int nc : {8, 16}) {
        const int t = (S + nc - 1) / nc;
        const int64_t pairs = (int64_t)t * plane / 2;
        const int pp = pairs <= kLegThreads ? 1 : 2;
        if (S < nc || pairs > (int64_t)pp * kLegThreads || (pp == 2 && sizeof(T) == 8)) continue;
        if (nc == 8 && pp == 2) continue;   // twice the CTAs rather than twice the cells per thread
        if (pp == 2 && dm == 3 && L.D.wall) continue;   // spills: 35 us a leg against 24 of launches (32 x 24 x 32)
        const int threads = (int)((pairs + pp - 1) / pp + 31) / 32 * 32;
        r.smem = (size_t)dm * ((size_t)(t + 2) * plane + 2 * pp * threads) * sizeof(T);
        if (r.smem > 200 * 1024) continue;
        r.nc = nc;
        r.pp = pp;
        r.threads = threads;
        return r;
    }
    return r;
}

// fits null: the launch; else asks whether the device can hold its cluster
template <class K, class A>
static cudaError_t launch_leg_k(K kernel, const A& args, const LegShape& sh, cudaStream_t s, bool* fits) {
    cudaError_t e = raise_smem_limit((const void*)kernel, std::max<size_t>(sh.smem, 49152));
    if (e != cudaSuccess) return e;
    if (sh.nc > 8) {
        e = cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return e;
    }
    const dim3 nc(sh.nc), block(sh.threads);   // one cluster
    if (fits) {
        *fits = cluster_fits((const void*)kernel, sh.nc, sh.threads, sh.smem);
        return cudaSuccess;
    }
    return launch_cluster(kernel, nc, block, nc, sh.smem, s, args);
}

template <class T, int DM, bool W, int PP>
static cudaError_t launch_leg_v(int visc, const LegArgs<T>& a, const LegShape& sh, cudaStream_t s, bool* fits) {
    switch (visc) {
        case -1: return launch_leg_k(k_level_leg<T, DM, -1, W, PP>, a, sh, s, fits);
        case -2: return launch_leg_k(k_level_leg<T, DM, -2, W, PP>, a, sh, s, fits);
        default: return launch_leg_k(k_level_leg<T, DM, -3, W, PP>, a, sh, s, fits);
    }
}
template <class T, int DM, bool W>
static cudaError_t launch_leg_p(int visc, const LegArgs<T>& a, const LegShape& sh, cudaStream_t s, bool* fits) {
    if constexpr (sizeof(T) == 4)
        if (sh.pp == 2) return launch_leg_v<T, DM, W, 2>(visc, a, sh, s, fits);
    return launch_leg_v<T, DM, W, 1>(visc, a, sh, s, fits);
}
template <class T>
static cudaError_t launch_leg(const LevelDev<T>& L, int visc, const LegArgs<T>& a, const LegShape& sh, cudaStream_t s, bool* fits) {
    if (L.D.dm == 2)
        return L.D.wall ? launch_leg_p<T, 2, true>(visc, a, sh, s, fits) : launch_leg_p<T, 2, false>(visc, a, sh, s, fits);
    return L.D.wall ? launch_leg_p<T, 3, true>(visc, a, sh, s, fits) : launch_leg_p<T, 3, false>(visc, a, sh, s, fits);
}

template <class T>
bool leg_supported(const LevelDev<T>& L, int visc) {
    const LegShape sh = leg_shape<T>(L, visc);
    bool fits = false;
    return sh.nc > 0 && launch_leg<T>(L, visc, LegArgs<T>{}, sh, nullptr, &fits) == cudaSuccess && fits;
}

template <class T>
cudaError_t launch_level_leg(const LevelDev<T>& L, const LevelDev<T>& Cc, int visc, bool up, int nsm, double omega, cudaStream_t s,
                             bool zero) {
    const LegShape sh = leg_shape<T>(L, visc);
    if (sh.nc == 0) return cudaErrorInvalidValue;
    LegArgs<T> a;
    memset(&a, 0, sizeof(a));
    a.D = L.D;
    a.Dc = Cc.D;
    a.dxsqinv = (T)(1.0 / (L.dx * L.dx));
    a.omega = (T)omega;
    a.C = L.coef();
    a.nsm = nsm;
    a.up = up ? 1 : 0;
    a.zero = zero ? 1 : 0;
    a.nc = sh.nc;
    for (int d = 0; d < L.D.dm; ++d) {
        a.phi[d] = L.phi[d];
        a.rhs[d] = L.rhs[d];
        a.tmp[d] = L.tmp[d];
        a.cphi[d] = Cc.phi[d];
        a.crhs[d] = Cc.rhs[d];
    }
    return launch_leg<T>(L, visc, a, sh, s, nullptr);
}

#define LMM_INSTANTIATE_LEG(T)                                                  \
    template bool leg_supported<T>(const LevelDev<T>&, int);                    \
    template bool launch_residual_pairs<T>(const LevelDev<T>&, int, const T* const[3], const T* const[3], T* const[3], cudaStream_t); \
    template void launch_prolong_add<T>(const LevelDev<T>&, const LevelDev<T>&, const T* const[3], T* const[3], cudaStream_t); \
    template cudaError_t launch_level_leg<T>(const LevelDev<T>&, const LevelDev<T>&, int, bool, int, double, cudaStream_t, bool);

}  // namespace lmm
