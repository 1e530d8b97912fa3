// wgrad_tile.cuh - weight gradient of the 3x3x3 periodic convolution from
// shared-memory halo tiles: dW[co][t][ci] += sum_v g[v][co] x[v + t][ci].
//
// A GEMM with K = voxels whose other two sides are small (27 Cin x Cout), so
// what bounds a plain implicit GEMM is forming its operand: every input voxel
// is gathered 27 times with its index arithmetic (k_conv3d_wgrad: the network's
// eleven layers at 2 x 64^3 took 2531 us, 30 TFLOP/s; 406 us here: 47 us for
// 16 -> 16 channels at 64^3, 66 for 32 -> 16, 21 for 32 -> 32 at 32^3).  Here a step stages P output-gradient planes and the
// P + 2 input halo planes of one 8 x 16 tile once, channel-group-major as
// conv_tile.cuh lays them out, [group of 8 channels][y][x][8 channels].  In
// MN-major form eight consecutive x voxels are the K rows of a core matrix,
// one halo row is the K stride and one channel group the M stride, so
//   - the nine (dy, dx) taps are shifted descriptors of the staged planes;
//   - the M = 128 rows run over the channel groups of consecutive planes
//     (a plane's groups continue the one before), the N columns over the P
//     gradient planes: one MMA forms the products of every (input plane a,
//     gradient plane b) and the three z taps are those with a - b = 0, 1, 2.
// Rows of products with another a - b, and rows past the staged planes, are
// accumulated and never read (a row of D depends on its own row of A alone).
// The accumulators (9 taps x MT row tiles x P NS columns <= 432 of the 512 TMEM
// columns) stay in TMEM over all the CTA's steps; at the end the P products
// of a tap are added in shared memory in the order of b and leave by one
// atomic per weight and CTA.
//
// P is the largest that keeps the accumulators within TMEM (Cin 8, 16: 3;
// Cin 32 with 16 output channels: 2; else 1); wider outputs go in slices of
// NS channels.  A ragged tile's gradient voxels past the grid are staged as
// zeros, so every grid size is taken.
//
// Roles: warps 0..7 copy (cp.async, kStagesWG stages, one mbarrier per stage
// filled by all 256 threads), warp 8's lane 0 issues the MMAs and commits each
// stage to its release barrier.  Waits are bounded as in conv_tile_ws.cuh.
#pragma once
#include "conv_tile.cuh"

namespace lmm {
namespace nn {

constexpr int kStagesWG = 2;
constexpr int kLoadersWG = 256;
constexpr int kThreadsWG = kLoadersWG + 32;
constexpr int kPlaneG = kTX * kTY * 16;   // bytes of one channel group of a gradient plane

__host__ __device__ constexpr int wg_xstage(int ng, int p) { return (p + 2) * ng * kGStride; }
__host__ __device__ constexpr int wg_gstage(int ns, int p) { return p * (ns / 8) * kPlaneG; }
__host__ __device__ constexpr int wg_mtiles(int ng, int p) { return ((p + 2) * ng + 15) / 16; }
// the operand stages, at least as much as the last stage's descriptors reach
// (16 channel groups per row tile), or the weights of the epilogue
__host__ __device__ constexpr int wg_data_bytes(int ng, int ns, int p) {
    const int st = kStagesWG * (wg_xstage(ng, p) + wg_gstage(ns, p));
    const int reach = (kStagesWG - 1) * wg_xstage(ng, p) + wg_mtiles(ng, p) * 16 * kGStride;
    const int w = 27 * ng * 8 * ns * 4;
    return st > reach ? (st > w ? st : w) : (reach > w ? reach : w);
}
__host__ __device__ constexpr int wg_smem_bytes(int ng, int ns, int p) { return wg_data_bytes(ng, ns, p) + 2 * kStagesWG * 8 + 16; }

struct WgradArgs {
    const bf16* x;    // input activations, Cin channels per voxel (on the half grid when up)
    const bf16* g;    // output gradient, Cg channels per voxel
    float* dw;        // [Cout][27 * Cin]
    int nx, ny, nz;   // output grid
    int up, B, Cg, Cout;
    int tiles_x, tiles_y, zsteps, steps;   // steps: tiles x ceil(nz / P)
};

template <int NG, int NS, int P>
__global__ void __launch_bounds__(kThreadsWG, 1) k_conv3d_wgrad_tile(WgradArgs A, int* err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr int CIN = NG * 8, MT = wg_mtiles(NG, P), N = P * NS;
    constexpr int XST = wg_xstage(NG, P), GST = wg_gstage(NS, P);
    constexpr int XU = XST / 16, GU = GST / 16, GG = NS / 8;
    constexpr uint32_t NCOLS = 512;
    static_assert(9 * MT * N <= 512 && N % 16 == 0 && N <= 256, "accumulators fit in TMEM");
    uint8_t* xs = smem;
    uint8_t* gs = smem + kStagesWG * XST;
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + wg_data_bytes(NG, NS, P));
    uint64_t* freed = full + kStagesWG;
    uint32_t* holder = reinterpret_cast<uint32_t*>(freed + kStagesWG);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(holder + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n0 = blockIdx.y * NS;
    const int start = (int)((int64_t)A.steps * blockIdx.x / gridDim.x), end = (int)((int64_t)A.steps * (blockIdx.x + 1) / gridDim.x);

    if (warp == 0) tc::tmem_alloc(holder, NCOLS);
    if (tid == 0) {
        for (int q = 0; q < kStagesWG; ++q) {
            tc::mbar_init(full + q, kLoadersWG);
            tc::mbar_init(freed + q, 1);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = *holder;

    auto wait_bar = [&](uint64_t* bar, unsigned parity) -> bool {
        const uint32_t a = tc::smem_u32(bar);
        for (unsigned it = 0; it < tc::kSpinLimit; ++it) {
            uint32_t done;
            asm volatile(
                "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                : "=r"(done)
                : "r"(a), "r"(parity)
                : "memory");
            if (done) return true;
            if ((it & 63) == 63) {
                if (*abort_flag) return false;
                __nanosleep(64);
            }
        }
        return false;
    };
    auto give_up = [&]() {
        *abort_flag = 1;
        atomicExch(err, 1);
    };

    if (warp == kLoadersWG / 32) {
        // ------------------------------------------------------------- MMA
        if (lane == 0) {
            const uint32_t idesc = tc::idesc_bf16(tc::kM, N, 1, 1);
            const uint32_t a_lo = (tc::smem_u32(xs) >> 4) | ((uint32_t)((kHX * 16) >> 4) << 16);
            const uint32_t a_hi = (uint32_t)(kGStride >> 4) | (1u << 14);
            const uint32_t b_lo = (tc::smem_u32(gs) >> 4) | ((uint32_t)((kTX * 16) >> 4) << 16);
            const uint32_t b_hi = (uint32_t)(kPlaneG >> 4) | (1u << 14);
            int last = -1;
            for (int st = start; st < end; ++st) {
                const int it = st - start, slot = it % kStagesWG;
                if (!wait_bar(full + slot, (unsigned)((it / kStagesWG) & 1))) {
                    give_up();
                    break;
                }
                tc::fence_async_smem();   // the copies (generic proxy) before the MMAs read them
                tc::tc_fence_after();
                const uint32_t al = a_lo + (uint32_t)(slot * (XST >> 4)), bl = b_lo + (uint32_t)(slot * (GST >> 4));
#pragma unroll
                for (int ks = 0; ks < kTY / 2; ++ks) {
                    const uint64_t bd = ((uint64_t)b_hi << 32) | (uint64_t)(bl + (uint32_t)(2 * ks * kTX));
#pragma unroll
                    for (int q = 0; q < 9; ++q)
#pragma unroll
                        for (int mt = 0; mt < MT; ++mt) {
                            const uint64_t ad =
                                ((uint64_t)a_hi << 32) |
                                (uint64_t)(al + (uint32_t)((q / 3 + 2 * ks) * kHX + q % 3 + mt * 16 * (kGStride >> 4)));
                            tc::mma_bf16(tmem + (uint32_t)((q * MT + mt) * N), ad, bd, idesc, (it > 0 || ks > 0) ? 1u : 0u);
                        }
                }
                tc::mma_commit(freed + slot);
                last = it;
            }
            // every MMA has completed (bounded, twice) before the accumulators are read or TMEM freed
            if (last >= 0 && !tc::mbar_wait(freed + last % kStagesWG, (unsigned)((last / kStagesWG) & 1)) &&
                !tc::mbar_wait(freed + last % kStagesWG, (unsigned)((last / kStagesWG) & 1)))
                give_up();
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------- copies
        const int nxi = A.nx >> A.up, nyi = A.ny >> A.up, nzi = A.nz >> A.up;
        for (int st = start; st < end; ++st) {
            const int it = st - start, slot = it % kStagesWG;
            if (it >= kStagesWG) {
                int w = 1;
                if (lane == 0) w = wait_bar(freed + slot, (unsigned)((it / kStagesWG - 1) & 1)) ? 1 : 0;
                if (!__shfl_sync(0xffffffffu, w, 0)) {
                    if (lane == 0) give_up();
                    break;
                }
            }
            int tile = st / A.zsteps;
            const int z0 = (st - tile * A.zsteps) * P;
            const int x0 = (tile % A.tiles_x) * kTX;
            tile /= A.tiles_x;
            const int y0 = (tile % A.tiles_y) * kTY, b = tile / A.tiles_y;
            // 16-byte units, channel groups fastest: a warp's copies cover whole sectors
            for (int u = tid; u < XU; u += kLoadersWG) {
                const int grp = u % NG, v = u / NG;
                const int a = v / kHalo, h = v - a * kHalo, hy = h / kHX, hx = h - hy * kHX;
                int xx = x0 - 1 + hx, yy = y0 - 1 + hy, zz = z0 - 1 + a;
                xx = xx < 0 ? xx + A.nx : (xx >= A.nx ? xx % A.nx : xx);
                yy = yy < 0 ? yy + A.ny : (yy >= A.ny ? yy % A.ny : yy);
                zz = zz < 0 ? zz + A.nz : (zz >= A.nz ? zz % A.nz : zz);
                const bf16* src =
                    A.x + ((((int64_t)b * nzi + (zz >> A.up)) * nyi + (yy >> A.up)) * nxi + (xx >> A.up)) * CIN + 8 * grp;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tc::smem_u32(xs + slot * XST + (a * NG + grp) * kGStride + h * 16)),
                             "l"(src)
                             : "memory");
            }
            for (int u = tid; u < GU; u += kLoadersWG) {
                const int grp = u % GG, v = u / GG;
                const int p = v / (kTX * kTY), h = v - p * (kTX * kTY), yy = y0 + h / kTX, xx = x0 + h % kTX, zz = z0 + p;
                const bool in = xx < A.nx && yy < A.ny && zz < A.nz && n0 + 8 * grp < A.Cg;
                const bf16* src = in ? A.g + ((((int64_t)b * A.nz + zz) * A.ny + yy) * A.nx + xx) * A.Cg + n0 + 8 * grp : A.g;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                                 tc::smem_u32(gs + slot * GST + (p * GG + grp) * kPlaneG + h * 16)),
                             "l"(src), "r"(in ? 16 : 0)
                             : "memory");
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(tc::smem_u32(full + slot)) : "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    if (start < end && !*abort_flag) {
        // row r of tile mt: channel (r & 7) of group (16 mt + r / 8) = a NG + group of input plane a
        float* w = reinterpret_cast<float*>(smem);   // [co][t][ci] of the slice
#pragma unroll 1
        for (int bb = 0; bb < P; ++bb) {
            if (warp < 4)
#pragma unroll 1
                for (int qm = 0; qm < 9 * MT; ++qm) {
                    const int q = qm / MT, mt = qm - q * MT;
                    const int row = 128 * mt + 32 * warp + lane, grp = row >> 3, a = grp / NG, ci = (grp - a * NG) * 8 + (row & 7);
                    const int tz = a - bb;
                    const bool use = tz >= 0 && tz <= 2;
#pragma unroll
                    for (int c0 = 0; c0 < NS; c0 += 16) {
                        float v[16];
                        tc::tmem_ld16(tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)(qm * N + bb * NS + c0), v);
                        if (use)
#pragma unroll
                            for (int e = 0; e < 16; ++e) {
                                float* d = w + (c0 + e) * 27 * CIN + (tz * 9 + q) * CIN + ci;
                                *d = bb == 0 ? v[e] : *d + v[e];
                            }
                    }
                }
            __syncthreads();
        }
        for (int e = tid; e < NS * 27 * CIN; e += kThreadsWG) {
            const int co = n0 + e / (27 * CIN);
            if (co < A.Cout) atomicAdd(A.dw + (int64_t)n0 * 27 * CIN + e, w[e]);
        }
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, NCOLS);
}

}  // namespace nn
}  // namespace lmm
