// wgrad_tc.cuh -- the weight gradient of a 3x3x3 convolution with 16 input
// and 16 output channels on the 5th-generation tensor cores.
//
//   dW[t][ci][co] = sum over cells c of G[c][co] * X[c + off(t)][ci]
//
// with X the layer's input activations and G the gradient with respect to its
// pre-activation, both in the two-plane BF16 layout of conv_tc.cuh, and
// off(t) = dx + dy*nx + dz*nx*ny.  As a GEMM the cells are the reduction
// (K) dimension: D[m][n] = sum_k A[m][k] B[n][k] with m = (tap, ci), n = co,
// k = cell, FP32 in tensor memory.
//
// Operands.  A line block of conv_tc.cuh -- 136 rows as [group][row][8
// channels] -- is also the no-swizzle MN-major operand layout: 8 rows x 16
// bytes form a 128-byte core matrix with the CHANNELS contiguous (channels on M
// or N, cells on K; K groups of 8 cells 128 bytes apart = LBO, channel groups
// 2176 bytes apart = SBO), and rows are 16 bytes apart throughout, so that a
// move of the start address by 16 bytes is the next cell.  Operand A of one
// MMA (M = 128) is 8 taps x 16 channels from 8 line blocks back to back.  A
// tile loads one block per (dy, dz), first row c0 - 1 + dy*nx + dz*nx*ny; the
// first 8 give the taps of dx = -1, 0, 1 at row offsets 0, 1, 2, three MMAs.
// The ninth pair's three taps are one MMA more, from three blocks whose first
// rows are one cell apart (its other rows read blocks of the same tile and are
// never used).  With operand B's (N = 16) that is 12 blocks a tile in 408 pieces
// of 128 bytes.  A block per tap and operand from channels-last cells, 36 a tile
// in 9216 pieces of 16 bytes, took 210 us for 16 crops of 34^3, bound by the
// pieces (12 thousand cycles a tile); now 34 (B200).  One MMA covers K = 16 cells
// (descriptor start + 256 bytes per step), 8 steps a tile of 128 cells.  Each of
// the four MMAs accumulates into its own 16 TMEM columns over every tile the
// CTA takes; at the end the four accumulators are the CTA's partial dW.
//
// Windows that start before the array or run past it read zeros.  Batched
// grids are consecutive in the array; a window crossing into the next member
// meets only G = 0 there (G vanishes off the interior, and an interior cell's
// 27 neighbours lie inside its own member).
//
// Warp roles (192 threads): warp 4 lane 0 issues the TMA loads, warp 5 the
// MMAs, warps 0-3 read the accumulators out at the end (TMEM lanes
// 32w..32w+31).  mbarriers: full[s] (a stage's 12 blocks landed), empty[s] (the
// MMAs reading the stage completed), done (every MMA completed).  Every wait
// is bounded; a role that gives up raises *err, and the producer and the MMA
// issuer still wait for their own copies and MMAs before the CTA leaves.
#pragma once

#include "conv_tc.cuh"

namespace piro {
namespace tc {

constexpr int kWgRows = 128;                   // cells per tile (8 MMAs of K = 16)
constexpr int kWgTaps = 8;                     // taps per MMA (M = 8 x 16)
constexpr int kWgAcc = 4;                      // accumulators: dx = -1, 0, 1 of 8 pairs (dy, dz); the ninth pair
constexpr int kWgBlocks = 12;                  // the ninth pair's 3 blocks, G's, the other 8 pairs'
constexpr int kWgG = 3 * kLineBytes, kWgX = 4 * kLineBytes;  // their places in a stage
constexpr int kWgStageBytes = kWgBlocks * kLineBytes;        // 51 KB
constexpr int kWgStages = 4;
constexpr int kWgThreads = 192;
constexpr int kWgBarOff = kWgStages * kWgStageBytes;
constexpr int kWgSmemBytes = kWgBarOff + (2 * kWgStages + 2) * 8 + 16 + 128;

// Instruction descriptor of kind::f16 with both operands MN-major (bits 15
// and 16): FP32 accumulator, BF16 A and B, N = 16, M = 128.
constexpr uint32_t kIdescMN = kIdesc | (1u << 15) | (1u << 16);

struct WgArgs {
    int nx;
    int64_t nxy;
    int64_t ntiles;   // tiles of kWgRows cells over all rows of the arrays
    int ci_n, co_n;   // channels kept in the partial layout (the layer's CI and CO)
    float *partials;  // [gridDim.x][27 * ci_n * co_n], per CTA: (t * ci_n + ci) * co_n + co
    int *err;
};

__global__ void __launch_bounds__(kWgThreads, 1) k_wgrad_tc(const __grid_constant__ CUtensorMap xmap,
                                                             const __grid_constant__ CUtensorMap gmap, WgArgs a)
{
    extern __shared__ unsigned char smem_raw[];
    unsigned char *sm = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~(uintptr_t)127);
    const uint32_t stage_s = smem_u32(sm);
    const uint32_t bar_s = stage_s + kWgBarOff;  // full[S], empty[S], done, drain
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(sm + kWgBarOff + (2 * kWgStages + 2) * 8);
    auto full = [&](int i) { return bar_s + 8u * i; };
    auto empty = [&](int i) { return bar_s + 8u * (kWgStages + i); };
    const uint32_t done_s = bar_s + 8u * (2 * kWgStages);
    const uint32_t drain_s = bar_s + 8u * (2 * kWgStages + 1);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // uniform, for the compiler
    const int64_t my_tiles = (int64_t)blockIdx.x < a.ntiles ? (a.ntiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kWgStages; ++i) {
            mbar_init(full(i), 1);
            mbar_init(empty(i), 1);
        }
        mbar_init(done_s, 1);
        mbar_init(drain_s, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(64)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t *>(tmem_slot), 0);
    bool mma_ok = my_tiles > 0;
    grid_launch_next();
    grid_wait();

    if (warp == 4) {
        if (lane == 0 && my_tiles > 0) {
            int64_t i = 0;
            for (; i < my_tiles; ++i) {
                const int s = (int)(i % kWgStages);
                if (i >= kWgStages && !mbar_wait(empty(s), (uint32_t)(((i / kWgStages) - 1) & 1), a.err)) break;
                const int64_t c0 = (blockIdx.x + i * gridDim.x) * kWgRows;
                const uint32_t st = stage_s + (uint32_t)s * kWgStageBytes;
                mbar_expect_tx(full(s), kWgStageBytes);
                for (int k = 0; k < 3; ++k) tma_load_rows(st + k * kLineBytes, &xmap, full(s), c0 - 1 + k + a.nx + a.nxy);
                tma_load_rows(st + kWgG, &gmap, full(s), c0);
                for (int k = 0; k < kWgTaps; ++k)
                    tma_load_rows(st + kWgX + k * kLineBytes, &xmap, full(s), c0 - 1 + (k % 3 - 1) * a.nx + (k / 3 - 1) * a.nxy);
            }
            // each stage's latest load is the only one that can still be in flight
            for (int64_t q = i - kWgStages < 0 ? 0 : i - kWgStages; q < i; ++q)
                mbar_drain(full((int)(q % kWgStages)), (uint32_t)((q / kWgStages) & 1));
        }
    } else if (warp == 5) {
        if (my_tiles > 0) {
            const uint32_t issue = elect_one();
            const uint64_t x0 = desc_nosw(stage_s, 128, kLineBytes / 2);  // a move of the start address adds to the low bits
            for (int64_t i = 0; i < my_tiles && mma_ok; ++i) {
                const int s = (int)(i % kWgStages);
                if (!(mma_ok = mbar_wait_warp(full(s), (uint32_t)((i / kWgStages) & 1), a.err))) break;
                fence_after();
                const uint64_t st = x0 + (uint32_t)s * (kWgStageBytes / 16);
#pragma unroll
                for (int d = 0; d < kWgAcc; ++d)
#pragma unroll
                    for (int ks = 0; ks < kWgRows / 16; ++ks)
                        mma_bf16(tmem + (uint32_t)(d * 16), st + ((d < 3 ? kWgX / 16 + d : 0) + ks * 16), st + (kWgG / 16 + ks * 16),
                                 (i > 0 || ks > 0) ? 1u : 0u, kIdescMN, issue);
                mma_commit(empty(s), issue);
            }
            mma_commit(done_s, issue);
            // every MMA issued here has completed before TMEM is read or released
            mma_commit(drain_s, issue);
            mbar_drain(drain_s, 0);
        }
    } else {
        // read-out: warp w holds accumulator rows m = 32w .. 32w+31, m = tl * 16 + ci
        const int m = warp * 32 + lane;
        const int tl = m / 16, ci = m % 16;
        float *pb = a.partials + (int64_t)blockIdx.x * 27 * a.ci_n * a.co_n;
        bool got = my_tiles > 0 && mbar_wait(done_s, 0, a.err);
        got = __all_sync(0xffffffffu, got);  // tcgen05.ld is warp-wide: the warp reads together or not at all
        if (got) fence_after();
        for (int d = 0; d < kWgAcc; ++d) {
            uint32_t v[16];
            if (got) {
                tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(d * 16), v);
            } else {
#pragma unroll
                for (int k = 0; k < 16; ++k) v[k] = 0u;  // a CTA without tiles contributes zeros
            }
            const int t = d < 3 ? 3 * tl + d : tl < 3 ? 3 * kWgTaps + tl : 27;
            if (t < 27 && ci < a.ci_n) {
#pragma unroll
                for (int co = 0; co < 16; ++co)
                    if (co < a.co_n) pb[((int64_t)t * a.ci_n + ci) * a.co_n + co] = __uint_as_float(v[co]);
            }
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 0) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(64) : "memory");
    }
}

}  // namespace tc
}  // namespace piro
