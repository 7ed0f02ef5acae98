// conv_tc.cuh -- the 3x3x3 convolution with 16 input and 16 output channels
// (the two middle layers of the learned preconditioner) as an implicit GEMM on
// the 5th-generation tensor cores: tcgen05.mma (kind::f16, BF16 operands,
// FP32 accumulation in tensor memory), operands staged by TMA.
//
// Activations are BF16 in two planes of 8 channels, [plane 2][cell][8], 16 bytes
// per cell and plane, on the ghost-inclusive grid; boundary cells hold zeros.
// A plane has act_rows(cells) rows: whole blocks of 8, and 8 more, zeros from
// the last cell on.  An output tile is 128 consecutive cells (MMA M = 128),
// N = 16 output channels, and the K loop is the 27 taps x 16 input channels:
// 27 MMAs of K = 16.
//
// Operand A of tap (dx, dy, dz) is the input at rows c0 + dx + dy*nx + dz*nx*ny
// + [0, 128).  For each (dy, dz) one "line block" of 136 rows (the tile, one row
// before it and 7 after) is loaded once; the three dx taps read it at row
// offsets 0, 1, 2.  The line block sits in shared memory in the no-swizzle
// K-major layout of the MMA -- [channel group 2][136 rows][8 channels], so an
// 8-row x 16-byte core matrix is 128 contiguous bytes, consecutive rows are 16
// bytes apart (SBO = 128 bytes per 8 rows) and the two channel groups
// LBO = 136*16 bytes apart -- and a row offset is a 16-byte move of the
// descriptor's start address.
//
// TMA writes that layout in 128-byte pieces of 8 rows from a 4-D view of the
// planes: (8 rows x 8 channels, first row 0..7 at 16 bytes, blocks of 8 rows,
// planes), box {64, 1, 17, 2} at (0, r mod 8, floor(r / 8), 0) for first row r.
// Blocks outside the planes read as zeros (TMA
// fill): before the array and after it there are at least 13 boundary cells,
// so the part of a block that lies in the array holds zeros too.
//
// The tiles are numbered along z within a column of 128 cells, the columns of
// one member after another, and a CTA takes an equal share of that sequence,
// three CTAs per SM.  Along z the 9 line blocks of tile z are the 3 of each of
// the planes z-1, z, z+1, so a tile after the first of a column (or of the
// share) loads 3 line blocks (one plane) while the others stay resident: a ring
// of 4 planes (3 in use, 1 loading).  L2 -> SM traffic is about 3 * 136/128 * 32
// bytes per output cell, against 27 * 32 for a load per tap.
//
// Bound by operand A's way from shared memory to the tensor pipe, 4 KB per MMA:
// 32 cycles each, 27 a tile, 48 us of 77 for a 128^3 layer (16128 tiles on 148
// SMs; B200).  CTAs of 16 tiles each, 2.3 per resident slot, whose MMAs one lane
// issued from a branch of its own, took 100 us: equal shares of the tiles give 95,
// and an MMA warp that runs its loops as one, so that the descriptors stay in
// uniform registers, 77.  Two CTAs per SM with 7 slots and 4 accumulators take
// 77 as well, one CTA 98, alternating the MMAs of two tiles 92.
//
// Batched grids (member b) are consecutive in the array: rows b*N .. b*N + N - 1.
//
// Warp roles (192 threads): warps 0-3 read the accumulator (TMEM lanes
// 32w..32w+31), apply GELU and store; warp 4 lane 0 issues the TMA loads;
// warp 5 issues the MMAs.  Two TMEM accumulators (2 x 16 columns)
// overlap a tile's epilogue with the next tile's MMAs (four measured slower).  mbarriers: full[slot]
// (TMA bytes landed), empty[slot] (the MMAs reading a plane completed),
// acc_full[b] (a tile's MMAs completed), acc_empty[b] (its epilogue read it).
// Every wait is bounded: on timeout the kernel raises *err and every role
// leaves its loop.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>

#include "common.cuh"

namespace piro {
namespace tc {

typedef __nv_bfloat16 bf16;

constexpr int kRows = 128;                    // output cells per tile (MMA M)
constexpr int kLineRows = kRows + 8;          // rows of a line block
constexpr int kLineBytes = kLineRows * 32;    // 4352: a multiple of 128, as TMA wants
constexpr int kSlots = 4;                     // planes resident (3 read by a tile, 1 loading)
constexpr int kPlaneBytes = 3 * kLineBytes;  // the 3 line blocks (dy = -1, 0, 1) of a plane
constexpr int kWBytes = 27 * 512;             // one layer's weights: per tap [group][co 16][8 ci] BF16
constexpr int kThreads = 192;
constexpr int kBarOff = kSlots * kPlaneBytes + kWBytes;
constexpr int kAcc = 2;                       // TMEM accumulators (16 columns each) per CTA
constexpr int kBarSlots = 2 * kSlots + 2 * kAcc + 1;  // full, empty, acc_full, acc_empty, drain
constexpr int kSmemBytes = kBarOff + kBarSlots * 8 + 16 + 128;  // + barriers, TMEM address, alignment slack
constexpr int kCtas = 3;                      // per SM
constexpr long long kSpin = 1ll << 24;        // polls before a wait gives up

// Rows of a plane of an activation array: the stride of its 8-row blocks divides it.
__host__ __device__ inline int64_t act_rows(int64_t cells) { return (cells + 7) / 8 * 8 + 8; }

struct Args {
    GridDiv g;
    int64_t N, nxy, ntiles;  // ntiles: members x columns x (nz - 2)
    int ncol;                // columns of 128 cells per member
    const bf16 *wpk;   // packed weights of this layer
    bf16 *out;         // output activations (epilogues 0, 2) or gradient (epilogue 3)
    float *zout;       // FP32 output channel 0 (epilogue 1)
    const double *rr;  // epilogue 1: output scale sqrt(rr[b] / n_int) (NULL: 1)
    double n_int;
    const int *skip;   // launch returns at once when set (may be NULL)
    int *err;          // raised on a timed-out wait
    int64_t cells, rows;  // cells of the whole array, rows of a plane of 8 channels
    bf16 *yout;        // epilogue 2: the pre-activation bf16(acc)
    const bf16 *yprev; // epilogue 3: the previous layer's pre-activation
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Programmatic dependent launch: the next kernel's blocks may come as this one's
// leave; a kernel waits for the one before it after its own set-up, before it
// reads or writes anything of the layers.  (The weights are packed two launches or
// more ahead.)  One training step's gradients, 18 launches: 485 us without, 429
// with (16 crops of 34^3, B200).
__device__ __forceinline__ void grid_launch_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Bounded wait for the phase with the given parity; false on timeout or when
// another role already gave up.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int *err)
{
    for (long long i = 0; i < kSpin; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 1023) == 1023 && *((volatile int *)err)) return false;
    }
    atomicExch(err, 1);
    return false;
}

// The same for a whole warp.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, int *err)
{
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, err));
}

// Wait for a phase that is certain to complete (copies or MMAs this CTA
// issued itself), with its own bound so that a role which gave up on a
// partner still leaves nothing in flight behind it.
__device__ __forceinline__ void mbar_drain(uint32_t bar, uint32_t parity)
{
    for (long long i = 0; i < kSpin; ++i)
        if (mbar_try_wait(bar, parity)) return;
}

// The line block of both planes whose first row is r.
__device__ __forceinline__ void tma_load_rows(uint32_t dst, const CUtensorMap *map, uint32_t bar, int64_t r)
{
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %3}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(0), "r"((int)(r & 7)), "r"((int)(r >> 3))
        : "memory");
}

// One cell's 16 channels, the planes' rows apart.
__device__ __forceinline__ void put_cell(bf16 *act, int64_t rows, int64_t c, uint4 lo, uint4 hi)
{
    *reinterpret_cast<uint4 *>(act + c * 8) = lo;
    *reinterpret_cast<uint4 *>(act + (rows + c) * 8) = hi;
}

// Shared-memory matrix descriptor, K-major, no swizzle: start address, LBO
// (between the two 8-element K groups), SBO (between 8-row groups), all in
// 16-byte units; bits 46-47 = 1 (the tcgen05 descriptor version).
__device__ __forceinline__ uint64_t desc_nosw(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | ((uint64_t)1 << 46);
}

// Instruction descriptor of kind::f16: FP32 accumulator (bits 4-5 = 1), BF16 A
// and B (bits 7-9 and 10-12 = 1), both K-major, N >> 3 at bits 17-22, M >> 4 at
// bits 24-28.
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((16u >> 3) << 17) | ((128u >> 4) << 24);

// The MMA warp runs its loops as one and the lane with `issue` set issues: the
// descriptors stay in uniform registers.  From a branch that one lane takes, an
// MMA cost its CTA about 100 cycles.
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t acc, uint32_t idesc,
                                         uint32_t issue)
{
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc), "r"(issue)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar, uint32_t issue)
{
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar), "r"(issue)
        : "memory");
}
__device__ __forceinline__ uint32_t elect_one()
{
    uint32_t e;
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(e));
    return e;
}
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// GELU in its tanh form (Hendrycks & Gimpel 2016): 0.5 x (1 + tanh(sqrt(2/pi)
// (x + 0.044715 x^3))), with the hardware tanh.approx (one instruction; the
// erf form costs several special-function operations per element and made
// this epilogue the kernel's bottleneck).
__device__ __forceinline__ float gelu_tc(float x)
{
    float t;
    const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(u));
    return 0.5f * x * (1.0f + t);
}

// GELU'(x) of the tanh form above: 0.5 (1 + t) + 0.5 x (1 - t^2) c (1 + 3 a x^2).
__device__ __forceinline__ float gelu_d_tc(float x)
{
    float t;
    const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(u));
    return 0.5f * (1.0f + t) + 0.5f * x * (1.0f - t * t) * 0.7978845608028654f * (1.0f + 0.134145f * x * x);
}

// A tile's place: member, column, plane; row: its first cell in the array.
struct Tile {
    int64_t b, row;
    int col, z;
    __device__ Tile(const Args &a, int64_t t)
    {
        const int planes = a.g.nz - 2;
        const int64_t q = t / planes;
        z = 1 + (int)(t % planes);
        b = q / a.ncol;
        col = (int)(q % a.ncol);
        row = b * a.N + z * a.nxy + (int64_t)col * kRows;
    }
    __device__ void next(const Args &a)
    {
        row += a.nxy;
        if (++z < a.g.nz - 1) return;
        z = 1;
        if (++col == a.ncol) {
            col = 0;
            ++b;
        }
        row = b * a.N + a.nxy + (int64_t)col * kRows;
    }
};

template <int kEpi>
__device__ __forceinline__ void put_zero(const Args &a, int64_t c)
{
    const uint4 z4 = make_uint4(0, 0, 0, 0);
    if (kEpi == 1) {
        a.zout[c] = 0.0f;
        return;
    }
    put_cell(a.out, a.rows, c, z4, z4);
    if (kEpi == 2) put_cell(a.yout, a.rows, c, z4, z4);
}

// kEpi 0: GELU, 16 BF16 channels out (hidden layers); 1: output channel 0 in
// FP32 times the batch member's scale (the last layer, N padded to 16);
// 2 (training forward): the pre-activation y = bf16(acc) to yout and GELU(y)
// to out; 3 (data gradient, run with the transposed, tap-reversed weights):
// out = bf16(acc * GELU'(yprev)), the gradient with respect to the previous
// layer's pre-activation.  Every epilogue writes zeros on non-interior cells.
template <int kEpi>
__global__ void __launch_bounds__(kThreads, kCtas) k_conv16_tc(const __grid_constant__ CUtensorMap xmap, Args a)
{
    if (a.skip) {
        grid_wait();
        if (*((volatile const int *)a.skip)) return;
    }
    extern __shared__ unsigned char smem_raw[];
    unsigned char *sm = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~(uintptr_t)127);
    const uint32_t planes_s = smem_u32(sm);
    const uint32_t w_s = planes_s + kSlots * kPlaneBytes;
    const uint32_t bar_s = planes_s + kBarOff;  // full[kSlots], empty[kSlots], acc_full[kAcc], acc_empty[kAcc], drain
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(sm + kBarOff + kBarSlots * 8);
    auto full = [&](int i) { return bar_s + 8u * i; };
    auto empty = [&](int i) { return bar_s + 8u * (kSlots + i); };
    auto accf = [&](int b) { return bar_s + 8u * (2 * kSlots + b); };
    auto acce = [&](int b) { return bar_s + 8u * (2 * kSlots + kAcc + b); };
    const uint32_t drain_s = bar_s + 8u * (2 * kSlots + 2 * kAcc);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // uniform, for the compiler
    const int64_t t0 = a.ntiles * blockIdx.x / gridDim.x;
    const int P = (int)(a.ntiles * (blockIdx.x + 1) / gridDim.x - t0);  // tiles of this CTA
    Tile tile(a, t0);

    // weights -> shared memory (generic proxy), then made visible to the tensor cores
    {
        const uint4 *src = reinterpret_cast<const uint4 *>(a.wpk);
        uint4 *dst = reinterpret_cast<uint4 *>(sm + kSlots * kPlaneBytes);
        for (int i = threadIdx.x; i < kWBytes / 16; i += kThreads) dst[i] = src[i];
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < kSlots; ++i) {
            mbar_init(full(i), 1);
            mbar_init(empty(i), 1);
        }
        for (int b = 0; b < kAcc; ++b) {
            mbar_init(accf(b), 1);
            mbar_init(acce(b), 4);
        }
        mbar_init(drain_s, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kAcc * 16)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t *>(tmem_slot), 0);

    grid_launch_next();
    grid_wait();
    if (P > 0) {
        if (warp == 4) {
            if (lane == 0) {
                // producer: a tile's new planes, three line blocks each
                int p = 0;  // planes loaded
                bool ok = true;
                for (int j = 0; j < P && ok; ++j, tile.next(a)) {
                    for (int k = j == 0 || tile.z == 1 ? 0 : 2; k < 3; ++k, ++p) {
                        const int slot = p % kSlots;
                        if (p >= kSlots && !(ok = mbar_wait(empty(slot), ((p / kSlots) - 1) & 1, a.err))) break;
                        mbar_expect_tx(full(slot), 3 * kLineBytes);
                        for (int dy = 0; dy < 3; ++dy)
                            tma_load_rows(planes_s + slot * kPlaneBytes + dy * kLineBytes, &xmap, full(slot),
                                          tile.row + (int64_t)(k - 1) * a.nxy - 1 + (int64_t)(dy - 1) * a.g.nx);
                    }
                }
                // no copy may land after the CTA has left, whatever the other
                // roles did: wait for each slot's latest load
                for (int q = p - kSlots < 0 ? 0 : p - kSlots; q < p; ++q) mbar_drain(full(q % kSlots), (q / kSlots) & 1);
            }
        } else if (warp == 5) {
            {
                const uint32_t issue = elect_one();
                // a move of the start address is an addition to the descriptor's low bits
                const uint64_t a0 = desc_nosw(planes_s, kLineRows * 16, 128), b0 = desc_nosw(w_s, 256, 128);
                int waited = 0, p = 0;  // p: the tile's first plane, in the order of loading
                bool ok = true;
                for (int j = 0; j < P && ok; ++j) {
                    while (ok && waited < p + 3) {
                        ok = mbar_wait_warp(full(waited % kSlots), (waited / kSlots) & 1, a.err);
                        ++waited;
                    }
                    const int buf = j % kAcc;
                    if (ok && j >= kAcc) ok = mbar_wait_warp(acce(buf), ((j / kAcc) - 1) & 1, a.err);
                    if (!ok) break;
                    fence_after();
                    const uint32_t d_tmem = tmem + (uint32_t)(buf * 16);
#pragma unroll
                    for (int dz = 0; dz < 3; ++dz) {
                        const uint64_t ab = a0 + (uint32_t)((p + dz) % kSlots) * (kPlaneBytes / 16);
#pragma unroll
                        for (int dy = 0; dy < 3; ++dy)
#pragma unroll
                            for (int dx = 0; dx < 3; ++dx) {
                                const int tap = dz * 9 + dy * 3 + dx;
                                mma_bf16(d_tmem, ab + (dy * kLineBytes / 16 + dx), b0 + tap * 32, tap > 0 ? 1u : 0u, kIdesc, issue);
                            }
                    }
                    mma_commit(accf(buf), issue);
                    // plane z-1 is read by no later tile; at the end of a column no plane is
                    tile.next(a);
                    mma_commit(empty(p++ % kSlots), issue);
                    if (tile.z == 1) {
                        mma_commit(empty(p++ % kSlots), issue);
                        mma_commit(empty(p++ % kSlots), issue);
                    }
                }
                // every MMA issued here has completed before TMEM is released
                mma_commit(drain_s, issue);
                mbar_drain(drain_s, 0);
            }
        } else {
            // epilogue: warp w holds tile rows 32w .. 32w+31
            float sc = 1.0f;
            int64_t sc_of = -1;  // the member whose scale that is
            for (int j = 0; j < P; ++j, tile.next(a)) {
                const int buf = j % kAcc;
                if (!mbar_wait(accf(buf), (j / kAcc) & 1, a.err)) break;
                fence_after();
                uint32_t v[16];
                tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(buf * 16), v);
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(acce(buf));
                const int64_t inplane = (int64_t)tile.col * kRows + warp * 32 + lane, boff = tile.b * a.N;
                const int64_t c = (int64_t)tile.z * a.nxy + inplane;
                // the boundary planes z = 0 and nz - 1 of a column hold zeros in every
                // output (no tile computes them; a buffer reused for another grid must
                // not keep values there), and so do the rows after the last cell (the
                // next layer's loads read them)
                if (inplane < a.nxy) {
                    if (tile.z == 1) put_zero<kEpi>(a, boff + inplane);
                    if (tile.z == a.g.nz - 2) put_zero<kEpi>(a, boff + c + a.nxy);
                }
                if (kEpi != 1 && t0 + j == a.ntiles - 1 && warp == 0 && a.cells + lane < a.rows)
                    put_cell(a.out, a.rows, a.cells + lane, make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0));
                if (kEpi == 1) {
                    if (c < a.N) {
                        if (a.rr && tile.b != sc_of) {  // an FP64 division and root: once per member
                            sc = (float)sqrt(a.rr[tile.b] / a.n_int);
                            sc_of = tile.b;
                        }
                        a.zout[boff + c] = a.g.interior(c) ? __uint_as_float(v[0]) * sc : 0.0f;
                    }
                } else if (kEpi == 3) {
                    if (c < a.N) {
                        uint32_t w[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                        if (a.g.interior(c)) {
                            const uint4 u0 = *reinterpret_cast<const uint4 *>(a.yprev + (boff + c) * 8);
                            const uint4 u1 = *reinterpret_cast<const uint4 *>(a.yprev + (a.rows + boff + c) * 8);
                            const uint32_t yw[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
#pragma unroll
                            for (int k = 0; k < 8; ++k) {
                                const float2 y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&yw[k]));
                                const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(v[2 * k]) * gelu_d_tc(y.x),
                                                                               __uint_as_float(v[2 * k + 1]) * gelu_d_tc(y.y));
                                w[k] = *reinterpret_cast<const uint32_t *>(&h);
                            }
                        }
                        put_cell(a.out, a.rows, boff + c, make_uint4(w[0], w[1], w[2], w[3]), make_uint4(w[4], w[5], w[6], w[7]));
                    }
                } else if (c < a.N) {
                    uint32_t w[8] = {0, 0, 0, 0, 0, 0, 0, 0}, yw[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                    if (a.g.interior(c)) {
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            const float y0 = __bfloat162float(__float2bfloat16_rn(__uint_as_float(v[2 * k])));
                            const float y1 = __bfloat162float(__float2bfloat16_rn(__uint_as_float(v[2 * k + 1])));
                            const __nv_bfloat162 h = __floats2bfloat162_rn(gelu_tc(y0), gelu_tc(y1));
                            w[k] = *reinterpret_cast<const uint32_t *>(&h);
                            if (kEpi == 2) {
                                const __nv_bfloat162 hy = __floats2bfloat162_rn(y0, y1);
                                yw[k] = *reinterpret_cast<const uint32_t *>(&hy);
                            }
                        }
                    }
                    put_cell(a.out, a.rows, boff + c, make_uint4(w[0], w[1], w[2], w[3]), make_uint4(w[4], w[5], w[6], w[7]));
                    if (kEpi == 2)
                        put_cell(a.yout, a.rows, boff + c, make_uint4(yw[0], yw[1], yw[2], yw[3]),
                                 make_uint4(yw[4], yw[5], yw[6], yw[7]));
                }
            }
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 0) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kAcc * 16) : "memory");
    }
}

}  // namespace tc
}  // namespace piro
