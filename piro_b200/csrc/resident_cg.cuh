// resident_cg.cuh -- backward-Euler solve of one 7-point problem by a team of
// CTAs that keep the whole Krylov state on chip.
//
// The method is the one of be_solver.cu and batched.cu: FP64 iterative
// refinement around FP32 Jacobi-PCG on the symmetric form of A = I -
// dt*diag(alpha)*L.  A team of `size` CTAs, one per SM, splits the interior
// x-lines (y, z) among them; a CTA holds its lines' vectors in shared memory
// and registers (at most kRcGroups groups of four cells).  Only z crosses
// CTAs, at the lines on a run's rim, through an exchange buffer in global
// memory that stays in L2.
//
// The symmetric form.  With s = r / alpha, S = diag(alpha)^-1 A_II has the
// diagonal D = A_rr / alpha and one constant off-diagonal -dt*vnb: the
// operator is D z + off * (sum of six neighbours), every dot product is
// unweighted, and no coefficient is formed in the loop.  alpha itself is only
// needed for |r|^2 of the inner stop test.
//
// CG with one all-reduce per iteration (Chronopoulos & Gear 1989), its
// vectors updated in one pass; r is not stored (s = z D):
//   H  the rim's neighbours received into shared memory
//   S  w = S z, kept in registers; all-reduce of <s, z>, <z, w>, |alpha s|^2
//   U  beta = <s, z> / <s, z>_old, <p, S p> = <z, w> - beta^2 <p, S p>_old,
//      a = <s, z> / <p, S p>; p = z + beta p, q = w + beta q, d += a p,
//      s = z D - a q, z = s / D; z of the run's rim sent
// Against the two all-reduces of the usual form one L2 round trip less is
// exposed, and the vectors pass through shared memory once, not twice.
//
// The sums' terms.  Where the launch with grid barriers takes the operator's and
// the update's dot products in groups of four cells (nx, and nx ny nz, a multiple
// of 4) their terms are FP32 products, four added in FP32; elsewhere each is an
// FP64 product (wide_s, wide_u), so that fields of 1e-25 or 1e20, whose FP32
// products vanish or overflow, are solved there.  <p, S p> by the recurrence below
// differs from the sum over the cells by what CG's orthogonality has lost.
//
// Lines are ordered in strips of h planes (y within a strip, z within h
// fastest), so that a run of consecutive lines is about square in (y, z) and
// most of its neighbours are its own.  A table gives for every line where its
// four neighbour lines sit in shared memory: in the run, in the halo, or the
// line of zeros (the boundary), so that S has no cases.  The rim's z travels
// as 16-byte words of two values and the round number, written by one 128-bit
// store: the reader polls the word it needs itself, and neither side waits
// for a fence (with a flag per CTA behind a fence, the fence alone took 1600
// cycles of an iteration with 148 CTAs at work).
//
// The loop's code is kept small (every loop but those over a thread's groups
// is rolled): with 140 to 220 KB of code per kernel the instruction cache
// missed in every phase, and phases without any memory access took several
// times their time.
//
// All-reduce: every CTA stores each partial with the round's number in one
// 16-byte word (a single 128-bit access, so value and tag arrive together) in
// a 128-byte line of its own, and every CTA polls the lines of all ranks, a
// lane per word, and adds them in rank order: one trip through L2 after the
// last arrival, no counter and no fence, the same sum in every CTA and on every
// run.  B200, cycles per all-reduce of 148 CTAs: 2450 (8 CTAs: 1300); several
// words in one line 5600; ranks packed in shared lines 5400 to 6500, the polls
// holding up the stores; a counter and a read of the partials 3450; a leader
// that sums and publishes the total 3100; a __nanosleep between polls adds
// 2400.  Rounds are numbered on from launch
// to launch, so that nothing has to be cleared.  Waits are bounded: on
// time-out the error flag is raised and every CTA leaves.
#pragma once

#include <algorithm>

#include "common.cuh"

namespace piro {

constexpr int kRcThreads = 512;
constexpr int kRcK = 7;                            // groups of 4 cells per thread, at most
constexpr int kRcGroups = kRcThreads * kRcK;       // and per CTA
// The words of a rank, each in a line of its own: the residual's four sums,
// the iteration's three (twice, alternating), x published.
enum : int { kRcWordR = 0, kRcWordSums = 4, kRcWordX = 10, kRcWords = 11 };
constexpr int kRcMaxTeam = 160;                    // ranks of a team (five polling warps)
constexpr size_t kRcSmemMax = 226 * 1024;          // dynamic shared memory of a CTA
constexpr int kRcRegK = 3;                         // up to so many groups per thread keep q and d in registers

struct RcSlot {
    double v;
    unsigned long long tag;
    double pad[14];
};
static_assert(sizeof(RcSlot) == 128, "a slot is a line");

// One problem.  Cells are indexed as everywhere (x + y nx + z nx ny, ghost-
// inclusive); zx and ax hold the interior lines, y fastest, each padded to
// whole groups.
struct RcProblem {
    int nx, ny, nz;
    int gx;          // groups per line
    int lines;       // interior lines (ny - 2)(nz - 2)
    int h, hlast, strips;            // planes of a strip, of the last one, strips
    FastDiv fgx, fst, fh, fhl, fly;  // by gx, (ny - 2) h, h, hlast, ny
    int groups, halo;                // of the CTA with the most: groups of its run, neighbour lines in other runs
    const float *alpha;     // per cell, or NULL: constant
    float alpha0;
    float mdt, vself, vnb;  // A = I + mdt * diag(alpha) * (vself, vnb)
    double cd64, co64;      // constant alpha: the FP64 operator of the residual
    const float *b;
    float *xout;
    double *x64;
    double *beff;  // b_I - A_IB b_B on the interior cells next to the boundary (not for constant alpha)
    uint4 *zx;              // two words per group: z.x, z.y (z.z, z.w), round, 0
    float4 *ax;             // alpha, where it does not fit beside the vectors (rc_stream_alpha)
    const int32_t *ib_ptr, *ib_col;  // interior-boundary entries of A (constant alpha: the stencil value)
    const float *ib_val;
    double rtol, inner_floor;
    int max_outer, max_inner;
    int wide_s, wide_u;  // FP64 terms in S and in U (read by the kWide instances alone)
};

struct RcTeam {
    RcSlot *slots;  // [kRcWords][size]
    unsigned long long *epoch;  // the last round used; slots, zx and epoch are zero at first and after a failed launch
    int rank, size;
    int *err;       // raised by the first wait that runs out
    long long spin_limit;
};

struct RcResult {
    int status, outer, inner;
    double rel;
    bool ok;  // false: a wait ran out
};

// A flexible CG iteration to go on with (kResume): its residual, last direction
// and that direction's A p, the correction so far (read and left), all on the
// grid; <p, S p>, the iterations so far (0: no direction yet) and the bounds.
struct RcResume {
    const float *r, *p, *q;
    float *d;
    double tol2, rr0, pq;
    int iters;
};

struct RcShared {
    double red[4 * 16];
    double tot[kRcMaxTeam / 32][4];  // per polling warp
    double out[4];
    int halo;      // neighbour lines in other runs
    int ok, ok_z;  // of the last all-reduce, and of the last wait for the neighbours' z
};

// The geometry of an nx*ny*nz grid solved by `size` CTAs: a strip is as high
// as the side of a square of one CTA's lines (the whole grid for one CTA).
inline RcProblem rc_geometry(int nx, int ny, int nz, int size)
{
    RcProblem P{};
    const int nyi = ny - 2, nzi = nz - 2;
    P.nx = nx;
    P.ny = ny;
    P.nz = nz;
    P.gx = (nx - 2 + 3) / 4;
    P.lines = nyi * nzi;
    P.h = nzi;
    if (size > 1) {
        int h = 1;
#pragma unroll 1
        while ((int64_t)(h + 1) * h * size <= P.lines) ++h;  // h (h + 1) <= lines per CTA: h near its root
        P.h = std::min(h, nzi);
    }
    P.strips = (nzi + P.h - 1) / P.h;
    P.hlast = nzi - (P.strips - 1) * P.h;
    P.fgx = FastDiv((uint32_t)P.gx);
    P.fst = FastDiv((uint32_t)(nyi * P.h));
    P.fh = FastDiv((uint32_t)P.h);
    P.fhl = FastDiv((uint32_t)P.hlast);
    P.fly = FastDiv((uint32_t)ny);
    // the largest run, and (a walk over the lines) the most neighbour lines outside a
    // run, which a grid too large for the chip needs no count of
    P.groups = (int)(cdiv(P.lines, size) * P.gx);
    P.halo = 0;
    if (size > 1 && P.groups <= kRcGroups) {
        int l = 0;
        for (int r = 0, st = 0, y = 0, zz = 0; r < size; ++r) {
            const int l0 = l, l1 = (int)((int64_t)P.lines * (r + 1) / size);
            int n = 0;
            for (; l < l1; ++l) {
                const int hs = st == P.strips - 1 ? P.hlast : P.h;
                n += (y > 0 && l - hs < l0) + (y < nyi - 1 && l + hs >= l1);
                n += zz > 0 ? l == l0 : st > 0;
                n += zz < hs - 1 ? l == l1 - 1 : st < P.strips - 1;
                if (++zz == hs) {
                    zz = 0;
                    if (++y == nyi) {
                        y = 0;
                        ++st;
                    }
                }
            }
            P.halo = std::max(P.halo, n);
        }
    }
    return P;
}

// Bytes of dynamic shared memory of rc_solve: z with the halo and a line of
// zeros, q and d (d alone, as a staging area, when both are in registers),
// alpha, and the tables of the lines.
inline size_t rc_smem(const RcProblem &P, bool constant, bool stream_alpha)
{
    const bool reg = cdiv(P.groups, kRcThreads) <= kRcRegK;
    const size_t vecs = 1 + (reg ? 1 : 2) + (constant || stream_alpha ? 0 : 1);
    const size_t nl = (size_t)P.groups / P.gx;
    return 16 * (vecs * P.groups + ((size_t)P.halo + 1) * P.gx) + 12 * nl + 4 * (size_t)P.halo + 64;
}

// Whether `size` CTAs hold the problem, and whether alpha has to be streamed.
inline bool rc_fits(const RcProblem &P, bool constant, bool &stream_alpha)
{
    stream_alpha = false;
    if (P.groups > kRcGroups) return false;
    if (rc_smem(P, constant, false) <= kRcSmemMax) return true;
    if (constant || P.groups <= kRcThreads * kRcRegK) return false;
    stream_alpha = true;
    return rc_smem(P, constant, true) <= kRcSmemMax;
}

inline size_t rc_slot_bytes(int size) { return sizeof(RcSlot) * kRcWords * size; }

inline size_t rc_exchange_bytes(int nx, int ny, int nz)
{
    return (size_t)(ny - 2) * (nz - 2) * ((nx - 2 + 3) / 4) * 2 * sizeof(uint4);
}

// By an exchange, which goes to L2 at once: a plain store lingered in the SM
// for about 1000 cycles (16 CTAs, an iteration of 33^3 cells: 10000 cycles with
// stores, 7300 with exchanges).
__device__ __forceinline__ void rc_put(RcSlot *p, double v, unsigned long long tag)
{
    asm volatile("{\n .reg .b128 t, o;\n mov.b128 t, {%1, %2};\n atom.relaxed.gpu.global.exch.b128 o, [%0], t;\n}" ::"l"(p),
                 "l"(__double_as_longlong(v)), "l"(tag)
                 : "memory");
}

__device__ __forceinline__ void rc_fence() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// Two values of z and their round, and back.
__device__ __forceinline__ void rc_send(uint4 *p, float a, float b, unsigned round)
{
    asm volatile("{\n .reg .b128 t;\n .reg .b64 lo, hi;\n mov.b64 lo, {%1, %2};\n mov.b64 hi, {%3, %4};\n"
                 " mov.b128 t, {lo, hi};\n st.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(p),
                 "r"(__float_as_uint(a)), "r"(__float_as_uint(b)), "r"(round), "r"(0)
                 : "memory");
}

__device__ __forceinline__ unsigned rc_recv(const uint4 *p, float &a, float &b)
{
    unsigned x, y, t, u;
    asm volatile("{\n .reg .b128 t;\n .reg .b64 lo, hi;\n ld.relaxed.gpu.global.b128 t, [%4];\n"
                 " mov.b128 {lo, hi}, t;\n mov.b64 {%0, %1}, lo;\n mov.b64 {%2, %3}, hi;\n}"
                 : "=r"(x), "=r"(y), "=r"(t), "=r"(u)
                 : "l"(p)
                 : "memory");
    a = __uint_as_float(x);
    b = __uint_as_float(y);
    return t;
}

__device__ __forceinline__ unsigned long long rc_get(const RcSlot *p, double &v)
{
    long long a;
    unsigned long long tag;
    asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
                 : "=l"(a), "=l"(tag)
                 : "l"(p)
                 : "memory");
    v = __longlong_as_double(a);
    return tag;
}

// The team's sums of n <= 4 values, round `tag`, words first..; left in sh.out
// for every thread.  Warp t adds the 16 warps' parts of value t and stores it;
// then a warp per value and 32 ranks waits for the ranks' words.  kSync: the
// CTAs' global writes before are visible to all of them afterwards.  False if
// a wait ran out (sh.ok is 1 on entry).  One copy of the code serves every
// sum: what a launch executes has to come through the instruction cache, and
// with 60 KB more of it a solve took 100 us longer.
static __device__ __noinline__ bool rc_allreduce(const RcTeam &T, RcShared &sh, int first, int n, unsigned long long tag,
                                                 double v0, double v1, double v2, double v3, bool sync)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (T.size + 31) >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v0 += __shfl_xor_sync(0xffffffffu, v0, o);
        v1 += __shfl_xor_sync(0xffffffffu, v1, o);
        v2 += __shfl_xor_sync(0xffffffffu, v2, o);
        v3 += __shfl_xor_sync(0xffffffffu, v3, o);
    }
    if (lane == 0) {
        sh.red[w] = v0;
        sh.red[16 + w] = v1;
        sh.red[32 + w] = v2;
        sh.red[48 + w] = v3;
    }
    __syncthreads();
    if (w < n) {
        if (sync) rc_fence();
        double s = (lane & 15) < kRcThreads / 32 ? sh.red[w * 16 + (lane & 15)] : 0.0;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) {
            if (T.size > 1) rc_put(T.slots + (first + w) * T.size + T.rank, s, tag);
            else sh.out[w] = s;
        }
        __syncwarp();  // the store before this warp's polls, not behind its lanes' spinning
    }
    if (T.size > 1) {
#pragma unroll 1
        for (int job = w; job < n * nw; job += kRcThreads / 32) {
            const int t = job / nw, j = job - t * nw, r = 32 * j + lane;
            double v = 0.0;
            if (r < T.size) {
                const RcSlot *p = T.slots + (first + t) * T.size + r;
                long long spins = 0;
#pragma unroll 1
                while (rc_get(p, v) != tag) {
                    if (++spins > T.spin_limit || ((spins & 63) == 0 && *((volatile int *)T.err))) {
                        atomicExch(T.err, 1);
                        sh.ok = 0;
                        break;
                    }
                }
            }
            __syncwarp();
            v = warp_sum(v);
            if (lane == 0) sh.tot[j][t] = v;
        }
        if (sync) rc_fence();
        __syncthreads();
        if (w == 0 && lane < n) {
            double a[kRcMaxTeam / 32];
#pragma unroll
            for (int j = 0; j < kRcMaxTeam / 32; ++j) a[j] = j < nw ? sh.tot[j][lane] : 0.0;
            sh.out[lane] = ((a[0] + a[1]) + (a[2] + a[3])) + a[4];
        }
    }
    __syncthreads();
    return sh.ok != 0;
}

// A vector of this thread's groups: in registers, or in shared memory at the
// group's index.
template <bool kReg, int kK>
struct RcVec {
    float4 r[kReg ? kK : 1];
    float4 *s;
    __device__ __forceinline__ float4 get(int k, int v) const { return kReg ? r[kReg ? k : 0] : s[v]; }
    __device__ __forceinline__ void put(int k, int v, float4 x)
    {
        if (kReg) r[kReg ? k : 0] = x;
        else s[v] = x;
    }
};

// The sum of a group's four products, each in FP64 (wide) or all in FP32.
template <bool kWide>
__device__ __forceinline__ double rc_dot(const float4 &a, const float4 &b, bool wide)
{
    if (kWide && wide)
        return ((double)a.x * (double)b.x + (double)a.y * (double)b.y) + ((double)a.z * (double)b.z + (double)a.w * (double)b.w);
    return (double)((a.x * b.x + a.y * b.y) + (a.z * b.z + a.w * b.w));
}

// Solve A x = b for one problem on this CTA's team.  Every CTA of the team
// runs it with the same arguments and takes the same branches.  kConst:
// constant alpha (the batched members: boundary neighbours enter the residual
// with their own value and the stencil's coefficient); else alpha per cell,
// and the interior-boundary block of A from ib_*.  kK: groups per thread
// (with at most kRcRegK, q and d fit in registers beside D, w and p).
// kStreamA: alpha is read from ax in every iteration.  kWide: the sums' terms as
// P.wide_s and P.wide_u say, else FP32 products (an instance of its own: the other
// widths keep their registers).  Prob: the problem by
// value (a kernel's parameter) or by reference (in shared memory).
// kResume: no refinement sweeps, but the iterations that follow U's up to its
// tolerance, from the state U on.  Its first direction is conjugate to U's p, and
// its residual orthogonal to p, as a CG iteration leaves them; from then on they are
// CG iterations.  R.inner counts U's iterations too, R.rel is |r|^2.
template <bool kConst, int kK, bool kStreamA, bool kWide, class Prob, bool kResume = false>
__device__ __forceinline__ void rc_solve(Prob P, const RcTeam T, RcShared &sh, float4 *smem, RcResult &R,
                                         const RcResume U = RcResume())
{
    constexpr bool kReg = kK <= kRcRegK;
    const int tid = threadIdx.x, lane = tid & 31;
    const int nxi = P.nx - 2, nyi = P.ny - 2, nzi = P.nz - 2, gx = P.gx, h = P.h;
    const int l0 = (int)((int64_t)P.lines * T.rank / T.size), l1 = (int)((int64_t)P.lines * (T.rank + 1) / T.size);
    const int nl = l1 - l0, ng = nl * gx;
    const int nx = P.nx, sxy = P.nx * P.ny;
    const float off = P.mdt * P.vnb;
    const int lx = nxi - 4 * (gx - 1);  // cells of a line's last group
    // shared memory: z [groups | halo | zeros], d, q, alpha, tables
    float4 *__restrict__ sz = smem;
    const int zero_line = P.groups + P.halo * gx;
    RcVec<kReg, kK> q, d;
    float4 *next = smem + zero_line + gx;
    d.s = next;
    next += P.groups;
    q.s = next;
    if (!kReg) next += P.groups;
    float4 *__restrict__ sa = next;
    if (!kConst && !kStreamA) next += P.groups;
    uint2 *nbr = reinterpret_cast<uint2 *>(next);                       // per line: groups of its y-, y+, z-, z+ lines
    int *nat = reinterpret_cast<int *>(nbr + P.groups / gx);            // per line: z nyi + y, top bit: others read it
    int *hsrc = nat + P.groups / gx;                                    // per halo line: its z nyi + y
    float *szf = reinterpret_cast<float *>(sz), *sdf = reinterpret_cast<float *>(d.s);

    // y and z of line l
    auto place = [&](int l, int &hs, int &y, int &z) {
        const int st = (int)P.fst.div((uint32_t)l), rem = l - st * nyi * h;
        const bool last = st == P.strips - 1;
        hs = last ? P.hlast : h;
        y = (int)(last ? P.fhl.div((uint32_t)rem) : P.fh.div((uint32_t)rem));
        z = st * h + rem - y * hs;
    };
    // cell c of this run (x fastest over padded lines): its x, y, z; past a
    // line's end or the run's, false, with the coordinates of another cell, so
    // that loads need no branch
    auto where = [&](int c, int &x, int &y, int &z) {
        const int ll = min((int)P.fgx.div((uint32_t)(c >> 2)), nl - 1);
        x = c - ll * 4 * gx;
        const bool in = x < nxi;
        x = min(x, nxi - 1);
        int hs;
        place(l0 + ll, hs, y, z);
        return in;
    };
    auto cell = [&](int x, int y, int z) { return (int64_t)(z + 1) * sxy + (int64_t)(y + 1) * nx + 1 + x; };

    if (tid == 0) {
        sh.ok = sh.ok_z = 1;
        sh.halo = 0;
    }
    // boundary cells: x = b; x64 = 0, or b for constant alpha (its residual reads them)
    if (!kResume) {
        const int total = P.ny * P.nz, w = tid >> 5, nw = kRcThreads / 32;
#pragma unroll 1
        for (int ln = T.rank * nw + w; ln < total; ln += T.size * nw) {
            const int z = (int)P.fly.div((uint32_t)ln), y = ln - z * P.ny;
            const int64_t i0 = (int64_t)ln * nx;
            const bool whole = y == 0 || y == P.ny - 1 || z == 0 || z == P.nz - 1;
            const int step = whole ? 1 : nx - 1;
#pragma unroll 1
            for (int x = lane * step; x < nx; x += 32 * step) {
                const float v = P.b[i0 + x];
                P.xout[i0 + x] = v;
                P.x64[i0 + x] = kConst ? (double)v : 0.0;
            }
        }
    }
    __syncthreads();
    // the tables
#pragma unroll 1
    for (int ll = tid; ll < nl; ll += kRcThreads) {
        int hs, y, z;
        place(l0 + ll, hs, y, z);
        const int zz = z - (int)P.fh.div((uint32_t)z) * h;
        bool rim = false;
        // the neighbour line dl lines away in its strip, or at natural index src in another run
        auto at = [&](bool in, bool same, int dl, int src) -> unsigned {
            if (!in) return (unsigned)zero_line;
            if (same && ll + dl >= 0 && ll + dl < nl) return (unsigned)((ll + dl) * gx);
            rim = true;
            const int slot = atomicAdd(&sh.halo, 1);
            hsrc[slot] = src;
            return (unsigned)(P.groups + slot * gx);
        };
        const int me = z * nyi + y;
        const unsigned ym = at(y > 0, true, -hs, me - 1), yp = at(y < nyi - 1, true, hs, me + 1);
        const unsigned zm = at(z > 0, zz > 0, -1, me - nyi), zp = at(z < nzi - 1, zz < hs - 1, 1, me + nyi);
        nbr[ll] = make_uint2(ym | yp << 16, zm | zp << 16);
        nat[ll] = rim ? me | (int)0x80000000 : me;
    }
    if (tid < gx) sz[zero_line + tid] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int g = tid + kRcThreads; g < gx; g += kRcThreads) sz[zero_line + g] = make_float4(0.f, 0.f, 0.f, 0.f);
    float D0 = 0.0f;
    if (kConst) D0 = __fadd_rn(1.0f, __fmul_rn(P.mdt, __fmul_rn(P.alpha0, P.vself))) / P.alpha0;
    // alpha of this run (1 past a line's end), and D = A_rr / alpha by way of d's memory
    // (batches of kB cells, their loads in flight together)
    constexpr int kB = 4;
    if (!kConst)
#pragma unroll 1
        for (int c0 = tid; c0 < 4 * ng; c0 += kB * kRcThreads) {
            float a[kB];
            int at[kB];
            bool in[kB];
#pragma unroll
            for (int j = 0; j < kB; ++j) {
                int x, y, z;
                in[j] = where(c0 + j * kRcThreads, x, y, z);
                at[j] = z * nyi + y;
                a[j] = __ldg(P.alpha + cell(x, y, z));
            }
#pragma unroll
            for (int j = 0; j < kB; ++j) {
                const int c = c0 + j * kRcThreads;
                if (c >= 4 * ng) break;
                const float v = in[j] ? a[j] : 1.0f;
                if (kStreamA) reinterpret_cast<float *>(P.ax)[(int64_t)4 * gx * at[j] + c % (4 * gx)] = v;
                else reinterpret_cast<float *>(sa)[c] = v;
                sdf[c] = __fadd_rn(1.0f, __fmul_rn(P.mdt, __fmul_rn(v, P.vself))) / v;
            }
        }
    __syncthreads();
    // beff: the two ends of every line, then the lines next to a face
    if (!kConst && !kResume) {
        auto fold = [&](int64_t i) {
            double be = (double)__ldg(P.b + i);
#pragma unroll 1
            for (int32_t e = P.ib_ptr[i]; e < P.ib_ptr[i + 1]; ++e)
                be -= (double)P.ib_val[e] * (double)__ldg(P.b + P.ib_col[e]);
            P.beff[i] = be;
        };
        const int ends = 2 * nl;
#pragma unroll 1
        for (int t = tid; t < ends + 4 * ng; t += kRcThreads) {
            const bool end = t < ends;
            int x, y, z;
            const bool here = where(end ? (t >> 1) * 4 * gx : t - ends, x, y, z);
            if (end) x = t & 1 ? nxi - 1 : 0;
            if (end || (here && x > 0 && x < nxi - 1 && (y == 0 || y == nyi - 1 || z == 0 || z == nzi - 1)))
                fold(cell(x, y, z));
        }
        __syncthreads();
    }
    float4 D[kK], p[kK], w[kK];
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < kK; ++k) {
        const int v = tid + k * kRcThreads;
        p[k] = w[k] = zero;
        if (v < ng) {
            if (!kConst) D[k] = d.s[v];
            q.put(k, v, zero);
            d.put(k, v, zero);
        }
    }
    if (kResume) {  // U's p, q / alpha (by way of z's memory) and d
        auto stage = [&](float *to, const float *from, bool over_alpha) {
            __syncthreads();
#pragma unroll 1
            for (int c = tid; c < 4 * ng; c += kRcThreads) {
                int x, y, z;
                const bool in = where(c, x, y, z);
                const float v = from[cell(x, y, z)], a = __ldg(P.alpha + cell(x, y, z));
                to[c] = in ? over_alpha ? v / a : v : 0.0f;
            }
            __syncthreads();
        };
        if (U.iters > 0) {
            stage(szf, U.p, false);
#pragma unroll
            for (int k = 0; k < kK; ++k)
                if (tid + k * kRcThreads < ng) p[k] = sz[tid + k * kRcThreads];
            stage(szf, U.q, true);
#pragma unroll
            for (int k = 0; k < kK; ++k)
                if (tid + k * kRcThreads < ng) q.put(k, tid + k * kRcThreads, sz[tid + k * kRcThreads]);
        }
        stage(sdf, U.d, false);
        if (kReg)
#pragma unroll
            for (int k = 0; k < kK; ++k)
                if (tid + k * kRcThreads < ng) d.put(k, 0, d.s[tid + k * kRcThreads]);
    }
    unsigned long long tag = T.size > 1 ? *((volatile unsigned long long *)T.epoch) : 0;
    unsigned round = (unsigned)tag, flip = 0;  // round: of z, never ahead of tag
    R.status = PIRO_ERR_NOT_CONVERGED;
    R.outer = 0;
    R.inner = 0;
    R.rel = INFINITY;
    R.ok = true;
    double prev_rel = INFINITY;
    bool corrected = false;  // x64 holds a sweep's result
    auto send = [&](int v, int ll, const float4 &z4) {
        const int n = nat[ll];
        if (n < 0) {
            uint4 *at = P.zx + 2 * ((int64_t)(n & 0x7fffffff) * gx + v - ll * gx);
            rc_send(at, z4.x, z4.y, round);
            rc_send(at + 1, z4.z, z4.w, round);
        }
    };
#pragma unroll 1
    for (int sweep = 0;; ++sweep) {
        // R: r = b - A x in FP64, z = s / D, a cell per thread (coalesced).
        // Sweep 0 has x = b, read from b itself.
        double rs[4] = {0.0, 0.0, 0.0, 0.0};
        if (kResume) {  // U's r; <s, z> and <z, S p> of its direction
#pragma unroll 1
            for (int c = tid; c < 4 * ng; c += kRcThreads) {
                int x, y, z;
                const bool here = where(c, x, y, z);
                const int64_t i = cell(x, y, z);
                const float a = __ldg(P.alpha + i), rf = U.r[i], qf = U.iters > 0 ? U.q[i] : 0.0f;
                const float c32 = __fadd_rn(1.0f, __fmul_rn(P.mdt, __fmul_rn(a, P.vself)));
                const float zz = here ? rf * rcp_approx(c32) : 0.0f;
                if (here) {
                    rs[2] += (double)rf / (double)a * (double)zz;
                    rs[1] += (double)zz * (double)qf / (double)a;
                }
                szf[c] = zz;
            }
        } else
#pragma unroll 1
        for (int c = tid; c < 4 * ng; c += kRcThreads) {
            int x, y, z;
            const bool here = where(c, x, y, z);
            const int64_t i = cell(x, y, z);
            const int64_t at[7] = {i, i - 1, i + 1, i - nx, i + nx, i - sxy, i + sxy};
            const bool in[7] = {true, x > 0, x < nxi - 1, y > 0, y < nyi - 1, z > 0, z < nzi - 1};
            const bool rim = !(in[1] && in[2] && in[3] && in[4] && in[5] && in[6]);
            const float bf = __ldg(P.b + i), a = kConst ? P.alpha0 : __ldg(P.alpha + i);
            double xv[7], fold = 0.0;
            if (!kConst && rim) fold = P.beff[i];
            // boundary neighbours: their own value for constant alpha, else folded in by beff
            if (sweep == 0) {
                float bn[7];
#pragma unroll
                for (int t = 0; t < 7; ++t) bn[t] = __ldg(P.b + at[t]);
#pragma unroll
                for (int t = 0; t < 7; ++t) xv[t] = kConst || in[t] ? (double)bn[t] : 0.0;
            } else {
#pragma unroll
                for (int t = 0; t < 7; ++t) xv[t] = P.x64[at[t]];
            }
            const double bi = (double)bf, be = !kConst && rim ? fold : bi;
            const double nb = (xv[1] + xv[2]) + (xv[3] + xv[4]) + (xv[5] + xv[6]);
            const float c32 = __fadd_rn(1.0f, __fmul_rn(P.mdt, __fmul_rn(a, P.vself)));
            const double cd = kConst ? P.cd64 : (double)c32;
            const double co = kConst ? P.co64 : (double)__fmul_rn(P.mdt, __fmul_rn(a, P.vnb));
            const double ri = be - (cd * xv[0] + co * nb);
            const float rf = (float)ri, zz = here ? rf * rcp_approx(c32) : 0.0f;
            if (here) {
                rs[0] += ri * ri;
                rs[1] += bi * bi;
                rs[2] += (kConst ? (double)rf : (double)rf / (double)a) * (double)zz;
                rs[3] += (double)rf * (double)rf;
            }
            szf[c] = zz;
        }
        if (kConst) rs[2] /= (double)P.alpha0;
        ++tag;
        ++round;
        __syncthreads();
        if (T.size > 1)
#pragma unroll 1
            for (int v = tid; v < ng; v += kRcThreads) send(v, (int)P.fgx.div((uint32_t)v), sz[v]);
        if (!rc_allreduce(T, sh, kRcWordR, 4, tag, rs[0], rs[1], rs[2], rs[3], false)) { R.ok = false; return; }
        const double rt[4] = {sh.out[0], sh.out[1], sh.out[2], sh.out[3]};
        double tol2 = U.tol2, rr0 = U.rr0, beta0 = 0.0, rz = rt[2], pq = 0.0;
        if (kResume) {
            R.status = PIRO_OK;
            R.inner = U.iters;
            if (U.iters > 0) {
                pq = U.pq;
                beta0 = -rt[1] / pq;
            }
        } else {
        const double bn = rt[1] > 0.0 ? sqrt(rt[1]) : 1.0;
        R.rel = sqrt(rt[0]) / bn;
        if (!isfinite(R.rel)) { R.status = PIRO_STATUS_STALLED; break; }
        if (R.rel <= P.rtol) { R.status = PIRO_OK; break; }
        if (sweep >= P.max_outer || R.inner >= P.max_inner) break;
        if (sweep > 0 && R.rel > 0.5 * prev_rel) { R.status = PIRO_STATUS_STALLED; break; }
        prev_rel = R.rel;
        R.outer = sweep + 1;
        double itol = 0.5 * P.rtol / R.rel;
        itol = itol > 0.1 ? 0.1 : itol;
        itol = itol < P.inner_floor ? P.inner_floor : itol;
        tol2 = itol * itol;
        rr0 = rt[3];
        }
        double sum[3] = {0.0, 0.0, 0.0};  // this thread's <s, z>, <z, w>, |alpha s|^2
        bool first = true, broken = kResume && !isfinite(beta0);
#pragma unroll 1
        while (rr0 > 0.0 && !broken) {
            // H: the halo's lines, two words per group, as they arrive
            if (T.size > 1) {
                const int nh = sh.halo * gx;
#pragma unroll 1
                for (int it = tid; it < nh; it += kRcThreads) {
                    const int j = (int)P.fgx.div((uint32_t)it);
                    const uint4 *at = P.zx + 2 * ((int64_t)hsrc[j] * gx + it - j * gx);
                    float4 o;
                    long long spins = 0;
                    while (true) {
                        const unsigned t0 = rc_recv(at, o.x, o.y), t1 = rc_recv(at + 1, o.z, o.w);
                        if (t0 == round && t1 == round) break;
                        if (++spins > T.spin_limit || ((spins & 63) == 0 && *((volatile int *)T.err))) {
                            atomicExch(T.err, 1);
                            sh.ok_z = 0;
                            break;
                        }
                    }
                    sz[P.groups + it] = o;
                }
            }
            __syncthreads();  // z of this run and the halo
            // S: w = D z + off * neighbours, 0 past a line's end; <z, w>
#pragma unroll
            for (int k = 0; k < kK; ++k) {
                const int v = tid + k * kRcThreads;
                if (k > 0 && k * kRcThreads >= ng) break;
                const float4 zc = v < ng ? sz[v] : zero;
                float zl = __shfl_up_sync(0xffffffffu, zc.w, 1), zr = __shfl_down_sync(0xffffffffu, zc.x, 1);
                if (v < ng) {
                    const int ll = (int)P.fgx.div((uint32_t)v), g = v - ll * gx;
                    const uint2 n = nbr[ll];
                    if (lane == 0 && g > 0) zl = szf[4 * v - 1];
                    if (lane == 31 && g < gx - 1) zr = szf[4 * v + 4];
                    if (g == 0) zl = 0.0f;
                    if (g == gx - 1) zr = 0.0f;
                    const float4 ym = sz[(n.x & 0xffffu) + g], yp = sz[(n.x >> 16) + g];
                    const float4 zm = sz[(n.y & 0xffffu) + g], zp = sz[(n.y >> 16) + g];
                    const float4 d4 = kConst ? make_float4(D0, D0, D0, D0) : D[k];
                    w[k].x = d4.x * zc.x + off * (((zl + zc.y) + (ym.x + yp.x)) + (zm.x + zp.x));
                    w[k].y = d4.y * zc.y + off * (((zc.x + zc.z) + (ym.y + yp.y)) + (zm.y + zp.y));
                    w[k].z = d4.z * zc.z + off * (((zc.y + zc.w) + (ym.z + yp.z)) + (zm.z + zp.z));
                    w[k].w = d4.w * zc.w + off * (((zc.z + zr) + (ym.w + yp.w)) + (zm.w + zp.w));
                    if (g == gx - 1) {
                        if (lx < 2) w[k].y = 0.0f;
                        if (lx < 3) w[k].z = 0.0f;
                        if (lx < 4) w[k].w = 0.0f;
                    }
                    sum[1] += rc_dot<kWide>(zc, w[k], kWide && P.wide_s);
                }
            }
            ++tag;
            const int first_word = kRcWordSums + 3 * (flip++ & 1);
            if (!rc_allreduce(T, sh, first_word, 3, tag, sum[0], sum[1], sum[2], 0.0, false) || !sh.ok_z) {
                R.ok = false;
                return;
            }
            const double st[3] = {sh.out[0], sh.out[1], sh.out[2]};
            double beta = beta0;
            if (!first) {
                ++R.inner;
                beta = st[0] / rz;
                rz = st[0];
                if (kResume) R.rel = st[2];
                if (!isfinite(st[2]) || !isfinite(beta)) { broken = !kConst; break; }
                if (st[2] <= tol2 * rr0 || R.inner >= P.max_inner) break;
            }
            pq = st[1] - beta * beta * pq;
            const double a = rz / pq;
            if (!isfinite(a) || pq <= 0.0) { broken = true; break; }
            first = false;
            // U
            const float fa = (float)a, fb = (float)beta;
            ++round;
            sum[0] = sum[1] = sum[2] = 0.0;
#pragma unroll
            for (int k = 0; k < kK; ++k) {
                const int v = tid + k * kRcThreads;
                if (v < ng) {
                    const int ll = (int)P.fgx.div((uint32_t)v);
                    const float4 zo = sz[v];
                    float4 al, qq = q.get(k, v), dd = d.get(k, v), s, zn;
                    if (!kConst) al = kStreamA ? P.ax[(int64_t)(nat[ll] & 0x7fffffff) * gx + v - ll * gx] : sa[v];
                    const float4 d4 = kConst ? make_float4(D0, D0, D0, D0) : D[k];
                    p[k].x = zo.x + fb * p[k].x; p[k].y = zo.y + fb * p[k].y;
                    p[k].z = zo.z + fb * p[k].z; p[k].w = zo.w + fb * p[k].w;
                    qq.x = w[k].x + fb * qq.x; qq.y = w[k].y + fb * qq.y;
                    qq.z = w[k].z + fb * qq.z; qq.w = w[k].w + fb * qq.w;
                    dd.x += fa * p[k].x; dd.y += fa * p[k].y; dd.z += fa * p[k].z; dd.w += fa * p[k].w;
                    s.x = zo.x * d4.x - fa * qq.x; s.y = zo.y * d4.y - fa * qq.y;
                    s.z = zo.z * d4.z - fa * qq.z; s.w = zo.w * d4.w - fa * qq.w;
                    zn.x = s.x * rcp_approx(d4.x); zn.y = s.y * rcp_approx(d4.y);
                    zn.z = s.z * rcp_approx(d4.z); zn.w = s.w * rcp_approx(d4.w);
                    q.put(k, v, qq);
                    d.put(k, v, dd);
                    sz[v] = zn;
                    if (T.size > 1) send(v, ll, zn);
                    sum[0] += rc_dot<kWide>(s, zn, kWide && P.wide_u);
                    if (!kConst) { s.x *= al.x; s.y *= al.y; s.z *= al.z; s.w *= al.w; }
                    sum[2] += rc_dot<kWide>(s, s, kWide && P.wide_u);
                }
            }
            if (kConst) sum[2] *= (double)P.alpha0 * (double)P.alpha0;
        }
        if (broken && !kConst) R.status = PIRO_STATUS_STALLED;
        if (broken && !kConst && !kResume) break;
        // X: x += d, a cell per thread (d through shared memory)
        if (kReg) {
#pragma unroll
            for (int k = 0; k < kK; ++k)
                if (tid + k * kRcThreads < ng) {
                    d.s[tid + k * kRcThreads] = d.get(k, 0);
                    d.put(k, 0, zero);
                }
        }
        __syncthreads();
#pragma unroll 1
        for (int c0 = tid; c0 < 4 * ng; c0 += kB * kRcThreads) {
            double xo[kB];
            int64_t ci[kB];
            bool in[kB];
#pragma unroll
            for (int j = 0; j < kB; ++j) {
                int x, y, z;
                in[j] = where(c0 + j * kRcThreads, x, y, z);
                ci[j] = cell(x, y, z);
                if (kResume) xo[j] = 0.0;
                else if (sweep > 0) xo[j] = P.x64[ci[j]];
                else xo[j] = (double)__ldg(P.b + ci[j]);
            }
#pragma unroll
            for (int j = 0; j < kB; ++j) {
                const int c = c0 + j * kRcThreads;
                if (c >= 4 * ng) break;
                if (kResume && in[j]) U.d[ci[j]] = sdf[c];
                else if (in[j]) P.x64[ci[j]] = xo[j] + (double)sdf[c];
                if (!kReg) sdf[c] = 0.0f;
            }
        }
        corrected = true;
        if (kResume) break;
        if (broken) { R.status = PIRO_STATUS_STALLED; break; }  // constant alpha: ends with the correction it has
        // every CTA's x64 before the next residual reads its neighbours
        ++tag;
        if (!rc_allreduce(T, sh, kRcWordX, 1, tag, 0.0, 0.0, 0.0, 0.0, true)) { R.ok = false; return; }
    }
    if (T.size > 1 && T.rank == 0 && tid == 0) *T.epoch = tag;  // every CTA has read it before its first sums
    if (kResume) return;
    // the interior from x64 (b itself if no sweep came to its end)
#pragma unroll 1
    for (int c = tid; c < 4 * ng; c += kRcThreads) {
        int x, y, z;
        if (!where(c, x, y, z)) continue;
        const int64_t i = cell(x, y, z);
        const bool have = kConst ? R.outer > 0 : corrected;  // a sweep begun is a sweep ended for constant alpha
        const double xv = have ? P.x64[i] : (double)P.b[i];
        if (!have) P.x64[i] = xv;
        P.xout[i] = (float)xv;
    }
}

}  // namespace piro
