// On-chip iteration loops of the whole-solve path for grids that fit into the SMs' shared
// memory and registers: one cooperative launch runs a whole loop (CG, Chebyshev, PPCG or
// Jacobi, and the FP32 inner CG, Chebyshev and PPCG solves) instead of a CUDA graph that launches
// one or more kernels per iteration.
//
// What bounds it.  On such grids a launch is all latency: reading the state, filling the
// row rings, the reduction's last block and the next launch take 6-12 us whatever the size,
// two launches an iteration (20.6 us per CG iteration at 512^2).  Here one block per SM
// owns a tile of the grid for the whole loop.  The stencil operand V (p, u or sd) sits in
// shared memory with a one-cell halo, the face coefficients beside it, the other vectors
// (r, w, p, u) in the registers of the threads that own the cells.  What is left of an
// iteration is the arithmetic, one exchange of the tile's rim and the dot products.
//
// Work split.  A warp owns up to RS consecutive rows of a strip 64 cells wide (two cells per
// lane), so that a row's y-neighbours and its lower face coefficient come from the registers
// of the row before.  A block has 16 warps for up to four rows each, 12 (of 168 registers a
// thread) for up to eight, and 16 again (with up to seven where that will do) only where 12
// are too few: beside 220 KB of shared memory the L1 cache is too small for spills, and CG at
// 850^2 takes 7.6 us an iteration with 12 warps and 12.0 with 16.  At the domain's faces a neighbour is the
// cell itself, as the reference's reflecting halo update gives it; only the faces shared by
// two tiles have halo cells.
//
// Exchange.  A rim value travels as one 16-byte word {value, epoch}: the owner stores it
// with one 128-bit store, the reader polls the word until it carries the epoch it needs, so
// no fence and no separate flag is needed.  Words are double-buffered by the epoch's parity:
// a block can be at most one epoch ahead of a neighbour, because it needs that neighbour's
// word of the same epoch to go on.
//
// Sums.  An all-to-all of the blocks' double-double partials through such words took 2400-2900
// cycles at 64-128 blocks, a counter that all blocks add to and poll 1400-1550 (148 blocks),
// so a dot product is formed by integer atomics: each thread's partial is cut into four 26-bit
// limbs at bit positions that all blocks know (from the last value of the same sum), the
// limbs add up exactly in any order, and each limb's 64-bit word counts its arrivals in
// its top byte, so that the poll that sees the last arrival has the sum.  The integer sums
// also replace five levels of double-double merges in a warp by four redux instructions.
// (Five 22-bit limbs, which 32 bits could sum over a block, and a chain of double-double adds
// behind the poll cost 3 % of an iteration more.)
// Every block then forms the rounded value and runs the scalar recurrence and the loop test
// itself.
//
// What the sums are worth.  The limbs hold a thread's double-double partial to 2^-95 of the scale,
// the sum's last value, and so the sum to 2^-76 of it.  Where that does not settle how the sum rounds
// (one in 2^23 where it is about as large as the last one; always where it has fallen by more than 2^23,
// or to 0), and where a partial lies beyond 2^8 of the scale (the terms of p.w may be far larger than
// p.w), the partials are merged again in double-double, as the per-launch kernels merge theirs: one
// more round through all blocks, and no more.  So a sum is the rounded sum of the threads' partials
// except within some 2^-100 of the terms' magnitude of a rounding boundary, as it is in the per-launch
// kernels, whose sums the tests find bit for bit.  Per cell the operations and their order are those
// of the per-call kernels.  (Against a loop that took every sum as the limbs gave it: CG at 512^2 0.9 %
// faster, by the compiler's schedule, PPCG at 1024^2 the same, Jacobi on 33 x 150 cells 1.7 % slower.)
//
// Clusters.  Up to 16 blocks with one row a warp (some 16000 cells) form one cluster: limbs and rim
// values go straight into the other blocks' shared memory, and an mbarrier there counts their
// bytes.  The rim buffers and the limbs' slots are double-buffered as above.  A CG iteration
// takes 2.6 us at 64^2 and 3.0 at 128^2 (through L2 3.9), a Jacobi one 1.5 and 1.9 (2.1), a
// Chebyshev one 1.0 and 1.2 (1.4).
//
// Every poll is bounded; a block that gives up raises a flag that ends the other blocks'
// polls too, and the host reports the solve as failed.
#pragma once

#include <math_constants.h>

#include "tea_fused.cuh"

namespace tea {

constexpr int RES_WARPS = 16;  // most warps of a block
// The kernels' forms: at most RS rows a warp, W warps a block; the blocks of the cluster form are one
// cluster, which exchanges through its shared memory.  It has one row a warp: with two, in 16 blocks,
// CG takes as long as with one in twice the blocks (3.65 us an iteration at 160^2 either way), and
// Chebyshev longer (1.67 against 1.42).
struct ResForm {
    int rows, warps;
    bool cluster;
};
constexpr ResForm RES_FORMS[] = {{1, 16, true},  {1, 16, false}, {2, 16, false},
                                 {4, 16, false}, {8, 12, false}, {7, 16, false}, {8, 16, false}};
constexpr int RES_FORM_COUNT = 7;
constexpr int RES_CLUSTER = 16;  // most blocks of a cluster
constexpr unsigned long long RES_BAR_NS = 2000000000ull;  // a wait at an mbarrier gives up after this time
constexpr unsigned long long RES_DRAIN_NS = 1000000ull;   // what is on its way in a cluster is given to arrive
constexpr int RES_POLLS = 1 << 21;  // rounds of polls before a wait gives up (a second or two)
constexpr int RES_LIMBS = 4;         // limbs of a sum, and one word of flags
constexpr int RES_SUM_STRIDE = 32;   // 64-bit words between two sums: a sum's words share a line
constexpr int RES_SUM_WORDS = 2 * 2 * RES_SUM_STRIDE;  // two sets of two parities
constexpr int RES_SLOTS = 256;       // blocks whose partials of a sum that is formed again lie behind the words, four
                                     // words each, by parity
constexpr size_t RES_SUM_BYTES = (RES_SUM_WORDS + 2 * RES_SLOTS * 4) * sizeof(unsigned long long);

struct ResWord {
    unsigned long long v, tag;
};

// How the grid is dealt to the blocks and a tile to the warps, and where things lie in shared
// memory.
struct ResPlan {
    int blocks = 0;           // 0: the grid does not fit
    int nbx = 1, nby = 1, nbz = 1;
    int warps = 1, form = 0;  // warps of a block, kernel form
    int tw = 0, th = 0, td = 0;  // largest tile
    int chunks = 1;           // a strip's rows are dealt to this many warps
    int sx = 0, kxs = 0, tws = 0;  // row strides of V, of Kx, and of the other arrays
    int halo = 0;             // most halo cells of a tile
    int pre = 0;              // with the preconditioner's diagonal
    int okx = 0, oky = 0, okz = 0, omi = 0, orh = 0, omh = 0;  // first elements of Kx, Ky, Kz, mi, halo r, halo mi
    int ox = 0;               // ... of one more vector of the loop, where there is room (else 0)
    int oh = 0, hst = 0;      // cluster: first element of the two buffers that the neighbours fill, and their stride
    int words = 0;            // elements of T before the halo table
    size_t bytes = 0;         // dynamic shared memory
};

struct SumArgs {
    unsigned long long* sums;  // RES_SUM_WORDS and the slots; this launch's set is zero, the other set's words
    int set;                   // are cleared for the next launch
    int blocks;                // at most 255 (the arrivals are counted in a byte)
    int polls;                 // rounds of polls before a wait gives up
    int* fail;
};

struct ResArgs {
    FusedArgs f;
    ResPlan p;
    const SolveState* start;  // the state the loop starts from, or null: s0
    SolveState s0;
    SolveState* host;  // the final state goes to *f.st and to the host's record
    ResWord* rim;    // [2][elems]: rim values by the cell's array index (from the allocation's start)
    long elems;
    SumArgs sum;
    unsigned long long epoch;  // the rim exchanges' last epoch before this launch
};

// First cell of part i of n parts of `cells` (in units of `unit` cells).
__host__ __device__ inline int res_split(int cells, int unit, int i, int n)
{
    const int units = (cells + unit - 1) / unit;
    const int c = (int)((long)i * units / n) * unit;
    return c < cells ? c : cells;
}

// ------------------------------------------------------------------ words

__device__ __forceinline__ void res_put(ResWord* p, unsigned long long v, unsigned long long tag)
{
    asm volatile("{\n .reg .b128 q;\n mov.b128 q, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], q;\n}\n" ::"l"(p), "l"(v),
                 "l"(tag)
                 : "memory");
}
__device__ __forceinline__ ResWord res_get(const ResWord* p)
{
    ResWord w;
    asm volatile("{\n .reg .b128 q;\n ld.relaxed.gpu.global.b128 q, [%2];\n mov.b128 {%0, %1}, q;\n}\n"
                 : "=l"(w.v), "=l"(w.tag)
                 : "l"(p)
                 : "memory");
    return w;
}
// The value of a word once it carries `tag`; after the poll limit, or when another block has
// given up, sets gave_up and returns whatever is there.
__device__ __forceinline__ unsigned long long res_wait(const ResWord* q, unsigned long long tag, int polls, int* fail,
                                                       bool& gave_up)
{
    ResWord w = res_get(q);
    for (int k = 0; w.tag != tag; ++k) {
        if (k >= polls || ((k & 1023) == 1023 && *(volatile int*)fail != 0)) {
            gave_up = true;
            break;
        }
        w = res_get(q);
    }
    return w.v;
}
__device__ __forceinline__ unsigned long long res_bits(double v) { return (unsigned long long)__double_as_longlong(v); }
__device__ __forceinline__ unsigned long long res_bits(float v) { return (unsigned long long)__float_as_uint(v); }
template <class T>
__device__ __forceinline__ T res_value(unsigned long long b);
template <>
__device__ __forceinline__ double res_value<double>(unsigned long long b) { return __longlong_as_double((long long)b); }
template <>
__device__ __forceinline__ float res_value<float>(unsigned long long b) { return __uint_as_float((unsigned)b); }

// ------------------------------------------------------------------ clusters

__device__ __forceinline__ unsigned res_shared(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
// The address in block `rank` of the cluster of what lies at `a` in this block.
__device__ __forceinline__ unsigned res_remote(unsigned a, int rank)
{
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
// Stores that count their bytes at an mbarrier of the block that they go to.
__device__ __forceinline__ void res_send(unsigned a, unsigned bar, double v)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(a),
                 "l"(__double_as_longlong(v)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void res_send(unsigned a, unsigned bar, float v)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(a),
                 "r"(__float_as_uint(v)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void res_send(unsigned a, unsigned bar, unsigned long long v0, unsigned long long v1)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(a), "l"(v0),
                 "l"(v1), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void res_expect(unsigned bar, int bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool res_arrived(unsigned bar, unsigned phase)
{
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(phase)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ unsigned long long res_now()
{
    unsigned long long ns;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(ns));
    return ns;
}
// Waits for a phase of an mbarrier; gives up as res_wait does, but by the clock: the hardware chooses how
// long a try takes.
__device__ __forceinline__ void res_wait_bar(unsigned bar, unsigned phase, int* fail, bool& gave_up)
{
    unsigned long long from = 0;
    for (int k = 0; !res_arrived(bar, phase); ++k)
        if ((k & 63) == 63) {
            const unsigned long long now = res_now();
            if (from == 0) from = now;
            if (now - from >= RES_BAR_NS || *(volatile int*)fail != 0) {
                gave_up = true;
                break;
            }
        }
}
__device__ __forceinline__ void res_cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// What the blocks of a cluster write into each other: the blocks' limbs of a sum (by the sum's
// parity), and per face that a tile shares the neighbour's buffer and mbarriers.
struct ResFace {
    unsigned data, bar;
};
template <bool CL>
struct ClusterShared {
    alignas(16) unsigned long long sums[2][RES_CLUSTER][4];
    unsigned long long sum_bar[2], rim_bar[2];
    ResFace face[6];
    int gone;  // a block of the cluster has given up
};
template <>
struct ClusterShared<false> {
};

// ------------------------------------------------------------------ sums

// Limb positions of a sum, from the biased exponent E of its expected magnitude m: a thread's
// partial may reach 2^8 m, the limbs are 26 bits apart (so that a warp's total of a limb is
// at most 2^30), the first one's unit is 2^-17 m and the last one's 2^-95 m.
constexpr int RES_E_MIN = 97, RES_E_MAX = 1980;  // expected exponents stay inside (units are normal numbers)
constexpr int RES_E_UNIT = -17, RES_E_STEP = 26, RES_E_ROOM = 7;
constexpr int RES_E_LOW = 46;    // a partial's low part is below 2^-45 m
constexpr int RES_E_SLACK = 76;  // the limbs give the sum of the partials to less than 2^-76 m
constexpr int RES_E_LIFT = 3;    // room above the largest partial of a sum that was formed again

__device__ __forceinline__ int res_exponent(double v) { return (__double2hiint(v) >> 20) & 0x7ff; }
__device__ __forceinline__ int res_clamp(int e) { return min(max(e, RES_E_MIN), RES_E_MAX); }
__device__ __forceinline__ double res_unit(int E, int limb)
{
    return __hiloint2double((E + RES_E_UNIT - RES_E_STEP * limb) << 20, 0);
}

// A lane's partial hi + lo cut into limbs: 1.5 * 2^52 units plus the rest has the limb in its
// low word.  lo, below 2^-45 m, joins after the second limb, whose rest is at most 2^-44 m: that
// sum rounds off at most 2^-97 m, and 2^-96 m is left below the last limb.  Over 2^17 threads (255
// blocks of 16 warps) that is at most 2^-78 m; adding the limbs up rounds off 2^-79 m (the totals of
// the two low ones are below 2^43 units).
__device__ __forceinline__ void res_limbs(double hi, double lo, int E, int (&v)[RES_LIMBS])
{
    double rest = hi;
#pragma unroll
    for (int i = 0; i < RES_LIMBS; ++i) {
        const double cut = __hiloint2double(((E + RES_E_UNIT + 52 - RES_E_STEP * i) << 20) | 0x00080000, 0);
        const double t = cut + rest;
        v[i] = __double2loint(t);
        rest = rest - (t - cut);
        if (i == 1) rest = rest + lo;
    }
}

// A sum in double-double, and the least scale at which the limbs take its partials.
struct Wide {
    DD s;
    int scale;
};
__device__ __forceinline__ void wide_add(Wide& a, const Wide& b)
{
    a.s = dd_merge(a.s, b.s);
    a.scale = max(a.scale, b.scale);
}
// Over the warp; the same in every lane.
__device__ __forceinline__ void wide_merge(Wide& a)
{
#pragma unroll 1
    for (int o = 16; o > 0; o >>= 1) {
        Wide b;
        b.s.hi = __shfl_xor_sync(0xffffffffu, a.s.hi, o);
        b.s.lo = __shfl_xor_sync(0xffffffffu, a.s.lo, o);
        b.scale = __shfl_xor_sync(0xffffffffu, a.scale, o);
        wide_add(a, b);
    }
}
// Over the block, by every thread; the result is valid in warp 0.
__device__ __forceinline__ Wide wide_block(DD acc, Wide* s)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    Wide a = {acc, max(res_exponent(acc.hi) - RES_E_ROOM, res_exponent(acc.lo) + RES_E_LOW)};
    wide_merge(a);
    if (lane == 0) s[warp] = a;
    __syncthreads();
    if (warp == 0) {
        if (lane >= (int)(blockDim.x >> 5)) a = {{0.0, 0.0}, 0};
        else a = s[lane];
        wide_merge(a);
    }
    return a;
}
// Over the blocks' four words each at `slots`, by one warp.
__device__ __forceinline__ Wide wide_grid(const unsigned long long* slots, int nb)
{
    Wide a = {{0.0, 0.0}, 0};
    for (int b = threadIdx.x & 31; b < nb; b += 32) {
        const volatile unsigned long long* q = slots + 4 * b;
        wide_add(a, {{res_value<double>(q[0]), res_value<double>(q[1])}, (int)q[2]});
    }
    wide_merge(a);
    return a;
}

// Out of line for the on-chip loops, which have no registers to spare (PPCG at 1024^2 0.7 % slower with
// these in line), and the streamed FP64 loop (CG phase of PPCG at 256^3: the timestep 0.4 % slower in
// line); in line for the streamed FP32 loop (CG at 256^3 0.9 % slower with calls).
__device__ __noinline__ Wide wide_block_call(DD acc, Wide* s) { return wide_block(acc, s); }
__device__ __noinline__ Wide wide_grid_call(const unsigned long long* slots, int nb) { return wide_grid(slots, nb); }

template <bool CL = false>
struct SumShared : ClusterShared<CL> {
    int limbs[RES_LIMBS][RES_WARPS];
    int scale[2];  // expected exponents of the loop's two sums
    int lift[2];   // ... above the exponents of their last values
    Wide wide[RES_WARPS];  // the warps' partials of a sum that is formed again
    int bad;       // a partial out of range (1) or not finite (2)
    int next;      // what follows a sum or an iteration: RN_*
    int lost;      // a wait of this block has given up
    double sum;    // the last sum
};
enum { RN_GO = 0, RN_STOP = 1, RN_AGAIN = 2, RN_FAIL = 4 };

// A block's part in the sums over the grid.
template <bool CL = false, bool CALL = false>
struct GridSum {
    const SumArgs& sa;
    SumShared<CL>& ss;
    int nw, warp, lane;
    unsigned long long seen0 = 0, seen1 = 0;  // this lane's word of the sums, as last read, by parity
    int parity = 0;
    unsigned phases = 0;  // of the cluster's sum barriers, a bit for each parity
    bool gave_up = false;

    __device__ __forceinline__ GridSum(const SumArgs& a, SumShared<CL>& s)
        : sa(a), ss(s), nw(blockDim.x >> 5), warp(threadIdx.x >> 5), lane(threadIdx.x & 31)
    {
    }
    __device__ __forceinline__ void start(double scale)  // one thread, before the first sum
    {
        ss.scale[0] = ss.scale[1] = res_clamp(res_exponent(scale));
        ss.lift[0] = ss.lift[1] = 0;
        ss.bad = 0;
        ss.next = RN_GO;
        ss.lost = 0;
    }
    // The other set's words, by one block at the end of the launch.
    __device__ __forceinline__ void clear_other_set() const
    {
        for (int i = threadIdx.x; i < RES_SUM_WORDS / 2; i += blockDim.x) sa.sums[(sa.set ^ 1) * (RES_SUM_WORDS / 2) + i] = 0;
    }

    // Sum number `which` of the loop over all blocks.  `meanwhile` runs in the other warps while
    // warp 0 waits.  With the rounded sum, `control` runs in warp 0's first lane before any
    // thread goes on (it returns whether the loop goes on), and `after` in the last warp's first
    // lane while the others go on.  Returns RN_GO, RN_STOP or RN_FAIL.
    // With FENCE, what the blocks wrote before the sum is visible to all of them after it.
    // All blocks see the same totals and flags, and so agree on whether the sum stands.
    template <bool FENCE = false, class M, class C, class N>
    __device__ __forceinline__ int reduce(const DD& acc, int which, M&& meanwhile, C&& control, N&& after)
    {
        const int E = ss.scale[which];
        if (max(res_exponent(acc.hi) - RES_E_ROOM, res_exponent(acc.lo) + RES_E_LOW) > E)
            atomicOr(&ss.bad, isfinite(acc.hi) ? 1 : 2);
        int v[RES_LIMBS];
        res_limbs(acc.hi, acc.lo, E, v);  // whatever they are for a partial out of range: the flag says so
#pragma unroll
        for (int i = 0; i < RES_LIMBS; ++i) v[i] = __reduce_add_sync(0xffffffffu, v[i]);
        if (lane == 0) {
#pragma unroll
            for (int i = 0; i < RES_LIMBS; ++i) ss.limbs[i][warp] = v[i];
        }
        parity ^= 1;
        __syncthreads();
        if (warp == 0) {
            unsigned bad = ss.bad;
            const int lift = ss.lift[which];
            long long tot[RES_LIMBS];
#pragma unroll
            for (int i = 0; i < RES_LIMBS; ++i) {
                // The halves of the warps' limbs apart: together they may exceed 32 bits.
                const int v = lane < nw ? ss.limbs[i][lane] : 0;
                const int low = __reduce_add_sync(0xffffffffu, v & 0xffff), high = __reduce_add_sync(0xffffffffu, v >> 16);
                tot[i] = (long long)high * 65536 + low;
            }
            constexpr long long bias = 1ll << 36;  // raises a block's limbs to be positive
            if constexpr (CL) {
                all_to_all(tot, bad, sa.blocks, bias);
            } else if (sa.blocks > 1) {
                long long mine = (long long)((bad & 1) + ((bad & 2) << 15));
#pragma unroll
                for (int i = 0; i < RES_LIMBS; ++i) mine = lane == i ? tot[i] : mine;
                mine = counted<FENCE>(mine + bias) - sa.blocks * bias;
#pragma unroll
                for (int i = 0; i < RES_LIMBS; ++i) tot[i] = __shfl_sync(0xffffffffu, mine, i);
                bad = (unsigned)__shfl_sync(0xffffffffu, (int)mine, RES_LIMBS);
                bad = ((bad & 0xffff) ? 1 : 0) | ((bad >> 16) ? 2 : 0);
            }
            // Each total is below 2^53, so exact; the sum of the two high ones is kept whole.
            static_assert(RES_LIMBS == 4, "the limbs summed here");
            DD s = {(double)tot[0] * res_unit(E, 0), 0.0};
            dd_add(s, (double)tot[1] * res_unit(E, 1));
            const double low = s.lo + ((double)tot[2] * res_unit(E, 2) + (double)tot[3] * res_unit(E, 3));
            if (lane == 0) {
                // The sum stands if it rounds the same wherever in the limbs' error it lies (0 never does).
                const double slack = __hiloint2double((E - RES_E_SLACK) << 20, 0);
                const double sum = s.hi + low;
                const bool doubtful = (s.hi + (low + slack)) != (s.hi + (low - slack));
                int next = RN_AGAIN;
                if (__builtin_expect(!doubtful && bad == 0, 1)) {
                    ss.scale[which] = res_clamp(res_exponent(sum) + lift);
                    ss.sum = sum;
                    next = control(sum) ? RN_GO : RN_STOP;
                } else if (bad & 2) {  // as the double-double merges make of it
                    next = control(CUDART_NAN) ? RN_GO : RN_STOP;
                    ss.sum = CUDART_NAN;
                }
                ss.bad = 0;
                ss.next = next;
            }
        }
        meanwhile();
        int next = finish();
        if (__builtin_expect(next == RN_AGAIN, 0)) {
            reduce_wide(acc, which, control);
            next = finish();
        }
        if (next & RN_FAIL) return RN_FAIL;
        if (threadIdx.x == 32 * (nw - 1)) after(ss.sum);
        return next;
    }
    // The sum again, from the partials as they are: double-double merges in the block, whose result goes to
    // all blocks, and each merges them in the same order.
    template <class C>
    __device__ __forceinline__ void reduce_wide(const DD& acc, int which, C&& control)
    {
        parity ^= 1;
        Wide s = CALL ? wide_block_call(acc, ss.wide) : wide_block(acc, ss.wide);
        if (warp != 0) return;
        const int nb = sa.blocks;
        if (nb > 1) {
            const unsigned long long* slots;
            if constexpr (CL) {
                slots = &ss.sums[parity][0][0];
                exchange(res_bits(s.s.hi), res_bits(s.s.lo), (unsigned long long)s.scale, 0, nb);
            } else {
                slots = sa.sums + RES_SUM_WORDS + (size_t)parity * RES_SLOTS * 4;
                if (lane == 0) {
                    volatile unsigned long long* q = const_cast<unsigned long long*>(slots) + 4 * blockIdx.x;
                    q[0] = res_bits(s.s.hi);
                    q[1] = res_bits(s.s.lo);
                    q[2] = (unsigned long long)s.scale;
                }
                counted<true>(0);
            }
            s = CALL ? wide_grid_call(slots, nb) : wide_grid(slots, nb);
        }
        if (lane == 0) {
            const double sum = dd_value(s.s);
            ss.next = control(sum) ? RN_GO : RN_STOP;
            if (isfinite(sum) && sum != 0.0) {
                const int e = res_exponent(sum);
                ss.lift[which] = max(s.scale + RES_E_LIFT - e, 0);
                ss.scale[which] = res_clamp(e + ss.lift[which]);
            }
            ss.sum = sum;
        }
    }
    // Adds `mine` (positive, below 2^48) to this lane's word of all blocks and returns the total: a count of
    // arrivals in the top byte, the total below it.  The warp stays together: a lane that polled before
    // another has added would wait for a word that the other blocks' same lanes wait for too.  The atomics
    // return a value so that the polls begin when this block's have arrived (1550 cycles a sum against 2050
    // at 64 blocks).  With FENCE, what the blocks wrote before is visible after it.
    template <bool FENCE>
    __device__ __forceinline__ long long counted(long long mine)
    {
        const bool has = lane <= RES_LIMBS;
        unsigned long long* q = sa.sums + (sa.set * 2 + parity) * RES_SUM_STRIDE + (has ? lane : RES_LIMBS);
        const unsigned long long add = (1ull << 56) + (unsigned long long)mine;
        const unsigned long long old = parity ? seen1 : seen0;
        unsigned long long now = old;
        if (FENCE) __threadfence();
        if (has) asm volatile("atom.relaxed.gpu.global.add.u64 %0, [%1], %2;" : "=l"(now) : "l"(q), "l"(add) : "memory");
        __syncwarp();
        now += add;
        for (int k = 0; __any_sync(0xffffffffu, has && (int)((now - old) >> 56) != sa.blocks); ++k) {
            if (k >= sa.polls || ((k & 1023) == 1023 && *(volatile int*)sa.fail != 0)) {
                gave_up = true;
                break;
            }
            asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(now) : "l"(q) : "memory");
        }
        if (FENCE) __threadfence();
        seen0 = parity ? seen0 : now;
        seen1 = parity ? now : seen1;
        return (long long)((now - old) & ((1ull << 56) - 1));
    }
    // The limbs and flags of all blocks of the cluster: each block sends its own to every block.
    __device__ __forceinline__ void all_to_all(long long (&tot)[RES_LIMBS], unsigned& bad, int nb, long long bias)
    {
        if constexpr (CL) {
            exchange((unsigned long long)(tot[0] + bias) | (unsigned long long)bad << 56, (unsigned long long)(tot[1] + bias),
                     (unsigned long long)(tot[2] + bias), (unsigned long long)(tot[3] + bias), nb);
            unsigned flags = 0;
            long long v[RES_LIMBS] = {0, 0, 0, 0};
            if (lane < nb) {
                const ulonglong2 *q = reinterpret_cast<const ulonglong2*>(&ss.sums[parity][lane][0]), a = q[0], b = q[1];
                flags = (unsigned)(a.x >> 56);
                v[0] = (long long)(a.x & ((1ull << 56) - 1)) - bias;
                v[1] = (long long)a.y - bias;
                v[2] = (long long)b.x - bias;
                v[3] = (long long)b.y - bias;
            }
            bad = __reduce_or_sync(0xffffffffu, flags);
#pragma unroll
            for (int i = 0; i < RES_LIMBS; ++i) {
                const int low = __reduce_add_sync(0xffffffffu, (int)(v[i] & 0xfffff)),
                          high = __reduce_add_sync(0xffffffffu, (int)(v[i] >> 20));
                tot[i] = (long long)high * (1 << 20) + low;
            }
        }
    }
    // Four words of this block to every block of the cluster, and theirs to ss.sums.
    __device__ __forceinline__ void exchange(unsigned long long v0, unsigned long long v1, unsigned long long v2,
                                             unsigned long long v3, int nb)
    {
        if constexpr (CL) {
            const unsigned bar = res_shared(&ss.sum_bar[parity]);
            if (lane == 0) res_expect(bar, 32 * nb);
            if (lane < nb) {
                const unsigned to = res_remote(res_shared(&ss.sums[parity][blockIdx.x][0]), lane), at = res_remote(bar, lane);
                res_send(to, at, v0, v1);
                res_send(to + 16, at, v2, v3);
            }
            __syncwarp();
            res_wait_bar(bar, phases >> parity & 1, sa.fail, gave_up);
            phases ^= 1u << parity;
        }
    }
    // The end of an exchange: after it every thread sees what the others have written and what
    // warp 0 has decided.
    __device__ __forceinline__ int finish()
    {
        if (gave_up) {
            *(volatile int*)sa.fail = 1;
            ss.lost = 1;
        }
        __syncthreads();
        return ss.lost ? RN_FAIL : ss.next;
    }
};

// ------------------------------------------------------------------ a block's tile

template <class T>
struct alignas(2 * sizeof(T)) Two {
    T x, y;
};
template <class T>
__device__ __forceinline__ Two<T> ld_two(const T* p) { return *reinterpret_cast<const Two<T>*>(p); }
template <class T>
__device__ __forceinline__ void st_two(T* p, T x, T y)
{
    Two<T> v;
    v.x = x;
    v.y = y;
    *reinterpret_cast<Two<T>*>(p) = v;
}


enum {
    RF_A0 = 1, RF_A1 = 2,                // the lane's cells exist
    RF_XM = 4, RF_XP0 = 8, RF_XP1 = 16,  // an x-neighbour is the cell itself (domain face)
    RF_P0 = 32, RF_P1 = 64,              // the cells of every row lie on the tile's rim
    RF_PFIRST = 128, RF_PLAST = 256,     // the first (last) row's do
    RF_WFIRST = 512, RF_WLAST = 1024,    // the row below the first (above the last) is itself
    // Cluster forms: the neighbours that the cells go to besides those of the first and last row.
    RF_SXM = 2048, RF_SX0 = 4096, RF_SX1 = 8192, RF_SZM = 16384, RF_SZP = 32768
};

template <bool CL>
struct ResShared {
    SolveState s;
    SumShared<CL> sum;
};

template <class T, int RS, bool CL>
struct ResTile : GridSum<CL, true> {
    using Base = GridSum<CL, true>;
    using Base::gave_up;
    using Base::lane;
    using Base::nw;
    using Base::sa;
    using Base::ss;
    using Base::warp;
    const ResArgs& A;
    const Geom& g;
    T* const V;   // shared memory: the operand, then the arrays at the plan's offsets
    int nh;       // halo cells of this tile
    int x0, y0, z0, tw, th, td;  // first cell (0-based inner) and extents
    int sx, plane;
    // The warp's rows: y .. y + rows - 1 of plane z, columns x and x + 1 of this lane.
    int rows, x, y, z;
    int o, okx, oky, okz;  // offsets of the first row in V, Kx, Ky and Kz
    long gi;               // its array index
    int fl;                // RF_* flags
    int dzm, dzp;          // offsets of the z-neighbours (0 at a domain face)
    unsigned long long tag;   // epoch of the last rim exchange

    __device__ __forceinline__ ResTile(const ResArgs& a, ResShared<CL>& s, T* mem)
        : Base(a.sum, s.sum), A(a), g(a.f.g), V(mem)
    {
        const ResPlan& p = a.p;
        const int b = blockIdx.x;
        const int bx = b % p.nbx, by = (b / p.nbx) % p.nby, bz = b / (p.nbx * p.nby);
        x0 = res_split(g.nx, 2, bx, p.nbx);
        tw = res_split(g.nx, 2, bx + 1, p.nbx) - x0;
        y0 = res_split(g.ny, 1, by, p.nby);
        th = res_split(g.ny, 1, by + 1, p.nby) - y0;
        z0 = res_split(g.nz, 1, bz, p.nbz);
        td = res_split(g.nz, 1, bz + 1, p.nbz) - z0;
        sx = p.sx;
        plane = (th + 2) * sx;
        tag = CL ? 0 : a.epoch;
        // The warp's strip, plane and rows.
        const int strips = (tw + 63) / 64;
        const int strip = warp % strips, rest = warp / strips;
        const int chunk = rest % p.chunks;
        z = rest / p.chunks;
        y = res_split(th, 1, chunk, p.chunks);
        rows = z < td ? res_split(th, 1, chunk + 1, p.chunks) - y : 0;
        if (rows == 0) y = z = 0;
        x = strip * 64 + 2 * lane;
        const bool a0 = rows > 0 && x < tw, a1 = rows > 0 && x + 1 < tw;
        const bool xl = x0 == 0, xr = x0 + tw == g.nx;
        const bool zrim = (z == 0 && z0 > 0) || (z == td - 1 && z0 + td < g.nz);
        fl = (a0 ? RF_A0 : 0) | (a1 ? RF_A1 : 0) | (x == 0 && xl ? RF_XM : 0) | (x == tw - 1 && xr ? RF_XP0 : 0) |
             (x + 1 == tw - 1 && xr ? RF_XP1 : 0) |
             (a0 && (zrim || (x == 0 && !xl) || (x == tw - 1 && !xr)) ? RF_P0 : 0) |
             (a1 && (zrim || (x + 1 == tw - 1 && !xr)) ? RF_P1 : 0) | (y == 0 && y0 > 0 ? RF_PFIRST : 0) |
             (y + rows == th && y0 + th < g.ny ? RF_PLAST : 0) | (y == 0 && y0 == 0 ? RF_WFIRST : 0) |
             (y + rows == th && y0 + th == g.ny ? RF_WLAST : 0);
        if (CL && a0)
            fl |= (x == 0 && !xl ? RF_SXM : 0) | (x == tw - 1 && !xr ? RF_SX0 : 0) | (x + 1 == tw - 1 && !xr ? RF_SX1 : 0) |
                  (z == 0 && z0 > 0 ? RF_SZM : 0) | (z == td - 1 && z0 + td < g.nz ? RF_SZP : 0);
        dzm = z == 0 && z0 == 0 ? 0 : plane;
        dzp = z == td - 1 && z0 + td == g.nz ? 0 : plane;
        const int row = z * th + y;
        o = ((DIM == 3 ? (z + 1) * (th + 2) : 0) + y + 1) * sx + x + 2;
        okx = p.okx + row * p.kxs + x;
        oky = p.oky + (row + z) * p.tws + x;
        okz = p.okz + row * p.tws + x;
        gi = fidx(g, HALO_PAD + x0 + x, HALO_PAD + y0 + y, DIM == 3 ? HALO_PAD + z0 + z : 0);
        build_table();
        if constexpr (CL) join(bx, by, bz);
    }
    // Set up the block's mbarriers and what it needs to know of its neighbours' buffers.
    __device__ void join(int bx, int by, int bz)
    {
        if constexpr (CL) {
            const ResPlan& p = A.p;
            if (threadIdx.x == 0) {
                for (int k = 0; k < 2; ++k) {
                    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(res_shared(&ss.sum_bar[k])) : "memory");
                    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(res_shared(&ss.rim_bar[k])) : "memory");
                }
                ss.gone = 0;
                asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            }
            if (threadIdx.x < 6) {
                // The neighbour at face f sees this tile at its face f ^ 1.
                const int f = threadIdx.x, d = (f & 1) ? 1 : -1;
                const int nx = bx + (f >> 1 == 0 ? d : 0), ny = by + (f >> 1 == 1 ? d : 0), nz = bz + (f >> 1 == 2 ? d : 0);
                if (nx >= 0 && nx < p.nbx && ny >= 0 && ny < p.nby && nz >= 0 && nz < p.nbz) {
                    const int w = res_split(g.nx, 2, nx + 1, p.nbx) - res_split(g.nx, 2, nx, p.nbx);
                    const int h = res_split(g.ny, 1, ny + 1, p.nby) - res_split(g.ny, 1, ny, p.nby);
                    const int e = res_split(g.nz, 1, nz + 1, p.nbz) - res_split(g.nz, 1, nz, p.nbz);
                    int base = 0;
                    for (int q = 0; q < (f ^ 1); ++q) base += face_cells(q, nx, ny, nz, w, h, e);
                    const int rank = (nz * p.nby + ny) * p.nbx + nx;
                    ss.face[f].data = res_remote(res_shared(V + p.oh + base), rank);
                    ss.face[f].bar = res_remote(res_shared(&ss.rim_bar[0]), rank);
                }
            }
            res_cluster_sync();
        }
    }
    // The end of a cluster's loop: nothing may be on its way to a block that has ended.  Where no wait has
    // given up, each block has waited for all that was sent to it.  Else no instruction waits for the
    // stores still under way: once no block sends any more, they are given a thousand times what they take.
    __device__ void leave() const
    {
        if constexpr (CL) {
            if (ss.lost && (int)threadIdx.x < sa.blocks)
                asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(res_remote(res_shared(&ss.gone), threadIdx.x)), "r"(1)
                             : "memory");
            __syncwarp();
            res_cluster_sync();
            if (*(volatile int*)&ss.gone) {
                const unsigned long long from = res_now();
                while (res_now() - from < RES_DRAIN_NS) __nanosleep(1000);
                __syncwarp();
                res_cluster_sync();
            }
        }
    }
    // Halo cells at face f of the tile of block (bx, by, bz), w x h x e cells.
    __device__ __forceinline__ int face_cells(int f, int bx, int by, int bz, int w, int h, int e) const
    {
        const int at = f >> 1 == 0 ? bx : (f >> 1 == 1 ? by : bz), n = f >> 1 == 0 ? A.p.nbx : (f >> 1 == 1 ? A.p.nby : A.p.nbz);
        if ((f & 1) ? at == n - 1 : at == 0) return 0;
        return f >> 1 == 0 ? h * e : (f >> 1 == 1 ? w * e : w * h);
    }

    __device__ __forceinline__ bool on(int k) const { return (fl & RF_A0) && k < rows; }
    __device__ __forceinline__ bool both() const { return fl & RF_A1; }
    __device__ __forceinline__ long gidx(int k) const { return gi + k * g.pitch; }
    __device__ __forceinline__ T* cell(int k) const { return V + o + k * sx; }
    __device__ __forceinline__ Two<T> mi_of(int k) const { return ld_two(V + okz + (A.p.omi - A.p.okz) + k * A.p.tws); }
    __device__ __forceinline__ T* own(int k) const { return V + okz + (A.p.ox - A.p.okz) + k * A.p.tws; }
    __device__ __forceinline__ int2* table() const { return reinterpret_cast<int2*>(V + A.p.words); }  // halo cells: {offset in V, array index}
    __device__ __forceinline__ T& halo_r(int h) const { return V[A.p.orh + h]; }
    __device__ __forceinline__ T& halo_mi(int h) const { return V[A.p.omh + h]; }

    // The tile's halo cells: the faces it shares with other tiles, without edges and corners.
    __device__ void build_table()
    {
        const int fx = th * td, fy = tw * td, fz = DIM == 3 ? tw * th : 0;
        const bool has[6] = {x0 > 0, x0 + tw < g.nx, y0 > 0, y0 + th < g.ny, DIM == 3 && z0 > 0, DIM == 3 && z0 + td < g.nz};
        const int cnt[3] = {fx, fy, fz};
        int base = 0;
        for (int f = 0; f < 6; ++f) {
            if (!has[f]) continue;
            const int n = cnt[f >> 1];
            for (int h = threadIdx.x; h < n; h += blockDim.x) {
                int hx, hy, hz;
                if (f < 2) {
                    hx = f == 0 ? -1 : tw;
                    hy = h % th;
                    hz = h / th;
                } else if (f < 4) {
                    hy = f == 2 ? -1 : th;
                    hx = h % tw;
                    hz = h / tw;
                } else {
                    hz = f == 4 ? -1 : td;
                    hx = h % tw;
                    hy = h / tw;
                }
                const int vr = DIM == 3 ? (hz + 1) * (th + 2) + hy + 1 : hy + 1;
                table()[base + h] = make_int2(vr * sx + hx + 2,
                                            (int)fidx(g, HALO_PAD + x0 + hx, HALO_PAD + y0 + hy,
                                                      DIM == 3 ? HALO_PAD + z0 + hz : 0));
            }
            base += n;
        }
        nh = base;
    }

    // Fill the coefficient arrays from the fields (mi in a preconditioned solve, else null).
    __device__ void load_coefs(const T* kx, const T* ky, const T* kz, const T* mi)
    {
        T *KX = V + A.p.okx, *KY = V + A.p.oky, *KZ = V + A.p.okz, *MI = V + A.p.omi;
        for (int r = warp; r < th * td; r += nw) {
            const int rz = r / th, ry = r - rz * th;
            const long i = fidx(g, HALO_PAD + x0, HALO_PAD + y0 + ry, DIM == 3 ? HALO_PAD + z0 + rz : 0);
            for (int c = lane; c <= tw; c += 32) KX[r * A.p.kxs + c] = kx[i + c];
            for (int c = lane; c < tw; c += 32) {
                KY[(r + rz) * A.p.tws + c] = ky[i + c];
                if (ry == th - 1) KY[(r + rz + 1) * A.p.tws + c] = ky[i + g.pitch + c];
                if (DIM == 3) {
                    KZ[r * A.p.tws + c] = kz[i + c];
                    if (rz == td - 1) KZ[(r + th) * A.p.tws + c] = kz[i + g.page + c];
                }
                if (mi) MI[r * A.p.tws + c] = mi[i + c];
            }
        }
    }
    // V and its halo from a field.
    __device__ void load_operand(const T* v)
    {
        for (int r = warp; r < th * td; r += nw) {
            const int rz = r / th, ry = r - rz * th;
            const long i = fidx(g, HALO_PAD + x0, HALO_PAD + y0 + ry, DIM == 3 ? HALO_PAD + z0 + rz : 0);
            const int vr = DIM == 3 ? (rz + 1) * (th + 2) + ry + 1 : ry + 1;
            for (int c = lane; c < tw; c += 32) V[vr * sx + c + 2] = v[i + c];
        }
        __syncthreads();  // the table
        for (int h = threadIdx.x; h < nh; h += blockDim.x) V[table()[h].x] = v[table()[h].y];
    }
    __device__ void load_halo_mi(const T* mi)
    {
        for (int h = threadIdx.x; h < nh; h += blockDim.x) halo_mi(h) = mi[table()[h].y];
    }

    // The operator's operands at the warp's rows in order: f(k, cell, nb, kx0, kx1, ky0, ky1,
    // kz0, kz1) for the two cells of each row.
    template <class F>
    __device__ __forceinline__ void sweep(F&& f) const
    {
        if (!(fl & RF_A0)) return;
        Two<T> ym = ld_two(V + o - ((fl & RF_WFIRST) ? 0 : sx)), c = ld_two(V + o), ky0 = ld_two(V + oky);
#pragma unroll
        for (int k = 0; k < RS; ++k)
            if (k < rows) {
                const T* vk = cell(k);
                const Two<T> yp = ld_two(vk + (k == rows - 1 && (fl & RF_WLAST) ? 0 : sx));
                const T l = vk[-1], r = vk[2];
                const T* kxp = V + okx + k * A.p.kxs;
                const Two<T> kx = ld_two(kxp);
                const T kx2 = kxp[2];
                const Two<T> ky1 = ld_two(V + oky + (k + 1) * A.p.tws);
                Two<T> zm = c, zp = c, kz0, kz1;
                kz0.x = kz0.y = kz1.x = kz1.y = (T)0;
                if (DIM == 3) {
                    zm = ld_two(vk - dzm);
                    zp = ld_two(vk + dzp);
                    kz0 = ld_two(V + okz + k * A.p.tws);
                    kz1 = ld_two(V + okz + (k + th) * A.p.tws);
                }
                NbT<T> nb;
                nb.c = c.x;
                nb.xm = (fl & RF_XM) ? c.x : l;
                nb.xp = (fl & RF_XP0) ? c.x : c.y;
                nb.ym = ym.x;
                nb.yp = yp.x;
                nb.zm = zm.x;
                nb.zp = zp.x;
                f(k, 0, nb, kx.x, kx.y, ky0.x, ky1.x, kz0.x, kz1.x);
                nb.c = c.y;
                nb.xm = c.x;
                nb.xp = (fl & RF_XP1) ? c.y : r;
                nb.ym = ym.y;
                nb.yp = yp.y;
                nb.zm = zm.y;
                nb.zp = zp.y;
                f(k, 1, nb, kx.y, kx2, ky0.y, ky1.y, kz0.y, kz1.y);
                ym = c;
                c = yp;
                ky0 = ky1;
            }
    }
    // The operand around the warp's rows: the rows below the first and above the last, and in lane k
    // (8 + k) the cell left (right) of row k.
    struct Around {
        Two<T> below, above;
        T side;
    };
    __device__ __forceinline__ Around around() const
    {
        Around e;
        e.below.x = e.below.y = e.above.x = e.above.y = e.side = (T)0;
        if (rows == 0) return e;
        const int first = o - 2 * lane, cols = min(64, tw - (x - 2 * lane)), k = lane & 7;
        const int at = (fl & RF_A0) ? o : first;
        e.below = ld_two(V + at - ((fl & RF_WFIRST) ? 0 : sx));
        e.above = ld_two(V + at + (rows - 1) * sx + ((fl & RF_WLAST) ? 0 : sx));
        if (lane < 16 && k < rows) e.side = V[first + k * sx + (lane < 8 ? -1 : cols)];
        return e;
    }
    // 2D: a sweep whose new operand takes the place of the old one row by row (after every warp has
    // formed its Around, and before the neighbours' values are collected).  Registers need not hold
    // the new rows until all warps have read the old ones.  f(k, c, nb0, nb1, kx0, kx1, kx2, ky0, ky1,
    // out) leaves the row's new cells in out, and they are published.  Every lane of a warp takes
    // part; those without cells work on lane 0's and store nothing.
    // Seven rows and 16 warps have no room for the new rows beside two more vectors: with u (PPCG) or
    // the right-hand side (Chebyshev) in L2 instead, an inner step moved 115 KB per SM through it.
    // PPCG at 1024^2 91.6 ms a timestep against 107.5, Chebyshev at 1000^2 42.6 against 47.2; the
    // 12-warp form, which has shared memory for the third vector, gains nothing (800^2: 49.9
    // against 48.7).
    template <class F>
    __device__ __forceinline__ void sweep_over(const Around& e, F&& f) const
    {
        if (rows == 0) return;
        const bool a0 = fl & RF_A0;
        const int back = a0 ? 0 : 2 * lane;
        const bool right = 2 * lane + 2 >= min(64, tw - (x - 2 * lane));
        Two<T> ym = e.below, c = ld_two(V + o - back), ky0 = ld_two(V + oky - back);
#pragma unroll
        for (int k = 0; k < RS; ++k)
            if (k < rows) {
                const T* vk = cell(k) - back;
                Two<T> yp = e.above;
                if (k < rows - 1) yp = ld_two(vk + sx);
                T l = vk[-1], r = vk[2];
                const T sl = __shfl_sync(0xffffffffu, e.side, k), sr = __shfl_sync(0xffffffffu, e.side, 8 + k);
                if (lane == 0) l = sl;
                if (right) r = sr;
                const T* kxp = V + okx - back + k * A.p.kxs;
                const Two<T> kx = ld_two(kxp);
                const T kx2 = kxp[2];
                const Two<T> ky1 = ld_two(V + oky - back + (k + 1) * A.p.tws);
                NbT<T> nb0, nb1;
                nb0.c = c.x;
                nb0.xm = (fl & RF_XM) ? c.x : l;
                nb0.xp = (fl & RF_XP0) ? c.x : c.y;
                nb0.ym = ym.x;
                nb0.yp = yp.x;
                nb1.c = c.y;
                nb1.xm = c.x;
                nb1.xp = (fl & RF_XP1) ? c.y : r;
                nb1.ym = ym.y;
                nb1.yp = yp.y;
                nb0.zm = nb0.zp = nb1.zm = nb1.zp = (T)0;
                Two<T> out;
                f(k, c, nb0, nb1, kx.x, kx.y, kx2, ky0, ky1, out);
                __syncwarp();  // every lane has read the row
                if (a0) {
                    store(k, out.x, out.y);
                    publish(k, out.x, out.y);
                }
                ym = c;
                c = yp;
                ky0 = ky1;
            }
    }
    // Adds cell q of row k to a thread's sum; the second cell of a row may not exist.
    __device__ __forceinline__ void add(DD& acc, int k, int q, double v) const
    {
        if (k == 0 && q == 0) acc.hi = v;
        else dd_add(acc, q == 0 || both() ? v : 0.0);
    }

    __device__ __forceinline__ void store(int k, T v0, T v1) const
    {
        // The second cell of a lane past the tile's edge may be a halo cell.
        if (both()) st_two(cell(k), v0, v1);
        else *cell(k) = v0;
    }
    // The next rim exchange.  In a cluster it is counted from 1, and fills buffer (tag - 1) & 1.
    __device__ __forceinline__ void next_exchange()
    {
        ++tag;
        if constexpr (CL)
            if (threadIdx.x == 0) res_expect(res_shared(&ss.rim_bar[turn()]), nh * (int)sizeof(T));
    }
    __device__ __forceinline__ int turn() const { return (int)(tag - 1) & 1; }
    __device__ __forceinline__ void send(int f, int i, T v) const
    {
        if constexpr (CL) {
            const ResFace q = ss.face[f];
            res_send(q.data + (turn() * A.p.hst + i) * (int)sizeof(T), q.bar + 8 * turn(), v);
        }
    }
    // Publish the rim cells of row k under the current exchange's epoch.
    __device__ __forceinline__ void publish(int k, T v0, T v1) const
    {
        if constexpr (CL) {
            const int ix = z * th + y + k, iy = z * tw + x, iz = (y + k) * tw + x;
            if (fl & RF_SXM) send(0, ix, v0);
            if (fl & (RF_SX0 | RF_SX1)) send(1, ix, (fl & RF_SX0) ? v0 : v1);
            if (k == 0 && (fl & RF_PFIRST)) {
                send(2, iy, v0);
                if (both()) send(2, iy + 1, v1);
            }
            if (k == rows - 1 && (fl & RF_PLAST)) {
                send(3, iy, v0);
                if (both()) send(3, iy + 1, v1);
            }
            if (DIM == 3 && (fl & RF_SZM)) {
                send(4, iz, v0);
                if (both()) send(4, iz + 1, v1);
            }
            if (DIM == 3 && (fl & RF_SZP)) {
                send(5, iz, v0);
                if (both()) send(5, iz + 1, v1);
            }
            return;
        }
        int rim = fl & (RF_P0 | RF_P1);
        if ((k == 0 && (fl & RF_PFIRST)) || (k == rows - 1 && (fl & RF_PLAST))) rim = RF_P0 | (both() ? RF_P1 : 0);
        if (rim) {
            ResWord* q = A.rim + (tag & 1) * A.elems + kLeadPad + gidx(k);
            if (rim & RF_P0) res_put(q, res_bits(v0), tag);
            if (rim & RF_P1) res_put(q + 1, res_bits(v1), tag);
        }
    }
    // The neighbours' values of the current exchange, through put(h, value); the warps from
    // `first` on share the halo cells.
    template <class F>
    __device__ __forceinline__ void collect(int first, F&& put)
    {
        if (nh == 0 || warp < first) return;
        if constexpr (CL) {
            const int h0 = (warp - first) * 32 + lane;
            if (h0 >= nh) return;
            res_wait_bar(res_shared(&ss.rim_bar[turn()]), (unsigned)(tag - 1) >> 1 & 1, sa.fail, gave_up);
            for (int h = h0; h < nh; h += (nw - first) * 32) put(h, V[A.p.oh + turn() * A.p.hst + h]);
            return;
        }
        const ResWord* q = A.rim + (tag & 1) * A.elems + kLeadPad;
        for (int h = (warp - first) * 32 + lane; h < nh; h += (nw - first) * 32) {
            put(h, res_value<T>(res_wait(q + table()[h].y, tag, sa.polls, sa.fail, gave_up)));
        }
    }
};

// Arrays of the FP64 solve and of the FP32 inner solves.
struct ResF64 {
    using T = double;
    static constexpr bool fp32 = false;
    __device__ static T* r(const FusedArgs& a) { return a.r; }
    __device__ static T* w(const FusedArgs& a) { return a.w; }
    __device__ static T* p(const FusedArgs& a) { return a.p[0]; }
    __device__ static T* u(const FusedArgs& a) { return a.u[0]; }
    __device__ static T* rhs(const FusedArgs& a) { return a.u0; }
    __device__ static const T* kx(const FusedArgs& a) { return a.kx; }
    __device__ static const T* ky(const FusedArgs& a) { return a.ky; }
    __device__ static const T* kz(const FusedArgs& a) { return a.kz; }
    __device__ static const T* mi(const FusedArgs& a, bool pre) { return pre ? a.mi : nullptr; }
};
struct ResF32 {
    using T = float;
    static constexpr bool fp32 = true;
    __device__ static T* r(const FusedArgs& a) { return a.r32; }
    __device__ static T* w(const FusedArgs& a) { return a.w32; }
    __device__ static T* p(const FusedArgs& a) { return a.p32[0]; }
    __device__ static T* u(const FusedArgs& a) { return a.d32; }
    __device__ static T* rhs(const FusedArgs& a) { return a.r32; }
    __device__ static const T* kx(const FusedArgs& a) { return a.kx32; }
    __device__ static const T* ky(const FusedArgs& a) { return a.ky32; }
    __device__ static const T* kz(const FusedArgs& a) { return a.kz32; }
    __device__ static const T* mi(const FusedArgs&, bool) { return nullptr; }
};

// A lane's two cells of an array (rows are padded, so the pair is always inside it).
template <class T>
__device__ __forceinline__ void ld_cells(const T* a, long i, T& x, T& y)
{
    const Two<T> v = ld_two(a + i);
    x = v.x;
    y = v.y;
}
template <class T>
__device__ __forceinline__ void st_cells(T* a, long i, bool both, T x, T y)
{
    if (both) st_two(a + i, x, y);
    else a[i] = x;
}

// A vector that the loop reads (or updates) at a warp's own cells only: u, or the right-hand
// side.  Up to four rows of it stay in registers; with more rows the two vectors that are live
// across a sum fill the registers, and it lies in shared memory where there is room, else in
// L2, from which all rows are loaded before any is stored.
template <class T, int RS, bool CL>
struct ResOwn {
    static constexpr bool kept = RS * sizeof(T) <= 32;
    T v[kept ? RS : 1][2];
    T* far;  // the array
    __device__ __forceinline__ ResOwn(const ResTile<T, RS, CL>& t, T* array) : far(array)
    {
#pragma unroll
        for (int k = 0; k < RS; ++k)
            if (t.on(k)) {
                if constexpr (kept) {
                    ld_cells(far, t.gidx(k), v[k][0], v[k][1]);
                } else if (t.A.p.ox) {
                    const Two<T> c = ld_two(far + t.gidx(k));
                    st_two(t.own(k), c.x, c.y);
                }
            }
    }
    // The rows, in `w` when they are not kept.
    __device__ __forceinline__ void load(const ResTile<T, RS, CL>& t, T (&w)[RS][2]) const
    {
        if constexpr (kept) {
#pragma unroll
            for (int k = 0; k < RS; ++k) {
                w[k][0] = v[k][0];
                w[k][1] = v[k][1];
            }
        } else {
#pragma unroll
            for (int k = 0; k < RS; ++k)
                if (t.on(k)) {
                    const Two<T> c = ld_two(t.A.p.ox ? t.own(k) : far + t.gidx(k));
                    w[k][0] = c.x;
                    w[k][1] = c.y;
                }
        }
    }
    __device__ __forceinline__ void store(const ResTile<T, RS, CL>& t, const T (&w)[RS][2])
    {
        if constexpr (kept) {
#pragma unroll
            for (int k = 0; k < RS; ++k) {
                v[k][0] = w[k][0];
                v[k][1] = w[k][1];
            }
        } else {
#pragma unroll
            for (int k = 0; k < RS; ++k)
                if (t.on(k)) {
                    if (t.A.p.ox) st_two(t.own(k), w[k][0], w[k][1]);
                    else st_cells(far, t.gidx(k), t.both(), w[k][0], w[k][1]);
                }
        }
    }
    // Back to the array at the end of a loop that updates it.
    __device__ __forceinline__ void write(const ResTile<T, RS, CL>& t) const
    {
#pragma unroll
        for (int k = 0; k < RS; ++k)
            if (t.on(k)) {
                if constexpr (kept) {
                    st_cells(far, t.gidx(k), t.both(), v[k][0], v[k][1]);
                } else if (t.A.p.ox) {
                    const Two<T> c = ld_two(t.own(k));
                    st_cells(far, t.gidx(k), t.both(), c.x, c.y);
                }
            }
    }
};

// Diagonals of the warp's cells: in registers where there is room, else formed again from the
// coefficients (four of the thirteen operations of the 2D operator).
template <class T, int RS, bool CL>
struct ResDiag {
    static constexpr bool kept = RS * sizeof(T) <= 16;
    T d[kept ? RS : 1][2];
    __device__ __forceinline__ void load(const ResTile<T, RS, CL>& t)
    {
        if constexpr (kept)
            t.sweep([&](int k, int q, const NbT<T>&, T kx0, T kx1, T ky0, T ky1, T kz0, T kz1) {
                d[k][q] = diag_k(kx0, kx1, ky0, ky1, kz0, kz1);
            });
    }
    __device__ __forceinline__ T smvp(int k, int q, const NbT<T>& nb, T kx0, T kx1, T ky0, T ky1, T kz0, T kz1) const
    {
        if constexpr (kept) return smvp_dk(d[k][q], nb, kx0, kx1, ky0, ky1, kz0, kz1);
        else return smvp_k(nb, kx0, kx1, ky0, ky1, kz0, kz1);
    }
};

// The scalars of a CG iteration after its sums, on the block's copy of the state: alpha after
// p.w; beta, the residual and the loop test after r.(r|z).  cg_note_* writes down what no
// thread waits for.
__device__ __forceinline__ bool cg_after_pw(SolveState& s, double v)
{
    s.alpha = s.rro / v;
    return true;
}
template <class P>
__device__ __forceinline__ void cg_note_pw(const FusedArgs& a, SolveState& s, double v)
{
    s.pw = v;
    if (!P::fp32 && blockIdx.x == 0) a.cg_alphas[s.n] = s.alpha;
    if (!isfinite(v)) s.nonfinite = 1;
}
template <class P>
__device__ __forceinline__ bool cg_after_rr(const FusedArgs& a, SolveState& s, double v)
{
    // The loop test first: the division's call hides what is behind it from the scheduler.
    const double rro = s.rro;
    if constexpr (P::fp32) {
        const int n = ++s.n_inner;
        const bool at_switch = s.switch_err > 0.0 && n >= s.switch_min && v <= s.switch_err;
        s.cont = isfinite(v) && v >= s.tol2 && n < s.inner_max && !at_switch;
    } else {
        s.error = v;
        end_iteration(a, s, PHASE_CG);
    }
    s.rro = v;
    s.last_beta = v / rro;
    return s.cont != 0;
}
template <class P>
__device__ __forceinline__ void cg_note_rr(const FusedArgs& a, SolveState& s, double v)
{
    // The iteration that has just ended: end_iteration steps n unless it converged.
    const int n = P::fp32 ? s.n_inner : (s.exit_reason == EXIT_CONVERGED ? s.n : s.n - 1);
    s.rrn = v;
    s.beta = s.last_beta;
    s.last_alpha = s.alpha;
    if (!isfinite(v)) s.nonfinite = 1;
    if (blockIdx.x == 0) {
        if (P::fp32) a.cg_alphas[n] = s.alpha;
        a.cg_betas[n] = s.beta;
    }
}

#define RES_PROLOGUE(P, RES_SCALE)                                                                 \
    using T = typename P::T;                                                                       \
    extern __shared__ __align__(16) unsigned char s_res_raw[];                                     \
    __shared__ ResShared<CL> sh;                                                                   \
    const FusedArgs& a = A.f;                                                                      \
    ResTile<T, RS, CL> t(A, sh, reinterpret_cast<T*>(s_res_raw));                                  \
    wait_for_previous(); /* up to here beside the launch before */                                 \
    if (threadIdx.x == 0) {                                                                        \
        sh.s = A.start ? *A.start : A.s0;                                                          \
        t.start(RES_SCALE);                                                                        \
    }                                                                                              \
    ResDiag<T, RS, CL> dg;                                                                         \
    SolveState& s = sh.s

#define RES_EPILOGUE()                                                                             \
    let_next_start();                                                                              \
    if constexpr (CL) t.leave();                                                                   \
    else __syncthreads();                                                                          \
    if (blockIdx.x == 0) {                                                                         \
        if (threadIdx.x == 0) *a.st = *A.host = s;                                                 \
        t.clear_other_set();                                                                       \
    }

// CG: per iteration p = beta p + (z|r), w = A p and p.w; u += alpha p, r -= alpha w and
// r.(r|z).  The neighbours' r arrives while the second sum is formed, and the halo of p follows
// by the same recurrence, so an iteration waits for two sums and nothing else.
template <class P, int RS, int W, bool CL>
__global__ void __launch_bounds__(32 * W, 1) k_res_cg(const __grid_constant__ ResArgs A)
{
    RES_PROLOGUE(P, sh.s.rro);
    const bool pre = !P::fp32 && A.p.pre;
    t.load_coefs(P::kx(a), P::ky(a), P::kz(a), P::mi(a, pre));
    t.load_operand(P::p(a));
    if (pre) t.load_halo_mi(P::mi(a, pre));
    T r[RS][2], w[RS][2];
    ResOwn<T, RS, CL> u(t, P::u(a));
#pragma unroll
    for (int k = 0; k < RS; ++k) {
        r[k][0] = r[k][1] = w[k][0] = w[k][1] = (T)0;
        if (t.on(k)) ld_cells(P::r(a), t.gidx(k), r[k][0], r[k][1]);
    }
    __syncthreads();
    dg.load(t);
    const int h0 = (int)threadIdx.x < t.nh ? t.table()[threadIdx.x].x : -1;
    for (bool pend = false;; pend = true) {
        if (pend) {
            const T beta = (T)s.last_beta;
            // The thread's halo cell is loaded beside its own cells.
            T hp = (T)0, hr = (T)0;
            if (h0 >= 0) {
                hp = t.V[h0];
                hr = t.halo_r(threadIdx.x);
                if (pre) hr = t.halo_mi(threadIdx.x) * hr;
            }
#pragma unroll
            for (int k = 0; k < RS; ++k)
                if (t.on(k)) {
                    const Two<T> c = ld_two(t.cell(k));
                    T q0 = r[k][0], q1 = r[k][1];
                    if (pre) {
                        const Two<T> m = t.mi_of(k);
                        q0 = m.x * q0;
                        q1 = m.y * q1;
                    }
                    t.store(k, beta * c.x + q0, beta * c.y + q1);
                }
            if (h0 >= 0) t.V[h0] = beta * hp + hr;
            for (int h = threadIdx.x + blockDim.x; h < t.nh; h += blockDim.x) {
                T q = t.halo_r(h);
                if (pre) q = t.halo_mi(h) * q;
                T* c = t.V + t.table()[h].x;
                *c = beta * *c + q;
            }
            __syncthreads();
        }
        DD acc = {0.0, 0.0};
        t.sweep([&](int k, int q, const NbT<T>& nb, T kx0, T kx1, T ky0, T ky1, T kz0, T kz1) {
            const T wv = dg.smvp(k, q, nb, kx0, kx1, ky0, ky1, kz0, kz1);
            w[k][q] = wv;
            t.add(acc, k, q, (double)wv * (double)nb.c);
        });
        if (t.reduce(
                acc, 0, [] {}, [&](double v) { return cg_after_pw(s, v); }, [&](double v) { cg_note_pw<P>(a, s, v); }) !=
            RN_GO)
            break;
        const T alpha = (T)s.alpha;
        acc.hi = acc.lo = 0.0;
        t.next_exchange();
#pragma unroll
        for (int k = 0; k < RS; ++k)
            if (t.on(k)) {
                r[k][0] = r[k][0] - alpha * w[k][0];
                r[k][1] = r[k][1] - alpha * w[k][1];
                t.publish(k, r[k][0], r[k][1]);
            }
        // w is free: it takes u.
        u.load(t, w);
#pragma unroll
        for (int k = 0; k < RS; ++k)
            if (t.on(k)) {
                const Two<T> c = ld_two(t.cell(k));
                T q0 = r[k][0], q1 = r[k][1];
                if (pre) {
                    const Two<T> m = t.mi_of(k);
                    q0 = m.x * q0;
                    q1 = m.y * q1;
                }
                t.add(acc, k, 0, (double)r[k][0] * (double)q0);
                t.add(acc, k, 1, (double)r[k][1] * (double)q1);
                w[k][0] = w[k][0] + alpha * c.x;
                w[k][1] = w[k][1] + alpha * c.y;
            }
        u.store(t, w);
        if (t.reduce(
                acc, 1, [&] { t.collect(1, [&](int h, T v) { t.halo_r(h) = v; }); },
                [&](double v) { return cg_after_rr<P>(a, s, v); }, [&](double v) { cg_note_rr<P>(a, s, v); }) != RN_GO)
            break;
    }
    __syncthreads();  // what the last sum left to be written down
    t.sweep([&](int k, int q, const NbT<T>& nb, T kx0, T kx1, T ky0, T ky1, T kz0, T kz1) {
        w[k][q] = dg.smvp(k, q, nb, kx0, kx1, ky0, ky1, kz0, kz1);
    });
    if (threadIdx.x == 0) s.pending_p = 1;
#pragma unroll
    for (int k = 0; k < RS; ++k)
        if (t.on(k)) {
            const long i = t.gidx(k);
            const Two<T> c = ld_two(t.cell(k));
            st_cells(P::p(a), i, t.both(), c.x, c.y);
            st_cells(P::r(a), i, t.both(), r[k][0], r[k][1]);
            st_cells(P::w(a), i, t.both(), w[k][0], w[k][1]);
            if constexpr (!P::fp32)
                if (pre) {
                    const Two<T> m = t.mi_of(k);
                    st_cells(a.z, i, t.both(), m.x * r[k][0], m.y * r[k][1]);
                }
        }
    u.write(t);
    RES_EPILOGUE();
}

// Chebyshev: r = rhs - A u, p = alpha p + beta (mi r | r), u += p.  Iterations between two
// checks only exchange the rim of u with the neighbouring tiles; r.r is summed where the loop
// checks it.
template <class P, int RS, int W, bool CL>
__global__ void __launch_bounds__(32 * W, 1) k_res_cheby(const __grid_constant__ ResArgs A)
{
    RES_PROLOGUE(P, P::fp32 ? sh.s.rro : sh.s.error);
    const bool pre = !P::fp32 && A.p.pre;
    t.load_coefs(P::kx(a), P::ky(a), P::kz(a), P::mi(a, pre));
    t.load_operand(P::u(a));
    T p[RS][2], un[RS][2];
    const ResOwn<T, RS, CL> b(t, P::rhs(a));
    // Where the rows of the right-hand side do not stay in registers beside p and the new u, the
    // sweep works in place, and un holds them for the whole loop.
    constexpr bool OVER = DIM == 2 && !ResOwn<T, RS, CL>::kept && W > 12;
#pragma unroll
    for (int k = 0; k < RS; ++k) {
        p[k][0] = p[k][1] = un[k][0] = un[k][1] = (T)0;
        if (t.on(k)) ld_cells(P::p(a), t.gidx(k), p[k][0], p[k][1]);
    }
    __syncthreads();
    dg.load(t);
    if constexpr (OVER) b.load(t, un);
    for (;;) {
        const int step = P::fp32 ? s.n_inner - 1 : s.cheby_calc_steps - 1;
        const T al = (T)a.ch_alphas[step], be = (T)a.ch_betas[step];
        const bool check = P::fp32 ? s.n_inner % 10 == 0 : (s.n >= s.est_itc && s.n % 10 == 0);
        DD acc = {0.0, 0.0};
        t.next_exchange();
        Two<T> m;
        m.x = m.y = (T)1;
        auto cell = [&](int k, int q, const NbT<T>& nb, T kx0, T kx1, T ky0, T ky1, T kz0, T kz1) {
            const T wv = dg.smvp(k, q, nb, kx0, kx1, ky0, ky1, kz0, kz1);
            const T rv = un[k][q] - wv;
            const T pv = al * p[k][q] + be * (pre ? (q == 0 ? m.x : m.y) * rv : rv);
            p[k][q] = pv;
            if (check && (!OVER || t.on(k))) t.add(acc, k, q, (double)rv * (double)rv);
            return nb.c + pv;
        };
        if constexpr (OVER) {
            const auto e = t.around();
            __syncthreads();  // every warp has read the old operand around its rows, and the state
            t.sweep_over(e, [&](int k, const Two<T>&, const NbT<T>& nb0, const NbT<T>& nb1, T kx0, T kx1, T kx2,
                                const Two<T>& ky0, const Two<T>& ky1, Two<T>& out) {
                if (pre && t.on(k)) m = t.mi_of(k);
                out.x = cell(k, 0, nb0, kx0, kx1, ky0.x, ky1.x, (T)0, (T)0);
                out.y = cell(k, 1, nb1, kx1, kx2, ky0.y, ky1.y, (T)0, (T)0);
            });
        } else {
            b.load(t, un);
            t.sweep([&](int k, int q, const NbT<T>& nb, T kx0, T kx1, T ky0, T ky1, T kz0, T kz1) {
                if (q == 0 && pre) m = t.mi_of(k);
                un[k][q] = cell(k, q, nb, kx0, kx1, ky0, ky1, kz0, kz1);
            });
#pragma unroll
            for (int k = 0; k < RS; ++k)
                if (t.on(k)) t.publish(k, un[k][0], un[k][1]);
            __syncthreads();  // every warp has read the old operand and the state
#pragma unroll
            for (int k = 0; k < RS; ++k)
                if (t.on(k)) t.store(k, un[k][0], un[k][1]);
        }
        auto halo = [&](int first) { t.collect(first, [&](int h, T v) { t.V[t.table()[h].x] = v; }); };
        auto finish = [&](double v) {
            if constexpr (P::fp32) {
                s.n_inner = s.n_inner + 1;
                OpCheby32::finish(a, s, check, v);
            } else {
                if (check) s.error = v;
                s.cheby_calc_steps = s.cheby_calc_steps + 1;
                end_iteration(a, s, PHASE_CHEBY);
            }
            return s.cont != 0;
        };
        int next;
        if (check) {
            next = t.reduce(acc, 0, [&] { halo(t.nw > 1 ? 1 : 0); }, finish, [](double) {});
        } else {
            if (threadIdx.x == 0) sh.sum.next = finish(0.0) ? RN_GO : RN_STOP;
            halo(0);
            next = t.finish();
        }
        if (next != RN_GO) break;
    }
    // Where CG takes over again it needs the last residual, which is not kept: the arrays stay as they
    // were, and the host runs the iterations again by the per-call kernels (restore_residual).
    if (P::fp32 || s.exit_reason != EXIT_PHASE) {
#pragma unroll
        for (int k = 0; k < RS; ++k)
            if (t.on(k)) {
                const Two<T> c = ld_two(t.cell(k));
                st_cells(P::u(a), t.gidx(k), t.both(), c.x, c.y);
                st_cells(P::p(a), t.gidx(k), t.both(), p[k][0], p[k][1]);
            }
    }
    RES_EPILOGUE();
}

// PPCG without the preconditioner: the CG sweep on p, then the inner steps on sd, each with
// one rim exchange; V holds p and then sd.
template <class P, int RS, int W, bool CL>
__global__ void __launch_bounds__(32 * W, 1) k_res_ppcg(const __grid_constant__ ResArgs A)
{
    RES_PROLOGUE(P, sh.s.rro);
    t.load_coefs(P::kx(a), P::ky(a), P::kz(a), nullptr);
    t.load_operand(P::p(a));
    constexpr bool PREG = RS * sizeof(T) <= 16;  // p waits in registers, else in its array, for the next outer iteration
    // Where u does not stay in registers beside r and w, the inner steps work in place, and w holds u
    // for all of them.
    constexpr bool OVER = DIM == 2 && !ResOwn<T, RS, CL>::kept && W > 12;
    T r[RS][2], w[RS][2], p[PREG ? RS : 1][2];
    ResOwn<T, RS, CL> u(t, P::u(a));
#pragma unroll
    for (int k = 0; k < RS; ++k) {
        r[k][0] = r[k][1] = w[k][0] = w[k][1] = (T)0;
        if (t.on(k)) {
            ld_cells(P::r(a), t.gidx(k), r[k][0], r[k][1]);
            if constexpr (PREG) ld_cells(P::p(a), t.gidx(k), p[k][0], p[k][1]);
        }
    }
    auto set_operand = [&](int k, T v0, T v1) {
        t.store(k, v0, v1);
        t.publish(k, v0, v1);
    };
    auto exchange = [&] {
        t.collect(0, [&](int h, T v) { t.V[t.table()[h].x] = v; });
        return t.finish();
    };
    __syncthreads();
    dg.load(t);
    const int inner = s.inner_steps;
    bool lost = false;
    for (bool pend = false;; pend = true) {
        if (pend) {
            const T beta = (T)s.last_beta;
            t.next_exchange();
            if constexpr (PREG) {
#pragma unroll
                for (int k = 0; k < RS; ++k) {
                    w[k][0] = p[k][0];
                    w[k][1] = p[k][1];
                }
            } else {
#pragma unroll
                for (int k = 0; k < RS; ++k)
                    if (t.on(k)) ld_cells(P::p(a), t.gidx(k), w[k][0], w[k][1]);
            }
#pragma unroll
            for (int k = 0; k < RS; ++k)
                if (t.on(k)) {
                    w[k][0] = beta * w[k][0] + r[k][0];
                    w[k][1] = beta * w[k][1] + r[k][1];
                    set_operand(k, w[k][0], w[k][1]);
                    if constexpr (PREG) {
                        p[k][0] = w[k][0];
                        p[k][1] = w[k][1];
                    } else {
                        st_cells(P::p(a), t.gidx(k), t.both(), w[k][0], w[k][1]);
                    }
                }
            if (exchange() != RN_GO) break;
        }
        DD acc = {0.0, 0.0};
        t.sweep([&](int k, int q, const NbT<T>& nb, T kx0, T kx1, T ky0, T ky1, T kz0, T kz1) {
            const T wv = dg.smvp(k, q, nb, kx0, kx1, ky0, ky1, kz0, kz1);
            w[k][q] = wv;
            t.add(acc, k, q, (double)wv * (double)nb.c);
        });
        if (t.reduce(
                acc, 0, [] {}, [&](double v) { return cg_after_pw(s, v); },
                [&](double v) {
                    s.pw = v;
                    if (!P::fp32 && blockIdx.x == 0) a.cg_alphas[s.n] = s.alpha;
                    if (!isfinite(v)) s.nonfinite = 1;
                }) != RN_GO)
            break;
        const T alpha = (T)s.alpha, theta = (T)s.theta;
        t.next_exchange();
#pragma unroll
        for (int k = 0; k < RS; ++k)
            if (t.on(k)) {
                r[k][0] = r[k][0] - alpha * w[k][0];
                r[k][1] = r[k][1] - alpha * w[k][1];
            }
        u.load(t, w);
#pragma unroll
        for (int k = 0; k < RS; ++k)
            if (t.on(k)) {
                const Two<T> c = ld_two(t.cell(k));
                w[k][0] = w[k][0] + alpha * c.x;
                w[k][1] = w[k][1] + alpha * c.y;
            }
        if constexpr (!OVER) u.store(t, w);
#pragma unroll
        for (int k = 0; k < RS; ++k)
            if (t.on(k)) set_operand(k, r[k][0] / theta, r[k][1] / theta);
        if (exchange() != RN_GO) break;
        acc.hi = acc.lo = 0.0;
        for (int m = 1; m <= inner; ++m) {
            const T al = (T)a.ch_alphas[m - 1], be = (T)a.ch_betas[m - 1];
            const bool last = m == inner;
            if constexpr (OVER) {
                if (!last) {
                    const auto e = t.around();
                    __syncthreads();  // every warp has read the old sd around its rows
                    t.next_exchange();
                    t.sweep_over(e, [&](int k, const Two<T>& c, const NbT<T>& nb0, const NbT<T>& nb1, T kx0, T kx1, T kx2,
                                        const Two<T>& ky0, const Two<T>& ky1, Two<T>& out) {
                        w[k][0] = w[k][0] + c.x;
                        w[k][1] = w[k][1] + c.y;
                        r[k][0] = r[k][0] - dg.smvp(k, 0, nb0, kx0, kx1, ky0.x, ky1.x, (T)0, (T)0);
                        r[k][1] = r[k][1] - dg.smvp(k, 1, nb1, kx1, kx2, ky0.y, ky1.y, (T)0, (T)0);
                        out.x = al * c.x + be * r[k][0];
                        out.y = al * c.y + be * r[k][1];
                    });
                    if (exchange() != RN_GO) {
                        lost = true;
                        break;
                    }
                    continue;
                }
            } else {
                // u += sd first: its rows pass through w, which then takes the new sd.
                u.load(t, w);
            }
#pragma unroll
            for (int k = 0; k < RS; ++k)
                if (t.on(k)) {
                    const Two<T> c = ld_two(t.cell(k));
                    w[k][0] = w[k][0] + c.x;
                    w[k][1] = w[k][1] + c.y;
                }
            u.store(t, w);
            t.sweep([&](int k, int q, const NbT<T>& nb, T kx0, T kx1, T ky0, T ky1, T kz0, T kz1) {
                const T rv = r[k][q] - dg.smvp(k, q, nb, kx0, kx1, ky0, ky1, kz0, kz1);
                r[k][q] = rv;
                if constexpr (!OVER) w[k][q] = al * nb.c + be * rv;
                if (last) t.add(acc, k, q, (double)rv * (double)rv);
            });
            if (last) break;
            __syncthreads();  // every warp has read the old sd
            t.next_exchange();
#pragma unroll
            for (int k = 0; k < RS; ++k)
                if (t.on(k)) set_operand(k, w[k][0], w[k][1]);
            if (exchange() != RN_GO) {
                lost = true;
                break;
            }
        }
        if (lost) break;
        if (t.reduce(
                acc, 1, [] {},
                [&](double v) {
                    s.last_beta = v / s.rro;
                    s.rro = v;
                    if constexpr (P::fp32) {
                        s.n_inner = s.n_inner + 1;
                        if (!isfinite(v)) s.inner_diverged = 1;  // the correction is dropped; CG takes over
                        s.cont = isfinite(v) && v >= s.tol2 && s.n_inner < s.inner_max;
                    } else {
                        s.error = v;
                        s.cheby_calc_steps = s.cheby_calc_steps + 1;
                        end_iteration(a, s, PHASE_PPCG);
                    }
                    return s.cont != 0;
                },
                [&](double v) {
                    s.rrn = v;
                    s.beta = s.last_beta;
                    if (!P::fp32 && !isfinite(v)) s.nonfinite = 1;
                }) != RN_GO)
            break;
    }
    __syncthreads();  // what the last sum left to be written down
    if (threadIdx.x == 0) {
        s.pending_p = 1;
        s.pending_u = 0;
    }
#pragma unroll
    for (int k = 0; k < RS; ++k)
        if (t.on(k)) {
            const long i = t.gidx(k);
            st_cells(P::r(a), i, t.both(), r[k][0], r[k][1]);
            if constexpr (PREG) st_cells(P::p(a), i, t.both(), p[k][0], p[k][1]);
        }
    u.write(t);
    RES_EPILOGUE();
}

// Jacobi: u_new = (rhs + sum K u) / diagonal and sum |u_new - u|; every 50th iteration the
// true residual instead.
template <class P, int RS, int W, bool CL>
__global__ void __launch_bounds__(32 * W, 1) k_res_jacobi(const __grid_constant__ ResArgs A)
{
    RES_PROLOGUE(P, sh.s.error);
    t.load_coefs(a.kx, a.ky, a.kz, nullptr);
    t.load_operand(a.u[0]);
    T un[RS][2];
    const ResOwn<T, RS, CL> b(t, a.u0);
#pragma unroll
    for (int k = 0; k < RS; ++k) un[k][0] = un[k][1] = (T)0;
    __syncthreads();
    dg.load(t);
    for (;;) {
        const bool residual = s.n % 50 == 0;
        DD acc = {0.0, 0.0};
        t.next_exchange();
        b.load(t, un);
        t.sweep([&](int k, int q, const NbT<T>& nb, T kx0, T kx1, T ky0, T ky1, T kz0, T kz1) {
            const T v = jacobi_k(un[k][q], nb, kx0, kx1, ky0, ky1, kz0, kz1);
            un[k][q] = v;
            t.add(acc, k, q, fabs(v - nb.c));
        });
#pragma unroll
        for (int k = 0; k < RS; ++k)
            if (t.on(k)) t.publish(k, un[k][0], un[k][1]);
        __syncthreads();  // every warp has read the old operand and the state
#pragma unroll
        for (int k = 0; k < RS; ++k)
            if (t.on(k)) t.store(k, un[k][0], un[k][1]);
        int next = t.reduce(
            acc, 0, [&] { t.collect(t.nw > 1 ? 1 : 0, [&](int h, T v) { t.V[t.table()[h].x] = v; }); },
            [&](double v) {
                s.error = v;
                if (!residual) end_iteration(a, s, PHASE_JACOBI);
                return residual || s.cont != 0;
            },
            [](double) {});
        if (next != RN_GO) break;
        if (residual) {
            acc.hi = acc.lo = 0.0;
            b.load(t, un);
            t.sweep([&](int k, int q, const NbT<T>& nb, T kx0, T kx1, T ky0, T ky1, T kz0, T kz1) {
                un[k][q] = un[k][q] - dg.smvp(k, q, nb, kx0, kx1, ky0, ky1, kz0, kz1);
                t.add(acc, k, q, un[k][q] * un[k][q]);
            });
#pragma unroll
            for (int k = 0; k < RS; ++k)
                if (t.on(k)) st_cells(a.r, t.gidx(k), t.both(), un[k][0], un[k][1]);
            next = t.reduce(
                acc, 1, [] {},
                [&](double v) {
                    s.error = v;
                    end_iteration(a, s, PHASE_JACOBI);
                    return s.cont != 0;
                },
                [](double) {});
            if (next != RN_GO) break;
        }
    }
#pragma unroll
    for (int k = 0; k < RS; ++k)
        if (t.on(k)) {
            const Two<T> c = ld_two(t.cell(k));
            st_cells(a.u[0], t.gidx(k), t.both(), c.x, c.y);
        }
    RES_EPILOGUE();
}

}  // namespace tea
