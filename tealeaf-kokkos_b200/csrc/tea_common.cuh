// Shared device-side infrastructure of the TeaLeaf B200 library: the field layout in
// HBM, the tile walk used by the per-call kernels, and the deterministic double-double
// grid reduction.  Compiled into both libtea2d_b200.so and libtea3d_b200.so
// (-DTEA_DIM=2 / -DTEA_DIM=3).  Build with -fmad=false: every multiply and add is
// rounded separately, exactly as the reference's C++ (and the oracle) evaluate them.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#ifndef TEA_DIM
#error "compile with -DTEA_DIM=2 or -DTEA_DIM=3"
#endif

namespace tea {

constexpr int DIM = TEA_DIM;
constexpr int HALO_PAD = 2;
// Field layout: element (kk, jj, ii) of a padded array (kk in [0, nx+4) etc., the
// reference's flat index kk + jj*X + ii*X*Y) lives at f[kk + jj*pitch + ii*page] with
// pitch = roundup(nx+4, 32) doubles and f = allocation + kLeadPad, so the first inner
// cell of every row (kk = 2) starts on a 256-byte boundary.
constexpr int kLeadPad = 30;
constexpr int kPitchAlign = 32;

// Per-call kernels walk the inner domain in 32 x 8 tiles (one z-plane per tile in 3D).
constexpr int TILE_X = 32;
constexpr int TILE_Y = 8;
constexpr int BLOCK = TILE_X * TILE_Y;
constexpr int MAX_RED = 4;  // values per reduction (field summary needs 4)

struct Geom {
    int nx, ny, nz;     // inner cells (nz = 1 in 2D)
    int X, Y, Z;        // padded extents (Z = 1 in 2D)
    long pitch, page;   // elements
    int tiles_x, tiles_y;
    long tiles_inner;   // tiles covering the inner domain
    int ftiles_x, ftiles_y;
    long tiles_full;    // tiles covering the whole padded array
};

__host__ __device__ inline long fidx(const Geom& g, int kk, int jj, int ii)
{
    return (long)kk + (long)jj * g.pitch + (long)ii * g.page;
}

// A launch with programmatic stream serialization may start before the launch in front of it has
// ended: once all its blocks have called let_next_start().  wait_for_previous() waits for its end;
// nothing it leaves is read, and nothing it uses is written, before that.
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ------------------------------------------------------------------ double-double sums

struct DD {
    double hi, lo;
};

// Knuth's TwoSum accumulation (cascaded summation): hi + lo carries the running sum to
// about twice the working precision, so the final hi + lo is the correctly rounded sum
// except within ~n*2^-106 of a rounding boundary, independent of the summation order.
__device__ __forceinline__ void dd_add(DD& a, double x)
{
    const double s = a.hi + x;
    const double bp = s - a.hi;
    const double e = (a.hi - (s - bp)) + (x - bp);
    a.hi = s;
    a.lo = a.lo + e;
}

__device__ __forceinline__ DD dd_merge(DD a, DD b)
{
    const double s = a.hi + b.hi;
    const double bp = s - a.hi;
    const double e = (a.hi - (s - bp)) + (b.hi - bp);
    DD r;
    r.hi = s;
    r.lo = (a.lo + b.lo) + e;
    return r;
}

__device__ __forceinline__ double dd_value(DD a) { return a.hi + a.lo; }

template <int NV>
struct DDVec {
    DD v[NV];
    __device__ __forceinline__ void zero()
    {
#pragma unroll
        for (int k = 0; k < NV; ++k) v[k].hi = v[k].lo = 0.0;
    }
};

// Grid reduction scratch: one DD per value per block, and an arrival counter.
struct RedScratch {
    DD* partials;           // [max_blocks * MAX_RED]
    unsigned int* counter;  // reset to 0 by the last block
    int max_blocks;
    unsigned long long* done;   // host memory: takes a word pair per result under `ticket` (null: none)
    unsigned long long ticket;
};

// A result for a host that polls: the value's bits and, in the same 16-byte store, a word that says
// which launch they belong to.  No fence orders anything: a pair of which the host sees only one half
// does not pass posted().
__host__ __device__ inline unsigned long long post_check(unsigned long long bits, unsigned long long ticket)
{
    return bits ^ (ticket * 0x9E3779B97F4A7C15ull);
}
__device__ __forceinline__ void post_result(unsigned long long* to, double v, unsigned long long ticket)
{
    const unsigned long long bits = (unsigned long long)__double_as_longlong(v);
    asm volatile("st.volatile.global.v2.u64 [%0], {%1, %2};" ::"l"(to), "l"(bits), "l"(post_check(bits, ticket)) : "memory");
}

template <int NV>
__device__ __forceinline__ void warp_merge(DDVec<NV>& a)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            DD b;
            b.hi = __shfl_xor_sync(0xffffffffu, a.v[k].hi, o);
            b.lo = __shfl_xor_sync(0xffffffffu, a.v[k].lo, o);
            a.v[k] = dd_merge(a.v[k], b);
        }
    }
}

// Merge over a block: butterflies in the warps, then over the warps' values in warp 0, through `s`
// (nwarps x NV, shared).  Called by every thread; the result is valid in warp 0.
template <int NV>
__device__ __forceinline__ DDVec<NV> block_merge(DDVec<NV> a, DD* s, int tid, int nwarps)
{
    const int lane = tid & 31, warp = tid >> 5;
    warp_merge<NV>(a);
    if (nwarps == 1) return a;
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) s[warp * NV + k] = a.v[k];
    }
    __syncthreads();
    if (warp == 0) {
        a.zero();
        if (lane < nwarps) {
#pragma unroll
            for (int k = 0; k < NV; ++k) a.v[k] = s[lane * NV + k];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            if (o >= nwarps) continue;
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                DD b;
                b.hi = __shfl_xor_sync(0xffffffffu, a.v[k].hi, o);
                b.lo = __shfl_xor_sync(0xffffffffu, a.v[k].lo, o);
                a.v[k] = dd_merge(a.v[k], b);
            }
        }
    }
    return a;
}

// The sum over the grid, valid in thread 0 of the block for which `last` comes back true (the last
// to arrive, which merges the blocks' partials).  The order depends only on the grid and block
// sizes; no block waits on another.  Called by every thread of the block.
//
// At the per-call kernels' sizes this tail is latency from end to end: with serial merges by one
// thread (the warps' values, twice), a fence on either side of the arrival and one more before the
// host's word a reduction took 2 us longer (ext_cg_calc_w_, call to result: 14.5 us on 10 x 10
// cells and 14.8 at 512 x 512, now 12.6 and 12.7).
template <int NV>
__device__ __forceinline__ DDVec<NV> grid_merge(const DDVec<NV>& acc, const RedScratch& rs, DD* s, int tid, int nwarps,
                                                bool& last)
{
    __shared__ bool s_last;
    DDVec<NV> b = block_merge<NV>(acc, s, tid, nwarps);
    const int nblk = (int)gridDim.x;
    last = true;
    if (nblk == 1) return b;
    if (tid == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) rs.partials[(long)blockIdx.x * MAX_RED + k] = b.v[k];
        unsigned int prev;
        asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(prev) : "l"(rs.counter) : "memory");
        s_last = prev == (unsigned)nblk - 1;
    }
    __syncthreads();
    last = s_last;
    if (!last) return b;
    // Every thread merges a strided share of the partials, four loads in flight.
    const int nthreads = nwarps * 32;
    b.zero();
    for (int blk0 = tid; blk0 < nblk; blk0 += 4 * nthreads) {
        DD p[4][NV];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int blk = blk0 + u * nthreads;
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                p[u][k].hi = blk < nblk ? __ldcg(&rs.partials[(long)blk * MAX_RED + k].hi) : 0.0;
                p[u][k].lo = blk < nblk ? __ldcg(&rs.partials[(long)blk * MAX_RED + k].lo) : 0.0;
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (u > 0 && blk0 + u * nthreads >= nblk) break;
#pragma unroll
            for (int k = 0; k < NV; ++k) b.v[k] = dd_merge(b.v[k], p[u][k]);
        }
    }
    if (tid == 0) *rs.counter = 0u;
    return block_merge<NV>(b, s, tid, nwarps);
}

// Reduce over the grid; the last block writes the rounded results to out[0..NV), or posts them to
// the host where it waits for them.  Must be called by every thread of the block.
template <int NV>
__device__ void grid_reduce(DDVec<NV> acc, const RedScratch& rs, double* out)
{
    __shared__ DD s_warp[BLOCK / 32][NV];
    const int tid = threadIdx.x + threadIdx.y * blockDim.x;
    bool last;
    const DDVec<NV> b = grid_merge<NV>(acc, rs, &s_warp[0][0], tid, (blockDim.x * blockDim.y) >> 5, last);
    if (last && tid == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            if (rs.done) post_result(rs.done + 2 * k, dd_value(b.v[k]), rs.ticket);
            else out[k] = dd_value(b.v[k]);
        }
    }
}

// As grid_reduce, but the last block's lane 0 hands the rounded values to `f` (the
// solver's scalar recurrence and loop control run there, with every other block done).
template <int NV, class F>
__device__ void grid_reduce_then(DDVec<NV> acc, const RedScratch& rs, F&& f)
{
    __shared__ DD s_warp2[32][NV];
    const int tid = threadIdx.x + threadIdx.y * blockDim.x;
    bool last;
    const DDVec<NV> b = grid_merge<NV>(acc, rs, &s_warp2[0][0], tid, (blockDim.x * blockDim.y) >> 5, last);
    if (last && tid == 0) {
        double vals[NV];
#pragma unroll
        for (int k = 0; k < NV; ++k) vals[k] = dd_value(b.v[k]);
        f(vals);
    }
}

}  // namespace tea
