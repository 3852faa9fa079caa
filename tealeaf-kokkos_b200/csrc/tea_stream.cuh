// The CG loop of grids that do not fit on the chip, as one cooperative launch.
//
// What bounds it.  Each of the two sweeps of a CG iteration streams the fields from HBM, and as
// launches of their own (k_ring2d / k_ring3d<OpSweepA> and k_cg_sweep_b) they spend 15 us of an
// iteration on what is not streaming: launch, the read of the state, filling the rings, and
// the reduction's last block.  That is a fifth of an iteration at 2048^2 and a third at 1400^2.
// Here one block per SM stays for the whole loop, the sums go through the counted words of
// tea_resident.cuh (GridSum), and every block runs the scalar recurrence itself.
//
// Sweep A streams as k_ring2d and k_ring3d do (cp.async rings; strips of 32 lanes x 16 bytes,
// in 3D 4-row tiles marching through z).  Sweep B takes the same cells back to front, so
// that the last rows of r and w that sweep A touched are still in L2 (126 MB), and the next sweep
// A meets the rows of r that sweep B touched last; a thread's w and r of sweep B are the ones it
// wrote itself, so only the second sum has to make writes visible.
//
// u is updated on every second iteration only, by two steps at once from the two p buffers
// (u = (u + alpha' p') + alpha p, the operations and the order of two single updates): 7.5 words
// per cell of sweep A instead of 8 (2D), 8.5 instead of 9 (3D).
//
// Measured per CG iteration, launches of their own -> this kernel (HBM time of 10.5 / 11.5 words
// at the copy peak): 1400^2 41 -> 25.7 us, 2047x2049 78.7 -> 59.3 (53.8), 4096^2 264.5 -> 226 (215),
// 256^3 294 -> 274 (236), 512^3 2260 -> 2210 (1887); FP32: 2047x2049 47.9 -> 30.5, 4096^2 138 -> 119,
// 256^3 154 -> 148, 320^3 344 -> 325; larger 3D FP32 grids keep the launches.  12 warps of 3 rows in flight beat 10 x 4, 14 x 2 and 16 x 2
// (2D, 227 us against 245, 229 and 239 at 4096^2); three groups of 4-row tiles two planes ahead
// beat 4 x 4 rows x 1 plane, 2 x 6 x 2, 2 x 8 x 1 and 1 x 12 x 2 (3D, 279 us against 339, 291, 321
// and 289 at 256^3).  Deeper rings where u is not updated and eight rows of sweep B in flight
// instead of four made no difference or spilled.
#pragma once

#include "tea_resident.cuh"

namespace tea {

struct StreamArgs {
    FusedArgs f;
    const SolveState* start;  // as in ResArgs
    SolveState s0;
    SolveState* host;
    SumArgs sum;
    int seg;        // rows (2D) or planes (3D) of a work unit
};

#if TEA_DIM == 2
constexpr int ST_WARPS = 12;  // independent warps of a block
constexpr int ST_RP = 3;      // rows in flight beyond row j + 1
#else
constexpr int ST_TY = 4;      // rows of a tile: a group of 4 warps marches through its planes
constexpr int ST_GROUPS = 3;  // independent groups of a block
constexpr int ST_WARPS = ST_TY * ST_GROUPS;
constexpr int ST_RP = 2;      // planes in flight beyond plane z + 1
constexpr long ST_FP32_CELLS = 40000000;  // most cells of the FP32 loop
#endif

constexpr int ST_BACK = 4;  // rows (planes) of sweep B that a thread has in flight

// Arrays of a ring row or slot.
enum { ST_P = 0, ST_Q = 1, ST_KX = 2, ST_KY = 3, ST_U = 4, ST_OLD = 5 };

// A warp's (2D) or group's (3D) ring, as large as the sweeps that update u need it.
template <class T>
struct StreamRing {
#if TEA_DIM == 2
    static constexpr int parts = ST_WARPS, rows = (ST_RP + 2) * 6;
#else
    static constexpr int parts = ST_GROUPS, rows = (ST_RP + 2) * (2 * (ST_TY + 2) + 5 * ST_TY + 1);
#endif
    static constexpr int elems = rows * RingGeom<T>::WIDTH;
    static constexpr size_t bytes = (size_t)parts * elems * sizeof(T) + 16;  // of which ring_start() leaves 0 or 16
    static_assert(RingGeom<T>::WIDTH * sizeof(T) % 32 == 0 && RingGeom<T>::OFF * sizeof(T) == 16, "see ring_start");
};

// One iteration's operands: p and the new p's buffer (which holds the p before), q = z or r
// (null before the first update of p), and what is done to u.
template <class T>
struct StreamStep {
    const T* p;
    T* pn;
    const T* q;
    T* u;
    T beta, a_old, a_last;  // where u is updated: u = (u + a_old pn) + a_last p
};

template <class T>
__device__ __forceinline__ void stream_store(T* a, long i, int n, const T* v)
{
    constexpr int VEC = RingGeom<T>::VEC;
    if (n >= VEC) {
        st_vec(a + i, v);
    } else {
#pragma unroll
        for (int q = 0; q < VEC; ++q)
            if (q < n) a[i + q] = v[q];
    }
}

// A lane's cells of one row in sweep A: the staged operand's neighbours and the coefficients in
// cv/mv/pv/..., p and the old p as they were.  Stores w, the new p and (when due) u.
template <class P, bool UPD, class T = typename P::T>
__device__ __forceinline__ void stream_cells(const FusedArgs& a, const StreamStep<T>& st, long i, int n, const T* cv,
                                             const T* w, const T* praw, const T* uv, const T* old, DD& acc)
{
    constexpr int VEC = RingGeom<T>::VEC;
#pragma unroll
    for (int q = 0; q < VEC; ++q) dd_add(acc, q < n ? (double)w[q] * (double)cv[q] : 0.0);
    if (n <= 0) return;
    stream_store(st.pn, i, n, cv);
    stream_store(P::w(a), i, n, w);
    if constexpr (UPD) {
        T un[VEC];
#pragma unroll
        for (int q = 0; q < VEC; ++q) un[q] = (uv[q] + st.a_old * old[q]) + st.a_last * praw[q];
        stream_store(st.u, i, n, un);
    }
}

#if TEA_DIM == 2

// Sweep A of a warp's strips: p = beta p + q, w = A p, p.w; rows j0 - 1 .. j1 of a segment go
// through a ring of RP + 2 rows.
template <class P, bool UPD, class T = typename P::T>
__device__ __forceinline__ void stream_sweep_a(const StreamArgs& A, const StreamStep<T>& st, T* ring, int gw, int nwarps,
                                               DD& acc)
{
    constexpr int VEC = RingGeom<T>::VEC, STRIP = RingGeom<T>::STRIP, OFF = RingGeom<T>::OFF, RWT = RingGeom<T>::WIDTH;
    constexpr int RP = ST_RP, RQ = RP + 2, NA = UPD ? 6 : 4;
    const FusedArgs& a = A.f;
    const Geom& g = a.g;
    const int lane = threadIdx.x & 31;
    const int xlast = g.X - HALO_PAD - 1, ylast = g.Y - HALO_PAD - 1;
    const int per_x = (g.nx + STRIP - 1) / STRIP;
    const int nseg = per_x * ((g.ny + A.seg - 1) / A.seg);
    const int cmax = (int)g.pitch - 2 * VEC + 2;  // copies stay inside the row
    const T* __restrict__ KX = P::kx(a);
    const T* __restrict__ KY = P::ky(a);
    const bool pend = st.q != nullptr;
    for (int sgi = gw; sgi < nseg; sgi += nwarps) {
        const int xs = sgi % per_x, ys = sgi / per_x;
        const int c0 = HALO_PAD + STRIP * xs, c = c0 + VEC * lane, cc = min(c, cmax);
        const int n = xlast - c + 1;  // the lane's inner cells (VEC or more: all)
        const int j0 = HALO_PAD + A.seg * ys, j1 = min(j0 + A.seg, ylast + 1);
        const int left = refl(c0 - 1, g.X), right_op = refl(min(c0 + STRIP, xlast + 1), g.X);
        const int right_k = min(c0 + STRIP, xlast + 1);
        auto slot = [&](int r) { return ring + ((r - j0 + 1) % RQ) * NA * RWT; };
        auto issue = [&](int r) {
            if (r <= j1) {
                T* base = slot(r);
                const long os = (long)refl(min(max(r, 1), ylast + 1), g.Y) * g.pitch;
                const long oi = (long)min(max(r, HALO_PAD), ylast + 1) * g.pitch;
                T* d = base + OFF + VEC * lane;
                cp_async_16(d + ST_P * RWT, st.p + os + cc);
                if (pend) cp_async_16(d + ST_Q * RWT, st.q + os + cc);
                cp_async_16(d + ST_KX * RWT, KX + oi + cc);
                cp_async_16(d + ST_KY * RWT, KY + oi + cc);
                if (UPD && r >= j0 && r < j1) {
                    cp_async_16(d + ST_U * RWT, st.u + oi + cc);
                    cp_async_16(d + ST_OLD * RWT, st.pn + oi + cc);
                }
                if (lane == 0) {
                    ring_copy_one(base + ST_P * RWT + OFF - 1, st.p + os + left);
                    if (pend) ring_copy_one(base + ST_Q * RWT + OFF - 1, st.q + os + left);
                }
                if (lane == 31) {
                    ring_copy_one(base + ST_P * RWT + OFF + STRIP, st.p + os + right_op);
                    if (pend) ring_copy_one(base + ST_Q * RWT + OFF + STRIP, st.q + os + right_op);
                    ring_copy_one(base + ST_KX * RWT + OFF + STRIP, KX + oi + right_k);
                }
            }
            cp_async_commit();
        };
        auto stage = [&](T p, T q) { return pend ? st.beta * p + q : p; };
        auto stage_row = [&](int r, T* v, T& ve) {
            const T* base = slot(r);
            T x[VEC], y[VEC];
            ld_vec(base + ST_P * RWT + OFF + VEC * lane, x);
            ld_vec(base + ST_Q * RWT + OFF + VEC * lane, y);
            const int e = lane == 0 ? OFF - 1 : OFF + STRIP;
#pragma unroll
            for (int q = 0; q < VEC; ++q) v[q] = stage(x[q], y[q]);
            ve = stage(base[ST_P * RWT + e], base[ST_Q * RWT + e]);
        };
        for (int r = j0 - 1; r <= j0 + RP; ++r) issue(r);
        cp_async_wait<RP>();
        __syncwarp();
        T mv[VEC], cv[VEC], ce;
        stage_row(j0 - 1, mv, ce);
        stage_row(j0, cv, ce);
        for (int j = j0; j < j1; ++j) {
            cp_async_wait<RP - 1>();
            __syncwarp();
            T pv[VEC], pe;
            stage_row(j + 1, pv, pe);
            const T* cur = slot(j);
            const T* nxt = slot(j + 1);
            const T up = __shfl_up_sync(0xffffffffu, cv[VEC - 1], 1);
            const T dn = __shfl_down_sync(0xffffffffu, cv[0], 1);
            T kx[VEC + 1], ky0[VEC], ky1[VEC], praw[VEC], uv[VEC], old[VEC], w[VEC];
            ld_vec(cur + ST_KX * RWT + OFF + VEC * lane, kx);
            const T kxn = __shfl_down_sync(0xffffffffu, kx[0], 1);
            kx[VEC] = lane == 31 ? cur[ST_KX * RWT + OFF + STRIP] : kxn;
            ld_vec(cur + ST_KY * RWT + OFF + VEC * lane, ky0);
            ld_vec(nxt + ST_KY * RWT + OFF + VEC * lane, ky1);
            ld_vec(cur + ST_P * RWT + OFF + VEC * lane, praw);
            if constexpr (UPD) {
                ld_vec(cur + ST_U * RWT + OFF + VEC * lane, uv);
                ld_vec(cur + ST_OLD * RWT + OFF + VEC * lane, old);
            }
#pragma unroll
            for (int q = 0; q < VEC; ++q) {
                NbT<T> nb;
                nb.c = cv[q];
                nb.xm = q == 0 ? (lane == 0 ? ce : up) : cv[q > 0 ? q - 1 : 0];
                nb.xp = c + q == xlast ? cv[q] : (q == VEC - 1 ? (lane == 31 ? ce : dn) : cv[q < VEC - 1 ? q + 1 : q]);
                nb.ym = mv[q];
                nb.yp = pv[q];
                nb.zm = nb.zp = (T)0;
                w[q] = smvp_k(nb, kx[q], kx[q + 1], ky0[q], ky1[q], (T)0, (T)0);
            }
            stream_cells<P, UPD>(a, st, fidx(g, c, j, 0), n, cv, w, praw, uv, old, acc);
#pragma unroll
            for (int q = 0; q < VEC; ++q) {
                mv[q] = cv[q];
                cv[q] = pv[q];
            }
            ce = pe;
            __syncwarp();
            issue(j + RP + 1);  // into the slot of row j - 1, which no lane reads any more
        }
        cp_async_wait<0>();
        __syncwarp();
    }
}

// The rows of a warp's segments from the last to the first, ST_BACK at a time: f(i, rows, step, n)
// with the array index of the lane's cells in the first of `rows` rows, `step` apart.
template <class T, class F>
__device__ __forceinline__ void stream_back(const StreamArgs& A, int gw, int nwarps, F&& f)
{
    constexpr int VEC = RingGeom<T>::VEC, STRIP = RingGeom<T>::STRIP;
    const Geom& g = A.f.g;
    const int xlast = g.X - HALO_PAD - 1, ylast = g.Y - HALO_PAD - 1;
    const int per_x = (g.nx + STRIP - 1) / STRIP;
    const int nseg = per_x * ((g.ny + A.seg - 1) / A.seg);
    if (gw >= nseg) return;
    for (int sgi = gw + (nseg - 1 - gw) / nwarps * nwarps; sgi >= 0; sgi -= nwarps) {
        const int c = HALO_PAD + STRIP * (sgi % per_x) + VEC * (int)(threadIdx.x & 31);
        const int j0 = HALO_PAD + A.seg * (sgi / per_x), j1 = min(j0 + A.seg, ylast + 1);
        if (c > xlast) continue;
        for (int j = j1 - 1; j >= j0; j -= ST_BACK) f(fidx(g, c, j, 0), min(ST_BACK, j - j0 + 1), -g.pitch, xlast - c + 1);
    }
}

#else

// Sweep A of a group's tiles: a group of ST_TY warps owns 32 lanes x 16 bytes by ST_TY rows and
// marches through the planes of its unit, as k_ring3d; the groups of a block only share its
// sums, so each has a named barrier of its own.
__device__ __forceinline__ void stream_group_sync(int group)
{
    asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(ST_TY * 32) : "memory");
}

template <class P, bool UPD, class T = typename P::T>
__device__ __forceinline__ void stream_sweep_a(const StreamArgs& A, const StreamStep<T>& st, T* ring, int first, int stride,
                                               DD& acc)
{
    constexpr int VEC = RingGeom<T>::VEC, STRIP = RingGeom<T>::STRIP, OFF = RingGeom<T>::OFF, RWT = RingGeom<T>::WIDTH;
    constexpr int TY = ST_TY, RP = ST_RP, RQ = RP + 2;
    // Row offsets of a slot: p and q with the rows below and above the tile, Kx, Ky with the row
    // above, Kz, u and the old p.
    constexpr int RP_ = 0, RQ_ = TY + 2, RX = 2 * (TY + 2), RY = RX + TY, RZ = RY + TY + 1, RU = RZ + TY, RO = RU + TY;
    constexpr int SLOT = (UPD ? RO + TY : RU) * RWT;
    const FusedArgs& a = A.f;
    const Geom& g = a.g;
    const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) % TY, group = (threadIdx.x >> 5) / TY;
    const int xlast = g.X - HALO_PAD - 1, ylast = g.Y - HALO_PAD - 1, zlast = g.Z - HALO_PAD - 1;
    const int per_x = (g.nx + STRIP - 1) / STRIP, per_y = (g.ny + TY - 1) / TY;
    const int txy = per_x * per_y, nunits = txy * ((g.nz + A.seg - 1) / A.seg);
    const int cmax = (int)g.pitch - 2 * VEC + 2;
    const T* __restrict__ KX = P::kx(a);
    const T* __restrict__ KY = P::ky(a);
    const T* __restrict__ KZ = P::kz(a);
    const bool pend = st.q != nullptr;
    for (int unit = first; unit < nunits; unit += stride) {
        const int zs = unit / txy, rxy = unit % txy, xs = rxy % per_x, ys = rxy / per_x;
        const int c0 = HALO_PAD + STRIP * xs, c = c0 + VEC * lane, cc = min(c, cmax);
        const int y0 = HALO_PAD + TY * ys, j = y0 + w;
        const int n = j <= ylast ? xlast - c + 1 : 0;
        const int z0 = HALO_PAD + A.seg * zs, z1 = min(z0 + A.seg, zlast + 1);
        const int left = refl(c0 - 1, g.X), right_op = refl(min(c0 + STRIP, xlast + 1), g.X);
        const int right_k = min(c0 + STRIP, xlast + 1);
        const long rj = (long)refl(min(j, ylast + 1), g.Y) * g.pitch, ij = (long)min(j, ylast + 1) * g.pitch;
        const long r_below = (long)refl(y0 - 1, g.Y) * g.pitch, r_above = (long)refl(min(y0 + TY, ylast + 1), g.Y) * g.pitch;
        const long i_above = (long)min(y0 + TY, ylast + 1) * g.pitch;
        auto slot = [&](int z) { return ring + ((z - z0 + 1) % RQ) * SLOT; };
        auto issue = [&](int z) {
            if (z <= z1) {
                T* base = slot(z);
                const bool seg = z >= z0 && z < z1;
                const long zr = (long)refl(min(z, zlast + 1), g.Z) * g.page, zi = (long)z * g.page;
                const int col = OFF + VEC * lane;
                auto operand = [&](T* d, const T* s) {
                    cp_async_16(d + (w + 1) * RWT + col, s + zr + rj + cc);
                    if (z >= z0) {
                        if (lane == 0) ring_copy_one(d + (w + 1) * RWT + OFF - 1, s + zr + rj + left);
                        if (lane == 31) ring_copy_one(d + (w + 1) * RWT + OFF + STRIP, s + zr + rj + right_op);
                    }
                    if (seg && w == 0) cp_async_16(d + col, s + zr + r_below + cc);
                    if (seg && w == TY - 1) cp_async_16(d + (TY + 1) * RWT + col, s + zr + r_above + cc);
                };
                operand(base + RP_ * RWT, st.p);
                if (pend) operand(base + RQ_ * RWT, st.q);
                if (seg) {
                    if (UPD) {
                        cp_async_16(base + (RU + w) * RWT + col, st.u + zi + ij + cc);
                        cp_async_16(base + (RO + w) * RWT + col, st.pn + zi + ij + cc);
                    }
                    cp_async_16(base + (RX + w) * RWT + col, KX + zi + ij + cc);
                    if (lane == 31) ring_copy_one(base + (RX + w) * RWT + OFF + STRIP, KX + zi + ij + right_k);
                    cp_async_16(base + (RY + w) * RWT + col, KY + zi + ij + cc);
                    if (w == TY - 1) cp_async_16(base + (RY + TY) * RWT + col, KY + zi + i_above + cc);
                }
                if (z >= z0) cp_async_16(base + (RZ + w) * RWT + col, KZ + zi + ij + cc);
            }
            cp_async_commit();
        };
        auto stage = [&](T p, T q) { return pend ? st.beta * p + q : p; };
        auto stage_row = [&](const T* base, int row, T* v) {
            T x[VEC], y[VEC];
            ld_vec(base + (RP_ + row) * RWT + OFF + VEC * lane, x);
            ld_vec(base + (RQ_ + row) * RWT + OFF + VEC * lane, y);
#pragma unroll
            for (int q = 0; q < VEC; ++q) v[q] = stage(x[q], y[q]);
        };
        auto stage_edge = [&](const T* base) {
            const int e = (w + 1) * RWT + (lane == 0 ? OFF - 1 : OFF + STRIP);
            return stage(base[RP_ * RWT + e], base[RQ_ * RWT + e]);
        };
        for (int z = z0 - 1; z <= z0 + RP; ++z) issue(z);
        cp_async_wait<RP>();
        stream_group_sync(group);
        T mv[VEC], cv[VEC];
        stage_row(slot(z0 - 1), w + 1, mv);
        stage_row(slot(z0), w + 1, cv);
        T ce = stage_edge(slot(z0));
        for (int z = z0; z < z1; ++z) {
            cp_async_wait<RP - 1>();
            stream_group_sync(group);
            issue(z + RP + 1);  // into the slot of plane z - 1, which no warp reads any more
            const T* cur = slot(z);
            const T* nxt = slot(z + 1);
            T pv[VEC], ym[VEC], yp[VEC];
            stage_row(nxt, w + 1, pv);
            const T pe = stage_edge(nxt);
            stage_row(cur, w, ym);
            stage_row(cur, w + 2, yp);
            const T up = __shfl_up_sync(0xffffffffu, cv[VEC - 1], 1);
            const T dn = __shfl_down_sync(0xffffffffu, cv[0], 1);
            T kx[VEC + 1], ky0[VEC], ky1[VEC], kz0[VEC], kz1[VEC], praw[VEC], uv[VEC], old[VEC], wv[VEC];
            const int col = OFF + VEC * lane;
            ld_vec(cur + (RX + w) * RWT + col, kx);
            const T kxn = __shfl_down_sync(0xffffffffu, kx[0], 1);
            kx[VEC] = lane == 31 ? cur[(RX + w) * RWT + OFF + STRIP] : kxn;
            ld_vec(cur + (RY + w) * RWT + col, ky0);
            ld_vec(cur + (RY + w + 1) * RWT + col, ky1);
            ld_vec(cur + (RZ + w) * RWT + col, kz0);
            ld_vec(nxt + (RZ + w) * RWT + col, kz1);
            ld_vec(cur + (RP_ + w + 1) * RWT + col, praw);
            if constexpr (UPD) {
                ld_vec(cur + (RU + w) * RWT + col, uv);
                ld_vec(cur + (RO + w) * RWT + col, old);
            }
#pragma unroll
            for (int q = 0; q < VEC; ++q) {
                NbT<T> nb;
                nb.c = cv[q];
                nb.xm = q == 0 ? (lane == 0 ? ce : up) : cv[q > 0 ? q - 1 : 0];
                nb.xp = c + q == xlast ? cv[q] : (q == VEC - 1 ? (lane == 31 ? ce : dn) : cv[q < VEC - 1 ? q + 1 : q]);
                nb.ym = ym[q];
                nb.yp = yp[q];
                nb.zm = mv[q];
                nb.zp = pv[q];
                wv[q] = smvp_k(nb, kx[q], kx[q + 1], ky0[q], ky1[q], kz0[q], kz1[q]);
            }
            stream_cells<P, UPD>(a, st, fidx(g, c, j, z), n, cv, wv, praw, uv, old, acc);
#pragma unroll
            for (int q = 0; q < VEC; ++q) {
                mv[q] = cv[q];
                cv[q] = pv[q];
            }
            ce = pe;
        }
        cp_async_wait<0>();
        stream_group_sync(group);  // the next unit's copies reuse slots other warps may still read
    }
}

// As in 2D: the planes of a warp's row of its group's units from the last to the first.
template <class T, class F>
__device__ __forceinline__ void stream_back(const StreamArgs& A, int first, int stride, F&& f)
{
    constexpr int VEC = RingGeom<T>::VEC, STRIP = RingGeom<T>::STRIP, TY = ST_TY;
    const Geom& g = A.f.g;
    const int w = (threadIdx.x >> 5) % TY;
    const int xlast = g.X - HALO_PAD - 1, ylast = g.Y - HALO_PAD - 1, zlast = g.Z - HALO_PAD - 1;
    const int per_x = (g.nx + STRIP - 1) / STRIP, per_y = (g.ny + TY - 1) / TY;
    const int txy = per_x * per_y, nunits = txy * ((g.nz + A.seg - 1) / A.seg);
    if (first >= nunits) return;
    for (int unit = first + (nunits - 1 - first) / stride * stride; unit >= 0; unit -= stride) {
        const int zs = unit / txy, rxy = unit % txy;
        const int c = HALO_PAD + STRIP * (rxy % per_x) + VEC * (int)(threadIdx.x & 31);
        const int j = HALO_PAD + TY * (rxy / per_x) + w;
        const int z0 = HALO_PAD + A.seg * zs, z1 = min(z0 + A.seg, zlast + 1);
        if (c > xlast || j > ylast) continue;
        for (int z = z1 - 1; z >= z0; z -= ST_BACK) f(fidx(g, c, j, z), min(ST_BACK, z - z0 + 1), -g.page, xlast - c + 1);
    }
}
#endif

// Loads the lane's cells of up to ST_BACK rows (whole vectors: rows are padded).
template <class T>
__device__ __forceinline__ void stream_load(const T* a, long i, int rows, long step, T (&v)[ST_BACK][RingGeom<T>::VEC])
{
#pragma unroll
    for (int k = 0; k < ST_BACK; ++k)
        if (k < rows) ld_vec(a + i + k * step, v[k]);
}

// Sweep B: r -= alpha w, z = mi r, r.(r|z).
template <class P, class T = typename P::T>
__device__ __forceinline__ void stream_sweep_b(const StreamArgs& A, T alpha, bool pre, int first, int stride, DD& acc)
{
    constexpr int VEC = RingGeom<T>::VEC;
    const FusedArgs& a = A.f;
    stream_back<T>(A, first, stride, [&](long i, int rows, long step, int n) {
        T r[ST_BACK][VEC], w[ST_BACK][VEC];
        stream_load(P::r(a), i, rows, step, r);
        stream_load(P::w(a), i, rows, step, w);
#pragma unroll
        for (int k = 0; k < ST_BACK; ++k)
            if (k < rows) {
                const long ik = i + k * step;
                T z[VEC];
                if constexpr (!P::fp32) {
                    if (pre) ld_vec(a.mi + ik, z);
                }
#pragma unroll
                for (int q = 0; q < VEC; ++q) {
                    const T rq = r[k][q] - alpha * w[k][q];
                    r[k][q] = rq;
                    z[q] = pre ? z[q] * rq : rq;
                    dd_add(acc, q < n ? (double)rq * (double)z[q] : 0.0);
                }
                stream_store(P::r(a), ik, n, r[k]);
                if constexpr (!P::fp32) {
                    if (pre) stream_store(a.z, ik, n, z);
                }
            }
    });
}

template <class P>
struct StreamP;
template <>
struct StreamP<ResF64> {
    __device__ static double* p(const FusedArgs& a, int b) { return a.p[b]; }
};
template <>
struct StreamP<ResF32> {
    __device__ static float* p(const FusedArgs& a, int b) { return a.p32[b]; }
};

// A row's strip starts 16 bytes behind the row.  It has to start on 32 bytes, as the sectors that the
// copies bring do (16 bytes off, an iteration takes 6-9 % longer), wherever the kernel's static part ends.
// (Not by the array's alignment: all kernels of the file share it, and others' rings would move.)
template <class T>
__device__ __forceinline__ T* ring_start(unsigned char* raw)
{
    return reinterpret_cast<T*>(raw + ((16 - res_shared(raw)) & 31));
}

template <class P>
__global__ void __launch_bounds__(ST_WARPS * 32, 1) k_stream_cg(const __grid_constant__ StreamArgs A)
{
    using T = typename P::T;
    extern __shared__ __align__(16) unsigned char s_stream_raw[];
    __shared__ ResShared<false> sh;
    const FusedArgs& a = A.f;
    SolveState& s = sh.s;
    GridSum<false, !P::fp32> sum(A.sum, sh.sum);
    if (threadIdx.x == 0) {
        s = A.start ? *A.start : A.s0;
        sum.start(s.rro);
    }
    constexpr int warps = ST_WARPS / StreamRing<T>::parts;  // that share a ring
    const int part = sum.warp / warps;
    const int first = blockIdx.x * StreamRing<T>::parts + part, stride = gridDim.x * StreamRing<T>::parts;
    T* ring = ring_start<T>(s_stream_raw) + part * StreamRing<T>::elems;
    __syncthreads();
    const bool pre = !P::fp32 && s.precond;
    int par = s.par_p, waiting = 0;  // p's buffer, steps of u not yet taken
    T a_old = (T)0, a_last = (T)0;
    for (bool pend = false;; pend = true) {
        StreamStep<T> st;
        st.p = StreamP<P>::p(a, par);
        st.pn = StreamP<P>::p(a, par ^ 1);
        st.q = nullptr;
        if (pend) {
            st.q = P::r(a);
            if constexpr (!P::fp32)
                if (pre) st.q = a.z;
        }
        st.u = P::u(a);
        st.beta = (T)s.last_beta;
        st.a_old = a_old;
        st.a_last = a_last;
        DD acc = {0.0, 0.0};
        if (waiting == 2) {
            waiting = 0;
            stream_sweep_a<P, true>(A, st, ring, first, stride, acc);
        } else {
            stream_sweep_a<P, false>(A, st, ring, first, stride, acc);
        }
        par ^= 1;
        if (sum.reduce(
                acc, 0, [] {}, [&](double v) { return cg_after_pw(s, v); }, [&](double v) { cg_note_pw<P>(a, s, v); }) !=
            RN_GO)
            break;
        const T alpha = (T)s.alpha;
        acc.hi = acc.lo = 0.0;
        stream_sweep_b<P>(A, alpha, pre, first, stride, acc);
        a_old = a_last;
        a_last = alpha;
        ++waiting;
        if (sum.template reduce<true>(
                acc, 1, [] {}, [&](double v) { return cg_after_rr<P>(a, s, v); },
                [&](double v) { cg_note_rr<P>(a, s, v); }) != RN_GO)
            break;
    }
    // The last step of u is left to whoever uses it next (pending_u); one before that is taken here.
    if (waiting == 2) {
        T* u = P::u(a);
        const T* old = StreamP<P>::p(a, par ^ 1);
        stream_back<T>(A, first, stride, [&](long i, int rows, long step, int n) {
            constexpr int VEC = RingGeom<T>::VEC;
            T x[ST_BACK][VEC], y[ST_BACK][VEC];
            stream_load(u, i, rows, step, x);
            stream_load(old, i, rows, step, y);
#pragma unroll
            for (int k = 0; k < ST_BACK; ++k)
                if (k < rows) {
#pragma unroll
                    for (int q = 0; q < VEC; ++q) x[k][q] = x[k][q] + a_old * y[k][q];
                    stream_store(u, i + k * step, n, x[k]);
                }
        });
    }
    __syncthreads();  // what the last sum left to be written down
    if (blockIdx.x == 0) {
        if (threadIdx.x == 0) {
            s.par_p = par;
            s.pending_p = s.pending_u = 1;
            *a.st = *A.host = s;
        }
        sum.clear_other_set();
    }
}

}  // namespace tea
