// The beginning and the end of a whole solve, one launch each.
//
// What bounds them.  On small grids a solve is launches and host round trips: the set-up was
// nine launches and one or two reads of a sum, the end eight launches, three copies and three
// waits, together 150 of the 210 us of a CG timestep at 10x10.  On large grids they are passes
// over memory: 24 words per cell in the set-up where 11 are needed (3D).  k_setup forms every field
// of the set-up from density and energy alone (and is then bound by instruction issue and latencies:
// 1.39 ms at 256^3, issue slots 55 % busy, DRAM at 16 % of its peak), so that nothing waits for a
// neighbour's value: a cell's coefficients and its residual are formed from the (reflected)
// densities and energies around it, with the operations of CGInitUW, CGInitK and CGCalcRRO in
// their order.  The starting state goes to device memory, from where the first loop takes it
// without the host.
#pragma once

#include "tea_fused.cuh"

namespace tea {

struct SetupArgs {
    Geom g;
    Fields f;
    Box full;
    int cond, precond;  // the coefficient is the density; diagonal preconditioner
    double rx, ry, rz;
    double eps_rel;     // > 0: eps = eps_rel^2 sum u0^2
    RedScratch red;
    SolveState s0;      // the starting state, without rro (and eps where eps_rel is set)
    SolveState* start;
    double* out;        // rro, sum u0^2
};

// Where a padded cell's density and energy come from once their halo (depth 2) is updated: the
// reflected inner cell; in 3D the halo's edges and corners are not updated.
__device__ __forceinline__ long setup_src(const Geom& g, int kk, int jj, int ii)
{
#if TEA_DIM == 2
    (void)ii;
    return fidx(g, refl(kk, g.X), refl(jj, g.Y), 0);
#else
    const int ko = kk < HALO_PAD || kk >= g.X - HALO_PAD, jo = jj < HALO_PAD || jj >= g.Y - HALO_PAD,
              io = ii < HALO_PAD || ii >= g.Z - HALO_PAD;
    return ko + jo + io > 1 ? fidx(g, kk, jj, ii) : fidx(g, refl(kk, g.X), refl(jj, g.Y), refl(ii, g.Z));
#endif
}

struct SetupCell {
    double u, w, r, p, mi, z;
};

// The start of an inner cell: u0, A u0, the residual and the CG start p (with mi and z).
__device__ __forceinline__ SetupCell setup_cell(const SetupArgs& a, int kk, int jj, int ii)
{
    const Geom& g = a.g;
    auto rho = [&](int k, int j, int i) { return a.f.density[setup_src(g, k, j, i)]; };
    auto wof = [&](double d) { return a.cond ? d : 1.0 / d; };
    auto uof = [&](int k, int j, int i, double d) { return a.f.energy[setup_src(g, k, j, i)] * d; };
    auto face = [](double rr, double lo, double hi) { return rr * (lo + hi) / (2.0 * lo * hi); };
    const double dc = rho(kk, jj, ii), dl = rho(kk - 1, jj, ii), dr = rho(kk + 1, jj, ii), db = rho(kk, jj - 1, ii),
                 dt = rho(kk, jj + 1, ii);
    const double wc = wof(dc);
    const double kx0 = face(a.rx, wof(dl), wc), kx1 = face(a.rx, wc, wof(dr));
    const double ky0 = face(a.ry, wof(db), wc), ky1 = face(a.ry, wc, wof(dt));
    double kz0 = 0.0, kz1 = 0.0;
    Nb nb;
    nb.c = uof(kk, jj, ii, dc);
    nb.xm = uof(kk - 1, jj, ii, dl);
    nb.xp = uof(kk + 1, jj, ii, dr);
    nb.ym = uof(kk, jj - 1, ii, db);
    nb.yp = uof(kk, jj + 1, ii, dt);
    nb.zm = nb.zp = 0.0;
    if (DIM == 3) {
        const double df = rho(kk, jj, ii - 1), dk = rho(kk, jj, ii + 1);
        kz0 = face(a.rz, wof(df), wc);
        kz1 = face(a.rz, wc, wof(dk));
        nb.zm = uof(kk, jj, ii - 1, df);
        nb.zp = uof(kk, jj, ii + 1, dk);
    }
    SetupCell c;
    c.u = nb.c;
    c.w = smvp_k(nb, kx0, kx1, ky0, ky1, kz0, kz1);
    c.r = c.u - c.w;
    c.p = c.r;
    c.mi = c.z = 0.0;
    if (a.precond) {
#if TEA_DIM == 2
        c.mi = 1.0 / (1.0 + (kx1 + kx0) + (ky1 + ky0));
#else
        c.mi = 1.0 / (1.0 + (kx1 + kx0) + (ky1 + ky0) + (kz1 + kz0));
#endif
        c.z = c.mi * c.r;
        c.p = c.z;
    }
    return c;
}

// The set-up of a CG, Chebyshev or PPCG solve (at least two cells along every axis): the depth-2
// halos of density and energy, u, u0, Kx, Ky(, Kz), w, r, p (with its depth-1 halo), mi and z,
// and the sums rro = r.p and u0.u0, as update_halo, ext_cg_solver_init_, update_halo,
// ext_solver_copy_u_ and ext_calculate_2norm_ leave them.
__global__ void __launch_bounds__(BLOCK) k_setup(const __grid_constant__ SetupArgs a)
{
    let_next_start();
    const Geom& g = a.g;
    const Fields& f = a.f;
    DDVec<2> acc;
    acc.zero();
    walk(a.full, [&](int kk, int jj, int ii) {
        const long i = fidx(g, kk, jj, ii), s = setup_src(g, kk, jj, ii);
        const double e = f.energy[s], d = f.density[s];
        if (s != i) {
            f.energy[i] = e;
            f.density[i] = d;
        }
        f.u[i] = e * d;
        auto beyond = [](int k, int n, int depth) { return k < HALO_PAD - depth || k >= n - HALO_PAD + depth; };
        const int out0 = beyond(kk, g.X, 0) + beyond(jj, g.Y, 0) + (DIM == 3 ? beyond(ii, g.Z, 0) : 0);
        const int out1 = beyond(kk, g.X, 1) + beyond(jj, g.Y, 1) + (DIM == 3 ? beyond(ii, g.Z, 1) : 0);
        // Kx, Ky(, Kz) on the inner cells and one beyond on the high sides, w one beyond on all.
        auto wat = [&](int k, int j, int l) {
            const double v = f.density[setup_src(g, k, j, l)];
            return a.cond ? v : 1.0 / v;
        };
        double wc = 0.0;
        if (out1 == 0) wc = wat(kk, jj, ii);
        if (kk >= HALO_PAD && kk < g.X - 1 && jj >= HALO_PAD && jj < g.Y - 1 && (DIM == 2 || (ii >= HALO_PAD && ii < g.Z - 1))) {
            const double wl = wat(kk - 1, jj, ii), wb = wat(kk, jj - 1, ii);
            f.kx[i] = a.rx * (wl + wc) / (2.0 * wl * wc);
            f.ky[i] = a.ry * (wb + wc) / (2.0 * wb * wc);
            if (DIM == 3) {
                const double wf = wat(kk, jj, ii - 1);
                f.kz[i] = a.rz * (wf + wc) / (2.0 * wf * wc);
            }
        }
        double p = 0.0, r = 0.0;
        // p's halo: the depth-1 ring, in 3D without its edges and corners.
        if (out0 == 0 || (out1 == 0 && (DIM == 2 || out0 == 1))) {
            const SetupCell c = setup_cell(a, refl(kk, g.X), refl(jj, g.Y), DIM == 3 ? refl(ii, g.Z) : 0);
            p = c.p;
            if (out0 == 0) {
                r = c.r;
                f.u0[i] = c.u;
                f.w[i] = c.w;
                if (a.precond) {
                    f.mi[i] = c.mi;
                    f.z[i] = c.z;
                }
                dd_add(acc.v[0], r * p);
                dd_add(acc.v[1], c.u * c.u);
            }
        }
        if (out0 != 0 && out1 == 0) f.w[i] = wc;
        f.p[i] = p;
        f.r[i] = r;
    });
    grid_reduce_then<2>(acc, a.red, [&](const double* v) {
        SolveState s = a.s0;
        s.rro = v[0];
        if (a.eps_rel > 0.0) s.eps = a.eps_rel * a.eps_rel * v[1];
        *a.start = s;
        a.out[0] = v[0];
        a.out[1] = v[1];
    });
}

// Brings u and p to the state the per-call kernels expect: pending updates applied (u +=
// last_alpha p, p = last_beta p + (z|r)), current values in the canonical buffers, the
// depth-1 halos of u and (with `p_halo`) of p reflected; with `energy` also ext_solver_finalise_
// (energy = u / density) and energy's depth-1 halo.  A cell's thread writes the halo cells that
// mirror it.  The state comes by value, or from *st where st is not null.
__global__ void __launch_bounds__(BLOCK) k_settle(FusedArgs a, Fields f, Box inner, SolveState s0, const SolveState* st,
                                                  int p_halo, int energy)
{
    wait_for_previous();
    const SolveState& s = st ? *st : s0;
    const Geom& g = a.g;
    const double* pc = a.p[s.par_p];
    const double* uc = a.u[s.par_u];
    const double alpha = s.last_alpha, beta = s.last_beta;
    const int pu = s.pending_u, pp = s.pending_p;
    const double* q = s.precond ? a.z : a.r;
    walk(inner, [&](int kk, int jj, int ii) {
        const long i = fidx(g, kk, jj, ii);
        const double po = pc[i];
        double u = uc[i], p = po, e = 0.0;
        if (pu) u = u + alpha * po;
        if (pp) p = beta * po + q[i];
        if (energy) e = u / f.density[i];
        auto put = [&](long to, bool inside) {
            a.u[0][to] = u;
            if (inside || p_halo) a.p[0][to] = p;
            if (energy) f.energy[to] = e;
        };
        put(i, true);
        // Mirrored cells: at most one on each side of an axis; in 2D the corners too.
        const bool l = kk == HALO_PAD, r = kk == g.X - HALO_PAD - 1;
        const bool b = jj == HALO_PAD, t = jj == g.Y - HALO_PAD - 1;
        if (l) put(i - 1, false);
        if (r) put(i + 1, false);
        if (b) put(i - g.pitch, false);
        if (t) put(i + g.pitch, false);
#if TEA_DIM == 2
        if (l && b) put(i - 1 - g.pitch, false);
        if (l && t) put(i - 1 + g.pitch, false);
        if (r && b) put(i + 1 - g.pitch, false);
        if (r && t) put(i + 1 + g.pitch, false);
#else
        if (ii == HALO_PAD) put(i - g.page, false);
        if (ii == g.Z - HALO_PAD - 1) put(i + g.page, false);
#endif
    });
}

}  // namespace tea
