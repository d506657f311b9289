// pointwise.cuh -- cell-local pieces of the RK3 substep: fluxes, SGS
// viscosity, RK update and the variable conversions.  Each piece is an
// argument struct plus a per-cell device function, so that the same body runs
// from a single-grid kernel (grid-stride loop) and from the batched
// persistent kernels that cover many grids in one launch.
#pragma once

#include "common.cuh"
#include "impeller.cuh"

namespace emix {

// Loop over cells with a grid-stride loop (grids are sized to the GPU).
#define EMIX_FOR_CELLS(q, n) \
    for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < (n); q += (long)gridDim.x * blockDim.x)

// 8 resident blocks of 256 threads per SM
inline int cells_grid(long n, int bs = 256) { return grid_cap(n, 8, bs); }

// ---- primitive variables: u = um(2..4)/um(1), pres = um(1)/Mach^2 ------------
// (varc_to_varnc, src/MSVSingle/herramientas_incomp2.f90:16-27)
struct PrimArgs {
    const double *um;
    double *u, *pres;
    double inv_m2;
    long n;               // cells (the component stride)
    long qbeg, qend;      // single-grid launches: cells [qbeg, qend) only (qend = 0: all)
};

EMIX_DEV void prim_cell(const PrimArgs &a, long q) {
    const long n = a.n;
    const double r = a.um[q];
    const double rr = rcp_fast(r);
    a.pres[q] = r * a.inv_m2;
    a.u[q] = a.um[n + q] * rr;
    a.u[n + q] = a.um[2 * n + q] * rr;
    a.u[2 * n + q] = a.um[3 * n + q] * rr;
}

// ---- fluxes of all five equations (flujos, solver/flujos_compact.f90:21-217) --
// Inviscid plus viscous, projected by J*dxi/dx (x), J*deta/dy (y), J*dzeta/dz (z):
//   F[3*m + d] = Jd * (inviscid_{m,d} + viscous_{m,d}),  m = 0..4, d = 0..2.
// jx/jy/jz are the static products jbn10*jbn1, jbn10*jbn5, jbn10*jbn9.
struct FluxArgs {
    double *F[15];
    const double *um;    // 5 fields
    const double *u;     // 3 fields
    const double *pres;
    const double *dvel;  // 9 fields
    const double *vis;
    const double *jbn;   // 11 fields (components 0, 4, 8 read)
    const double *jx, *jy, *jz;
    long n;
};

// ---- velocity-gradient pieces shared by the SGS viscosity and the fluxes ----
// The physical normal gradients sxx = ux, syy = vy, szz = wz (dvel times the
// metric terms jbn1, jbn5, jbn9) and the shear sums sxy = uy + vx, sxz = uz +
// wx, syz = vz + wy (flujos_compact.f90:68-70, :79-81, :123-125).
struct Strain {
    double sxx, syy, szz, sxy, sxz, syz;
};

EMIX_DEV Strain strain_cell(const double *__restrict__ jbn, const double *__restrict__ dvel, long n, long q) {
    const double j1 = jbn[q], j5 = jbn[4 * n + q], j9 = jbn[8 * n + q];
    const double *dv = dvel + q;
    Strain s;
    s.sxx = j1 * dv[0];
    s.syy = j5 * dv[4 * n];
    s.szz = j9 * dv[8 * n];
    s.sxy = fma(j5, dv[3 * n], j1 * dv[n]);
    s.sxz = fma(j9, dv[6 * n], j1 * dv[2 * n]);
    s.syz = fma(j9, dv[7 * n], j5 * dv[5 * n]);
    return s;
}

// fluxes of the cell from its strain pieces and viscosity vs
EMIX_DEV void flux_from(const FluxArgs &a, long q, const Strain &s, double vs) {
    const long n = a.n;
    const double um2 = a.um[n + q], um3 = a.um[2 * n + q], um4 = a.um[3 * n + q],
                 um5 = a.um[4 * n + q];
    const double u1 = a.u[q], u2 = a.u[n + q], u3 = a.u[2 * n + q];
    const double p = a.pres[q];
    const double JX = a.jx[q], JY = a.jy[q], JZ = a.jz[q];
    const double vs2 = vs + vs;   // the normal viscous terms' 2 vis
    // um = rho u: each shear term stands in two equations (58 -> 55 FP64
    // operations a cell, and the FP64 pipe is 87% busy: 256^3 1.77 -> 1.70 ms)
    const double txy = fma(-um3, u1, vs * s.sxy);
    const double txz = fma(-um4, u1, vs * s.sxz);
    const double tyz = fma(-um4, u2, vs * s.syz);
    // equation 1
    a.F[0][q] = JX * (-um2);
    a.F[1][q] = JY * (-um3);
    a.F[2][q] = JZ * (-um4);
    // equation 2
    a.F[3][q] = JX * fma(vs2, s.sxx, fma(-um2, u1, -p));
    a.F[4][q] = JY * txy;
    a.F[5][q] = JZ * txz;
    // equation 3
    a.F[6][q] = JX * txy;
    a.F[7][q] = JY * fma(vs2, s.syy, fma(-um3, u2, -p));
    a.F[8][q] = JZ * tyz;
    // equation 4
    a.F[9][q] = JX * txz;
    a.F[10][q] = JY * tyz;
    a.F[11][q] = JZ * fma(vs2, s.szz, fma(-um4, u3, -p));
    // equation 5
    a.F[12][q] = JX * (-u1 * um5);
    a.F[13][q] = JY * (-u2 * um5);
    a.F[14][q] = JZ * (-u3 * um5);
}

EMIX_DEV void flux_cell(const FluxArgs &a, long q) {
    flux_from(a, q, strain_cell(a.jbn, a.dvel, a.n, q), a.vis[q]);
}

// ---- Smagorinsky: amut = (Cs*Delta)^2 sqrt(2 S_ij S_ij), vis = c4 + amut ------
// 2 S_ij S_ij = 2 (ux^2 + vy^2 + wz^2) + sxy^2 + sxz^2 + syz^2
struct SmagArgs {
    const double *dvel, *jbn, *dxyz;
    double cs, c4;
    double *amut, *vis;
    long n;
};

EMIX_DEV double smag_amut(const Strain &s, double cs, double delta) {
    const double nn = fma(s.szz, s.szz, fma(s.syy, s.syy, s.sxx * s.sxx));
    const double sh = fma(s.syz, s.syz, fma(s.sxz, s.sxz, s.sxy * s.sxy));
    const double cd = cs * delta;
    return (cd * cd) * sqrt_fast(fma(2.0, nn, sh));
}

EMIX_DEV void smag_cell(const SmagArgs &a, long q) {
    const double am = smag_amut(strain_cell(a.jbn, a.dvel, a.n, q), a.cs, a.dxyz[q]);
    if (a.amut) a.amut[q] = am;
    a.vis[q] = a.c4 + am;
}

// Smagorinsky and the fluxes of one cell from one set of strain pieces (the
// two launches of a substep as one: the same values as smag_cell followed by
// flux_cell, bit for bit, with the strain pieces formed once)
EMIX_DEV void smag_flux_cell(const SmagArgs &sa, const FluxArgs &fa, long q) {
    const Strain s = strain_cell(fa.jbn, fa.dvel, fa.n, q);
    const double am = smag_amut(s, sa.cs, sa.dxyz[q]);
    if (sa.amut) sa.amut[q] = am;
    const double vs = sa.c4 + am;
    sa.vis[q] = vs;
    flux_from(fa, q, s, vs);
}

// ---- selective structure-function model (solver/sgdm_incomp.f90) ------------
// f_structura + amu0*sqrt*Delta (:131-137, :166-298)
struct SfArgs {
    const double *u, *ratios, *dxyz;
    double amu0;
    double *amut;
    int nx, ny, nz;
    long n;
};

EMIX_DEV void sf_cell(const SfArgs &a, long q) {
    const int nx = a.nx, ny = a.ny, nz = a.nz;
    const long n = a.n;
    const double *U = a.u, *V = a.u + n, *W = a.u + 2 * n;
    const double *ratios = a.ratios;
    const long sy = nx, sz = (long)nx * ny;
    int i, j, k;
    cell_of(q, n, nx, ny, i, j, k);
    double x, y, z, s;
    long p, m;
    // the six one-sided increments in the order of f_structura
    p = i < nx - 1 ? q + 1 : q; m = i < nx - 1 ? q : q - 1;
    double r = ratios[q];
    x = (U[p] - U[m]) * r; y = (V[p] - V[m]) * r; z = (W[p] - W[m]) * r;
    s = x * x + y * y + z * z;
    if (i > 0) { p = q - 1; m = q; } else { p = q + 1; m = q; }
    r = ratios[n + q];
    x = (U[p] - U[m]) * r; y = (V[p] - V[m]) * r; z = (W[p] - W[m]) * r;
    s = s + x * x + y * y + z * z;
    if (j < ny - 1) { p = q + sy; m = q; } else { p = q; m = q - sy; }
    r = ratios[2 * n + q];
    x = (U[p] - U[m]) * r; y = (V[p] - V[m]) * r; z = (W[p] - W[m]) * r;
    s = s + x * x + y * y + z * z;
    if (j > 0) { p = q - sy; m = q; } else { p = q; m = q + sy; }
    r = ratios[3 * n + q];
    x = (U[p] - U[m]) * r; y = (V[p] - V[m]) * r; z = (W[p] - W[m]) * r;
    s = s + x * x + y * y + z * z;
    if (k < nz - 1) { p = q + sz; m = q; } else { p = q; m = q - sz; }
    r = ratios[4 * n + q];
    x = (U[p] - U[m]) * r; y = (V[p] - V[m]) * r; z = (W[p] - W[m]) * r;
    s = s + x * x + y * y + z * z;
    if (k > 0) { p = q - sz; m = q; } else { p = q; m = q + sz; }
    r = ratios[5 * n + q];
    x = (U[p] - U[m]) * r; y = (V[p] - V[m]) * r; z = (W[p] - W[m]) * r;
    s = s + x * x + y * y + z * z;
    s = s * (1.0 / 6.0);
    a.amut[q] = a.amu0 * sqrt_fast(s) * a.dxyz[q];
}

// VORT (:330-341)
struct VortArgs {
    const double *dvel, *jbn;
    double *w;
    long n;
};

EMIX_DEV void vort_cell(const VortArgs &a, long q) {
    const long n = a.n;
    const double j1 = a.jbn[q], j5 = a.jbn[4 * n + q], j9 = a.jbn[8 * n + q];
    const double *dv = a.dvel + q;
    a.w[q] = j5 * dv[7 * n] - j9 * dv[5 * n];
    a.w[n + q] = j9 * dv[2 * n] - j1 * dv[6 * n];
    a.w[2 * n + q] = j1 * dv[3 * n] - j5 * dv[n];
}

// SELECTIVO (:346-395) and viscosidad (vis = c4 + amut)
struct SelArgs {
    const double *w;
    double *amut, *vis;
    double cutoff, c4;
    int nx, ny, nz;
    long n;
};

EMIX_DEV void select_cell(const SelArgs &a, long q) {
    const int nx = a.nx, ny = a.ny, nz = a.nz;
    const long n = a.n;
    const double *wx = a.w, *wy = a.w + n, *wz = a.w + 2 * n;
    const long sy = nx, sz = (long)nx * ny;
    int i, j, k;
    cell_of(q, n, nx, ny, i, j, k);
    const long a1 = i < nx - 1 ? q + 1 : q, a2 = i > 0 ? q - 1 : q;
    const long a3 = k < nz - 1 ? q + sz : q, a4 = k > 0 ? q - sz : q;
    const long a5 = j < ny - 1 ? q + sy : q, a6 = j > 0 ? q - sy : q;
    const double wxn = wx[a1] + wx[a2] + wx[a3] + wx[a4] + wx[a5] + wx[a6];
    const double wyn = wy[a1] + wy[a2] + wy[a3] + wy[a4] + wy[a5] + wy[a6];
    const double wzn = wz[a1] + wz[a2] + wz[a3] + wz[a4] + wz[a5] + wz[a6];
    const double x = wx[q], y = wy[q], z = wz[q];
    double wn = x * x + y * y + z * z;
    wn = sqrt(wn * (wxn * wxn + wyn * wyn + wzn * wzn));
    const double s1 = (x * wxn + y * wyn + z * wzn) / wn;
    double am = a.amut[q];
    if (s1 > a.cutoff) am = 0.0;
    a.amut[q] = am;
    a.vis[q] = a.c4 * 1.0 + am;
}

// ---- RK stage + conversions ------------------------------------------------------
// rs = jbn11*R; RK stage s; varc_to_varnc, clip to [-6,6], mask, varc_to_varnc;
// rebuild um1(1) = pres*Mach*Mach, um1(2..4) = u*um1(1)
// (solver/rungek_ico.f90:83-138,150-198,210-267)
struct RkArgs {
    const double *R;      // 5 fields
    const double *um0;    // 5
    const double *um;     // 5 (previous substep)
    double *out;          // 5 (may alias um or um0: read-before-write per cell)
    double *u;            // 3
    double *pres;
    const double *jbn;
    const double *mask;
    double dt, mach, inv_m2;
    int stage;
    int walls;            // 1: frontera_z/y/x_val between the RK combination and the conversions
    int faces;            // with walls: 0 = cells no wall rule touches, 1 = the wall cells
    int nx, ny, nz;
    long n;
    ImpGeom imp;          // impeller forcing after the walls (imp.on = 0: none)
    const double *xyz;    // coordinates (3 fields), read when imp.on
    const double *clock;  // impeller clock (k_imp_clock), read when imp.on
    const unsigned char *impflag;   // cells the impeller can reach (k_imp_flags)
    long qbeg, qend;      // single-grid launches: cells [qbeg, qend) only (qend = 0: all)
};

// Wall cells: z = 0, nz-2, nz-1 (frontera_z), y = 0, ny-1 (frontera_y),
// x = 0, nx-1 (frontera_x).  Enumerated as the three z planes, then the two
// y planes for z in [1, nz-3], then the two x planes for y in [1, ny-2].
__host__ __device__ inline long rk_face_count(int nx, int ny, int nz) {
    return 3L * nx * ny + 2L * nx * (nz - 3) + 2L * (ny - 2) * (nz - 3);
}

__host__ __device__ inline long rk_count(const RkArgs &a) {
    return (a.walls && a.faces) ? rk_face_count(a.nx, a.ny, a.nz) : a.n;
}

// RK3 combination of one cell (rungek_ico.f90:89-90, 153-154, 217-220), up to
// the factor rk_scale: um0 + dt R; 3 um0 + um + dt R (of 1/4);
// um0 + 2 um + 2 dt R (of 1/3).  The FP64 pipe bounds the update, and the
// factor cancels in the velocities, so it is left to the density and the last
// equation (27 -> 23 FP64 operations a cell).
EMIX_DEV double rk_scale(int stage) { return stage == 1 ? 1.0 : (stage == 2 ? 0.25 : 1.0 / 3.0); }

EMIX_DEV void rk_sums(const RkArgs &a, long q, double v[5]) {
    const long n = a.n;
    // the substep's weight of dt*R times the metric factor jbn(11), once per cell
    const double w = a.stage == 3 ? 2.0 * a.dt : a.dt;
    const double cj = w * a.jbn[10 * n + q];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
        const double u0 = a.um0[m * n + q];
        double b;
        if (a.stage == 1)
            b = u0;
        else if (a.stage == 2)
            b = fma(3.0, u0, a.um[m * n + q]);
        else
            b = fma(2.0, a.um[m * n + q], u0);
        v[m] = fma(cj, a.R[m * n + q], b);
    }
}

EMIX_DEV void rk_combine(const RkArgs &a, long q, double v[5]) {
    rk_sums(a, q, v);
    if (a.stage == 1) return;
    const double c = rk_scale(a.stage);
#pragma unroll
    for (int m = 0; m < 5; ++m) v[m] *= c;
}

// fmax(-6, fmin(6, x)) by integer compares on the bit pattern (|x| > 6 takes
// 6 with x's sign; a NaN also becomes +-6)
EMIX_DEV double clip6(double x) {
    const long long b = __double_as_longlong(x);
    const long long six = 0x4018000000000000LL;   // 6.0
    return (b & 0x7fffffffffffffffLL) > six ? __longlong_as_double((b & (long long)0x8000000000000000ULL) | six)
                                            : x;
}

// varc_to_varnc + clip + mask + varc_to_varnc (:104-124), then the rebuild
// after the level-set call site (:127-138), of the combined values v c
EMIX_DEV void rk_convert(const RkArgs &a, long q, double v[5], double c) {
    const long n = a.n;
    double pc = a.inv_m2 * c;
    if (a.imp.on && a.impflag[q]) {
        // rushton(stage) after the walls (rungek_ico.f90:102); cells the
        // impeller cannot reach are left as they are
        double f[5];
#pragma unroll
        for (int m = 0; m < 5; ++m) f[m] = v[m] * c;
        c = 1.0;
        pc = a.inv_m2;
        impeller_force_cell(a.imp, a.clock + 2 + 2 * (a.stage - 1) * kImpMaxBlades, a.xyz[q],
                            a.xyz[n + q], a.xyz[2 * n + q], f, nullptr);
#pragma unroll
        for (int m = 0; m < 5; ++m) v[m] = f[m];
    }
    const double r = v[0];
    const double rr = rcp_fast(r);
    const double mk = a.mask[q];
    // velocity, clipped and masked; the reference's masked momentum u r mk
    // divided by r again is u mk.  A mask of exactly 1 or +0 (the usual
    // case) applies by bit operations: c * 1 = c, and c * 0 = +-0 with c's
    // sign for the finite clipped c; any other mask value multiplies
    double uu[3];
    const long long mb = __double_as_longlong(mk);
    if (mb == 0x3FF0000000000000LL || mb == 0) {
        const long long keep = mb ? -1LL : (long long)0x8000000000000000ULL;
#pragma unroll
        for (int d = 0; d < 3; ++d)
            uu[d] = __longlong_as_double(__double_as_longlong(clip6(v[d + 1] * rr)) & keep);
    } else {
#pragma unroll
        for (int d = 0; d < 3; ++d) uu[d] = clip6(v[d + 1] * rr) * mk;
    }
    const double p = r * pc;
    const double r1 = p * (a.mach * a.mach);
    a.out[q] = r1;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        a.out[(d + 1) * n + q] = uu[d] * r1;
        a.u[d * n + q] = uu[d];
    }
    a.out[4 * n + q] = a.stage == 1 ? v[4] : v[4] * c;
    a.pres[q] = p;
}

// Values after frontera_z_val (src/MSVSingle/frontera_z.f90:231-259): z = 0
// copies z = 1 with um(4) = 0; z = nz-2, nz-1 take um(1) = 1, um(4) = 0 and
// the rest from z = nz-3.
EMIX_DEV void wall_z(const RkArgs &a, int i, int j, int k, double v[5]) {
    const int nx = a.nx, ny = a.ny, nz = a.nz;
    const int ks = k == 0 ? 1 : (k >= nz - 2 ? nz - 3 : k);
    rk_combine(a, i + (long)nx * (j + (long)ny * ks), v);
    if (k == 0) v[3] = 0.0;
    else if (k >= nz - 2) { v[0] = 1.0; v[3] = 0.0; }
}

// then frontera_y_val (frontera_y.f90:231-245): y walls copy um(1), um(5)
// from the neighbour plane, momentum 0
EMIX_DEV void wall_y(const RkArgs &a, int i, int j, int k, double v[5]) {
    const int ny = a.ny;
    const bool w = j == 0 || j == ny - 1;
    wall_z(a, i, j == 0 ? 1 : (j == ny - 1 ? ny - 2 : j), k, v);
    if (w) { v[1] = 0.0; v[2] = 0.0; v[3] = 0.0; }
}

// then frontera_x_val (frontera_x.f90:235-253): the same on the x walls
EMIX_DEV void wall_x(const RkArgs &a, int i, int j, int k, double v[5]) {
    const int nx = a.nx;
    const bool w = i == 0 || i == nx - 1;
    wall_y(a, i == 0 ? 1 : (i == nx - 1 ? nx - 2 : i), j, k, v);
    if (w) { v[1] = 0.0; v[2] = 0.0; v[3] = 0.0; }
}

EMIX_DEV void rk_cell(const RkArgs &a, long q) {
    double v[5];
    if (!a.walls) {
        rk_sums(a, q, v);
        rk_convert(a, q, v, rk_scale(a.stage));
        return;
    }
    // 32-bit indices (a context of 2^32 cells does not fit in memory): the
    // conversions of 64-bit divisions run at the FP64 pipe's rate
    const unsigned nx = a.nx, ny = a.ny, nz = a.nz;
    unsigned i, j, k, r = (unsigned)q;
    if (!a.faces) {
        const unsigned row = r / nx;
        k = row / ny;
        j = row - k * ny;
        i = r - row * nx;
        if (i == 0 || i == nx - 1 || j == 0 || j == ny - 1 || k == 0 || k >= nz - 2) return;
        rk_sums(a, q, v);
        rk_convert(a, q, v, rk_scale(a.stage));
        return;
    }
    const unsigned pz = nx * ny, py = nx * (nz - 3), px = (ny - 2) * (nz - 3);
    if (r < 3 * pz) {
        const unsigned pl = r / pz;
        r -= pl * pz;
        j = r / nx;
        i = r - j * nx;
        k = pl == 0 ? 0 : nz - 3 + pl;
    } else if (r < 3 * pz + 2 * py) {
        r -= 3 * pz;
        const unsigned pl = r / py;
        r -= pl * py;
        k = r / nx;
        i = r - k * nx;
        ++k;
        j = pl == 0 ? 0 : ny - 1;
    } else {
        r -= 3 * pz + 2 * py;
        const unsigned pl = r / px;
        r -= pl * px;
        k = r / (ny - 2);
        j = 1 + r - k * (ny - 2);
        ++k;
        i = pl == 0 ? 0 : nx - 1;
    }
    // the wall rules read only cells no rule writes (k = 1, nz-3; j = 1,
    // ny-2; i = 1, nx-2 after the earlier rules), recomputed here from the RK
    // inputs, which this launch does not overwrite: it runs before the launch
    // over the other cells, and writes only wall cells
    wall_x(a, i, j, k, v);
    rk_convert(a, i + (long)nx * (j + (long)ny * k), v, 1.0);
}

// ---- kernels ------------------------------------------------------------------
__global__ void k_prim(PrimArgs a);
__global__ void k_flux_all(FluxArgs a);
__global__ void k_sgs_smag(SmagArgs a);
__global__ void k_smag_flux(SmagArgs s, FluxArgs f);
__global__ void k_sgs_sf(SfArgs a);
__global__ void k_vort(VortArgs a);
__global__ void k_selective(SelArgs a);
__global__ void k_rk_post(RkArgs a);

// flujos(neq) one equation at a time (the emix_flux_dev entry point)
__global__ void k_flux_one(int neq, double *__restrict__ e, double *__restrict__ f,
                           double *__restrict__ g, double *__restrict__ ev,
                           double *__restrict__ fv, double *__restrict__ gv,
                           const double *__restrict__ um, const double *__restrict__ u,
                           const double *__restrict__ pres, const double *__restrict__ dvel,
                           const double *__restrict__ jbn, const double *__restrict__ vis, long n);

// INISGDM (solver/sgdm_incomp.f90:20-108)
__global__ void k_sgs_setup(const double *__restrict__ xyz, double *__restrict__ dxyz,
                            double *__restrict__ ratios, int nx, int ny, int nz);

} // namespace emix
