// impeller.cuh -- the rotating impeller as a volumetric forcing: the linked
// rushton(sub_step) without its blade-edge interpolation
// (src/Geometry/rush_ruth_me.f90:2-108; makeAspa :519-593; addMaskCil and
// addAngularVel, src/Geometry/rotating.f90:110-205).
//
// Per cell: the impeller mask m (0 inside a blade, the hub disc or the shaft,
// 1 elsewhere) at the substep's time, then
//   um2 = ((1-m) ue + m um2/um1) um1,  um3 likewise with ve,  um4 = m um4,
// with (ue, ve) the rigid rotation at the cell.  The blade angles of the three
// substeps of a step are computed once per step on the device (k_imp_clock)
// from t = t0 + k dt, so graph replays advance the impeller.
//
// The plane tests and the angle arithmetic use explicitly rounded operations
// (no contraction) so the mask is decided exactly as written.
#pragma once

#include "common.cuh"

namespace emix {

constexpr int kImpMaxBlades = 16;
// clock buffer: [0] t0, [1] steps taken, then per substep s and blade b the
// pair (cos, sin) of the blade angle at index 2 + 2 (s kImpMaxBlades + b)
constexpr int kImpClockLen = 2 + 2 * 3 * kImpMaxBlades;

struct ImpGeom {
    int on, nblades;
    double omega, theta0;
    double r1, r2, z1, z2, half_thick;
    double hub_r, hub_z1, hub_z2;
    double shaft_r, shaft_z0, shaft_z1;
};

struct ImpClockArgs {
    double *clock;
    double dt;
    ImpGeom g;
};

// mask of one cell; cs = the (cos, sin) pairs of this substep's blades.  A
// cell is in a blade when the four plane distances -t' - h, t' - h, u - r2 and
// r1 - u (t' = sin x - cos y, u = cos x + sin y) are not positive; a rounded
// difference of doubles has the sign of the exact one, so they are compared
// directly, the blade's length only for cells within its thickness.  Few lanes
// of a warp have cells the impeller reaches, so its operations cost the update
// as much as a full warp's.
EMIX_DEV double impeller_mask(const ImpGeom &g, const double *cs, double x, double y, double z) {
    double m = 1.0;
    if (z >= g.z1 && z <= g.z2) {
        for (int b = 0; b < g.nblades; ++b) {
            const double c = cs[2 * b], sn = cs[2 * b + 1];
            const double t = __dadd_rn(__dmul_rn(sn, x), -__dmul_rn(c, y));
            if (fabs(t) <= g.half_thick) {
                const double u = __dadd_rn(__dmul_rn(c, x), __dmul_rn(sn, y));
                if (u <= g.r2 && u >= g.r1) m = 0.0;
            }
        }
    }
    const bool hub = z >= g.hub_z1 && z <= g.hub_z2;
    const bool shaft = z >= g.shaft_z0 && z <= g.shaft_z1;
    if (hub || shaft) {
        // radio <= R decided on sqrt(x^2 + y^2) as written; the square is only
        // a filter (with a margin far above rounding) that skips the root
        const double r2 = __dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y));
        const double R = fmax(hub ? g.hub_r : 0.0, shaft ? g.shaft_r : 0.0) * (1.0 + 1e-12);
        if (r2 <= R * R) {
            const double radio = sqrt(r2);
            if (hub && radio <= g.hub_r) m = 0.0;
            if (shaft && radio <= g.shaft_r) m = 0.0;
        }
    }
    return m;
}

// body velocity of addAngularVel (rotating.f90:163-186): the rotation by the
// polar angle a = atan(|y/x|), turned into its quadrant with 3.141592 for pi
// (and 3.1415926 / 2 for a on the y axis).  radio cos a = |x| and radio sin a =
// |y|, so the angle itself is not formed: with (sp, cp) = (sin, cos) of the
// quadrant's turn P, radio sin(P - a) = sp |x| - cp |y| and radio cos(P - a) =
// cp |x| + sp |y|.  With the atan, sine, cosine and root, all sixteen plane
// operations a blade and the clock's angles in one thread, the updates and the
// clock of a 40^3 step took 137 us, now 90 (256^3: 2.90 -> 2.73 ms).
EMIX_DEV double2 impeller_velocity(double omega, double x, double y) {
    double rc = fabs(x), rs = fabs(y);
    if (x == 0.0) {
        rc = rs * 2.6794896585028633e-08;   // cos, sin of 3.1415926 / 2
        rs = rs * 0.9999999999999997;
    }
    double sp = 0.0, cp = 1.0;
    if (x < 0.0) {                          // 3.141592 - a (y > 0) or + a
        sp = 6.535897930762419e-07;
        cp = -0.9999999999997864;
        if (!(y > 0.0)) rs = -rs;
    } else if (y < 0.0) {                   // 2 x 3.141592 - a
        sp = -1.3071795861522044e-06;
        cp = 0.9999999999991457;
    } else {
        rs = -rs;
    }
    return make_double2(-omega * fma(sp, rc, -cp * rs), omega * fma(cp, rc, sp * rs));
}

// the forcing on the conserved values v[5] of one cell
EMIX_DEV void impeller_force_cell(const ImpGeom &g, const double *cs, double x, double y, double z,
                                  double v[5], double *mask_out) {
    const double m = impeller_mask(g, cs, x, y, z);
    if (mask_out) *mask_out = m;
    // outside the impeller the forcing is the identity (up to the reference's
    // u/rho*rho round trip, which is left out)
    if (m == 1.0) return;
    // inside (m = 0): the body's velocity; a NaN or infinite momentum stays
    const double2 uv = impeller_velocity(g.omega, x, y);
    v[1] = fma(m, v[1], uv.x) * v[0];
    v[2] = fma(m, v[2], uv.y) * v[0];
    v[3] = m * v[3];
}

// t = t0 + k dt at the start of the step; the substeps are at t, t + dt/2,
// t + dt (rush_ruth_me.f90:52-54); then k += 1.  One warp, an angle a lane (18
// of them one after another took 18 us a step).
EMIX_DEV void imp_clock_tick(const ImpClockArgs &a, int lane) {
    const double t0 = a.clock[0], k = a.clock[1];
    const double t = __dadd_rn(t0, __dmul_rn(k, a.dt));
    const int nb = a.g.nblades;
    const double two_pi = 2.0 * 3.14159265358979323846;
    for (int e = lane; e < 3 * nb; e += 32) {
        const int s = e / nb, b = e - s * nb;
        const double ts = __dadd_rn(t, s == 0 ? 0.0 : (s == 1 ? 0.5 * a.dt : a.dt));
        const double th = __dadd_rn(__dadd_rn(a.g.theta0, __dmul_rn(a.g.omega, ts)),
                                    __dmul_rn((double)b, two_pi / nb));
        double sn, c;
        sincos(th, &sn, &c);
        a.clock[2 + 2 * (s * kImpMaxBlades + b)] = c;
        a.clock[3 + 2 * (s * kImpMaxBlades + b)] = sn;
    }
    __syncwarp();   // every lane has read k
    if (lane == 0) a.clock[1] = k + 1.0;
}

__global__ void k_imp_clock(ImpClockArgs a);

// the blade-edge interpolation (impeller_interp.cu)
struct ImpInterpArgs {
    ImpGeom g;
    const double *xyz, *clock, *mask;
    double *out, *u;        // the substep's um output and u output, updated in place
    int nx, ny, nz;
    long n;
    double rango;           // grid diagonal (getInterpolData :357-361)
    int stage, phase;       // phase 0: geometry, 1: lists, 2: apply
    unsigned char *status;  // per blade and plane cell
    signed char *face;
    double *geo;            // 11 per blade and plane cell: matrix, surface point
    int *nb;                // 2 per blade and plane cell: neighbour cells
    int *list, *count;
};
__global__ void k_interp_geom(ImpInterpArgs a);
__global__ void k_interp_list(ImpInterpArgs a);
__global__ void k_interp_apply(ImpInterpArgs a);

// 1 where some blade angle could put the cell inside the impeller (blade
// band within reach of a blade corner, hub disc, shaft), 0 elsewhere: the RK
// kernel tests only flagged cells.  The margin 1e-9 is far above rounding.
__global__ void k_imp_flags(const double *xyz, ImpGeom g, long n, unsigned char *flag);

} // namespace emix
