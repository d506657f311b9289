// reinit.cu -- Sussman reinitialisation of the level set, the device form of
// cuReinitLsJB (src/LevelSet/lsTransportEc.cu:420-676) with the right-hand
// side reini_RS_WENOJB (src/LevelSet/lsTools.cu:824-902):
//
//   per iteration: mirror the ghost layers of phi, phi0 = phi, then three
//   TVD-RK3 stages of  d(phi)/dtau = -S(phi0) (|grad phi| - 1),
//   S = phi0 / sqrt(phi0^2 + dmin^2),  dtau = deltamin / 2,
//   |grad phi| by the Godunov upwinding of the left- and right-biased WENO5
//   derivatives (PhiDevPlus/MinusParameterJB, lsTools.cu:587-770).
//
// One fused kernel per stage, marching in z like the advection stage
// (weno_march.cuh): a block owns a 16 x 16 column, the z differences live in a
// register window, the x and y differences, second differences and scaled
// third differences in shared tiles formed once per position; both WENO5
// reconstructions of each direction read them (weno5s), then the Godunov
// combination, the speed and the stage update.  Cells near the padded grid's
// edges follow the edge rules of the stencil (weno5).  The metric pairs
// (C, eps / C^2) are formed once per call and the smoothed sign once per
// iteration.  Stages ping-pong between two scratch fields so that stencil
// reads never meet a write.
//
// FP64 bounds it: about 201 operations per cell and stage, 280 with every
// cell forming its own differences, metric pairs and sign.  140 x 128 x 116 cells,
// 10 iterations: 38.7 -> 26.7 ms, 30 x 34 x 41: 2.11 -> 1.35.
#include "weno_march.cuh"

namespace emix {

namespace {

struct ReinitArgs {
    const double *src;    // field the derivatives are taken of
    const double *phi;    // iteration start (the sign's field, the TVD combination's phi_n)
    const double2 *ce;    // per direction and cell: C = jbn / h and eps / C^2
    const double *dmins;  // padded smoothing widths (stage 1)
    double *sgn;          // smoothed sign of phi: written by stage 1, read by the others
    double *out;
    int nxg, nyg, nzg;
    double dt;
    int stage, ref_bugs;
};

// max(x, 0) and max(-x, 0) by the sign bit; the larger of two non-negative
// doubles (their bit patterns order as integers)
EMIX_DEV double pos_part(double x) { return __double_as_longlong(x) > 0 ? x : 0.0; }
EMIX_DEV double neg_mag(double x) {
    const long long b = __double_as_longlong(x);
    return b < 0 ? __longlong_as_double(b & 0x7fffffffffffffffLL) : 0.0;
}
EMIX_DEV double larger(double a, double b) { return __double_as_longlong(a) >= __double_as_longlong(b) ? a : b; }
// x with its sign bit flipped where c has one
EMIX_DEV double with_sign_of(double x, double c) {
    return __longlong_as_double(__double_as_longlong(x) ^
                                (__double_as_longlong(c) & (long long)0x8000000000000000ull));
}

// (C, eps / C^2) of every cell and direction (components 1, 5, 9 of jbn)
__global__ void k_reinit_scales(const double *__restrict__ jbn, double2 *__restrict__ ce, double sx, double sy,
                                double sz, long ng) {
    for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < ng; q += (long)gridDim.x * blockDim.x) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double C = (d == 0 ? sx : (d == 1 ? sy : sz)) * jbn[4 * d * ng + q];
            ce[d * ng + q] = make_double2(C, kWenoEps4 * rcp_fast(C * C));
        }
    }
}

// both reconstructions from the five second differences A0..A4 around the
// cell, the scaled third differences S1..S4 between them and the two central
// differences
EMIX_DEV void both_sides(double vl, double vr, double A0, double A1, double A2, double A3, double A4, double S1,
                         double S2, double S3, double S4, double eps, double &am, double &bp) {
    am = weno5s(vl, A0, A1, A2, A3, S1, S2, S3, eps, 6.0);    // phi^-: D(c), A(c-1..c+2)
    bp = weno5s(vr, A4, A3, A2, A1, S4, S3, S2, eps, -6.0);   // phi^+: D(c+1), -A(c+3..c)
}

__global__ void __launch_bounds__(kNT, 3) k_reinit_stage(const ReinitArgs a) {
    __shared__ double P[kPY][kPX];
    __shared__ double Dx[kMY][kMX + 5];      // positions x0-2 .. x0+kMX+2
    __shared__ double Ax[kMY][kMX + 4];      // positions x0-1 .. x0+kMX+2
    __shared__ double Tx[kMY][kMX + 3];      // positions x0 .. x0+kMX+2
    __shared__ double Dy[kMY + 5][kMX];      // rows alike
    __shared__ double Ay[kMY + 4][kMX];
    __shared__ double Ty[kMY + 3][kMX];
    const int nxg = a.nxg, nyg = a.nyg, nzg = a.nzg;
    const long sxy = (long)nxg * nyg, ng = sxy * nzg;
    const double *__restrict__ phi = a.src;
    const int tid = threadIdx.x, tx = tid % kMX, ty = tid / kMX;
    const int x0 = blockIdx.x * kMX, y0 = blockIdx.y * kMY;
    const int chunk = (nzg + gridDim.z - 1) / gridDim.z;
    const int zs = blockIdx.z * chunk, ze = min(zs + chunk, nzg);
    const int X = x0 + tx, Y = y0 + ty;
    const bool active = X < nxg && Y < nyg;
    const long col = (long)X + (long)nxg * Y;
    // warps (two rows of 16 cells) with a cell whose x or y stencil follows an
    // edge rule take that rule's form for all their cells
    const bool wedge_x = __any_sync(0xffffffffu, active && (X < 2 || X > nxg - 4));
    const bool wedge_y = __any_sync(0xffffffffu, active && (Y < 2 || Y > nyg - 4));
    auto ld = [&](int z) { return (active && z >= 0 && z < nzg) ? phi[col + sxy * z] : 0.0; };
    // Dz[t] = D(Z - 2 + t); Az[t] = A(Z - 1 + t); Tz[t] = S(Z + t); fz = phi(Z + 3)
    double Dz[6], Az[5], Tz[4], fz;
    {
        double f[7];
#pragma unroll
        for (int t = 0; t < 7; ++t) f[t] = ld(zs - 3 + t);
#pragma unroll
        for (int t = 0; t < 6; ++t) Dz[t] = (zs - 2 + t == 0) ? ld(1) - ld(0) : f[t + 1] - f[t];
#pragma unroll
        for (int t = 0; t < 5; ++t) Az[t] = Dz[t + 1] - Dz[t];
#pragma unroll
        for (int t = 0; t < 4; ++t) Tz[t] = kSqrt13_3 * (Az[t + 1] - Az[t]);
        fz = f[6];
    }
    Plane pl;
    if (zs < ze) load_plane(phi, x0, y0, zs, nxg, nyg, nzg, sxy, tid, pl);
    for (int Z = zs; Z < ze; ++Z) {
        // this plane's tile (loaded during the previous plane), then its
        // differences, second and third differences
#pragma unroll
        for (int r = 0; r < kPR; ++r) {
            const int t = tid + r * kNT;
            if (t < kPN) (&P[0][0])[t] = pl.v[r];
        }
        __syncthreads();
        if (Z + 1 < ze) load_plane(phi, x0, y0, Z + 1, nxg, nyg, nzg, sxy, tid, pl);
        const double fnext = ld(Z + 4);
        for (int t = tid; t < kMY * (kMX + 5); t += kNT) {
            const int i = t % (kMX + 5), j = t / (kMX + 5);
            Dx[j][i] = x0 - 2 + i == 0 ? P[j + 3][i + 2] - P[j + 3][i + 1] : P[j + 3][i + 1] - P[j + 3][i];
        }
        for (int t = tid; t < (kMY + 5) * kMX; t += kNT) {
            const int i = t % kMX, j = t / kMX;
            Dy[j][i] = y0 - 2 + j == 0 ? P[j + 2][i + 3] - P[j + 1][i + 3] : P[j + 1][i + 3] - P[j][i + 3];
        }
        const double pin = active ? P[ty + 3][tx + 3] : 0.0;
        __syncthreads();
        for (int t = tid; t < kMY * (kMX + 4); t += kNT) {
            const int i = t % (kMX + 4), j = t / (kMX + 4);
            Ax[j][i] = Dx[j][i + 1] - Dx[j][i];
        }
        for (int t = tid; t < (kMY + 4) * kMX; t += kNT) {
            const int i = t % kMX, j = t / kMX;
            Ay[j][i] = Dy[j + 1][i] - Dy[j][i];
        }
        __syncthreads();
        for (int t = tid; t < kMY * (kMX + 3); t += kNT) {
            const int i = t % (kMX + 3), j = t / (kMX + 3);
            Tx[j][i] = kSqrt13_3 * (Ax[j][i + 1] - Ax[j][i]);
        }
        for (int t = tid; t < (kMY + 3) * kMX; t += kNT) {
            const int i = t % kMX, j = t / kMX;
            Ty[j][i] = kSqrt13_3 * (Ay[j + 1][i] - Ay[j][i]);
        }
        __syncthreads();
        if (active) {
            const long id = col + sxy * Z;
            double p0 = 0.0, sg;
            if (a.stage == 1) {
                p0 = a.phi[id];
                const double dm = a.dmins[id];
                sg = p0 * rsqrt_fast(fma(p0, p0, dm * dm));
                a.sgn[id] = sg;
            } else {
                sg = a.sgn[id];
            }
            // sign of phi (0 for zero and NaN), by its bits
            const long long sb = __double_as_longlong(sg), sm = sb & 0x7fffffffffffffffLL;
            const int tsg = sm == 0 || sm > 0x7ff0000000000000LL ? 0 : (sb < 0 ? -1 : 1);
            double r = 0.0;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const double2 ce = a.ce[d * ng + id];
                const int c = d == 0 ? X : (d == 1 ? Y : Z), L = d == 0 ? nxg : (d == 1 ? nyg : nzg);
                double am, bp;
                if (d == 2 ? c >= 2 && c <= L - 4 : !(d == 0 ? wedge_x : wedge_y)) {
                    if (d == 0)
                        both_sides(Dx[ty][tx + 2], Dx[ty][tx + 3], Ax[ty][tx], Ax[ty][tx + 1], Ax[ty][tx + 2],
                                   Ax[ty][tx + 3], Ax[ty][tx + 4], Tx[ty][tx],
                                   Tx[ty][tx + 1], Tx[ty][tx + 2], Tx[ty][tx + 3], ce.y,
                                   am, bp);
                    else if (d == 1)
                        both_sides(Dy[ty + 2][tx], Dy[ty + 3][tx], Ay[ty][tx], Ay[ty + 1][tx], Ay[ty + 2][tx],
                                   Ay[ty + 3][tx], Ay[ty + 4][tx], Ty[ty][tx],
                                   Ty[ty + 1][tx], Ty[ty + 2][tx], Ty[ty + 3][tx], ce.y,
                                   am, bp);
                    else
                        both_sides(Dz[2], Dz[3], Az[0], Az[1], Az[2], Az[3], Az[4], Tz[0], Tz[1], Tz[2], Tz[3], ce.y,
                                   am, bp);
                } else {
                    // edge rules: the differences at the rule's positions
                    double vl[5], vr[5];
                    if (d == 2) {
                        weno_z_general(phi, id, Z, nzg, true, a.ref_bugs && Z == nzg - 1, nxg, sxy, vl);
                        weno_z_general(phi, id, Z, nzg, false, false, nxg, sxy, vr);
                    } else {
                        int p[5];
                        stencil_left(c, L, p);
                        for (int k = 0; k < 5; ++k) vl[k] = d == 0 ? Dx[ty][p[k] - (x0 - 2)] : Dy[p[k] - (y0 - 2)][tx];
                        stencil_right(c, L, p);
                        for (int k = 0; k < 5; ++k) vr[k] = d == 0 ? Dx[ty][p[k] - (x0 - 2)] : Dy[p[k] - (y0 - 2)][tx];
                    }
                    am = weno5(vl[0], vl[1], vl[2], vl[3], vl[4], ce.y);
                    bp = weno5(vr[0], vr[1], vr[2], vr[3], vr[4], ce.y);
                }
                // Godunov: phi0 > 0 takes max(max(a-, 0)^2, min(b+, 0)^2), phi0 < 0
                // max(max(b+, 0)^2, min(a-, 0)^2), phi0 = 0 their mean; the larger
                // of two non-negative magnitudes squared, the magnitudes picked by
                // sign and compared as integers (squaring is monotone, and so is
                // the metric's factor, which only the larger is multiplied by)
                am = with_sign_of(am, ce.x);
                bp = with_sign_of(bp, ce.x);
                if (tsg != 0) {
                    const double u = tsg > 0 ? am : bp, v = tsg > 0 ? bp : am;
                    const double m = ce.x * larger(pos_part(u), neg_mag(v));
                    r = fma(m, m, r);
                } else {
                    const double m1 = ce.x * larger(pos_part(am), neg_mag(bp));
                    const double m2 = ce.x * larger(pos_part(bp), neg_mag(am));
                    r += fma(0.5 * m2, m2, 0.5 * m1 * m1);
                }
            }
            const double rs = sg * (sqrt_fast(r) - 1.0);
            const double t = pin - a.dt * rs;
            double o;
            if (a.stage == 1) o = t;
            else if (a.stage == 2) o = 0.75 * a.phi[id] + 0.25 * t;
            else o = fma(2.0, t, a.phi[id]) * (1.0 / 3.0);
            a.out[id] = o;
        }
        // advance the z window
#pragma unroll
        for (int t = 0; t < 5; ++t) Dz[t] = Dz[t + 1];
        Dz[5] = fnext - fz;   // D(Z + 4); Z + 4 > 0
        fz = fnext;
#pragma unroll
        for (int t = 0; t < 4; ++t) Az[t] = Az[t + 1];
        Az[4] = Dz[5] - Dz[4];
#pragma unroll
        for (int t = 0; t < 3; ++t) Tz[t] = Tz[t + 1];
        Tz[3] = kSqrt13_3 * (Az[4] - Az[3]);
        __syncthreads();
    }
}

// The stage by cells, each with differences, metric pairs and sign of its own: 280
// FP64 operations, two fields of scratch, any extent.
__global__ void __launch_bounds__(256) k_reinit_cells(const ReinitArgs a, const double *__restrict__ jbn, double sx, double sy,
                                                      double sz) {
    const int nxg = a.nxg, nyg = a.nyg, nzg = a.nzg;
    const long sxy = (long)nxg * nyg, ng = sxy * nzg;
    for (long id = blockIdx.x * (long)blockDim.x + threadIdx.x; id < ng; id += (long)gridDim.x * blockDim.x) {
        int c3[3];
        cell_of(id, ng, nxg, nyg, c3[0], c3[1], c3[2]);
        const int L3[3] = {nxg, nyg, nzg};
        const long s3[3] = {1, nxg, sxy};
        const double sc[3] = {sx, sy, sz};
        const double p0 = a.phi[id];
        const int tsg = (p0 > 0.0) - (p0 < 0.0);
        double r = 0.0;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double C = sc[d] * jbn[4 * d * ng + id];
            const double eps = kWenoEps4 * rcp_fast(C * C);
            const long s = s3[d], base = id - c3[d] * s;
            const int c = c3[d];
            auto diff = [&](int p) {
                const long q = base + (p == 0 ? 1 : p) * s;
                return a.src[q] - a.src[q - s];
            };
            double am, bp;
            if (c >= 2 && c <= L3[d] - 4) {
                double v[6];
#pragma unroll
                for (int k = 0; k < 6; ++k) v[k] = diff(c - 2 + k);
                const double A0 = v[1] - v[0], A1 = v[2] - v[1], A2 = v[3] - v[2], A3 = v[4] - v[3], A4 = v[5] - v[4];
                both_sides(v[2], v[3], A0, A1, A2, A3, A4, kSqrt13_3 * (A1 - A0), kSqrt13_3 * (A2 - A1),
                           kSqrt13_3 * (A3 - A2), kSqrt13_3 * (A4 - A3), eps, am, bp);
            } else {
                int p[5];
                double v[5];
                stencil_left(c, L3[d], p);
                for (int k = 0; k < 5; ++k) v[k] = diff(p[k]);
                if (d == 2 && a.ref_bugs && c == nzg - 1) {
                    // lsTools.cu:636: id_kp2 = id_jm1 at the top layer
                    const long ib = c3[1] == 0 ? id : id - nxg;
                    v[4] = a.src[ib] - a.src[ib - sxy];
                }
                am = weno5(v[0], v[1], v[2], v[3], v[4], eps);
                stencil_right(c, L3[d], p);
                for (int k = 0; k < 5; ++k) v[k] = diff(p[k]);
                bp = weno5(v[0], v[1], v[2], v[3], v[4], eps);
            }
            // Godunov, as in k_reinit_stage
            am *= C;
            bp *= C;
            const double m1 = larger(pos_part(am), neg_mag(bp)), m2 = larger(pos_part(bp), neg_mag(am));
            r += tsg > 0 ? m1 * m1 : (tsg < 0 ? m2 * m2 : fma(0.5, m2 * m2, 0.5 * (m1 * m1)));
        }
        const double dm = a.dmins[id];
        const double rs = (p0 * rsqrt_fast(fma(p0, p0, dm * dm))) * (sqrt_fast(r) - 1.0);
        const double t = a.src[id] - a.dt * rs;
        double o;
        if (a.stage == 1) o = t;
        else if (a.stage == 2) o = 0.75 * a.phi[id] + 0.25 * t;
        else o = fma(2.0, t, a.phi[id]) * (1.0 / 3.0);
        a.out[id] = o;
    }
}

// ghost layers of a padded field from its own interior (mirror images)
__global__ void k_mirror_inplace(double *f, int g, int nx, int ny, int nz) {
    const int nxg = nx + 2 * g, nyg = ny + 2 * g, nzg = nz + 2 * g;
    const long ng = (long)nxg * nyg * nzg;
    for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < ng; q += (long)gridDim.x * blockDim.x) {
        int X, Y, Z;
        cell_of(q, ng, nxg, nyg, X, Y, Z);
        if (X >= g && X < nx + g && Y >= g && Y < ny + g && Z >= g && Z < nz + g) continue;
        const long src = (mirror(X, g, nx) + g) + (long)nxg * ((mirror(Y, g, ny) + g) + (long)nyg * (mirror(Z, g, nz) + g));
        f[q] = f[src];
    }
}

int grid_r(long n) { return grid_cap(n, 8); }

} // namespace

// Whether the stages go by cells: where a launch's grid does not reach, and on
// small grids whose one-plane blocks are a few more than one for each SM, or than
// the three an SM holds, so that a second one or round runs for those few, while
// the cells by themselves are less (one block of theirs an SM, or the second
// round).  ms a call of 10 iterations, marching / by cells: 30 x 30 x 40 1.43 /
// 1.12, 37 x 50 x 42 2.48 / 1.97, 49 x 50 x 30 2.24 / 1.86; 55 x 55 x 35 2.45 / 2.8.
static bool by_cells(long cols, int gy, int nzg, long ng) {
    const long sms = device_sms(), blocks = cols * nzg;
    return gy > 65535 || (blocks > sms && ng <= 256 * sms) || (blocks > 3 * sms && blocks <= 4 * sms && ng < 600 * sms);
}

int reinit_impl(double *phi, const double *jbn, const double *dmins, double dX, double dY, double dZ,
                int nxg, int nyg, int nzg, int g, double deltamin, int iters, int ref_bugs,
                cudaStream_t st) {
    const long ng = (long)nxg * nyg * nzg;
    const int gx = (nxg + kMX - 1) / kMX, gy = (nyg + kMY - 1) / kMY;
    double *scr;
    bool cells = by_cells((long)gx * gy, gy, nzg, ng);
    // a call whose nine fields do not fit goes by cells, in two
    int rc = device_scratch((size_t)(cells ? 2 : 9) * ng * sizeof(double), &scr);
    if (rc == EMIX_ERR_ALLOC && !cells) {
        cells = true;
        rc = device_scratch((size_t)2 * ng * sizeof(double), &scr);
    }
    if (rc) return rc;
    double *A = cells ? scr : scr + 6 * ng, *B = A + ng;   // the pairs first, 16-byte aligned
    const int nx = nxg - 2 * g, ny = nyg - 2 * g, nz = nzg - 2 * g;
    ReinitArgs a{};
    a.phi = phi; a.dmins = dmins;
    a.nxg = nxg; a.nyg = nyg; a.nzg = nzg;
    a.dt = 0.5 * deltamin; a.ref_bugs = ref_bugs;
    dim3 grid(1);
    if (!cells) {
        a.ce = reinterpret_cast<const double2 *>(scr);
        a.sgn = B + ng;
        grid = dim3(gx, gy, march_chunks((long)gx * gy, nzg, 3));
        k_reinit_scales<<<grid_r(ng), 256, 0, st>>>(jbn, reinterpret_cast<double2 *>(scr), 1.0 / dX, 1.0 / dY, 1.0 / dZ, ng);
    }
    auto stage = [&](int q, const double *src, double *out) {
        a.src = src;
        a.out = out;
        a.stage = q;
        if (cells) k_reinit_cells<<<grid_r(ng), 256, 0, st>>>(a, jbn, 1.0 / dX, 1.0 / dY, 1.0 / dZ);
        else k_reinit_stage<<<grid, kNT, 0, st>>>(a);
    };
    for (int it = 0; it < iters; ++it) {
        if (g > 0) k_mirror_inplace<<<grid_r(ng), 256, 0, st>>>(phi, g, nx, ny, nz);
        stage(1, phi, A);
        stage(2, A, B);
        stage(3, B, phi);
    }
    EMIX_CUDA_TRY(cudaGetLastError());
    return EMIX_OK;
}

} // namespace emix

using namespace emix;

extern "C" {

int emix_reinit_dev(double *phi, const double *jbn, const double *dmins, double deltaX, double deltaY,
                    double deltaZ, int nxg, int nyg, int nzg, int gcells, double deltamin, int iters,
                    int ref_bugs, void *stream) {
    if (!phi || !jbn || !dmins || gcells < 0 || nxg - 2 * gcells < 1 || nyg - 2 * gcells < 1 ||
        nzg - 2 * gcells < 1 || nxg < 4 || nyg < 4 || nzg < 4 || iters < 0 || !(deltaX > 0) ||
        !(deltaY > 0) || !(deltaZ > 0) || (ref_bugs != 0 && ref_bugs != 1))
        return EMIX_ERR_ARG;
    return reinit_impl(phi, jbn, dmins, deltaX, deltaY, deltaZ, nxg, nyg, nzg, gcells, deltamin, iters,
                       ref_bugs, (cudaStream_t)stream);
}

} // extern "C"
