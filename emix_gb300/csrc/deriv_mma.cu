// deriv_mma.cu -- the compact first derivative on the tensor cores
// (tcgen05.mma, f16 operands, f32 sums in tensor memory).
//
// The FP64 pipe (2 lanes per clock and SM) bounds the factored Thomas sweeps
// at 3 clocks per cell and field.  Here D f is a contraction of the dense
// operator, which falls off so fast that 96 differences reach 16 outputs
// (deriv_mma.cuh), and its products are formed on the tensor cores: each
// pencil's differences are turned into fixed-point numbers (relative to the
// pencil's largest difference, to 2^-60 of it) of six balanced digits to the base
// 1024, the operator into digits of the same kind, and the sums of digit products
// are integers in f32 (the error-free splitting of K. Ozaki et al., Numerical
// Algorithms 59, 2012, applied to a banded operator).  Products of digit orders
// i + j <= 5 are kept; the sums of the first four orders are below 2^24 and exact,
// those of the last two round in the worst case, by 2^-54 of the result
// (deriv_table.cu).
//
// Errors, relative to the pencil's largest difference over h: 2^-57 from the
// products dropped, up to 2^-55.8 from the operator's cut at 40 rows.  The sweeps
// err by a few 2^-53 of the differences nearby, so a pencil may be quiet nowhere:
// one with a window of rows (16, along x 32) whose largest difference is below
// 2^-kMmaSpan of the pencil's takes the sweep (deriv.cuh's arithmetic), and so do
// infinities, NaN and magnitudes whose sums or results could leave the FP64 range.
// A window's error is then at most 2^-45.5 of its largest difference over h, about
// 2^-47 on average.  2^10: in a tank's first steps at 256^3 1 to 7% of the pencils
// span more, 30 to 50% more than 2^8 and nearly all more than 2^4, since the walls'
// no-slip jump is among them.  Over whole smooth fields the error against a dense
// solve is no larger than the sweeps' (192 x 160 x 192, 2-norm: A 5.4e-15 ->
// 3.9e-15, B 1.2e-15 -> 1.1e-15, cyclic 9.8e-16 -> 9.4e-16, C 5.7e-15 -> 3.4e-15).
//
// One CTA per SM walks tiles of 128 pencils (one per tensor-memory lane), its
// warps in four roles that meet on mbarriers:
//   seven warps read the next tile once for each pencil's largest difference and
//     its quietest window's (the first tile is shared by all);
//   eight warps convert the tile's differences to digits, 16 rows (a group) at
//     a time, into tensor memory, where they are the instruction's A operand;
//   one warp issues the products of a block of 16 outputs: 28 instructions,
//     since the operator's digits 0 .. 5-j lie next to each other and one
//     instruction adds all products of the differences' digit j;
//   eight warps combine the finished block's six sums per output.
// Whole tiles while they fill every SM, the rest cut into segments of blocks.  A
// tile of which every pencil takes the sweep is left out of the last three roles;
// the sweeps follow the CTA's last tile, a thread a pencil, or a warp if they are
// few.
//
// What bounds it: the scanning warps (loads from DRAM, and the differences on the
// FP64 pipe: 64 clocks of a quarter of the SM each) and the tensor-core warp (28
// instructions a block at 80 clocks each whatever their width up to 128 columns;
// 16 outputs a block are what tensor memory holds beside the digits) about alike,
// with the ALU pipe 55% busy.  The instructions' operands stay in uniform registers
// (elect.sync, branches on shuffled values): y 0.58 -> 0.52 ms.
// Measured, ms for 5 fields of 256^3, sweeps -> here: closed x 1.001 -> 0.594,
// y 0.993 -> 0.519, z 0.993 -> 0.522; cyclic 1.216 -> 0.631, 1.073 -> 0.580, 1.070
// -> 0.583.  Where 1% of the pencils take the sweep x 0.64, y 0.58; 30% 1.16, 1.03;
// all 2.05, 1.33.
#include "deriv_mma.cuh"
#include "tma.cuh"

#include <cuda_fp16.h>

#include <algorithm>
#include <cstdio>
#include <type_traits>
#include <vector>

namespace emix {
namespace {

__device__ int g_mma_timeouts = 0;
__device__ int g_mma_drop = 0;              // test hook: finished blocks are not signalled

constexpr int kMmaPencils = 128;            // per tile: the lanes of tensor memory
constexpr int kRpt = 8;                     // rows of a group (outputs of a block) a thread takes at a time
constexpr int kScanWarps = 7;               // warps that find the next tile's magnitudes
constexpr int kScan = 16;                   // rows a step of theirs
constexpr int scan_parts(bool xax) { return xax ? 1 : 4; }   // parts a pencil is scanned in
constexpr int kRole = 2 * kMmaPencils;      // converting threads, and as many for the results
constexpr int kRoleWarps = kRole / 32;
constexpr int kMmaThreads = 2 * kRole + 32 * (1 + kScanWarps);   // and the warp that drives the tensor core
// tensor memory, in columns: two sets of f32 sums, then the digits of the last
// groups, two f16 rows per column.  A block reads six groups and the seventh
// is being converted; of the outer two it reads the three leading digits at
// most, so the others are held for six groups only.
constexpr int kAccCols = kMmaDig * kMmaRows;
constexpr int kHighRing = 7, kLowRing = 6;
constexpr int kHighCol = 2 * kAccCols, kLowCol = kHighCol + kHighRing * 24;
constexpr int kTmemCols = 512;
// Kinds of pencils: closed, cyclic, and short cyclic ones of whole groups, all of
// whose groups are held in tensor memory at once and read round the cycle by the
// blocks, instead of five of them converted twice.  At least three groups (which
// wrap once) and at most four (which leave two places for the next tile's).  5
// fields of 64^3, us: x 28.2 -> 22.6, y and z 25.1 -> 20.7.  A kind of its own:
// tested at run time it costs the other cyclic pencils 2% (256^3 562 -> 574).
constexpr int kClosed = 0, kCyclic = 1, kRound = 2;
constexpr int kMmaRoundN = 64;
static_assert(kMmaMinN > 2 * kMmaRows && kMmaRoundN / kMmaRows < kLowRing, "kMmaRoundN");
// x: tiles of finished blocks.  A closed table's seven block types leave 28 KB of
// L1 beside two of them, 60 KB beside one, and what is in flight lives there: 5
// fields of 256^3 0.610 ms with two, 0.537 with one and another barrier a block.
constexpr int out_tiles(int kind) { return kind == kClosed ? 1 : 2; }
int kind_of(int n, bool periodic) {
    return !periodic ? kClosed : (n % kMmaRows == 0 && n <= kMmaRoundN ? kRound : kCyclic);
}
constexpr int kMmaWaitNs = 10000, kMmaWaitLimit = 1 << 15;   // a wait's slices, and their number
constexpr int kMmaSpan = 10;                // a window's largest difference to the pencil's, in powers of two
constexpr int kMmaSweepJobs = 128;          // jobs of a CTA whose sweeps wait for its last tile
// the sweeps a warp each where they are few: a warp takes 20 us for one at 256 rows,
// 10 at 40, a thread 170 and 14
constexpr int kSweepWarps = kMmaThreads / 32;
constexpr int kMmaShared = 120 * 1024;      // least shared memory a CTA asks for
constexpr int kXPitch = 17;                 // x pencils' staging tile: 17 rows, odd pitch
constexpr int kXTileDoubles = kMmaPencils * kXPitch;
static_assert(kLowCol + kLowRing * 24 <= kTmemCols, "tensor memory");

// issued by the one lane with `lead` (the whole warp keeps the operands, so
// that they stay in uniform registers)
EMIX_DEV void mma_f16(unsigned d, unsigned a, unsigned long long b, unsigned idesc, unsigned acc, unsigned lead) {
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %4, 0;\n\tsetp.ne.u32 q, %5, 0;\n\t"
                 "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 :: "r"(d), "r"(a), "l"(b), "r"(idesc), "r"(acc), "r"(lead) : "memory");
}

EMIX_DEV void tm_st4(unsigned addr, unsigned a, unsigned b, unsigned c, unsigned d) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};"
                 :: "r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

EMIX_DEV void tm_ld8(unsigned addr, float (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "r"(addr));
}

// v 2^(62 - (E - 1023)) modulo 2^64, its magnitude truncated before a negative one's
// bits are inverted: differences up to the biased exponent E come out below 2^63
EMIX_DEV unsigned long long to_fixed(double v, int E) {
    const int hi = __double2hiint(v), lo = __double2loint(v);
    const int up = ((hi >> 20) & 0x7ff) - E + 10;   // left shift of the mantissa
    const int sl = max(up, 0), sr = max(-up, 0);
    const unsigned mh = ((unsigned)hi & 0xfffffu) | 0x100000u;
    // 64-bit shifts: a funnel's is clamped at 32
    const unsigned h = __funnelshift_lc(0u, __funnelshift_lc((unsigned)lo, mh, sl), max(up - 32, 0));
    const unsigned l = __funnelshift_lc(0u, (unsigned)lo, sl);
    const unsigned neg = (unsigned)(hi >> 31);
    const unsigned rh = __funnelshift_rc(h, 0u, sr) ^ neg;
    const unsigned rl = __funnelshift_rc(__funnelshift_rc(l, h, sr), 0u, max(-32 - up, 0)) ^ neg;
    return ((unsigned long long)rh << 32) | rl;
}

// the differences of one pencil, or a part of it, by their high words without sign
struct Spread {
    int top;             // the largest
    int least;           // of the windows' largest, the smallest
    unsigned low;        // low words, or-ed (zero test)
};
EMIX_DEV int size_of(double d) { return __double2hiint(d) & 0x7fffffff; }

// the ten-bit digits at bit P of two rows' words as two f16: the two bytes
// they lie in, shifted down; 0x6400 | x is 1024 + x, and x carries a bias of 512
template <int P>
EMIX_DEV unsigned digit_pair(unsigned a, unsigned b) {
    constexpr unsigned i = P / 8, sel = i | (i + 1) << 4 | (i + 4) << 8 | (i + 5) << 12;
    const unsigned x = ((__byte_perm(a, b, sel) >> (P % 8)) & 0x03ff03ffu) | 0x64006400u;
    const __half2 h = __hsub2(*reinterpret_cast<const __half2 *>(&x), __float2half2_rn(1536.0f));
    return *reinterpret_cast<const unsigned *>(&h);
}

// digit P of a thread's rows as pairs of f16
template <int P>
EMIX_DEV void digits(unsigned (&d)[kRpt / 2], const unsigned (&w)[kRpt]) {
#pragma unroll
    for (int q = 0; q < kRpt / 2; ++q) d[q] = digit_pair<P>(w[2 * q], w[2 * q + 1]);
}

// one pencil's magnitudes, once known: the exponent its differences are fixed to,
// and whether it takes the scalar sweep: a window whose largest difference is below
// 2^-kMmaSpan of the pencil's, infinities, NaN, and exponents whose sums or whose
// results would leave the FP64 range
struct Scale {
    int E;
    bool scalar;
};

EMIX_DEV Scale scale_of(const Spread &a, int se) {
    Scale r{1023, false};
    if (a.top == 0 && a.low == 0) return r;   // all alike
    const int e = a.top >> 20;
    r.E = (a.top + 0x1000) >> 20;             // above 1 - 2^-8 of the next power of two: that one
    r.scalar = e < 256 || e > 1790 || r.E - se < 16 || r.E - se > 1960 || a.top - a.least > kMmaSpan << 20;
    return r;
}

// D f (EPI_STORE) or out += D f (EPI_ACCUM) along one pencil, as deriv_pencil with
// rows in runs of R: a run's loads are in flight while the one before it is walked.
// Few warps sweep here, and a run of a row's neighbours along x shares its sectors.
template <int EPI, bool PER>
__device__ __noinline__ void sweep_pencil(const DerivTable &T, const double *__restrict__ in, double *w, double *out, long s) {
    constexpr bool ACC = EPI == EPI_ACCUM;
    constexpr int R = 8;
    const int n = T.n;
    const DerivRow *rows = T.rows;
    const DerivRowU *ur = T.urows;
    double up = 0.0, y0 = 0.0;
    int i = 0;
    auto closure = [&]() {
        up = rhs_row(T, in, s, i) - (ACC ? __ldg(&ur[i].mu) : __ldg(&rows[i].m)) * up;
        w[i * s] = up;
    };
    if (!PER)
        for (; i < T.nlo; ++i) closure();
    const int iend = PER ? n : n - T.nhi, ku = PER ? min(T.ku, n) : 0;
    double fm2 = in[(PER ? n - 2 : i - 2) * s], fm1 = in[(PER ? n - 1 : i - 1) * s], f0 = in[i * s], fp1 = in[(i + 1) * s];
    double nf[R];   // f(i + 2) of the next run's rows
    auto fetch = [&](int b) {
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const int j = b + q + 2;
            nf[q] = in[(PER ? (j >= n ? j - n : j) : min(j, n - 1)) * s];
        }
    };
    fetch(i);
    for (; i < iend; i += R) {
        double f[R];
#pragma unroll
        for (int q = 0; q < R; ++q) f[q] = nf[q];
        if (i + R < iend) fetch(i + R);
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const int k = i + q;
            if (k >= iend) break;
            const double fp2 = f[q];
            double v;
            if constexpr (ACC)
                v = fma(__ldg(&ur[k].c), fp2 - fm2, fp1 - fm1) - __ldg(&ur[k].mu) * up;
            else
                v = __ldg(&rows[k].A) * (fp1 - fm1) + __ldg(&rows[k].B) * (fp2 - fm2) - __ldg(&rows[k].m) * up;
            w[k * s] = v;
            if (PER && k < ku) y0 += __ldg(ACC ? &T.u0s[k] : &T.u0[k]) * v;
            up = v;
            fm2 = fm1; fm1 = f0; f0 = fp1; fp1 = fp2;
        }
    }
    if (!PER)
        for (i = iend; i < n; ++i) closure();

    const double fact = PER ? (y0 + (ACC ? T.sm1s : T.sm1) * up) * T.sm2 : 0.0;
    double zn = 0.0, nw[R], no[R];
    auto fetch_back = [&](int b) {
#pragma unroll
        for (int q = 0; q < R; ++q) {
            nw[q] = w[max(b - q, 0) * s];
            if (ACC) no[q] = out[max(b - q, 0) * s];
        }
    };
    fetch_back(n - 1);
    for (i = n - 1; i >= 0; i -= R) {
        double v[R], old[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
            v[q] = nw[q];
            if (ACC) old[q] = no[q];
        }
        if (i >= R) fetch_back(i - R);
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const int k = i - q;
            if (k < 0) break;
            zn = v[q] - __ldg(ACC ? &ur[k].gu : &rows[k].g) * zn;
            const bool corr = PER && (k >= T.zhi || k < T.zlo);
            if constexpr (ACC) {
                double acc = old[q];
                if (corr) acc -= fact * __ldg(&T.zz[k]);
                out[k * s] = fma(__ldg(&ur[k].k), zn, acc);
            } else {
                out[k * s] = corr ? zn - fact * __ldg(&T.zz[k]) : zn;
            }
        }
    }
}

// the same by one warp, a lane a run of rows: each recurrence is an affine map of
// the value its lane starts from; the maps are composed by a scan and the runs
// walked again from their values.  row: n doubles of the warp's own.  False (and
// nothing stored) for infinities and NaN, which composed maps would spread.
template <int EPI, bool PER>
__device__ __noinline__ bool sweep_warp(const DerivTable &T, const double *__restrict__ in, double *out, long s,
                                        double *row, int lane) {
    constexpr bool ACC = EPI == EPI_ACCUM;
    constexpr unsigned kAll = 0xffffffffu;
    const int n = T.n, R = ((n + 31) / 32) | 1;   // odd: no bank conflicts
    const int first = min(lane * R, n), end = min(first + R, n);
    const DerivRow *rows = T.rows;
    const DerivRowU *ur = T.urows;
    bool finite = true;
    for (int i = lane; i < n; i += 32) {
        const double f = in[i * s];
        finite = finite && size_of(f) < 0x7ff00000;
        row[i] = f;
    }
    if (!__all_sync(kAll, finite)) return false;
    // what other runs hold, before they are overwritten
    auto at = [&](int i) { return row[PER ? (i < 0 ? i + n : (i >= n ? i - n : i)) : min(max(i, 0), n - 1)]; };
    double fm2 = at(first - 2), fm1 = at(first - 1), f0 = at(first), fp1 = at(first + 1);
    const double e0 = at(end), e1 = at(end + 1);
    double lo[4], hi[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        lo[q] = row[q];
        hi[q] = row[n - 1 - q];
    }
    __syncwarp();
    // right-hand sides, and each run from zero
    double a = 1.0, b = 0.0;
    for (int i = first; i < end; ++i) {
        const double fp2 = i + 2 < end ? row[i + 2] : (i + 2 == end ? e0 : e1);
        double r;
        if (!PER && (i < T.nlo || i >= n - T.nhi)) {
            const bool top = i >= T.nlo;
            const double *c = top ? T.chi + 4 * (n - 1 - i) : T.clo + 4 * i;
            r = c[0] * (top ? hi[0] : lo[0]) + c[1] * (top ? hi[1] : lo[1]) + c[2] * (top ? hi[2] : lo[2]) +
                c[3] * (top ? hi[3] : lo[3]);
        } else if constexpr (ACC) {
            r = fma(__ldg(&ur[i].c), fp2 - fm2, fp1 - fm1);
        } else {
            r = __ldg(&rows[i].A) * (fp1 - fm1) + __ldg(&rows[i].B) * (fp2 - fm2);
        }
        const double m = ACC ? __ldg(&ur[i].mu) : __ldg(&rows[i].m);
        b = r - m * b;
        a *= -m;
        row[i] = r;
        fm2 = fm1; fm1 = f0; f0 = fp1; fp1 = fp2;
    }
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
        const double pa = __shfl_up_sync(kAll, a, d), pb = __shfl_up_sync(kAll, b, d);
        if (lane >= d) {
            b = fma(a, pb, b);
            a *= pa;
        }
    }
    double v = __shfl_up_sync(kAll, b, 1), y0 = 0.0;
    if (lane == 0) v = 0.0;
    for (int i = first; i < end; ++i) {
        v = row[i] - (ACC ? __ldg(&ur[i].mu) : __ldg(&rows[i].m)) * v;
        row[i] = v;
        if (PER && i < T.ku) y0 += __ldg(ACC ? &T.u0s[i] : &T.u0[i]) * v;
    }
    double fact = 0.0;
    if constexpr (PER) {
#pragma unroll
        for (int d = 16; d; d /= 2) y0 += __shfl_xor_sync(kAll, y0, d);
        fact = (y0 + (ACC ? T.sm1s : T.sm1) * __shfl_sync(kAll, v, (n - 1) / R)) * T.sm2;
    }
    a = 1.0;
    b = 0.0;
    for (int i = end - 1; i >= first; --i) {
        const double g = ACC ? __ldg(&ur[i].gu) : __ldg(&rows[i].g);
        b = row[i] - g * b;
        a *= -g;
    }
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
        const double pa = __shfl_down_sync(kAll, a, d), pb = __shfl_down_sync(kAll, b, d);
        if (lane + d < 32) {
            b = fma(a, pb, b);
            a *= pa;
        }
    }
    double z = __shfl_down_sync(kAll, b, 1);
    if (lane == 31) z = 0.0;
    for (int i = end - 1; i >= first; --i) {
        z = row[i] - (ACC ? __ldg(&ur[i].gu) : __ldg(&rows[i].g)) * z;
        row[i] = z;
    }
    __syncwarp();
    for (int i = lane; i < n; i += 32) {
        const double corr = PER && (i >= T.zhi || i < T.zlo) ? fact * __ldg(&T.zz[i]) : 0.0;
        if constexpr (ACC) out[i * s] = fma(__ldg(&ur[i].k), row[i], out[i * s] - corr);
        else out[i * s] = row[i] - corr;
    }
    __syncwarp();
    return true;
}

// a tile of pencils as one thread sees it
struct Tile {
    const double *in;    // y, z: this thread's pencil; x: the field
    double *out;         // likewise
    long wofs;           // the pencil's offset in the field
    int p0, field;
    int b0, b1, ga, gb;  // blocks [b0, b1) of it, groups ga .. gb
    bool live;
};

// magnitudes of the 128 x pencils from p0 of field f: P at a time, two rows a
// lane, kScan / P / 2 rounds of 64 rows (two windows) each (P = 1: as many as it takes)
template <int P, bool PER>
EMIX_DEV void scan_x(const double *f, int p0, int np, int n, int uw, int step, int lane, Spread *to) {
    constexpr int C = kScan / P;
    constexpr bool kBefore = P == 1 || (PER && P <= 4);   // the value before the pencil: loaded, or among its rows
    constexpr int kB = kBefore ? P : 1;
    const int steps = P == 1 ? (n + 32 * C - 1) / (32 * C) : 1;
    double sv[kScan], before[kB], last = 0.0;   // last: P = 1, the rows' last value so far
    int top = 0, least = 0;
    unsigned low = 0;
    auto load = [&](int u, int st) {
        const int r = st * 32 * C + 2 * lane;
#pragma unroll
        for (int i = 0; i < P; ++i) {
            const double *fp = f + (long)min(p0 + u * P + i, np - 1) * n;
            if (kBefore && st == 0) before[i < kB ? i : 0] = fp[PER ? n - 1 : 0];
#pragma unroll
            for (int q = 0; q < C; ++q) sv[i * C + q] = fp[min(r + 64 * (q >> 1) + (q & 1), n - 1)];
        }
    };
    int u = uw, st = 0;
    if (u < kMmaPencils / P) load(u, 0);
    while (u < kMmaPencils / P) {
#pragma unroll
        for (int i = 0; i < P; ++i) {
            if (st == 0) {
                top = 0;
                least = 0x7fffffff;
                low = 0;
                if constexpr (kBefore) last = before[i < kB ? i : 0];
                else if constexpr (PER) {   // 64 rows at most
                    const double x = __shfl_sync(0xffffffffu, sv[i * C], (n - 1) >> 1);
                    last = __shfl_sync(0xffffffffu, sv[i * C + 1], (n - 1) >> 1);
                    if ((n - 1) % 2 == 0) last = x;
                } else {
                    last = __shfl_sync(0xffffffffu, sv[i * C], 0);
                }
            }
#pragma unroll
            for (int q = 0; q < C; q += 2) {
                const double x = sv[i * C + q], y = sv[i * C + q + 1];
                const double d = x - __shfl_sync(0xffffffffu, lane == 31 ? last : y, (lane + 31) & 31), e = y - x;
                last = y;
                low |= (unsigned)__double2loint(d) | (unsigned)__double2loint(e);
                const int m = max(size_of(d), size_of(e));
                // the lower and the upper 16 lanes' rows
                const int w0 = __reduce_max_sync(0xffffffffu, lane < 16 ? m : 0);
                const int w1 = __reduce_max_sync(0xffffffffu, lane < 16 ? 0 : m);
                top = max(top, max(w0, w1));
                // the rows after the last whole window count with it
                const int r = 32 * (st * C + q);
                if (r + 32 <= n) least = min(least, w0);
                if (r + 64 <= n) least = min(least, w1);
            }
            if (st == steps - 1) {
                const unsigned lw = __reduce_or_sync(0xffffffffu, low);
                if (lane == 0) to[u * P + i] = Spread{top, least, lw};
            }
        }
        if (++st == steps) {
            st = 0;
            u += step;
        }
        if (u < kMmaPencils / P) load(u, st);
    }
}

// XAX: pencils along x (rows contiguous, brought through a shared tile);
// otherwise along y or z (pencils contiguous along x)
// CTA `cta` of the I.ncta that share the item
template <bool XAX, int EPI, int KIND>
EMIX_DEV void mma_body(const MmaItem &I, int cta, const QuietGate *gate) {
    constexpr bool PER = KIND == kCyclic || KIND == kRound;
    constexpr int kScanParts = scan_parts(XAX);
    const MmaTable &M = I.M;
    const PencilFields &F = I.F;
    const int np = I.np, ntile = I.ntile, nf = I.nf, whole = I.whole, segs = I.segs, nx = I.nx, ncta = I.ncta;
    const long s = I.s, os = I.os;
    extern __shared__ __align__(1024) unsigned char dyn[];
    __shared__ unsigned s_tmem;
    __shared__ int s_fail;
    // full[a]: the tensor core has finished a block in sum buffer a; drained[a]:
    // all warps have read it; conv[q]: group q (mod 8) is in tensor memory;
    // done[b]: block b (mod 8) is finished, for the converting warps, which lag
    // by up to five blocks at a tile's end; scaled[t]: tile t's (mod 2)
    // magnitudes are in s_part; read[t]: every warp that wants them has them
    __shared__ __align__(8) unsigned long long s_full[2], s_drained[2], s_conv[8], s_done[8],
        s_scaled[2], s_read[2], s_table;
    __shared__ Spread s_part[2][kScanParts][kMmaPencils];   // by the tile's parity
    __shared__ unsigned char s_scalar[kMmaPencils];
    __shared__ unsigned s_sweep[kMmaSweepJobs][4];   // pencils of the CTA's jobs that take the scalar sweep
    __shared__ int s_sweeps;                          // their number
    const int tid = threadIdx.x, lane = tid & 31;
    // through a shuffle: the roles' branches are then known to be uniform, and
    // the instruction operands stay in uniform registers
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int n = M.n;

    if (tid == 0) {
        s_fail = 0;
        s_sweeps = 0;
        for (int q = 0; q < 2; ++q) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&s_full[q])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(&s_drained[q])), "r"(kRoleWarps) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(&s_scaled[q])), "r"(kScanWarps) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(&s_read[q])), "r"(2 * kRoleWarps + 1) : "memory");
        }
        for (int q = 0; q < 8; ++q) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(&s_conv[q])), "r"(kRoleWarps) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&s_done[q])) : "memory");
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&s_table)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        // the operator's digits, by bulk copies that land during the first scan
        // (four steps of a 40^3 tank: 1363 us, 1408 with loads before it)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                     :: "r"(smem_u32(&s_table)), "r"(M.ntype * kMmaTypeBytes) : "memory");
        for (int q = 0; q < M.ntype; ++q)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         :: "r"(smem_u32(dyn + q * kMmaTypeBytes)),
                            "l"(reinterpret_cast<const unsigned char *>(M.b) + (size_t)q * kMmaTypeBytes),
                            "r"(kMmaTypeBytes), "r"(smem_u32(&s_table)) : "memory");
    }
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_u32(&s_tmem)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // all columns were asked for, so they begin at 0: a constant, which keeps
    // the tensor-core instructions' operands in uniform registers
    constexpr unsigned tm = 0;
    const int nblk = M.nblk;
    const int g0 = PER ? -2 : 0;                                   // first and last group of a tile
    const int g1 = PER ? nblk + 2 : (n + 6) / kMmaRows;
    int jobs = whole + (ntile * nf - whole) * segs;
    constexpr bool round = KIND == kRound;
    constexpr int kOutTiles = out_tiles(KIND);
    bool ok = true;                                                // false: a wait ran out; nothing is stored any more

    // bounded wait; once one has run out no further one is waited for, and
    // the loops below run out by themselves
    auto wait = [&](unsigned long long *bar, unsigned parity) {
        if (!ok) return;   // the same in all lanes
        const unsigned addr = smem_u32(bar);
        for (int it = 0; it < kMmaWaitLimit; ++it) {
            unsigned done;
            asm volatile("{\n\t.reg .pred p;\n\t"
                         "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
                         "selp.u32 %0, 1, 0, p;\n\t}"
                         : "=r"(done) : "r"(addr), "r"(parity), "r"(kMmaWaitNs) : "memory");
            if (__all_sync(0xffffffffu, done)) return;
            if (__any_sync(0xffffffffu, *(volatile int *)&s_fail)) break;
        }
        *(volatile int *)&s_fail = 1;
        ok = false;
    };
    auto arrive = [&](unsigned long long *bar) {
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(smem_u32(bar)) : "memory");
    };
    auto row_sync = [](int id) { asm volatile("bar.sync %0, %1;" :: "r"(id), "n"(kRole) : "memory"); };

    // row of a pencil: wrapped (cyclic), or clamped to the ends, where the
    // repeated value makes the differences beyond them zero
    auto row_of = [&](int k) {
        if constexpr (PER) {
            while (k < 0) k += n;
            while (k >= n) k -= n;
            return k;
        }
        return min(max(k, 0), n - 1);
    };
    // job: a whole tile, or (from `whole` on) one of `segs` segments of one
    auto tile_of = [&](int job, int slot_p) {
        Tile t;
        int id = job, seg = 0, cut = 1;
        if (job >= whole) {
            id = whole + (job - whole) / segs;
            seg = (job - whole) % segs;
            cut = segs;
        }
        t.b0 = nblk * seg / cut;
        t.b1 = nblk * (seg + 1) / cut;
        t.ga = round ? 0 : max(g0, t.b0 - 2);
        t.gb = round ? nblk - 1 : min(g1, t.b1 + 2);
        t.field = id / ntile;
        t.p0 = (id - t.field * ntile) * kMmaPencils;
        const int p = min(t.p0 + slot_p, np - 1);
        t.live = t.p0 + slot_p < np;
        t.wofs = XAX ? (long)p * n : (long)(p % nx) + (long)(p / nx) * os;
        t.in = pick(F.in, t.field) + (XAX ? 0 : t.wofs);
        t.out = pick(F.out, t.field) + (XAX ? 0 : t.wofs);
        return t;
    };

    // magnitudes of a tile's pencils into s_part[buf]: this warp takes units
    // uw, uw + step, ...; kScan values a lane and step, loaded a step ahead
    auto scan_tile = [&](int job, int buf, int uw, int step) {
        if constexpr (!XAX) {
            // units of 32 pencils (lanes) by a part of the rows
            const int part = (n + kScanParts - 1) / kScanParts, steps = (part + kScan - 1) / kScan;
            double sv[kScan], before = 0.0, prev = 0.0;   // before: the value before the unit's first row
            const double *fp = nullptr;
            int ra = 0, rb = 0, top = 0, least = 0;
            unsigned low = 0;
            int rows = 0;                      // rows loaded that are the part's
            bool window = false;               // they are one that counts by itself
            auto load = [&](int u, int st) {
                if (st == 0) {
                    fp = tile_of(job, (u & 3) * 32 + lane).in;
                    ra = min((u >> 2) * part, n - 1);
                    rb = min(ra + part, n) - 1;
                    before = fp[(long)row_of(ra - 1) * s];
                }
                const int r = ra + st * kScan;
                const double *q0 = fp + (long)r * s;
                // fewer rows count with the window before them
                rows = min(kScan, rb - r + 1);
                window = rows == kScan || st == 0;
                if (r + kScan <= n) {
#pragma unroll
                    for (int q = 0; q < kScan; ++q) sv[q] = q0[q * s];
                } else {
#pragma unroll
                    for (int q = 0; q < kScan; ++q) sv[q] = fp[(long)min(r + q, rb) * s];
                }
            };
            int u = uw, st = 0;
            if (u < 4 * kScanParts) load(u, 0);
            while (u < 4 * kScanParts) {
                if (st == 0) {
                    top = 0;
                    least = 0x7fffffff;
                    low = 0;
                    prev = before;
                }
                int w = 0;
                auto take = [&](int q) {
                    const double d = sv[q] - prev;
                    prev = sv[q];
                    w = max(w, size_of(d));
                    low |= (unsigned)__double2loint(d);
                };
                if (rows == kScan) {
#pragma unroll
                    for (int q = 0; q < kScan; ++q) take(q);
                } else {
#pragma unroll
                    for (int q = 0; q < kScan; ++q) {
                        if (q >= rows) break;
                        take(q);
                    }
                }
                top = max(top, w);
                if (window) least = min(least, w);
                const int uu = u;
                if (++st == steps) {
                    st = 0;
                    u += step;
                }
                if (u < 4 * kScanParts) load(u, st);
                if (u != uu) s_part[buf][uu >> 2][(uu & 3) * 32 + lane] = Spread{top, least, low};
            }
        } else {
            const Tile tl = tile_of(job, 0);
            Spread *to = s_part[buf][0];
            if (n <= 32 * (kScan / 8)) scan_x<8, PER>(tl.in, tl.p0, np, n, uw, step, lane, to);
            else if (n <= 32 * (kScan / 4)) scan_x<4, PER>(tl.in, tl.p0, np, n, uw, step, lane, to);
            else if (n <= 32 * (kScan / 2)) scan_x<2, PER>(tl.in, tl.p0, np, n, uw, step, lane, to);
            else scan_x<1, PER>(tl.in, tl.p0, np, n, uw, step, lane, to);
        }
    };
    // slot's pencil of tile t (from p0), once its magnitudes are known; skip: every
    // pencil of the tile takes the sweep, and the roles leave it out
    auto scale_wait = [&](int t, int p0, int slot, bool &skip) {
        if (t > 0) wait(&s_scaled[t & 1], (unsigned)((t - 1) >> 1) & 1);
        auto scale = [&](int q) {
            Spread a = s_part[t & 1][0][q];
#pragma unroll
            for (int i = 1; i < kScanParts; ++i) {
                const Spread b = s_part[t & 1][i][q];
                a.top = max(a.top, b.top);
                a.least = min(a.least, b.least);
                a.low |= b.low;
            }
            return scale_of(a, M.se);
        };
        const Scale sc = scale(slot);
        bool all = __all_sync(0xffffffffu, sc.scalar || p0 + slot >= np);
#pragma unroll 1
        for (int q = lane; q < kMmaPencils && all; q += 32)
            all = __all_sync(0xffffffffu, scale(q).scalar || p0 + q >= np);
        skip = __shfl_sync(0xffffffffu, (int)all, 0);   // known to be uniform
        arrive(&s_read[t & 1]);
        return sc;
    };
    // the sweep of the caller's pencil of a tile
    auto sweep = [&](const Tile &t) {
        const long x = XAX ? t.wofs : 0;
        double *w = pick(F.w, t.field) + t.wofs;
        sweep_pencil<EPI, PER>(I.T, t.in + x, w, t.out + x, s);
    };
    constexpr int kPencilWarps = 2 * kRoleWarps + kScanWarps;   // all but the tensor core's
    wait_for_previous();   // what is read so far is constant
    if (gate && gate->sweeps) jobs = 0;   // nothing to do, past the setup
    if (warp != 2 * kRoleWarps && jobs > 0) {
        // the first tile's, by all of them
        scan_tile(cta, 0, warp < 2 * kRoleWarps ? warp : warp - 1, kPencilWarps);
    }
    // (the barriers, tensor memory and the operator are on their way meanwhile)
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (s_tmem != tm && tid == 0) s_fail = 1;

    if (warp == 2 * kRoleWarps) {
        // ---- the tensor core's warp ----------------------------------------
        {
            unsigned leader;
            asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(leader));
            int B = 0, first = 0;     // block, and the tile's first group, counted over the tiles
            int seen = 0;             // groups known to be in tensor memory
            const bool signal = leader && !*(volatile int *)&g_mma_drop;
            wait(&s_table, 0);
            int t = 0;
            for (int job = cta; job < jobs; job += ncta, ++t) {
                const Tile jt = tile_of(job, 0);
                bool skip;
                scale_wait(t, jt.p0, lane, skip);
                if (skip) continue;
                for (int b = jt.b0; b < jt.b1; ++b, ++B) {
                    for (const int need = first + min(b + 3, jt.gb) - jt.ga; seen <= need; ++seen)
                        wait(&s_conv[seen & 7], (unsigned)(seen >> 3) & 1);
                    if (B >= 2) wait(&s_drained[B & 1], (unsigned)((B - 2) >> 1) & 1);
                    if (!ok) continue;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const int ty = b < M.nlow ? b : (b >= nblk - M.nhigh ? M.ntype - (nblk - b) : M.nlow);
                    const unsigned base = smem_u32(dyn) + (unsigned)(ty * kMmaTypeBytes);
                    // the K-major operand without swizzle: 8 x 16-byte core
                    // matrices, 128 bytes apart along the rows, kMmaStack x 16
                    // along the columns
                    constexpr unsigned long long desc0 =
                        (1ull << 46) | ((unsigned long long)(128 >> 4) << 32) |
                        ((unsigned long long)((kMmaStack * 16) >> 4) << 16);
                    const unsigned sums = tm + (unsigned)(B & 1) * kAccCols;
                    constexpr int kLead[kMmaWin] = {kMmaLead0, kMmaLead1, 0, 0, kMmaLead1, kMmaLead0};
                    // the group in window place w: its digits' columns and operand
                    unsigned ah[kMmaWin], al[kMmaWin], lo[kMmaWin];
#pragma unroll
                    for (int w = 0; w < kMmaWin; ++w) {
                        int g = b - 2 + w;
                        if (round) g += g < 0 ? nblk : (g >= nblk ? -nblk : 0);
                        const unsigned c = (unsigned)(first + g - jt.ga + kHighRing * kLowRing);
                        ah[w] = tm + kHighCol + (c % kHighRing) * 24;
                        al[w] = tm + kLowCol + (c % kLowRing) * 24;
                        lo[w] = ((base + w * kMmaGroupBytes + kLead[w] * (kMmaRows * 16)) >> 4) & 0x3fff;
                    }
                    // digit j of the group in place w; the block's own group (w = 2)
                    // comes first and sets every sum
                    auto product = [&](int w, int j) {
                        const unsigned idesc = (1u << 4) | ((unsigned)((kMmaDig - kLead[w] - j) * kMmaRows >> 3) << 17) |
                                               ((kMmaPencils >> 4) << 24);
                        mma_f16(sums + (kLead[w] + j) * kMmaRows, j < 3 ? ah[w] + j * 8 : al[w] + (j - 3) * 8,
                                desc0 | lo[w], idesc, !(w == 2 && j == 0), leader);
                    };
                    constexpr int kOrder[kMmaWin] = {2, 0, 1, 3, 4, 5};
                    if (round || (b - 2 >= jt.ga && b + 3 <= jt.gb)) {
                        // digit by digit: instructions on the same sums follow one
                        // another (1900 clocks a block alone, 2180 group by group)
#pragma unroll
                        for (int j = 0; j < kMmaDig; ++j)
#pragma unroll
                            for (int q = 0; q < kMmaWin; ++q)
                                if (j < kMmaDig - kLead[kOrder[q]]) product(kOrder[q], j);
                    } else {
#pragma unroll
                        for (int q = 0; q < kMmaWin; ++q) {
                            const int w = kOrder[q], g = b - 2 + w;
                            if (g < jt.ga || g > jt.gb) continue;
#pragma unroll
                            for (int j = 0; j < kMmaDig - kLead[w]; ++j) product(w, j);
                        }
                    }
                    __syncwarp();
                    if (signal)
                        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t"
                                     "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%1];"
                                     :: "r"(smem_u32(&s_full[B & 1])), "r"(smem_u32(&s_done[B & 7])) : "memory");
                }
                first += jt.gb - jt.ga + 1;
            }
        }
    } else if (warp > 2 * kRoleWarps) {
        // ---- magnitudes of the tiles' pencils, one tile ahead ------------------
        int t = 1;
        for (int job = cta + ncta; job < jobs; job += ncta, ++t) {
            if (t >= 2) wait(&s_read[t & 1], (unsigned)((t - 2) >> 1) & 1);   // s_part's turn
            scan_tile(job, t & 1, warp - 2 * kRoleWarps - 1, kScanWarps);
            arrive(&s_scaled[t & 1]);
        }
    } else {
        // ---- the pencils' warps: converting, or the results --------------------
        const bool results = warp >= kRoleWarps;
        const int rtid = results ? tid - kRole : tid, rwarp = results ? warp - kRoleWarps : warp;
        const int quarter = warp & 3;                     // tensor-memory lanes 32 quarter ..
        const int rg = rwarp >> 2;                        // rows kRpt rg .. of a group or block
        const int slot_p = quarter * 32 + lane;           // this thread's pencil in the tile
        const unsigned tml = tm + ((unsigned)(quarter * 32) << 16);
        double *xin = reinterpret_cast<double *>(dyn + (size_t)M.ntype * kMmaTypeBytes);
        double *xout = xin + 2 * kXTileDoubles;
        if (!results) {
            // ---- a group's rows to digits, loaded one group ahead ---------------
            double v[kRpt + 1];   // y, z: the thread's rows; x: staged values
            auto load = [&](const Tile &t, int g) {
                int k = kMmaRows * g - 8;
                if constexpr (PER) {
                    // once for the group; its rows then wrap at most once (a loop
                    // for each: 5 fields of 64^3 31 us, here 25; 128^3 105, 91)
                    while (k < 0) k += n;
                    while (k >= n) k -= n;
                }
                auto wrap = [&](int r) {
                    if constexpr (PER) return r >= n ? r - n : r;
                    return min(max(r, 0), n - 1);
                };
                if constexpr (!XAX) {
                    if (k >= 0 && k + kMmaRows < n) {
                        const double *fp = t.in + (long)(k + kRpt * rg) * s;
#pragma unroll
                        for (int q = 0; q <= kRpt; ++q) v[q] = fp[q * s];
                    } else {
#pragma unroll
                        for (int q = 0; q <= kRpt; ++q) v[q] = t.in[(long)wrap(k + kRpt * rg + q) * s];
                    }
                } else {
                    const int row = wrap(k + (rtid & 15));
#pragma unroll
                    for (int q = 0; q < kRpt; ++q)
                        v[q] = t.in[(long)min(t.p0 + (rtid >> 4) + (kRole / 16) * q, np - 1) * n + row];
                    if (rtid < kMmaPencils) v[kRpt] = t.in[(long)min(t.p0 + rtid, np - 1) * n + wrap(k + 16)];
                }
            };
            auto stage = [&](int c) {   // x: into the tile of group c
                double *t = xin + (c & 1) * kXTileDoubles;
#pragma unroll
                for (int q = 0; q < kRpt; ++q) t[((rtid >> 4) + (kRole / 16) * q) * kXPitch + (rtid & 15)] = v[q];
                if (rtid < kMmaPencils) t[rtid * kXPitch + 16] = v[kRpt];
            };
            // the staged rows' (x: tile c's) digits
            unsigned dg[kMmaDig][kRpt / 2];
            auto convert = [&](int c, const Scale &sc) {
                unsigned w1[kRpt], w2[kRpt];
                const double *t = xin + (c & 1) * kXTileDoubles + slot_p * kXPitch + kRpt * rg;
                unsigned long long a = to_fixed(XAX ? t[0] : v[0], sc.E);
#pragma unroll
                for (int q = 0; q < kRpt; ++q) {
                    const unsigned long long b = to_fixed(XAX ? t[q + 1] : v[q + 1], sc.E);
                    // digits at bits 4 + 10 j, biased by 512; half of the bits dropped below
                    const unsigned long long y = b - a + 0x8020080200802008ull;
                    a = b;
                    w1[q] = (unsigned)(y >> 32);
                    w2[q] = (unsigned)(y >> 4);
                }
                digits<22>(dg[0], w1);
                digits<12>(dg[1], w1);
                digits<2>(dg[2], w1);
                digits<20>(dg[3], w2);
                digits<10>(dg[4], w2);
                digits<0>(dg[5], w2);
            };
            auto put = [&](int c) {
                const unsigned ah = tml + kHighCol + (unsigned)(c % kHighRing) * 24 + rg * (kRpt / 2);
                const unsigned al = tml + kLowCol + (unsigned)(c % kLowRing) * 24 + rg * (kRpt / 2);
#pragma unroll
                for (int j = 0; j < kMmaDig; ++j)
                    tm_st4((j < 3 ? ah : al) + j % 3 * 8, dg[j][0], dg[j][1], dg[j][2], dg[j][3]);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                arrive(&s_conv[c & 7]);
            };
            int c = 0, done = 0, t = 0, B = 0;   // groups, finished blocks, jobs, the job's first block
            int job = cta;
            Tile cur = tile_of(job, slot_p), last = cur;
            // the last block (counted over the jobs) that reads group `pos` of a
            // job, `reach` groups behind it at most; of one before the previous
            // job, the last of that
            auto last_use = [&](int pos, int reach) {
                if (round) reach = nblk;
                if (pos >= 0) return B + min(cur.ga + pos + reach, cur.b1 - 1) - cur.b0;
                const int Bl = B - (last.b1 - last.b0);
                if (!B) return -1;
                pos += last.gb - last.ga + 1;
                return pos >= 0 ? Bl + min(last.ga + pos + reach, last.b1 - 1) - last.b0 : Bl - 1;
            };
            load(cur, cur.ga);
            for (; job < jobs; job += ncta, ++t) {
                bool skip;
                const Scale sc = scale_wait(t, cur.p0, slot_p, skip);
                const bool more = job + ncta < jobs;
                Tile nxt = cur;
                if (more) nxt = tile_of(job + ncta, slot_p);
                const int ng = cur.gb - cur.ga + 1;
                if (skip) {
                    // (as many barriers as of other tiles: a wait that ran out may have
                    // left the warps of different minds)
                    if constexpr (XAX)
                        for (int k = 0; k < ng; ++k) row_sync(1);
                    if (more) load(nxt, nxt.ga);
                    cur = nxt;
                    continue;
                }
                for (int k = 0; k < ng; ++k, ++c) {
                    // the rings' places are free once the blocks that read them are done
                    const int need = max(last_use(k - kHighRing, 2), last_use(k - kLowRing, 1));
                    if constexpr (XAX) {
                        stage(c);
                        row_sync(1);
                        if (k + 1 < ng) load(cur, cur.ga + k + 1);
                        else if (more) load(nxt, nxt.ga);
                    }
                    // the arithmetic first, so that only the stores wait for the blocks
                    convert(c, sc);
                    if constexpr (!XAX) {
                        if (k + 1 < ng) load(cur, cur.ga + k + 1);
                        else if (more) load(nxt, nxt.ga);
                    }
                    for (; done <= need; ++done) wait(&s_done[done & 7], (unsigned)(done >> 3) & 1);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    put(c);
                }
                B += cur.b1 - cur.b0;
                last = cur;
                cur = nxt;
            }
        } else {
            // sums of the digit orders 0..5 combined exactly (weights 2^42, 2^32,
            // 2^22, 2^12, 2^2 and 2^-8), then scaled
            auto combine = [](const float (&acc)[kMmaDig][kRpt], int q, int escale) {
                const int a0 = __float2int_rn(acc[0][q]), a1 = __float2int_rn(acc[1][q]);
                const int a2 = __float2int_rn(acc[2][q]), a3 = __float2int_rn(acc[3][q]);
                const int a4 = __float2int_rn(acc[4][q]), a5 = __float2int_rn(acc[5][q]);
                long long r = (long long)(a4 * 4 + (a5 >> 8));
                r += (long long)a3 * 4096;
                r += (long long)a2 * (1 << 22);
                const unsigned hi = (unsigned)(r >> 32) + (unsigned)(a0 * 1024 + a1);
                const double d = (double)(long long)(((unsigned long long)hi << 32) | (unsigned)r);
                const int dh = __double2hiint(d);
                return __hiloint2double(dh ? dh + escale : 0, __double2loint(d));
            };

            // ---- the stream of blocks ----------------------------------------------
            int B = 0, t = 0;
            for (int job = cta; job < jobs; job += ncta, ++t) {
                const Tile cur = tile_of(job, slot_p);
                bool skip;
                const Scale sc = scale_wait(t, cur.p0, slot_p, skip);
                const int escale = (sc.E - 1023 - M.se) * (1 << 20);
                if (XAX && rg == 0) s_scalar[slot_p] = sc.scalar;
                // the pencils that take the sweep: after the tiles, by all warps
                // (those of jobs past the record's end: now)
                if (rg == 0) {
                    const bool mine = sc.scalar && cur.live && ok && cur.b0 == 0;
                    const unsigned m = __ballot_sync(0xffffffffu, mine);
                    if (t < kMmaSweepJobs) {
                        if (lane == 0) s_sweep[t][quarter] = m;
                    } else if (mine) {
                        sweep(cur);
                    }
                }
                if (skip) {
                    if constexpr (XAX)
                        for (int q = (cur.b1 - cur.b0) * (3 - kOutTiles); q >= 0; --q) row_sync(2);
                    continue;
                }
                for (int b = cur.b0; b < cur.b1; ++b, ++B) {
                    const int row = kMmaRows * b + kRpt * rg;
                    double old[kRpt];
                    if constexpr (EPI == EPI_ACCUM && !XAX) {
#pragma unroll
                        for (int q = 0; q < kRpt; ++q) old[q] = cur.out[(long)min(row + q, n - 1) * s];
                    }
                    wait(&s_full[B & 1], (unsigned)(B >> 1) & 1);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    float acc[kMmaDig][kRpt];
#pragma unroll
                    for (int j = 0; j < kMmaDig; ++j)
                        tm_ld8(tml + (unsigned)(B & 1) * kAccCols + j * kMmaRows + kRpt * rg, acc[j]);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    // the sums are not touched before the wait
#pragma unroll
                    for (int j = 0; j < kMmaDig; ++j)
                        asm volatile("" : "+f"(acc[j][0]), "+f"(acc[j][1]), "+f"(acc[j][2]), "+f"(acc[j][3]),
                                          "+f"(acc[j][4]), "+f"(acc[j][5]), "+f"(acc[j][6]), "+f"(acc[j][7]));
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    arrive(&s_drained[B & 1]);
                    if constexpr (!XAX) {
                        if (cur.live && !sc.scalar && ok) {
                            double *o = cur.out + (long)row * s;
                            if (row + kRpt <= n) {
#pragma unroll
                                for (int q = 0; q < kRpt; ++q) {
                                    double r = combine(acc, q, escale);
                                    if constexpr (EPI == EPI_ACCUM) r += old[q];
                                    o[q * s] = r;
                                }
                            } else {
#pragma unroll
                                for (int q = 0; q < kRpt; ++q) {
                                    double r = combine(acc, q, escale);
                                    if constexpr (EPI == EPI_ACCUM) r += old[q];
                                    if (row + q < n) o[q * s] = r;
                                }
                            }
                        }
                    } else {
                        double *tl = xout + (kOutTiles == 2 ? B & 1 : 0) * kXTileDoubles;
#pragma unroll
                        for (int q = 0; q < kRpt; ++q) tl[slot_p * kXPitch + kRpt * rg + q] = combine(acc, q, escale);
                        row_sync(2);
                        // the block's tile to memory, rows along the lanes
                        const int frow = kMmaRows * b + (rtid & 15);
                        double *o = cur.out + (long)(cur.p0 + (rtid >> 4)) * n + frow;
#pragma unroll
                        for (int q = 0; q < kRpt; ++q) {
                            const int pp = (rtid >> 4) + (kRole / 16) * q;
                            if (frow < n && cur.p0 + pp < np && !s_scalar[pp] && ok) {
                                double r = tl[pp * kXPitch + (rtid & 15)];
                                if (EPI == EPI_ACCUM) r += *o;
                                *o = r;
                            }
                            o += (long)(kRole / 16) * n;
                        }
                        if constexpr (kOutTiles == 1) row_sync(2);   // the tile is free
                    }
                }
                if constexpr (XAX) row_sync(2);   // s_scalar is free
            }
        }
    }
    // a wait that ran out: counted; tensor memory goes only after what the
    // tensor core still has in flight (bounded)
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (s_fail) {
        if (tid == 0) atomicAdd(&g_mma_timeouts, 1);
        for (int q = 0; q < 1 << 16; ++q) __nanosleep(256);
    }
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tm), "r"(kTmemCols));
    // the sweeps: their list, then a row buffer for each warp, in dyn, which nothing
    // reads any more
    static_assert(kMmaSweepJobs * 4 <= kMmaThreads && kMmaSweepJobs * kMmaPencils <= 65536, "s_sweep");
    const int mine = (jobs - cta + ncta - 1) / ncta;
    unsigned bits = tid < 4 * min(mine, kMmaSweepJobs) && !s_fail ? s_sweep[tid >> 2][tid & 3] : 0;
    if (!__syncthreads_or(bits != 0)) return;
    unsigned short *list = reinterpret_cast<unsigned short *>(dyn);
    if (bits) {
        int at = atomicAdd(&s_sweeps, __popc(bits));
        for (; bits; bits &= bits - 1) list[at++] = (unsigned short)(32 * tid + __ffs((int)bits) - 1);
    }
    __syncthreads();
    const int count = s_sweeps;
    if (count > kSweepWarps * max(1, n / 96)) {
        for (int q = tid; q < count; q += kMmaThreads) sweep(tile_of(cta + (list[q] >> 7) * ncta, list[q] & 127));
        return;
    }
    constexpr int kListBytes = kSweepWarps * (kTableMaxN / 96) * 2;
    const int warps = min((kMmaShared - kListBytes) / (8 * n), kSweepWarps);
    if (warp >= warps) return;
    double *row = reinterpret_cast<double *>(dyn + kListBytes) + (size_t)warp * n;
    for (int q = warp; q < count; q += warps) {
        const Tile t = tile_of(cta + (list[q] >> 7) * ncta, list[q] & 127);
        const long x = XAX ? t.wofs : 0;
        if (!sweep_warp<EPI, PER>(I.T, t.in + x, t.out + x, s, row, lane) && lane == 0) sweep(t);
    }
}

// 32 neighbouring pencils a block, each group's `every`-th: which of them are quiet
// somewhere (windows as of the scan, 16 rows or along x 32)
template <bool XAX>
__global__ void __launch_bounds__(256) k_quiet_sample(PencilFields F, int nf, int n, int np, int nx, long s, long os,
                                                      int limit, QuietGate *gate) {
    __shared__ int s_top[8][32], s_least[8][32];
    wait_for_previous();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int per = (np + 31) / 32, id = (int)((long)blockIdx.x * per * nf / gridDim.x);
    const int f = id / per, p0 = (id - f * per) * 32;
    int top = 0, least = 0x7fffffff;
    if constexpr (!XAX) {
        const int p = min(p0 + lane, np - 1);
        const double *in = pick(F.in, f) + p % nx + (long)(p / nx) * os;
        for (int r = 16 * warp; r < n; r += 128) {
            double prev = in[(long)max(r - 1, 0) * s], v[16];
#pragma unroll
            for (int q = 0; q < 16; ++q) v[q] = in[(long)min(r + q, n - 1) * s];
            int w = 0;
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                w = max(w, size_of(v[q] - prev));
                prev = v[q];
            }
            top = max(top, w);
            if (r + 16 <= n) least = min(least, w);
        }
        s_top[warp][lane] = top;
        s_least[warp][lane] = least;
    } else {
        for (int q = warp; q < 32; q += 8) {
            const double *in = pick(F.in, f) + (long)min(p0 + q, np - 1) * n;
            int t = 0, l = 0x7fffffff;
            for (int r0 = 0; r0 < n; r0 += 32) {
                const int r = min(r0 + lane, n - 1);
                const int w = __reduce_max_sync(0xffffffffu, size_of(in[r] - in[max(r - 1, 0)]));
                t = max(t, w);
                if (r0 + 32 <= n) l = min(l, w);
            }
            if (lane < 8) {
                s_top[lane][q] = t;
                s_least[lane][q] = l;
            }
        }
    }
    __syncthreads();
    if (warp != 0) return;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        top = max(top, s_top[q][lane]);
        least = min(least, s_least[q][lane]);
    }
    const unsigned quiet = __ballot_sync(0xffffffffu, p0 + lane < np && top - least > kMmaSpan << 20);
    if (lane == 0) {
        atomicAdd(&gate->sum, __popc(quiet));
        __threadfence();
        if (atomicAdd(&gate->done, 1) == (int)gridDim.x - 1) {   // the last block
            __threadfence();
            gate->sweeps = atomicExch(&gate->sum, 0) > limit;
            gate->done = 0;
        }
    }
}

template <bool XAX, int EPI, int KIND>
__global__ void __launch_bounds__(kMmaThreads, 1) k_deriv_mma(const __grid_constant__ MmaItem I) {
    mma_body<XAX, EPI, KIND>(I, blockIdx.x, I.gate);
}

// many grids' derivatives: the SMs are divided between the items (mma_split)
template <bool XAX, int EPI, int KIND>
__global__ void __launch_bounds__(kMmaThreads, 1) k_batch_deriv_mma(const MmaItem *__restrict__ items, int count) {
    __shared__ MmaItem s_item;
    int g = 0;
    for (int hi = count - 1; g < hi;) {
        const int mid = (g + hi + 1) >> 1;
        if (items[mid].cta0 <= (int)blockIdx.x) g = mid; else hi = mid - 1;
    }
    static_assert(sizeof(MmaItem) % sizeof(int) == 0, "copied by words");
    for (int q = threadIdx.x; q < (int)(sizeof(MmaItem) / sizeof(int)); q += kMmaThreads)
        reinterpret_cast<int *>(&s_item)[q] = reinterpret_cast<const int *>(items + g)[q];
    __syncthreads();
    mma_body<XAX, EPI, KIND>(s_item, (int)blockIdx.x - s_item.cta0, nullptr);
}

// tensor memory is taken whole: at least 116 KB of shared memory keeps a
// second CTA off the SM
template <bool XAX, int KIND>
int shared_bytes(int ntype) {
    const int shm = ntype * kMmaTypeBytes + (XAX ? (2 + out_tiles(KIND)) * kXTileDoubles * (int)sizeof(double) : 0);
    return shm < kMmaShared ? kMmaShared : shm;
}

// divides item I between at most `n` CTAs (I.ncta: those that get work):
// whole tiles while they fill every CTA; what is left is cut into the number
// of segments (each with five more groups to convert) that ends first.
// Returns the blocks and starts the most loaded CTA walks
long divide(MmaItem &I, int n) {
    const int tiles = I.ntile * I.nf, rest = tiles % n;
    I.whole = tiles - rest;
    I.segs = 1;
    long best = 0;
    for (int c = 1; rest > 0 && c <= I.M.nblk && c <= 64; ++c) {
        const long rounds = ((long)rest * c + n - 1) / n, t = rounds * ((I.M.nblk + c - 1) / c + 6);
        if (c == 1 || t < best) { best = t; I.segs = c; }
    }
    const long jobs = I.whole + (long)rest * I.segs;
    I.ncta = (int)(jobs < n ? jobs : n);
    return best + (long)(I.whole / n) * (I.M.nblk + 6);
}

template <bool XAX, int EPI, int KIND>
int launch(const MmaItem &I, cudaStream_t st) {
    const int shm = shared_bytes<XAX, KIND>(I.M.ntype);
    auto kernel = k_deriv_mma<XAX, EPI, KIND>;
    EMIX_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, shm));
    EMIX_CUDA_TRY(launch_early(kernel, I.ncta, kMmaThreads, (size_t)shm, st, I));
    return EMIX_OK;
}

template <bool XAX, int EPI, int KIND>
int launch(const MmaBatch &b, cudaStream_t st) {
    const int shm = shared_bytes<XAX, KIND>(b.ntype);
    auto kernel = k_batch_deriv_mma<XAX, EPI, KIND>;
    EMIX_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, shm));
    EMIX_CUDA_TRY(launch_early(kernel, b.ctas, kMmaThreads, (size_t)shm, st, b.items, b.count));
    return EMIX_OK;
}

// the variant for an item or a batch of items
template <bool XAX, int EPI, class W>
int launch_kind(int kind, const W &w, cudaStream_t st) {
    if constexpr (std::is_same<W, MmaItem>::value)   // (a batch holds pencils of all lengths)
        if (kind == kRound) return launch<XAX, EPI, kRound>(w, st);
    return kind == kCyclic ? launch<XAX, EPI, kCyclic>(w, st) : launch<XAX, EPI, kClosed>(w, st);
}

template <class W>
int launch_variant(bool xax, int epi, int kind, const W &w, cudaStream_t st) {
    if (xax) return epi == EPI_STORE ? launch_kind<true, EPI_STORE>(kind, w, st) : launch_kind<true, EPI_ACCUM>(kind, w, st);
    return epi == EPI_STORE ? launch_kind<false, EPI_STORE>(kind, w, st) : launch_kind<false, EPI_ACCUM>(kind, w, st);
}

} // namespace

MmaItem mma_item(const DerivTable &T, const MmaTable &M, int axis, const PencilFields &F, int nf, int nx, int ny,
                 int nz) {
    MmaItem I{};
    I.T = T;
    I.M = M;
    I.F = F;
    I.nf = nf;
    I.nx = nx;
    I.np = axis == 0 ? ny * nz : nx * (axis == 1 ? nz : ny);
    I.s = axis == 0 ? 1 : (axis == 1 ? (long)nx : (long)nx * ny);
    I.os = axis == 0 ? 0 : (axis == 1 ? (long)nx * ny : (long)nx);
    I.ntile = (I.np + kMmaPencils - 1) / kMmaPencils;
    return I;
}

MmaBatch mma_split(MmaItem *items, int count) {
    // one CTA each, then one at a time to the item that would end last
    const int sms = device_sms();
    std::vector<int> n(count, 1);
    std::vector<long> t(count);
    for (int g = 0; g < count; ++g) t[g] = divide(items[g], 1);
    for (int left = sms - count; left > 0; --left) {
        const int g = (int)(std::max_element(t.begin(), t.end()) - t.begin());
        t[g] = divide(items[g], ++n[g]);
    }
    MmaBatch b{nullptr, count, 0, 0};
    for (int g = 0; g < count; ++g) {
        items[g].cta0 = b.ctas;
        b.ctas += items[g].ncta;
        b.ntype = std::max(b.ntype, items[g].M.ntype);
    }
    return b;
}

int launch_deriv_mma_batch(const MmaBatch &b, bool xax, int epi, bool periodic, cudaStream_t st) {
    return launch_variant(xax, epi, periodic ? kCyclic : kClosed, b, st);
}

static PencilFields fields_of(int nf, const double *const *in, double *const *w, double *const *out) {
    PencilFields F{};
    for (int f = 0; f < nf; ++f) {
        F.in[f] = in[f];
        F.w[f] = w[f];
        F.out[f] = out[f];
    }
    return F;
}

int launch_deriv_mma(const DerivTable &T, const MmaTable &M, int axis, int epi, int nf, const double *const *in,
                     double *const *w, double *const *out, int nx, int ny, int nz, cudaStream_t st,
                     const QuietGate *gate) {
    MmaItem I = mma_item(T, M, axis, fields_of(nf, in, w, out), nf, nx, ny, nz);
    I.gate = gate;
    divide(I, device_sms());
    return launch_variant(axis == 0, epi, kind_of(T.n, M.periodic != 0), I, st);
}

int launch_quiet_sample(int axis, int nf, const double *const *in, int nx, int ny, int nz, QuietGate *gate,
                        cudaStream_t st) {
    PencilFields F{};
    for (int f = 0; f < nf; ++f) F.in[f] = in[f];
    const int n = axis == 0 ? nx : (axis == 1 ? ny : nz), np = axis == 0 ? ny * nz : nx * (axis == 1 ? nz : ny);
    const long s = axis == 1 ? (long)nx : (long)nx * ny, os = axis == 1 ? (long)nx * ny : (long)nx;
    const int groups = (np + 31) / 32 * nf, sms = device_sms(), blocks = std::min(groups, 2 * sms);
    // A launch gains 5 to 8 ps a cell and field over the sweeps; the quiet pencils of an
    // SM, once more than its warps take one by one, cost it a thread's walk, 0.6 to 1.2
    // us a row.  1200 pencils an SM is where a launch gains the walk: with more, a fifth
    // of them may be quiet (256^3, ms, 5 fields: x 0.82 at 10%, 1.17 at 30%, sweeps 1.00;
    // y 0.89, 1.03, 0.99), with fewer, as many as the warps take (128^3: x 0.10 at 1%,
    // 0.17 at 10%, sweeps 0.15; y 0.09, 0.17, 0.17).
    const long all = (long)np * nf, most = all >= 1200L * sms ? all / 5 : (long)kSweepWarps * std::max(1, n / 96) * sms;
    const int limit = (int)(most * 32 * blocks / all);
    auto kernel = axis == 0 ? k_quiet_sample<true> : k_quiet_sample<false>;
    EMIX_CUDA_TRY(launch_early(kernel, blocks, 256, 0, st, F, nf, n, np, nx, s, os, limit, gate));
    return EMIX_OK;
}

int deriv_mma_timeouts(int *count) {
    EMIX_CUDA_TRY(cudaMemcpyFromSymbol(count, g_mma_timeouts, sizeof(int)));
    return EMIX_OK;
}

int TimeoutWatch::note(int at, cudaStream_t st) {
    if (!h_) {
        if (cudaHostAlloc((void **)&h_, 4 * sizeof(int), cudaHostAllocPortable) != cudaSuccess) {
            cudaGetLastError();
            h_ = nullptr;
            set_last_message("cudaHostAlloc of the timeout counters failed");
            return EMIX_ERR_ALLOC;
        }
    }
    EMIX_CUDA_TRY(cudaMemcpyFromSymbolAsync(h_ + at, g_mma_timeouts, sizeof(int), 0, cudaMemcpyDeviceToHost, st));
    return pencil_tma_timeouts_async(h_ + at + 1, st);
}

int TimeoutWatch::result(const char *call) const {
    if (h_[2] == h_[0] && h_[3] == h_[1]) return EMIX_OK;
    char text[160];
    snprintf(text, sizeof text, "%s: pencil blocks gave up waiting for the tensor core or for TMA row copies; its results "
             "are incomplete", call);
    set_last_message(text);
    return EMIX_ERR_TIMEOUT;
}

TimeoutWatch::~TimeoutWatch() {
    if (h_) cudaFreeHost(h_);
}

} // namespace emix

extern "C" int emix_deriv_mma_test_drop(int on) {
    if (on != 0 && on != 1) return EMIX_ERR_ARG;
    EMIX_CUDA_TRY(cudaMemcpyToSymbol(emix::g_mma_drop, &on, sizeof(int)));
    EMIX_CUDA_TRY(cudaDeviceSynchronize());
    return EMIX_OK;
}
