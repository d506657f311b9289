// deriv_mma.cu -- the compact first derivative on the tensor cores
// (tcgen05.mma, f16 operands, f32 sums in tensor memory).
//
// The FP64 pipe (2 lanes per clock and SM) bounds the factored Thomas sweeps
// at 3 clocks per cell and field.  Here D f is a contraction of the dense
// operator, which falls off so fast that 96 differences reach 16 outputs
// (deriv_mma.cuh), and its products are formed exactly on the tensor cores:
// each pencil's differences are turned into fixed-point numbers (relative to
// the pencil's largest difference) of six balanced digits to the base 1024,
// the operator into digits of the same kind, and the f32 sums of digit
// products are integers below 2^24 and so exact (the error-free splitting of
// K. Ozaki et al., Numerical Algorithms 59, 2012, applied to a banded
// operator).  Products of digit orders i + j <= 5 are kept; what is dropped
// is 2^-57 of the largest term, an FP64 sum of the same terms rounds at
// 2^-53.
//
// One CTA per SM walks tiles of 128 pencils (one per tensor-memory lane), its
// warps in four roles that meet on mbarriers:
//   three warps read the next tile once for each pencil's largest exponent and
//     largest difference (the first tile is shared by all);
//   eight warps convert the tile's differences to digits, 16 rows (a group) at
//     a time, into tensor memory, where they are the instruction's A operand;
//   one warp issues the products of a block of 16 outputs: 28 instructions,
//     since the operator's digits 0 .. 5-j lie next to each other and one
//     instruction adds all products of the differences' digit j;
//   eight warps combine the finished block's six sums per output.
// Whole tiles while they fill every SM, the rest cut into segments of blocks.
//
// What bounds it: the scanning warps (their loads come from DRAM, 12 KB in
// flight per SM: a quarter of the scan took y from 0.514 to 0.434 ms) and the
// tensor-core warp (28 instructions a block at 80 clocks each whatever their
// width up to 128 columns; 16 outputs a block are what tensor memory holds
// beside the digits) about alike, with the ALU pipe 55% busy (conversion 45
// instructions a row, results 30, scan 11).  Two things made the issue of the
// instructions cheap: elect.sync with warp-uniform operands (0.569 -> 0.522)
// and a straight run of them, digit by digit, for the blocks whose six groups
// all exist (-> 0.492).  More or fewer rows a scan step, L2 prefetch of the
// rows to come, non-allocating loads and the scan spread over the other warps
// (0.62) measured no better or worse.
// Measured, ms for 5 fields of 256^3, sweeps -> here: closed x 1.001 -> 0.537,
// y 0.991 -> 0.492, z 0.991 -> 0.498; cyclic 1.215 -> 0.557, 1.071 -> 0.567,
// 1.069 -> 0.571.  Error against a dense solve, 192 x 160 x 192 smooth fields,
// 2-norm: A 5.4e-15 -> 3.9e-15, B 1.2e-15 -> 1.1e-15, cyclic 9.8e-16 ->
// 9.4e-16, C 5.7e-15 -> 3.4e-15.
//
// Pencils with infinities or NaN, or of magnitudes whose fixed-point
// exponents would leave the FP64 range, take the scalar sweep (deriv.cuh)
// after the tile.
#include "deriv_mma.cuh"
#include "tma.cuh"

#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>
#include <vector>

namespace emix {
namespace {

__device__ int g_mma_timeouts = 0;

constexpr int kMmaPencils = 128;            // per tile: the lanes of tensor memory
constexpr int kRpt = 8;                     // rows of a group (outputs of a block) a thread takes at a time
constexpr int kScanWarps = 3;               // warps that find the next tile's magnitudes
constexpr int kScan = 16;                   // rows a step of theirs
constexpr int kScanParts = 4;               // parts a pencil (y, z) is scanned in
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

// v 2^(62 - (E - 1023) + sh) modulo 2^64, truncated towards zero before the
// shift by sh: below 2^61 in magnitude before it for E two above v's biased
// exponent
EMIX_DEV unsigned long long to_fixed(double v, int E, int sh) {
    const int hi = __double2hiint(v), lo = __double2loint(v);
    const int r = E - ((hi >> 20) & 0x7ff);
    const unsigned mh = ((unsigned)hi & 0xfffffu) | 0x100000u;
    const unsigned h = __funnelshift_l((unsigned)lo, mh, 10), l = (unsigned)lo << 10;
    // 64-bit right shift: the funnel's shift is clamped at 32
    const unsigned neg = (unsigned)(hi >> 31);
    const unsigned rh = __funnelshift_rc(h, 0u, r) ^ neg;
    const unsigned rl = __funnelshift_rc(__funnelshift_rc(l, h, r), 0u, max(r - 32, 0)) ^ neg;
    const unsigned long long t = (((unsigned long long)rh << 32) | rl) + (neg & 1u);
    return ((unsigned long long)__funnelshift_l((unsigned)t, (unsigned)(t >> 32), sh) << 32) | ((unsigned)t << sh);
}

// a value's high word to about 20 bits as a float (2^-126 and less as 2^-126;
// meaningful for values whose exponents fit)
EMIX_DEV float rough(int hi) {
    const unsigned t = (unsigned)max(hi & 0x7fffffff, 897 << 20) * 8u - (896u << 23);
    return __uint_as_float((t & 0x7fffffffu) | ((unsigned)hi & 0x80000000u));
}

struct Spread {          // of one pencil, or a part of it
    int top;             // largest |high word|
    unsigned low;        // low words, or-ed (zero test)
    float diff;          // largest rough difference
};

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

// one pencil's magnitudes, once known: the exponent its values are fixed to,
// the left shift of their differences, and whether it takes the scalar sweep
struct Scale {
    int E, sh;
    bool scalar;
};

EMIX_DEV Scale scale_of(const Spread &a) {
    Scale r{1023, 0, false};
    if (a.top == 0 && a.low == 0) return r;   // all zero
    const int e = a.top >> 20;
    r.scalar = e < 256 || e > 1790;
    r.E = e + 2;
    if (e >= 930 && e <= 1140) {
        // differences are below B: shift them up to 63 bits
        const float B = fmaf(a.diff, 1.01f, __uint_as_float((unsigned)(e - 896 + 1 - 18) << 23));
        r.sh = min(max(r.E - 1023 - ((int)(__float_as_uint(B) >> 23) - 127), 0), 25);
    }
    return r;
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

// magnitudes of the 128 x pencils from p0 of field f: P at a time, lanes along
// the rows, kScan / P rounds of 32 rows each (P = 1: as many as it takes)
template <int P, bool PER>
EMIX_DEV void scan_x(const double *f, int p0, int np, int n, int uw, int step, int lane, Spread *to) {
    constexpr int C = kScan / P;
    const int steps = P == 1 ? (n + 32 * C - 1) / (32 * C) : 1;
    double sv[kScan], before[P];
    int top[P];
    unsigned low[P];
    float diff[P], prev[P];
    auto load = [&](int u, int st) {
        const int r = st * 32 * C + lane;
#pragma unroll
        for (int i = 0; i < P; ++i) {
            const double *fp = f + (long)min(p0 + u * P + i, np - 1) * n;
            if (st == 0) before[i] = fp[PER ? n - 1 : 0];
#pragma unroll
            for (int q = 0; q < C; ++q) sv[i * C + q] = fp[min(r + 32 * q, n - 1)];
        }
    };
    int u = uw, st = 0;
    if (u < kMmaPencils / P) load(u, 0);
    while (u < kMmaPencils / P) {
        if (st == 0) {
#pragma unroll
            for (int i = 0; i < P; ++i) {
                top[i] = 0;
                low[i] = 0;
                diff[i] = 0.0f;
                prev[i] = rough(__double2hiint(before[i]));
            }
        }
        int hi[kScan];
#pragma unroll
        for (int q = 0; q < kScan; ++q) {
            hi[q] = __double2hiint(sv[q]);
            low[q / C] |= (unsigned)__double2loint(sv[q]);
        }
        const int uu = u;
        if (++st == steps) {
            st = 0;
            u += step;
        }
        if (u < kMmaPencils / P) load(u, st);
#pragma unroll
        for (int q = 0; q < kScan; ++q) {
            const int i = q / C;
            top[i] = max(top[i], hi[q] & 0x7fffffff);
            const float x = rough(hi[q]);
            const float pr = __shfl_sync(0xffffffffu, lane == 31 ? prev[i] : x, (lane + 31) & 31);
            diff[i] = fmaxf(diff[i], fabsf(x - pr));
            prev[i] = x;
        }
        if (u != uu) {
#pragma unroll
            for (int i = 0; i < P; ++i) {
                const int tp = __reduce_max_sync(0xffffffffu, top[i]);
                const unsigned lw = __reduce_or_sync(0xffffffffu, low[i]);
                const unsigned d = __reduce_max_sync(0xffffffffu, __float_as_uint(diff[i]));   // not negative
                if (lane == 0) to[uu * P + i] = Spread{tp, lw, __uint_as_float(d)};
            }
        }
    }
}

// XAX: pencils along x (rows contiguous, brought through a shared tile);
// otherwise along y or z (pencils contiguous along x)
// CTA `cta` of the I.ncta that share the item
template <bool XAX, int EPI, int KIND>
EMIX_DEV void mma_body(const MmaItem &I, int cta) {
    constexpr bool PER = KIND == kCyclic || KIND == kRound;
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
    const int tid = threadIdx.x, lane = tid & 31;
    // through a shuffle: the roles' branches are then known to be uniform, and
    // the instruction operands stay in uniform registers
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int n = M.n;

    if (tid == 0) {
        s_fail = 0;
        for (int q = 0; q < 2; ++q) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&s_full[q])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(&s_drained[q])), "r"(kRoleWarps) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(&s_scaled[q])), "r"(kScanWarps) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(&s_read[q])), "r"(2 * kRoleWarps) : "memory");
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
    const int jobs = whole + (ntile * nf - whole) * segs;
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
            double sv[kScan], before = 0.0;    // before: the value before the unit's first row
            const double *fp = nullptr;
            int ra = 0, rb = 0, top = 0;
            unsigned low = 0;
            float diff = 0.0f, prev = 0.0f;
            auto load = [&](int u, int st) {
                if (st == 0) {
                    fp = tile_of(job, (u & 3) * 32 + lane).in;
                    ra = min((u >> 2) * part, n - 1);
                    rb = min(ra + part, n) - 1;
                    before = fp[(long)row_of(ra - 1) * s];
                }
                const int r = ra + st * kScan;
                const double *q0 = fp + (long)r * s;
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
                    low = 0;
                    diff = 0.0f;
                    prev = rough(__double2hiint(before));
                }
                int hi[kScan];
#pragma unroll
                for (int q = 0; q < kScan; ++q) {
                    hi[q] = __double2hiint(sv[q]);
                    low |= (unsigned)__double2loint(sv[q]);
                }
                const int uu = u;
                if (++st == steps) {
                    st = 0;
                    u += step;
                }
                if (u < 4 * kScanParts) load(u, st);
#pragma unroll
                for (int q = 0; q < kScan; ++q) {
                    top = max(top, hi[q] & 0x7fffffff);
                    const float x = rough(hi[q]);
                    diff = fmaxf(diff, fabsf(x - prev));
                    prev = x;
                }
                if (u != uu) s_part[buf][uu >> 2][(uu & 3) * 32 + lane] = Spread{top, low, diff};
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
    constexpr int kPencilWarps = 2 * kRoleWarps + kScanWarps;   // all but the tensor core's
    wait_for_previous();   // what is read so far is constant
    if (warp != 2 * kRoleWarps) {
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
            wait(&s_table, 0);
            for (int job = cta; job < jobs; job += ncta) {
                const Tile jt = tile_of(job, 0);
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
                    if (leader)
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
        // this thread's pencil of tile t, once its magnitudes are known
        auto scale_wait = [&](int t) {
            if (t > 0) wait(&s_scaled[t & 1], (unsigned)((t - 1) >> 1) & 1);
            Spread a = s_part[t & 1][0][slot_p];
            if constexpr (!XAX) {
#pragma unroll
                for (int q = 1; q < kScanParts; ++q) {
                    const Spread b = s_part[t & 1][q][slot_p];
                    a.top = max(a.top, b.top);
                    a.low |= b.low;
                    a.diff = fmaxf(a.diff, b.diff);
                }
            }
            arrive(&s_read[t & 1]);
            return scale_of(a);
        };
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
                unsigned long long a = to_fixed(XAX ? t[0] : v[0], sc.E, sc.sh);
#pragma unroll
                for (int q = 0; q < kRpt; ++q) {
                    const unsigned long long b = to_fixed(XAX ? t[q + 1] : v[q + 1], sc.E, sc.sh);
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
                if (t == 0) return -1;
                pos += last.gb - last.ga + 1;
                return pos >= 0 ? Bl + min(last.ga + pos + reach, last.b1 - 1) - last.b0 : Bl - 1;
            };
            load(cur, cur.ga);
            for (; job < jobs; job += ncta, ++t) {
                const Scale sc = scale_wait(t);
                const bool more = job + ncta < jobs;
                Tile nxt = cur;
                if (more) nxt = tile_of(job + ncta, slot_p);
                const int ng = cur.gb - cur.ga + 1;
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
                const Scale sc = scale_wait(t);
                const int escale = (sc.E - 1023 - M.se - sc.sh) * (1 << 20);
                if (XAX && rg == 0) s_scalar[slot_p] = sc.scalar;
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
                // the pencils outside the fixed-point range
                if (rg == 0 && sc.scalar && cur.live && ok && cur.b0 == 0) {
                    const long x = XAX ? cur.wofs : 0;
                    double *w = pick(F.w, cur.field) + cur.wofs;
                    deriv_pencil<EPI>(I.T, cur.in + x, w, cur.out + x, s);
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
}

template <bool XAX, int EPI, int KIND>
__global__ void __launch_bounds__(kMmaThreads, 1) k_deriv_mma(const __grid_constant__ MmaItem I) {
    mma_body<XAX, EPI, KIND>(I, blockIdx.x);
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
    mma_body<XAX, EPI, KIND>(s_item, (int)blockIdx.x - s_item.cta0);
}

// tensor memory is taken whole: at least 116 KB of shared memory keeps a
// second CTA off the SM
template <bool XAX, int KIND>
int shared_bytes(int ntype) {
    const int shm = ntype * kMmaTypeBytes + (XAX ? (2 + out_tiles(KIND)) * kXTileDoubles * (int)sizeof(double) : 0);
    return shm < 120 * 1024 ? 120 * 1024 : shm;
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
                     double *const *w, double *const *out, int nx, int ny, int nz, cudaStream_t st) {
    MmaItem I = mma_item(T, M, axis, fields_of(nf, in, w, out), nf, nx, ny, nz);
    divide(I, device_sms());
    return launch_variant(axis == 0, epi, kind_of(T.n, M.periodic != 0), I, st);
}

int deriv_mma_timeouts(int *count) {
    EMIX_CUDA_TRY(cudaMemcpyFromSymbol(count, g_mma_timeouts, sizeof(int)));
    return EMIX_OK;
}

} // namespace emix
