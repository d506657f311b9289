// deriv_mma.cuh -- the compact first derivative on the tensor cores
// (deriv_mma.cu): exact fixed-point digits of the pencils times exact digits
// of the dense operator.
#pragma once

#include "deriv.cuh"

namespace emix {

// The operator D = A^{-1} B / h acting on first differences: with
// d_k = f_{k+1} - f_k, (D f)_i = sum_k E_{ik} d_k, E_{ik} = sum_{m>k} D_{im}
// (the rows of D sum to zero).  |E_{ik}| falls by the root of the scheme's
// characteristic polynomial (0.38 or 0.27) per row away from the diagonal:
// 2^-55 of its largest entry 40 rows away, where it is cut (what is cut off is
// added to the last entry kept, so that row sums, and with them the
// derivative of a linear function, stay exact).
//
// Outputs go in blocks of 16 rows.  Block b reads the differences
// 16b-40 .. 16b+55, in six groups of 16: group g holds 16g-8 .. 16g+7, block b
// reads groups b-2 .. b+3.  Away from the ends every block has the same
// entries, so a table holds few distinct block types (at most 8; one for the
// cyclic scheme).
//
// Entries are fixed-point numbers of kMmaDig balanced digits to the base 1024
// (60 bits): E 2^sE = sum_i D_i 1024^(kMmaDig-1-i), -512 <= D_i <= 511, held
// as f16.  `b` has, per type, group and 8 columns of the group, the digits of
// 16 rows, i-major (kMmaDig x 16 rows of 8 f16: the no-swizzle K-major
// operand of tcgen05.mma).
constexpr int kMmaDig = 6;
constexpr int kMmaRows = 16;                                    // outputs of a block, differences of a group
constexpr int kMmaWin = 6;                                      // groups a block reads
constexpr int kMmaStack = kMmaDig * kMmaRows;                   // operand rows of a group
constexpr int kMmaGroupBytes = 2 * kMmaStack * 16;              // one group of one type
constexpr int kMmaTypeBytes = kMmaWin * kMmaGroupBytes;
constexpr int kMmaMaxTypes = 8;
// leading digits of the entries that vanish over a block's outer two groups
// (24 rows away and more: below 2^-30) and over the two within
constexpr int kMmaLead0 = 3, kMmaLead1 = 1;
constexpr int kMmaMaxBlocks = kTableMaxN / kMmaRows;

struct MmaTable {
    int n, periodic;
    int nblk;             // blocks of 16 outputs
    int ntype;
    int nlow, nhigh;      // blocks of their own type at the ends; type nlow is the interior's
    int se;               // scale exponent of the entries
    const unsigned short *b;   // ntype x kMmaTypeBytes, f16
};

// Tensor-core table of (scheme, n, sign h) (kept for the life of the
// process); null below kMmaMinN rows and where the operator does not fit the
// form above (the callers then keep the sweeps).
int get_mma_table(int scheme, int n, double h, double sign, const MmaTable **out);

// Whether a derivative goes to the tensor cores: by the length of its
// pencils.  Measured against the sweeps (us for 5 fields, closed / cyclic, x and y):
// n = 40 on 48 x 48 pencils x 25 / 31 -> 17 / 19, y 19 / 23 -> 17 / 17, on 256 x 256
// x 177 / 220 -> 145 / 202, y 152 / 192 -> 125 / 204 (the one loss); n = 64 x 33 / 43 ->
// 18 / 18, y 27 / 33 -> 16 / 16, and 261 / 333 -> 170 / 187, 240 / 299 -> 155 / 159;
// n = 256 x 1001 / 1212 -> 592 / 631, y 991 / 1071 -> 513 / 576.  n = 32, when the line
// was drawn: x 17 / 21 -> 16 / 18 at 32^3 but 134 -> 200 at 32 x 128 x 512 (3 fields), y
// and z 16 / 19 -> 16 / 19.  Shorter pencils have more blocks at an end and groups to
// convert per output than the sweeps have to lose.
constexpr int kMmaMinN = 40;
inline bool deriv_on_mma(const DerivTable &T) { return T.mma != nullptr; }

// launch_deriv on the tensor cores
int launch_deriv_mma(const DerivTable &T, const MmaTable &M, int axis, int epi, int nf, const double *const *in,
                     double *const *w, double *const *out, int nx, int ny, int nz, cudaStream_t st,
                     const QuietGate *gate = nullptr);

// Sets `gate` from a sample of the pencils: to the sweeps where more of them are
// quiet somewhere than the tensor cores' form gains from (those take a sweep there
// too, after a scan, and less well spread over the SM).
int launch_quiet_sample(int axis, int nf, const double *const *in, int nx, int ny, int nz, QuietGate *gate,
                        cudaStream_t st);
// Cells of a step's grid from which its derivatives are gated.  A step then has 24
// launches more, 0.12 ms (ms, ungated / gated: tanks in motion 128^3 4.19 / 4.31, 160^3
// 7.63 / 7.75, 256^3 28.10 / 28.25), which the states with many quiet pencils repay:
// a tank from rest 128^3 5.1-6.2 / 4.9-5.2, 256^3 36-43.6 / 33-33.8; bench.py's after 125
// steps 37.8 / 33.8 (the sweeps everywhere: 5.05, 34.5, 34.7).  Smaller grids would pay more
// than the states that last gain: 96^3 in motion 2.05 / 2.15, developed 2.32 / 2.32, from
// rest 2.6-3.2 / 2.4-2.7 (sweeps 2.56).
constexpr long kGateCells = 1L << 21;

// One derivative of nf fields of a grid, and the CTAs that walk its tiles.
struct MmaItem {
    DerivTable T;
    MmaTable M;
    PencilFields F;
    int np, ntile, nf, nx;    // pencils, tiles of them, fields
    int whole, segs;          // whole tiles, and segments each of the others is cut into
    int cta0, ncta;           // CTAs [cta0, cta0 + ncta) of the launch
    long s, os;               // strides along a pencil, and between lines of pencils
    const QuietGate *gate;    // null: none
};
MmaItem mma_item(const DerivTable &T, const MmaTable &M, int axis, const PencilFields &F, int nf, int nx, int ny,
                 int nz);

// Many items (all along x or none, all cyclic or none) as one launch.
struct MmaBatch {
    const MmaItem *items;     // on the device
    int count, ctas, ntype;   // items, CTAs of the launch, most block types of a table
};
// divides the SMs between the items, by their work (an item is at least one
// CTA); `items` of the result is left to the caller
MmaBatch mma_split(MmaItem *items, int count);
int launch_deriv_mma_batch(const MmaBatch &b, bool xax, int epi, bool periodic, cudaStream_t st);

// blocks that gave up a bounded wait since the library was loaded
int deriv_mma_timeouts(int *count);
// the sweeps' counter, copied on a stream (deriv_tma.cu)
int pencil_tma_timeouts_async(int *count, cudaStream_t st);

// Whether pencil blocks gave up a wait between two points of a stream's work: the
// counters are copied at both, and read once the caller has synchronised.  (Blocks of
// other streams' launches meanwhile count too.)
class TimeoutWatch {
public:
    TimeoutWatch() = default;
    TimeoutWatch(const TimeoutWatch &) = delete;
    TimeoutWatch &operator=(const TimeoutWatch &) = delete;
    ~TimeoutWatch();
    int begin(cudaStream_t st) { return note(0, st); }
    int end(cudaStream_t st) { return note(2, st); }
    int result(const char *call) const;   // EMIX_OK or EMIX_ERR_TIMEOUT

private:
    int note(int at, cudaStream_t st);
    int *h_ = nullptr;                    // pinned: tensor core and TMA, at the beginning and at the end
};

} // namespace emix
