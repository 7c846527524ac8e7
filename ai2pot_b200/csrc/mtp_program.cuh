// Compiled form of the MTP alpha tables, shared by the MTP kernels.
//
// The reference walks alpha_index_basic / alpha_index_times row by row for every atom
// (source/descriptor/mtpr/include/mtpBasis.h:472-528, linearMtp.h:292-306). Here the tables are
// analysed once on the host:
//  * basic moments (mu, ax, ay, az) are mapped onto a dense, degree-major canonical monomial
//    numbering per mu, so the kernels evaluate them with compile-time exponents;
//  * product rows (a, b, mult, dst) are grouped by destination and by dependency depth, so a
//    warp runs all destinations of one depth in parallel (forward), and the adjoint sweep is
//    turned into a gather per source moment (reverse).
#pragma once
#include "common.cuh"

namespace ai2b {

constexpr int MTP_MAX_MU = 8;
constexpr int MTP_MAX_DEG = 8;
constexpr int MTP_MAX_LEV = 16;

struct MtpProgramDev {
    int nm, nb, nt, ns, nmus, kmax, ndense, nlev;
    int kmu[MTP_MAX_MU];            // highest monomial degree used with radial function mu
    int doff[MTP_MAX_MU + 1];       // dense offset of mu: doff[mu] + canonical index
    int fwd_lev_off[MTP_MAX_LEV + 1];  // destinations of depth 1..nlev
    int rev_lev_off[MTP_MAX_LEV + 1];  // source moments of depth nlev-1..0
    const int *basic_dense;         // [nb] dense index of basic row i
    const int *dense_basic;         // [ndense] basic row of dense index d (-1: the tables have no such moment)
    const int4 *e4d;                // [ndense] dense indices holding {value, d/dx, d/dy, d/dz} sources (-1: none)
    const int4 *e4g;                // [ndense] basic row holding {value, d/dx, d/dy, d/dz} source (-1: none)
    const int *e4m;                 // [ndense] packed multipliers (ax+1) | (ay+1)<<8 | (az+1)<<16
    const int4 *fwd_dst;            // {dst, row_begin, row_end, -}
    const int2 *fwd_rows;           // [nt] {a | b<<16, multiplier as float bits}: one 8-byte load per row
    const int2 *rev_ents;           // [adjoint_rows()] {other | dst<<16, multiplier as float bits}
    // flat row streams for the lanes-as-atoms kernel: rows of one depth are contiguous, a flag marks the
    // last row of each destination, so any contiguous share of a depth's rows can be given to a worker
    const int2 *fwd_flat;           // [nt]   {a | b<<16, mult | last<<8 | dst<<16}
    const int2 *rev_flat;           // [adjoint_rows()] {other | dst<<16, mult | last<<8 | source<<16}
    int fwd_lev_row[MTP_MAX_LEV + 1];
    int rev_lev_row[MTP_MAX_LEV + 1];
    const int4 *rev_mom;            // {m, entry_begin, entry_end, -}
    const int *map;                 // [ns] alpha_moment_mapping
    // Row streams of the lanes-as-atoms contractions (tiles of 16 or 32 atoms, 16 bytes of atoms per lane, GL lanes per row, so
    // a warp works on 32 / GL rows at a time). Phase p < nlev is product depth p + 1 (rows {a, b}: M[dst] = sum mult * M[a] *
    // M[b]); phase nlev + k gathers the adjoints of the source moments of depth nlev - 1 - k (rows {dst, other}: E[src] =
    // seed + sum mult * E[dst] * M[other]). Every moment belongs to one group of lanes, or in pieces to all groups of one
    // warp (those with many rows, at the front of the warp's rows), and its rows are consecutive, so there are no atomics.
    // A row is {x | y << 16, multiplier with the moment that it completes + 1 in its low 11 bits (0: more rows follow) and
    // MTP_PAIR_WIDE if that moment is in pieces}; the multiplier is the high word of a double or a float, whose low bits are
    // zero for integers up to 255. The groups of a warp have equally many rows in a phase (empty ones where needed).
    struct Stream {
        const int2 *row_d, *row_f;      // [nrows][groups of a warp]
        const int2 *warp;               // [2 nlev][warps] {first row, rows}
        int nrows;                      // 0: the tables do not fit the encoding, or have too many rows for few warps
    } stream[4];                        // GL = 16, GL = 8 for MTP_PAIR_WARPS warps; the same for MTP_PAIR_FEW
    const int *constant;            // [n_adj_const] moments whose adjoint is only their seed (no product reads them), then, up to
    int n_adj_const, n_constant;    // n_constant, moments that are neither basic nor a product: zero
    // two per product, one for the square of a moment (unless twice its multiplier exceeds 255)
    __host__ __device__ int adjoint_rows() const { return rev_lev_row[nlev]; }
};

// A row with its moment indices scaled to element offsets in [moment][LD] (index * LD fits 16 bits); FLAT: the moment in the high half
// of the second word too.
template <int LD, bool FLAT>
struct ScaledRow {
    __host__ __device__ int2 operator()(int2 r) const
    {
        return make_int2(((r.x & 0xffff) * LD) | (((r.x >> 16) & 0xffff) * LD) << 16,
                         FLAT ? (r.y & 0xffff) | (((r.y >> 16) & 0xffff) * LD) << 16 : r.y);
    }
};
// Product rows, then (if `adjoints`) adjoint rows to to[0 .. nt + adjoint_rows()), by thread t of n.
template <typename Rows, typename Scale>
__host__ __device__ inline void stage_product_rows(const MtpProgramDev &P, Rows fwd, Rows rev, bool adjoints, int2 *to, int t, int n, Scale scale)
{
#pragma unroll 4
    for (int i = t; i < P.nt; i += n) to[i] = scale(fwd[i]);
    if (adjoints)
#pragma unroll 4
        for (int i = t; i < P.adjoint_rows(); i += n) to[P.nt + i] = scale(rev[i]);
}
// Warps of a block of the contractions. A phase of a small table is over before 32 warps have met: where there are more tiles than
// SMs such tables (levels up to 10, of 42 products; level 16 has 969 and fills 32 warps) take blocks of eight warps, four of which share
// an SM. Level 10, whole call, us, 32 / 8 warps: fp64 6,000 atoms 51.6 / 48.5, 13,824 atoms 73.2 / 67.2, 100,000 atoms 361 / 303; with a
// tile per SM 32 warps are sooner over it (2,500 atoms 34.8 / 37.2). Tables whose moments leave room for fewer than three such blocks
// stay with 32 warps: 20,000 atoms, fp64, 100 products, 230 moments 155 us with eight warps, 142 with 32; 128 products, 90 moments 104 / 113.
constexpr int MTP_PAIR_WARPS = 32, MTP_PAIR_FEW = 8, MTP_PAIR_FEW_ROWS = 128;
constexpr size_t MTP_PAIR_BYTES = 226 * 1024, MTP_PAIR_FEW_BYTES = 75 * 1024;      // shared memory of a block at most
constexpr int MTP_PAIR_WIDE = 0x800;
constexpr int MTP_TILE = 32;        // atoms per tile of the workspace

}  // namespace ai2b

struct ai2b_mtp_program {
    ai2b::MtpProgramDev dev;
    void *d_blob;       // one device allocation holding every table
    size_t blob_bytes;
    int device;
};
