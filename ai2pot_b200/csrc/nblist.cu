// Cell-list neighbour build on sm_100a, bit-compatible with the reference's CPU list.
//
// Reference semantics (source/nblist/include/structure.h:589-710, binLinkedList.h:658-696,983-1031,
// neighborList.h:532-578): the cell is replicated over images n_k in [-e_k, e_k],
// e_k = ceil(rcut / interplanar distance) on periodic axes; image position
// ((r_j + a0*nx) + a1*ny) + a2*nz; (j, n) is a neighbour of i iff 1e-3 < d2 < rcut^2 with
// d = image - r_i (squares accumulated in double when T = float); row = index j, rcs = d;
// padding -1 / 0. The order inside a row is not part of the contract.
//
// Here: atoms are binned by their fractional coordinates wrapped into the cell, in bins at least a cutoff
// thick. A TEAM of warps owns one bin: the candidates of its 27 neighbouring bins are brought into shared
// memory once, as single-precision positions relative to the bin with their squared length, and every atom of
// the bin is then tested against them with three fused multiply-adds per candidate. Survivors (the hits and a
// handful more) take the exact route: the reference's predicate with the reference's operation order (no FMA
// contraction). A row is put together in shared memory, padding included, and leaves as 16-byte stores.
// Bins that follow one another along the third axis are contiguous in bin order, so a column of bins is ONE
// range of atoms: the table of a bin holds 9 ranges (plus the wrapped remainders next to a periodic face).
// Binning is one launch of one block for systems of up to 2,048 atoms, else a chain of set-up, count, scan and fill
// (launch_chained() in common.cuh).
#include "nep_setup.cuh"
#include <cooperative_groups.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdlib>
#include <cstring>

namespace ai2b {

template <typename T> struct Vec4;
template <> struct Vec4<double> { using type = double4; };
template <> struct Vec4<float> { using type = float4; };
// Lattice wraps packed into one word, 10 bits per axis with bias 512: sums and differences of packed
// words are field-wise sums and differences as long as every true field stays inside +-511. The fourth
// component of a bin-ordered position carries the atom's packed wrap.
constexpr int NB_WRAP_MAX = 127;
constexpr int NB_PACK_ZERO = 512 | (512 << 10) | (512 << 20);
__host__ __device__ inline int nb_pack3(int a, int b, int c) { return (a + 512) | ((b + 512) << 10) | ((c + 512) << 20); }
__device__ __forceinline__ float nb_bits_to(float, int v) { return __int_as_float(v); }
__device__ __forceinline__ double nb_bits_to(double, int v) { return __longlong_as_double((long long)v); }
__device__ __forceinline__ int nb_bits_of(float v) { return __float_as_int(v); }
__device__ __forceinline__ int nb_bits_of(double v) { return (int)__double_as_longlong(v); }

struct NbGrid {          // lives in the workspace; written by the binning kernels
    int nb[3];           // bins per fractional axis
    int R[3];            // bins to search on each side
    int total;
    int zmerge;          // the bins of a column along the third axis are taken as one range (needs nb[2] >= 2 R[2] + 1 if periodic)
    float pre_err;       // rounding error of the single-precision pre-test on d^2, for atoms at most one period outside the cell
    int maxwrap;         // most lattice periods an atom lies outside the cell, if more than one (else 0)
    double lo[3];        // non-periodic axes: lowest fractional coordinate
    double scale[3];     // bin = (s - lo) * scale
};

template <typename T>
struct NbParams {
    T cell[9];           // rows = lattice vectors (as given, type T)
    double inv[9];       // inverse cell: frac_k = sum_c r_c * inv[3*c + k]
    double dplane[3];    // interplanar distances (double, for bin sizing only)
    int per[3], e[3];
    int nbh[3];          // bins of the periodic axes (host-computed); cap for the others
    double rcut_m;       // rcut with a safety margin, for bin sizing
    double rc2;          // rcut^2 as the reference forms it
    float rc2_lo, rc2_hi, eps_lo, eps_hi;   // the two thresholds -/+ 2e-6 relative (float builds)
    int n, umax, maxbins, is_cart;
    int ncentre;         // rows are built for atoms [cbegin, ncentre); the rest are neighbours only (ghosts)
    int cbegin;          // first centre; its row is row 0 of the outputs
};

__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }

template <typename T>
struct Pos3 { T x, y, z; };
// Cartesian position of atom i; fractional input with the reference's operation order (structure.h:561-581)
template <typename T>
__device__ __forceinline__ Pos3<T> position_of(const NbParams<T> &P, const T *__restrict__ coords, int i)
{
    const T f0 = coords[3 * i], f1 = coords[3 * i + 1], f2 = coords[3 * i + 2];
    if (P.is_cart) return {f0, f1, f2};
    return {add_rn(add_rn(mul_rn(f0, P.cell[0]), mul_rn(f1, P.cell[3])), mul_rn(f2, P.cell[6])),
            add_rn(add_rn(mul_rn(f0, P.cell[1]), mul_rn(f1, P.cell[4])), mul_rn(f2, P.cell[7])),
            add_rn(add_rn(mul_rn(f0, P.cell[2]), mul_rn(f1, P.cell[5])), mul_rn(f2, P.cell[8]))};
}

template <typename T>
__device__ __forceinline__ void frac_of(const NbParams<T> &P, const Pos3<T> &p, double *s)
{
    const double x = p.x, y = p.y, z = p.z;
#pragma unroll
    for (int k = 0; k < 3; k++) s[k] = x * P.inv[k] + y * P.inv[3 + k] + z * P.inv[6 + k];
}

__device__ __forceinline__ unsigned long long enc_double(double d)
{
    unsigned long long u = (unsigned long long)__double_as_longlong(d);
    return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}
__device__ __forceinline__ double dec_double(unsigned long long u)
{
    u = (u >> 63) ? (u & 0x7fffffffffffffffull) : ~u;
    return __longlong_as_double((long long)u);
}

// extents of the fractional coordinates (large systems with an open axis whose extent the caller does not know)
template <typename T>
__global__ void nb_extent_kernel(NbParams<T> P, const T *__restrict__ coords, unsigned long long *__restrict__ ext)
{
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < P.n; i += gridDim.x * blockDim.x) {
        double s[3];
        frac_of(P, position_of(P, coords, i), s);
#pragma unroll
        for (int k = 0; k < 3; k++) { lo[k] = fmin(lo[k], s[k]); hi[k] = fmax(hi[k], s[k]); }
    }
#pragma unroll
    for (int k = 0; k < 3; k++) {
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) {
            lo[k] = fmin(lo[k], __shfl_xor_sync(FULL_MASK, lo[k], o));
            hi[k] = fmax(hi[k], __shfl_xor_sync(FULL_MASK, hi[k], o));
        }
        if ((threadIdx.x & 31) == 0) {
            atomicMin(ext + k, enc_double(lo[k]));
            atomicMax(ext + 3 + k, enc_double(hi[k]));
        }
    }
}

__global__ void nb_init_kernel(unsigned long long *ext)
{
    if (threadIdx.x < 3) { ext[threadIdx.x] = ~0ull; ext[3 + threadIdx.x] = 0ull; }
}

// Error bound of the single-precision pre-test. It works on float copies of the positions wrapped into the cell plus
// the float image shift of the candidate's bin; with coordinates bounded by reach = sum_k (max|s_k| + 2) |a_k| every
// difference carries at most ~6 ulp(reach), so d^2 near the cutoff is off by less than 64 eps reach rcut. (The rounding of
// the positions themselves grows with the periods an atom lies outside the cell: see maxwrap.)
template <typename T>
__host__ __device__ inline void nb_pretest_bounds(const NbParams<T> &P, NbGrid *g)
{
    double reach = 0.0;
    for (int k = 0; k < 3; k++) {
        const double len = sqrt((double)P.cell[3 * k] * (double)P.cell[3 * k] + (double)P.cell[3 * k + 1] * (double)P.cell[3 * k + 1] +
                                (double)P.cell[3 * k + 2] * (double)P.cell[3 * k + 2]);
        double smax = 1.0;
        if (!P.per[k]) {
            const double hi = g->lo[k] + g->nb[k] / g->scale[k];
            smax = fmax(fabs(g->lo[k]), fabs(hi));
        }
        reach += (smax + 2.0) * len;
    }
    g->pre_err = (float)(64.0 * 6e-8 * reach * sqrt(P.rc2) + 1e-6 * P.rc2);
}

// The bin grid of a system: periodic axes from the host's numbers, open axes from the extents ext[0..2] .. ext[3..5].
// An open axis of the host-side form may be given bounds that are a little off: atoms outside are clamped into the edge bins.
template <typename T>
__host__ __device__ inline void nb_make_grid(const NbParams<T> &P, const double *ext, NbGrid *g)
{
    long total = 1;
    for (int k = 0; k < 3; k++) {
        if (P.per[k]) {
            g->nb[k] = P.nbh[k];
            g->R[k] = (int)ceil(P.rcut_m / (P.dplane[k] / P.nbh[k]));
            g->lo[k] = 0.0;
            g->scale[k] = (double)P.nbh[k];
        } else {
            const double lo = ext[k], span = fmax(ext[3 + k] - lo, 1e-12);
            const double want = floor(span * P.dplane[k] / P.rcut_m);
            const int nb = want < 1.0 ? 1 : (want > (double)P.nbh[k] ? P.nbh[k] : (int)want);
            g->nb[k] = nb;
            g->R[k] = 1;
            g->lo[k] = lo;
            g->scale[k] = nb / span;
        }
        total *= g->nb[k];
    }
    g->total = (int)total;   // <= maxbins by construction of nbh
    g->zmerge = (!P.per[2] || g->nb[2] >= 2 * g->R[2] + 1) ? 1 : 0;
    g->maxwrap = 0;
    nb_pretest_bounds(P, g);
}

template <typename T>
__global__ void nb_grid_kernel(NbParams<T> P, const unsigned long long *__restrict__ ext, NbGrid *__restrict__ g, int *__restrict__ status)
{
    if (threadIdx.x != 0) return;
    double e[6];
    for (int k = 0; k < 3; k++) { e[k] = dec_double(ext[k]); e[3 + k] = dec_double(ext[3 + k]); }
    nb_make_grid(P, e, g);
    status[0] = 0; status[1] = 0;
}

// bin and lattice wrap of an atom
template <typename T>
__device__ __forceinline__ int bin_of(const NbParams<T> &P, const NbGrid &g, const double *s, int *w)
{
    int b[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        if (P.per[k]) {
            double fl = floor(s[k]);
            w[k] = (int)fl;
            int bb = (int)((s[k] - fl) * g.scale[k]);
            b[k] = min(max(bb, 0), g.nb[k] - 1);
        } else {
            w[k] = 0;
            int bb = (int)((s[k] - g.lo[k]) * g.scale[k]);
            b[k] = min(max(bb, 0), g.nb[k] - 1);
        }
    }
    return (b[0] * g.nb[1] + b[1]) * g.nb[2] + b[2];
}
// (an atom out of the range of an int, or at infinity, counts as 2^31 - 1 periods away)
__device__ __forceinline__ int wrap_reach(const int *w)
{
    return max(abs(max(w[0], -INT_MAX)), max(abs(max(w[1], -INT_MAX)), abs(max(w[2], -INT_MAX))));
}

// What the row kernel reads of an atom, in bin order: spos = position (type T) and index, sposw = position brought
// into the cell in single precision and packed wrap; full wraps only when some wrap does not fit the packed form.
template <typename T>
__device__ __forceinline__ void store_binned(const NbParams<T> &P, int k, int i, const Pos3<T> &p, const int *w, bool bigwrap,
                                             typename Vec4<T>::type *__restrict__ spos, float4 *__restrict__ sposw, int4 *__restrict__ sinfo)
{
    typename Vec4<T>::type q;
    q.x = p.x; q.y = p.y; q.z = p.z;
    q.w = nb_bits_to(T(0), i);
    spos[k] = q;
    const double w0 = w[0], w1 = w[1], w2 = w[2];
    float4 f;
    f.x = (float)((double)p.x - (w0 * (double)P.cell[0] + w1 * (double)P.cell[3] + w2 * (double)P.cell[6]));
    f.y = (float)((double)p.y - (w0 * (double)P.cell[1] + w1 * (double)P.cell[4] + w2 * (double)P.cell[7]));
    f.z = (float)((double)p.z - (w0 * (double)P.cell[2] + w1 * (double)P.cell[5] + w2 * (double)P.cell[8]));
    f.w = __int_as_float(nb_pack3(w[0], w[1], w[2]));
    sposw[k] = f;
    if (bigwrap) sinfo[k] = make_int4(i, w[0], w[1], w[2]);
}

// ---- binning of systems of up to 2,048 atoms: one block, one launch -----------------------------------
// Counters and bin starts live in shared memory; an atom's place in its bin is what its counting atomic returns. About 4 us
// at 1,000 atoms, where a chain of set-up, count, scan and fill is bound by the latency of its launches (10 us).
constexpr int BINB_THREADS = 1024;
constexpr int BINB_ITEMS = 2;                 // atoms (and bins) per thread at most
constexpr int BINB_MAX_ATOMS = BINB_THREADS * BINB_ITEMS;
constexpr int BINB_MAX_BINS = BINB_THREADS * BINB_ITEMS;

// lowest and highest fractional coordinates over the threads of a block of 1,024 -> ext[6] (shared memory)
__device__ __forceinline__ void block_extent(double (&lo)[3], double (&hi)[3], double (*wext)[6], double *ext)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 3; k++) {
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) {
            lo[k] = fmin(lo[k], __shfl_xor_sync(FULL_MASK, lo[k], o));
            hi[k] = fmax(hi[k], __shfl_xor_sync(FULL_MASK, hi[k], o));
        }
        if (lane == 0) { wext[warp][k] = lo[k]; wext[warp][3 + k] = hi[k]; }
    }
    __syncthreads();
    if (warp < 6) {
        double v = wext[lane][warp];
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) {
            const double u = __shfl_xor_sync(FULL_MASK, v, o);
            v = warp < 3 ? fmin(v, u) : fmax(v, u);
        }
        if (lane == 0) ext[warp] = v;
    }
    __syncthreads();
}
// exclusive sum over the threads of a block; *all = total
__device__ __forceinline__ int block_exclusive_sum(int v, int *ws, int *all)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { int n = __shfl_up_sync(FULL_MASK, inc, o); if (lane >= o) inc += n; }
    if (lane == 31) ws[warp] = inc;
    __syncthreads();
    int w = lane < nw ? ws[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { int n = __shfl_up_sync(FULL_MASK, w, o); if (lane >= o) w += n; }
    const int before = __shfl_sync(FULL_MASK, w, max(warp - 1, 0));
    *all = __shfl_sync(FULL_MASK, w, 31);
    return inc - v + (warp > 0 ? before : 0);
}

template <typename T>
__global__ void __launch_bounds__(BINB_THREADS, 1)
nb_bin_block_kernel(NbParams<T> P, NbGrid host_grid, int have_grid, const T *__restrict__ coords, NbGrid *__restrict__ gp,
                    int *__restrict__ bin_start, typename Vec4<T>::type *__restrict__ spos, float4 *__restrict__ sposw,
                    int4 *__restrict__ sinfo, int *__restrict__ status, const NepSetup side)
{
    if (blockIdx.x > 0) {      // blocks of another kernel's set-up
        chain_release();
        chain_wait();
        nep_setup_any(side, blockIdx.x - 1);
        return;
    }
    __shared__ int cnt[BINB_MAX_BINS];           // counters, then the starts of the bins
    __shared__ int ws[32];
    __shared__ double wext[32][6], bext[6];
    __shared__ int block_wrap;
    __shared__ NbGrid sg;
    chain_release();
    for (int k = threadIdx.x; k < BINB_MAX_BINS; k += BINB_THREADS) cnt[k] = 0;
    if (threadIdx.x == 0) { block_wrap = 0; if (have_grid) sg = host_grid; }
    chain_wait();
    if (!have_grid) {     // extents of the atoms along the open axes
        double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
        for (int i = threadIdx.x; i < P.n; i += BINB_THREADS) {
            double s[3];
            frac_of(P, position_of(P, coords, i), s);
#pragma unroll
            for (int k = 0; k < 3; k++) { lo[k] = fmin(lo[k], s[k]); hi[k] = fmax(hi[k], s[k]); }
        }
        block_extent(lo, hi, wext, bext);
        if (threadIdx.x == 0) nb_make_grid(P, bext, &sg);
    }
    __syncthreads();
    // count; every atom keeps its bin and its place in it
    int bin[BINB_ITEMS], off[BINB_ITEMS], reach = 0;
#pragma unroll
    for (int u = 0; u < BINB_ITEMS; u++) {
        const int i = threadIdx.x + u * BINB_THREADS;
        bin[u] = off[u] = 0;
        if (i < P.n) {
            double s[3];
            int w[3];
            frac_of(P, position_of(P, coords, i), s);
            bin[u] = bin_of(P, sg, s, w);
            reach = max(reach, wrap_reach(w));
            off[u] = atomicAdd(cnt + bin[u], 1);
        }
    }
    if (reach > 1) atomicMax(&block_wrap, reach);
    __syncthreads();
    const int total = sg.total, base = threadIdx.x * BINB_ITEMS;
    int v[BINB_ITEMS], sum = 0, all;
#pragma unroll
    for (int k = 0; k < BINB_ITEMS; k++) { v[k] = base + k < total ? cnt[base + k] : 0; sum += v[k]; }
    int start = block_exclusive_sum(sum, ws, &all);
#pragma unroll
    for (int k = 0; k < BINB_ITEMS; k++)
        if (base + k < total) { bin_start[base + k] = start; cnt[base + k] = start; start += v[k]; }
    const int wmax = block_wrap;
    if (threadIdx.x == 0) {
        NbGrid out = sg;
        out.maxwrap = wmax;
        *gp = out;
        bin_start[total] = P.n;
        status[0] = 0; status[1] = 0;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < BINB_ITEMS; u++) {
        const int i = threadIdx.x + u * BINB_THREADS;
        if (i < P.n) {
            const Pos3<T> p = position_of(P, coords, i);
            double s[3];
            int wr[3];
            frac_of(P, p, s);
#pragma unroll
            for (int k = 0; k < 3; k++) wr[k] = P.per[k] ? (int)floor(s[k]) : 0;
            store_binned(P, cnt[bin[u]] + off[u], i, p, wr, wmax > NB_WRAP_MAX, spos, sposw, sinfo);
        }
    }
}

// ---- binning of larger systems: set-up, count, scan + fill --------------------------------------------
// the grid parameters are known on the host: one kernel zeroes the bin counters, resets the status words and writes the grid
__global__ void nb_setup_kernel(NbGrid host_grid, NbGrid *__restrict__ g, int *__restrict__ count, int ncount, int *__restrict__ status)
{
    chain_release();
    chain_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < ncount) count[i] = 0;
    if (i == 0) {
        status[0] = 0; status[1] = 0;
        *g = host_grid;
    }
}
// the same when an axis is open and its extent is not known: a cluster of blocks looks at all atoms first (a cluster keeps
// this one launch; systems of more than SETUP_OPEN_ATOMS atoms take nb_extent_kernel, which fills the chip)
constexpr int SETUP_CLUSTER = 8;
constexpr int SETUP_OPEN_ATOMS = 200000;
template <typename T>
__global__ void __cluster_dims__(SETUP_CLUSTER, 1, 1) __launch_bounds__(BINB_THREADS, 1)
nb_setup_open_kernel(NbParams<T> P, const T *__restrict__ coords, NbGrid *__restrict__ gp, int *__restrict__ count, int *__restrict__ status)
{
    namespace cg = cooperative_groups;
    __shared__ double wext[32][6], bext[6];
    __shared__ NbGrid sg;
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    chain_release();
    chain_wait();
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    for (int i = rank * BINB_THREADS + threadIdx.x; i < P.n; i += SETUP_CLUSTER * BINB_THREADS) {
        double s[3];
        frac_of(P, position_of(P, coords, i), s);
#pragma unroll
        for (int k = 0; k < 3; k++) { lo[k] = fmin(lo[k], s[k]); hi[k] = fmax(hi[k], s[k]); }
    }
    block_extent(lo, hi, wext, bext);
    cl.sync();
    if (threadIdx.x < 6) {
        double v = bext[threadIdx.x];
        for (int r = 0; r < SETUP_CLUSTER; r++) {
            const double u = *cl.map_shared_rank(&bext[threadIdx.x], r);
            v = threadIdx.x < 3 ? fmin(v, u) : fmax(v, u);
        }
        wext[0][threadIdx.x] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        nb_make_grid(P, wext[0], &sg);
        if (rank == 0) { *gp = sg; status[0] = 0; status[1] = 0; }
    }
    __syncthreads();
    for (int i = rank * BINB_THREADS + threadIdx.x; i < sg.total; i += SETUP_CLUSTER * BINB_THREADS) count[i] = 0;
    cl.sync();      // no block leaves while another may still read its extents
}

// bin of every atom and its place in the bin, bin populations
template <typename T>
__global__ void nb_count_kernel(NbParams<T> P, NbGrid *gp, const T *__restrict__ coords, int2 *__restrict__ ainfo, int *__restrict__ bin_count)
{
    chain_release();
    chain_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.n) return;
    const NbGrid g = *gp;
    double s[3];
    int w[3];
    frac_of(P, position_of(P, coords, i), s);
    const int bin = bin_of(P, g, s, w);
    const int reach = wrap_reach(w);
    if (reach > 1) atomicMax(&gp->maxwrap, reach);
    ainfo[i] = make_int2(bin, atomicAdd(bin_count + bin, 1));
}

// Exclusive scan of in[0 .. total) -> out[0 .. total] by one cluster: every block scans a chunk that its threads load along
// the array, scan eight counters each by themselves, and combine with one block-wide scan; the blocks' totals are read from
// each other's shared memory. Longer arrays take several rounds.
constexpr int SCAN_BLOCK = 1024;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_CLUSTER = 8;
__global__ void __cluster_dims__(SCAN_CLUSTER, 1, 1) __launch_bounds__(SCAN_BLOCK)
nb_scan_kernel(const NbGrid *__restrict__ gp, const int *__restrict__ in, int *__restrict__ out)
{
    namespace cg = cooperative_groups;
    __shared__ int buf[SCAN_BLOCK * (SCAN_ITEMS + 1)];
    __shared__ int ws[32];
    __shared__ int block_total[2];
    cg::cluster_group cl = cg::this_cluster();
    chain_release();
    chain_wait();
    const int rank = (int)cl.block_rank();
    const int total = gp->total;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int carry = 0, turn = 0;
    for (int round = 0; round <= total; round += SCAN_CLUSTER * SCAN_BLOCK * SCAN_ITEMS, turn ^= 1) {
        const int base = round + rank * SCAN_BLOCK * SCAN_ITEMS;
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; k++) {
            const int e = k * SCAN_BLOCK + threadIdx.x, i = base + e;
            buf[(e / SCAN_ITEMS) * (SCAN_ITEMS + 1) + e % SCAN_ITEMS] = i < total ? in[i] : 0;
        }
        __syncthreads();
        int v[SCAN_ITEMS], sum = 0;
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; k++) {
            v[k] = sum;
            sum += buf[threadIdx.x * (SCAN_ITEMS + 1) + k];
        }
        int inc = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { int n = __shfl_up_sync(FULL_MASK, inc, o); if (lane >= o) inc += n; }
        if (lane == 31) ws[warp] = inc;
        __syncthreads();
        int w = ws[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { int n = __shfl_up_sync(FULL_MASK, w, o); if (lane >= o) w += n; }
        const int before = __shfl_sync(FULL_MASK, w, max(warp - 1, 0)), all = __shfl_sync(FULL_MASK, w, 31);
        if (threadIdx.x == 0) block_total[turn] = all;
        cl.sync();
        int off = carry + inc - sum + (warp > 0 ? before : 0);
        for (int r = 0; r < SCAN_CLUSTER; r++) {
            const int t = *cl.map_shared_rank(&block_total[turn], r);
            if (r < rank) off += t;
            carry += t;
        }
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; k++) buf[threadIdx.x * (SCAN_ITEMS + 1) + k] = off + v[k];
        __syncthreads();
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; k++) {
            const int e = k * SCAN_BLOCK + threadIdx.x, i = base + e;
            if (i <= total) out[i] = buf[(e / SCAN_ITEMS) * (SCAN_ITEMS + 1) + e % SCAN_ITEMS];
        }
        __syncthreads();     // the buffer is reused by the next round (the totals alternate between two words)
    }
    cl.sync();      // no block leaves while another may still read its total
}

// Atoms into bin order. SCAN: the bins are few (at most FILL_SCAN_BINS), and every block sums their populations up by
// itself, which is cheaper than another launch between counting and filling; block 0 writes the starts down.
constexpr int FILL_SCAN_BINS = 8192;
constexpr int FILL_THREADS = 256;
template <typename T, bool SCAN>
__global__ void __launch_bounds__(FILL_THREADS)
nb_fill_kernel(NbParams<T> P, const T *__restrict__ coords, const int2 *__restrict__ ainfo, const int *__restrict__ bin_count,
               int *__restrict__ bin_start, typename Vec4<T>::type *__restrict__ spos, float4 *__restrict__ sposw, int4 *__restrict__ sinfo,
               const NbGrid *__restrict__ gp, int own, const NepSetup side)
{
    if ((int)blockIdx.x >= own) {      // blocks of another kernel's set-up
        chain_release();
        chain_wait();
        nep_setup_any(side, blockIdx.x - own);
        return;
    }
    __shared__ int s_start[SCAN ? FILL_SCAN_BINS : 1];
    __shared__ int ws[32];
    chain_release();
    chain_wait();
    const int i = blockIdx.x * FILL_THREADS + threadIdx.x;
    int2 a = make_int2(0, 0);
    Pos3<T> p = {T(0), T(0), T(0)};
    if (i < P.n) { a = ainfo[i]; p = position_of(P, coords, i); }
    if constexpr (SCAN) {
        const int total = gp->total, items = (total + FILL_THREADS - 1) / FILL_THREADS;
        for (int b = threadIdx.x; b < total; b += FILL_THREADS) s_start[b] = bin_count[b];
        __syncthreads();
        const int b0 = threadIdx.x * items, b1 = min(total, b0 + items);
        int sum = 0, all;
        for (int b = b0; b < b1; b++) sum += s_start[b];
        int start = block_exclusive_sum(sum, ws, &all);
        for (int b = b0; b < b1; b++) { const int c = s_start[b]; s_start[b] = start; start += c; }
        __syncthreads();
        if (blockIdx.x == 0) {
            for (int b = threadIdx.x; b < total; b += FILL_THREADS) bin_start[b] = s_start[b];
            if (threadIdx.x == 0) bin_start[total] = all;
        }
    }
    if (i >= P.n) return;
    double s[3];
    int w[3];
    frac_of(P, p, s);
#pragma unroll
    for (int k = 0; k < 3; k++) w[k] = P.per[k] ? (int)floor(s[k]) : 0;
    const int first = SCAN ? s_start[a.x] : bin_start[a.x];
    store_binned(P, first + a.y, i, p, w, gp->maxwrap > NB_WRAP_MAX, spos, sposw, sinfo);
}

// Is an image of candidate pj a neighbour of centre pi? d = image - centre. The image is given as packed periods per axis
// (nw) or, if those do not fit, as plain ones (n0, n1, n2).
template <typename T>
__device__ __forceinline__ bool nb_exact(const NbParams<T> &P, const typename Vec4<T>::type &pj, const typename Vec4<T>::type &pi, bool packed,
                                         int nw, int n0, int n1, int n2, bool have, T &d0, T &d1, T &d2)
{
    bool covered = have;
    T ix = pj.x, iy = pj.y, iz = pj.z;
    // The home image needs no arithmetic: x + a*0 is x bit for bit, except for x = -0.0 (whose
    // sum with +0 is +0), so exact zeros take the full path.
    const bool away = packed ? nw != NB_PACK_ZERO : (n0 | n1 | n2) != 0;
    if (away || ix == T(0) || iy == T(0) || iz == T(0)) {
        if (packed) { n0 = (nw & 1023) - 512; n1 = ((nw >> 10) & 1023) - 512; n2 = ((nw >> 20) & 1023) - 512; }
        covered = have && abs(n0) <= P.e[0] && abs(n1) <= P.e[1] && abs(n2) <= P.e[2];
        const T f0 = T(n0), f1 = T(n1), f2 = T(n2);
        ix = add_rn(add_rn(add_rn(pj.x, mul_rn(P.cell[0], f0)), mul_rn(P.cell[3], f1)), mul_rn(P.cell[6], f2));
        iy = add_rn(add_rn(add_rn(pj.y, mul_rn(P.cell[1], f0)), mul_rn(P.cell[4], f1)), mul_rn(P.cell[7], f2));
        iz = add_rn(add_rn(add_rn(pj.z, mul_rn(P.cell[2], f0)), mul_rn(P.cell[5], f1)), mul_rn(P.cell[8], f2));
    }
    d0 = sub_rn(ix, pi.x); d1 = sub_rn(iy, pi.y); d2 = sub_rn(iz, pi.z);
    // Reference predicate: squares accumulate in double for both types (pow(T,int) promotes
    // float), the sum is rounded to T and compared with rc^2 and 1e-3. For float a
    // single-precision sum is within a few ulp of that value, so it decides every pair outside
    // a 2e-6 relative band around the two thresholds; only pairs inside the band take the
    // exact route.
    bool hit = false, undecided = covered;
    if (sizeof(T) == 4) {
        const float sq = (float)d0 * (float)d0 + (float)d1 * (float)d1 + (float)d2 * (float)d2;
        hit = covered && sq < P.rc2_lo && sq > P.eps_hi;
        undecided = covered && !hit && !(sq > P.rc2_hi || sq < P.eps_lo);
    }
    if (undecided) {
        const double dd = add_rn(add_rn(mul_rn((double)d0, (double)d0), mul_rn((double)d1, (double)d1)), mul_rn((double)d2, (double)d2));
        const double ddT = (double)(T)dd;
        hit = (ddT < P.rc2) && (ddT > 1e-3);
    }
    return hit;
}

// ---- rows --------------------------------------------------------------------------------------------
// A team of WPC warps per bin, CAP candidates of it in shared memory at a time. What bounds it is instruction issue: 700 warp
// instructions per atom at 13,824 atoms (280 candidates, 30 survivors), 540 at 1,048,576 of a sparser crystal, half of them exact
// predicate and row. One warp per atom with bins of half a cutoff and a table per atom took 1,750.
// TO = element type of the rcs rows (T, or float rows from double positions: what an MD host that keeps
// double coordinates and a single-precision model does on the CPU).
template <int WPC> __host__ __device__ constexpr int nbc_warps() { return WPC > 4 ? WPC : 4; }    // warps per block
constexpr int NBC_STAGE_BYTES = 7 * 1024;     // longest row that is put together in shared memory
template <typename TO, int WPC, int CAP>
__host__ __device__ inline size_t nbc_smem(int umax, bool staged)
{
    constexpr int NBC_WARPS = nbc_warps<WPC>(), TEAMS = NBC_WARPS / WPC;
    return (size_t)TEAMS * CAP * (sizeof(float4) + 2 * sizeof(int)) + (size_t)NBC_WARPS * CAP * sizeof(unsigned short) +
           (staged ? (size_t)NBC_WARPS * umax * (sizeof(int) + 3 * sizeof(TO)) : 0);
}

// two single-precision fused multiply-adds in one instruction
__device__ __forceinline__ unsigned long long pack2(float a, float b)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c)
{
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

template <typename T, typename TO, int WPC, int CAP>
__global__ void __launch_bounds__(nbc_warps<WPC>() * 32, WPC == 8 ? 4 : 9)
nb_rows_kernel(NbParams<T> P, const NbGrid *__restrict__ gp, const int *__restrict__ bin_start, const typename Vec4<T>::type *__restrict__ spos,
               const float4 *__restrict__ sposw, const int4 *__restrict__ sinfo, int *__restrict__ numneigh, int *__restrict__ firstneigh,
               TO *__restrict__ rcs, int *__restrict__ status, int staged, int splits)
{
    constexpr int NBC_WARPS = nbc_warps<WPC>(), TEAMS = NBC_WARPS / WPC, TT = WPC * 32;
    extern __shared__ __align__(16) unsigned char nbc_smem_raw[];
    __shared__ int s_start[TEAMS][32], s_pre[TEAMS][33], s_shift[TEAMS][32];
    __shared__ float4 s_sv[TEAMS][32];        // image shift of a table entry as a single-precision vector
    __shared__ float s_n2[NBC_WARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int team = warp / WPC, tw = warp % WPC, tt = threadIdx.x - team * TT;
    // candidates e and e + 32 of every 64 side by side, positions relative to the bin: 32 x {x, x', y, y'}, 32 x {z, z', q^2, q'^2}
    ulonglong2 *cq = reinterpret_cast<ulonglong2 *>(nbc_smem_raw) + team * CAP;
    int *caj = reinterpret_cast<int *>(reinterpret_cast<float4 *>(nbc_smem_raw) + TEAMS * CAP) + team * CAP;    // a candidate's place in bin order
    int *csh = caj + TEAMS * CAP;                                            // its image, less its own wrap
    unsigned char *p_list = nbc_smem_raw + (size_t)TEAMS * CAP * (sizeof(float4) + 2 * sizeof(int));
    TO *rowp = reinterpret_cast<TO *>(p_list) + (size_t)warp * 3 * P.umax;   // (staged only)
    int *rowi = reinterpret_cast<int *>(reinterpret_cast<TO *>(p_list) + (size_t)NBC_WARPS * 3 * P.umax) + warp * P.umax;
    unsigned short *list = reinterpret_cast<unsigned short *>(p_list + (staged ? (size_t)NBC_WARPS * P.umax * (sizeof(int) + 3 * sizeof(TO)) : 0)) + warp * CAP;
    // The teams of a block walk over different numbers of bins (empty ones are skipped) and tables of different length, so a
    // barrier is the team's own (numbers as constants: a number in a register would claim all sixteen).
    static_assert(WPC == 1 || TEAMS <= 2, "a barrier per team");
    auto sync_team = [&]() {
        __syncwarp();
        if constexpr (WPC > 1) {
            if constexpr (TEAMS == 1) __syncthreads();
            else if (team == 0) asm volatile("bar.sync 1, %0;" ::"n"(TT) : "memory");
            else asm volatile("bar.sync 2, %0;" ::"n"(TT) : "memory");
        }
    };
    // no chain_release(): blocks of the next kernel that become resident now only take slots and issue cycles from this one
    // (13,824 atoms: a NEP evaluation 85.7 -> 74.5 us, an MTP evaluation 143.9 -> 127.7 us)
    chain_wait();
    const NbGrid g = *gp;
    const bool packed = g.maxwrap <= NB_WRAP_MAX;   // every wrap fits the packed form
    const float pre_hi = (float)((P.rc2 + (double)g.pre_err * (1.0 + g.maxwrap)) * (1.0 + 1e-6));
    const int nx = 2 * g.R[0] + 1, ny = 2 * g.R[1] + 1, nz = 2 * g.R[2] + 1;
    const bool zmerge = g.zmerge != 0;
    const int nnb_full = zmerge ? nx * ny : nx * ny * nz;   // table entries of a bin away from the third axis' faces
    const unsigned lt_mask = (1u << lane) - 1u;
    int local_max = 0;
    // offsets of table entry `lane` (the table of most bins is that of the first 32 entries)
    int ent0 = 0, ent1 = 0, ent2 = 0;
    {
        const int kk = zmerge && lane >= nnb_full ? lane - nnb_full : lane;
        if (zmerge) { ent0 = kk / ny - g.R[0]; ent1 = kk % ny - g.R[1]; }
        else { ent0 = kk / (ny * nz) - g.R[0]; ent1 = (kk / nz) % ny - g.R[1]; ent2 = kk % nz - g.R[2]; }
    }

    for (int unit = blockIdx.x * TEAMS + team; unit < g.total * splits; unit += gridDim.x * TEAMS) {
        const int cell = unit / splits, part = unit - cell * splits;      // (splits > 1: small systems)
        const int a_begin = bin_start[cell], a_end = bin_start[cell + 1];
        if (a_begin + part * WPC >= a_end) continue;
        const int col = cell / g.nb[2], bz = cell - col * g.nb[2], bx = col / g.nb[1], by = col - bx * g.nb[1];
        // With merged columns a bin within R bins of a periodic face of the third axis has, per column, a second
        // range: the part of its 2R+1 bins that lies across the face (entries nnb_full .. 2 nnb_full - 1).
        const bool zsplit = zmerge && P.per[2] && (bz - g.R[2] < 0 || bz + g.R[2] >= g.nb[2]);
        const int nnb = zsplit ? 2 * nnb_full : nnb_full;
        float4 org = sposw[a_begin];
        if (!(fabsf(org.x) + fabsf(org.y) + fabsf(org.z) < 1e15f)) org = make_float4(0.f, 0.f, 0.f, 0.f);   // an atom that has flown off

        // up to 32 table entries (columns of bins, or bins) from entry `base` on, by the team's first warp; returns their candidates
        auto make_entries = [&](int base) -> int {
            if (tw == 0) {
                int start = 0, len = 0, shift = 0;
                float4 sv = make_float4(0.f, 0.f, 0.f, 0.f);
                const int k = base + lane;
                if (k < nnb) {
                    int d[3] = {ent0, ent1, ent2}, b[3], m[3];
                    if (base > 0) {
                        const int kk = zmerge && k >= nnb_full ? k - nnb_full : k;
                        if (zmerge) { d[0] = kk / ny - g.R[0]; d[1] = kk % ny - g.R[1]; d[2] = 0; }
                        else { d[0] = kk / (ny * nz) - g.R[0]; d[1] = (kk / nz) % ny - g.R[1]; d[2] = kk % nz - g.R[2]; }
                    }
                    b[0] = bx + d[0]; b[1] = by + d[1]; b[2] = bz + d[2];
                    bool ok = true;
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        m[c] = 0;
                        if (b[c] < 0 || b[c] >= g.nb[c]) {      // across a face of the cell
                            if (P.per[c]) {
                                int q = b[c] < 0 ? -1 : 1;      // one period off unless the grid is tiny
                                if (b[c] < -g.nb[c] || b[c] >= 2 * g.nb[c]) q = b[c] >= 0 ? b[c] / g.nb[c] : -((-b[c] + g.nb[c] - 1) / g.nb[c]);
                                m[c] = q; b[c] -= q * g.nb[c];
                            } else {
                                ok = false;
                            }
                        }
                    }
                    int zlo = b[2], zhi = b[2];          // bins of the third axis this entry covers (inside the grid)
                    if (zmerge) {
                        zlo = bz - g.R[2]; zhi = bz + g.R[2];
                        if (k < nnb_full) {              // the part inside the cell
                            zlo = max(zlo, 0); zhi = min(zhi, g.nb[2] - 1);
                        } else if (zlo < 0) {            // the part below the face: bins nb + zlo .. nb - 1 of the image one period down
                            zlo += g.nb[2]; zhi = g.nb[2] - 1; m[2] = -1;
                        } else {                         // the part above the face
                            zhi -= g.nb[2]; zlo = 0; m[2] = 1;
                        }
                    }
                    if (ok) {
                        const int c0 = (b[0] * g.nb[1] + b[1]) * g.nb[2];
                        start = bin_start[c0 + zlo];
                        len = bin_start[c0 + zhi + 1] - start;
                        shift = nb_pack3(m[0], m[1], m[2]);
                        const float f0 = (float)m[0], f1 = (float)m[1], f2 = (float)m[2];
                        sv.x = f0 * (float)P.cell[0] + f1 * (float)P.cell[3] + f2 * (float)P.cell[6];
                        sv.y = f0 * (float)P.cell[1] + f1 * (float)P.cell[4] + f2 * (float)P.cell[7];
                        sv.z = f0 * (float)P.cell[2] + f1 * (float)P.cell[5] + f2 * (float)P.cell[8];
                    }
                }
                int inc = len;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) { int n = __shfl_up_sync(FULL_MASK, inc, o); if (lane >= o) inc += n; }
                s_start[team][lane] = start;
                s_pre[team][lane] = inc - len;
                s_shift[team][lane] = shift;
                s_sv[team][lane] = sv;
                if (lane == 31) s_pre[team][32] = inc;
            }
            sync_team();
            return s_pre[team][32];
        };
        // candidates c0 .. c0 + count of the entries into shared memory (the tail of the last 64 filled with far-away
        // points); returns the widening of the pre-test: rounding of |q_j|^2 - 2 q_i q_j + |q_i|^2
        auto load_candidates = [&](int c0, int count) -> float {
            float n2max = 0.f;
            for (int s = tt; s < ((count + 63) & ~63) / 2; s += TT) {
                float qx[2], qy[2], qz[2], qw[2];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int e = (s & ~31) * 2 + (s & 31) + 32 * h;
                    qx[h] = qy[h] = qz[h] = 0.f; qw[h] = 3e38f;
                    if (e < count) {
                        const int c = c0 + e;
                        int lo = 0;             // largest slot with pre[slot] <= c
#pragma unroll
                        for (int st = 16; st >= 1; st >>= 1) if (s_pre[team][lo + st] <= c) lo += st;
                        const int aj = s_start[team][lo] + (c - s_pre[team][lo]);
                        const float4 pw = sposw[aj], sv = s_sv[team][lo];
                        qx[h] = (pw.x + sv.x) - org.x; qy[h] = (pw.y + sv.y) - org.y; qz[h] = (pw.z + sv.z) - org.z;
                        qw[h] = qx[h] * qx[h] + qy[h] * qy[h] + qz[h] * qz[h];
                        n2max = fmaxf(n2max, qw[h]);
                        caj[e] = aj;
                        csh[e] = packed ? s_shift[team][lo] - __float_as_int(pw.w) : s_shift[team][lo];
                    }
                }
                ulonglong2 *dst = cq + 2 * (s & ~31) + (s & 31);
                dst[0] = make_ulonglong2(pack2(qx[0], qx[1]), pack2(qy[0], qy[1]));
                dst[32] = make_ulonglong2(pack2(qz[0], qz[1]), pack2(qw[0], qw[1]));
            }
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) n2max = fmaxf(n2max, __shfl_xor_sync(FULL_MASK, n2max, o));
            if constexpr (WPC > 1) {
                if (lane == 0) s_n2[warp] = n2max;
                sync_team();
#pragma unroll
                for (int k = 0; k < WPC; k++) n2max = fmaxf(n2max, s_n2[team * WPC + k]);
            } else {
                __syncwarp();
            }
            return 2e-6f * n2max;
        };

        // tests atom `a` of the bin against the candidates in shared memory and appends its hits behind `count`
        auto scan_centre = [&](int a, int ncand, float slack, int count, int *frow, TO *rrow) -> int {
            const float4 pw = sposw[a];
            const typename Vec4<T>::type pi = spos[a];
            const float qx = pw.x - org.x, qy = pw.y - org.y, qz = pw.z - org.z;
            // below the padding's 3e38 whatever the atoms are (infinite or undefined: the exact predicate decides about all others)
            const float limit = fminf(pre_hi + slack - (qx * qx + qy * qy + qz * qz), 1e38f);
            const unsigned long long mx = pack2(-2.f * qx, -2.f * qx), my = pack2(-2.f * qy, -2.f * qy), mz = pack2(-2.f * qz, -2.f * qz);
            unsigned mine = 0;      // bit k: candidate 32 k + lane survives
            const ulonglong2 *cl = cq + lane;
#pragma unroll 2
            for (int k = 0; 32 * k < ncand; k += 2, cl += 64) {
                const ulonglong2 a2 = cl[0], b2 = cl[32];
                float v0, v1;
                unpack2(fma2(mx, a2.x, fma2(my, a2.y, fma2(mz, b2.x, b2.y))), v0, v1);
                if (v0 < limit) mine |= 1u << k;
                if (v1 < limit) mine |= 2u << k;
            }
            int inc = __popc(mine);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { int n = __shfl_up_sync(FULL_MASK, inc, o); if (lane >= o) inc += n; }
            const int nsurv = __shfl_sync(FULL_MASK, inc, 31);
            for (unsigned short *l = list + inc; mine; mine &= mine - 1) *--l = (unsigned short)((__ffs(mine) - 1) * 32 + lane);
            __syncwarp();
            int4 si = make_int4(0, 0, 0, 0);
            if (!packed) si = sinfo[a];
            const int wi = __float_as_int(pw.w);
            for (int c0 = 0; c0 < nsurv; c0 += 32) {
                const int c = c0 + lane;
                const bool have = c < nsurv;
                const int e = have ? list[c] : 0;
                const int aj = caj[e], sh = csh[e];
                const typename Vec4<T>::type pj = spos[aj];
                // periods between the candidate's stored position and the image this entry means: bin shift - candidate's
                // wrap + centre's wrap, all three axes in one word if they fit
                int n0 = 0, n1 = 0, n2 = 0;
                if (!packed) {
                    const int4 sj = sinfo[aj];
                    n0 = (sh & 1023) - 512 - sj.y + si.y;
                    n1 = ((sh >> 10) & 1023) - 512 - sj.z + si.z;
                    n2 = ((sh >> 20) & 1023) - 512 - sj.w + si.w;
                }
                T d0, d1, d2;
                const bool hit = nb_exact<T>(P, pj, pi, packed, sh + wi, n0, n1, n2, have, d0, d1, d2);
                const unsigned bal = __ballot_sync(FULL_MASK, hit);
                if (hit) {
                    const int p = count + __popc(bal & lt_mask);
                    if (p < P.umax) {
                        frow[p] = nb_bits_of(pj.w);
                        rrow[3 * p] = (TO)d0; rrow[3 * p + 1] = (TO)d1; rrow[3 * p + 2] = (TO)d2;
                    }
                }
                count += __popc(bal);
            }
            __syncwarp();
            return count;
        };
        auto pad_row = [&](int count, int *frow, TO *rrow) {
            for (int k = count + lane; k < P.umax; k += 32) {
                frow[k] = -1;
                rrow[3 * k] = TO(0); rrow[3 * k + 1] = TO(0); rrow[3 * k + 2] = TO(0);
            }
        };

        int total = make_entries(0);
        if (nnb <= 32 && total <= CAP) {     // the usual case: one table serves all atoms of the bin
            const float slack = load_candidates(0, total);
            for (int a = a_begin + part * WPC + tw; a < a_end; a += WPC * splits) {
                const int i = nb_bits_of(spos[a].w);
                if (i >= P.ncentre || i < P.cbegin) continue;
                int *frow = firstneigh + (size_t)(i - P.cbegin) * P.umax;
                TO *rrow = rcs + (size_t)(i - P.cbegin) * P.umax * 3;
                int count;
                if (staged) {
                    count = scan_centre(a, total, slack, 0, rowi, rowp);
                    pad_row(count, rowi, rowp);
                    __syncwarp();
                    for (int k = lane; k < P.umax / 4; k += 32) reinterpret_cast<int4 *>(frow)[k] = reinterpret_cast<const int4 *>(rowi)[k];
                    for (int k = lane; k < 3 * P.umax * (int)sizeof(TO) / 16; k += 32)
                        reinterpret_cast<int4 *>(rrow)[k] = reinterpret_cast<const int4 *>(rowp)[k];
                    __syncwarp();
                } else {
                    count = scan_centre(a, total, slack, 0, frow, rrow);
                    pad_row(count, frow, rrow);
                }
                if (lane == 0) numneigh[i - P.cbegin] = min(count, P.umax);
                local_max = max(local_max, count);
            }
            sync_team();      // the table is rebuilt for the next bin
        } else {
            // cells narrower than the cutoff or crowded bins: the candidates come in pieces. Up to 32 atoms of the bin per
            // sweep over the pieces, lane l of the team's warp keeps the count of the l-th atom that the warp owns
            for (int ab = a_begin + part * WPC; ab < a_end; ab += 32 * WPC * splits) {
                int counts = 0;
                for (int base = 0; base < nnb; base += 32) {
                    sync_team();
                    total = make_entries(base);
                    for (int c0 = 0; c0 < total; c0 += CAP) {
                        sync_team();
                        const int ncand = min(CAP, total - c0);
                        const float slack = load_candidates(c0, ncand);
                        for (int l = 0; l < 32; l++) {
                            const int a = ab + l * WPC * splits + tw;
                            if (a >= a_end) break;
                            const int i = nb_bits_of(spos[a].w);
                            if (i >= P.ncentre || i < P.cbegin) continue;
                            int *frow = firstneigh + (size_t)(i - P.cbegin) * P.umax;
                            TO *rrow = rcs + (size_t)(i - P.cbegin) * P.umax * 3;
                            const int c = scan_centre(a, ncand, slack, __shfl_sync(FULL_MASK, counts, l), frow, rrow);
                            if (lane == l) counts = c;
                        }
                    }
                }
                for (int l = 0; l < 32; l++) {
                    const int a = ab + l * WPC * splits + tw;
                    if (a >= a_end) break;
                    const int i = nb_bits_of(spos[a].w);
                    if (i >= P.ncentre || i < P.cbegin) continue;
                    const int count = __shfl_sync(FULL_MASK, counts, l);
                    pad_row(count, firstneigh + (size_t)(i - P.cbegin) * P.umax, rcs + (size_t)(i - P.cbegin) * P.umax * 3);
                    if (lane == 0) numneigh[i - P.cbegin] = min(count, P.umax);
                    local_max = max(local_max, count);
                }
            }
            sync_team();
        }
    }
    if (lane == 0 && local_max > 0) {
        atomicMax(status, local_max);
        if (local_max > P.umax) status[1] = 1;
    }
}

// optional pass 4: order each row by distance (the reference's sort=true, neighborList.h:290-335:
// std::sort on sqrt(dx^2+dy^2+dz^2)). Stable rank sort, one warp per row; ties keep build order.
template <typename T>
__global__ void nb_sort_rows_kernel(int n, int umax, const int *__restrict__ numneigh, int *__restrict__ firstneigh, T *__restrict__ rcs)
{
    extern __shared__ __align__(16) unsigned char sort_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    T *key = reinterpret_cast<T *>(sort_smem) + (size_t)warp * umax * 4;
    T *val = key + umax;                                   // 3 * umax
    int *idx = reinterpret_cast<int *>(reinterpret_cast<T *>(sort_smem) + (size_t)wpb * umax * 4) + (size_t)warp * umax;
    for (int i = blockIdx.x * wpb + warp; i < n; i += gridDim.x * wpb) {
        const int nn = min(numneigh[i], umax);
        int *frow = firstneigh + (size_t)i * umax;
        T *rrow = rcs + (size_t)i * umax * 3;
        for (int k = lane; k < nn; k += 32) {
            T a = rrow[3 * k], b = rrow[3 * k + 1], c = rrow[3 * k + 2];
            val[3 * k] = a; val[3 * k + 1] = b; val[3 * k + 2] = c;
            idx[k] = frow[k];
            key[k] = (T)sqrt((double)a * (double)a + (double)b * (double)b + (double)c * (double)c);
        }
        __syncwarp();
        for (int k = lane; k < nn; k += 32) {
            const T kk = key[k];
            int rank = 0;
            for (int m = 0; m < nn; m++) rank += (key[m] < kk || (key[m] == kk && m < k)) ? 1 : 0;
            frow[rank] = idx[k];
            rrow[3 * rank] = val[3 * k]; rrow[3 * rank + 1] = val[3 * k + 1]; rrow[3 * rank + 2] = val[3 * k + 2];
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------------------------
struct NbLayout {
    size_t grid, ext, ainfo, count, start, spos, sinfo, sposw, total;
};
template <typename T>
static NbLayout nb_layout(int n, int maxbins)
{
    NbLayout L;
    size_t o = 0;
    auto take = [&](size_t bytes) { size_t r = o; o += (bytes + 255) & ~size_t(255); return r; };
    L.grid = take(sizeof(NbGrid));
    L.ext = take(6 * sizeof(unsigned long long));
    L.ainfo = take(sizeof(int2) * (size_t)n);
    L.count = take(sizeof(int) * ((size_t)maxbins + 1));
    L.start = take(sizeof(int) * ((size_t)maxbins + 2));
    L.spos = take(sizeof(typename Vec4<T>::type) * (size_t)n);
    L.sinfo = take(sizeof(int4) * (size_t)n);
    L.sposw = take(sizeof(float4) * (size_t)n);
    L.total = o;
    return L;
}
// Bins at most: a structure has about one bin per four to ten atoms, sparse cells up to one per atom.
static int nb_maxbins(int n) { return n <= BINB_MAX_ATOMS ? BINB_MAX_BINS : n + 4096; }

template <typename T>
static void plane_distances(const T *cell, T *d)
{
    // interplanar distances in type T, same operations as structure.h:818-843
    for (int k = 0; k < 3; k++) {
        const T *a = cell + 3 * ((k == 0) ? 1 : 0), *b = cell + 3 * ((k == 2) ? 1 : 2);
        T n[3] = {a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]};
        T len = (T)std::sqrt((double)(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]));
        T u[3] = {n[0] / len, n[1] / len, n[2] / len};
        const T *c = cell + 3 * k;
        d[k] = (T)std::fabs((double)(c[0] * u[0] + c[1] * u[1] + c[2] * u[2]));
    }
}

constexpr int NBC_SMALL_ATOMS = 8000;
template <typename T, typename TO, int WPC, int CAP>
static int launch_rows(const NbParams<T> &P, const NbGrid *grid, const int *start, const typename Vec4<T>::type *spos, const float4 *sposw,
                       const int4 *sinfo, int *numneigh, int *firstneigh, TO *rcs, int *status, int staged, long bins, int splits, cudaStream_t st)
{
    auto kern = nb_rows_kernel<T, TO, WPC, CAP>;
    const size_t smem = nbc_smem<TO, WPC, CAP>(P.umax, staged != 0);
    static KernelSetup setup;
    int per_sm = 1;
    if (int rc = kernel_setup(setup, kern, smem, nbc_warps<WPC>() * 32, &per_sm)) return rc;
    constexpr int NBC_WARPS = nbc_warps<WPC>(), TEAMS = NBC_WARPS / WPC;
    long blocks = (bins * splits + TEAMS - 1) / TEAMS;
    if (blocks > (long)sm_count() * per_sm) blocks = (long)sm_count() * per_sm;
    AI2B_CUDA(launch_chained(kern, (unsigned)blocks, NBC_WARPS * 32, smem, st, P, grid, start, spos, sposw, sinfo, numneigh, firstneigh, rcs,
                             status, staged, splits));
    return AI2B_OK;
}

// Rows for the centres [cbegin, ncentre) of the n atoms. reuse_bins: the workspace still holds the bins of an
// earlier call with the same atoms, cell, cutoff and flags, so only the row pass runs (d_status is then
// accumulated into, not reset).
template <typename T, typename TO = T>
static int nblist_build(int n, int ncentre, const T *h_cell, const T *d_coords, int is_cart, double rcut_in, const int *pbc, int umax,
                        int *d_numneigh, int *d_firstneigh, TO *d_rcs, int *d_status, void *ws, size_t ws_bytes, cudaStream_t st,
                        int cbegin = 0, bool reuse_bins = false, const double *open_ext = nullptr, const NepSetup &side = NepSetup())
{
    AI2B_REQUIRE(h_cell && pbc && d_status, AI2B_ERR_INVALID, "ai2b_nblist_build: NULL argument");
    AI2B_REQUIRE(n >= 0 && umax >= 0 && rcut_in > 0 && ncentre >= 0 && ncentre <= n && cbegin >= 0 && cbegin <= ncentre,
                 AI2B_ERR_INVALID, "ai2b_nblist_build: bad size, centre range or cutoff");
    if (n == 0 || ncentre == cbegin) return AI2B_OK;
    AI2B_REQUIRE(d_coords && d_numneigh && d_firstneigh && d_rcs, AI2B_ERR_INVALID, "ai2b_nblist_build: NULL argument");
    const int maxbins = nb_maxbins(n);
    const NbLayout L = nb_layout<T>(n, maxbins);
    AI2B_REQUIRE(ws && ws_bytes >= L.total, AI2B_ERR_WORKSPACE, "nblist workspace too small: %zu < %zu bytes", ws_bytes, L.total);

    NbParams<T> P;
    memset(&P, 0, sizeof(P));
    const T rcut = (T)rcut_in;                 // the float build casts rcut first (nblist_bind.cc:133)
    for (int k = 0; k < 9; k++) P.cell[k] = h_cell[k];
    // inverse cell in double
    double a[9];
    for (int k = 0; k < 9; k++) a[k] = (double)h_cell[k];
    double det = a[0] * (a[4] * a[8] - a[5] * a[7]) - a[1] * (a[3] * a[8] - a[5] * a[6]) + a[2] * (a[3] * a[7] - a[4] * a[6]);
    AI2B_REQUIRE(std::fabs(det) > 1e-300, AI2B_ERR_INVALID, "ai2b_nblist_build: singular cell");
    // inv = A^{-1}, with r = f A  =>  f = r A^{-1}
    double c[9] = {a[4] * a[8] - a[5] * a[7], a[2] * a[7] - a[1] * a[8], a[1] * a[5] - a[2] * a[4],
                   a[5] * a[6] - a[3] * a[8], a[0] * a[8] - a[2] * a[6], a[2] * a[3] - a[0] * a[5],
                   a[3] * a[7] - a[4] * a[6], a[1] * a[6] - a[0] * a[7], a[0] * a[4] - a[1] * a[3]};
    for (int k = 0; k < 9; k++) P.inv[k] = c[k] / det;
    T dT[3];
    plane_distances<T>(h_cell, dT);
    P.rcut_m = (double)rcut * 1.0001 + 1e-6;
    P.rc2 = (double)rcut * (double)rcut;
    if (sizeof(T) == 8) { volatile double r2 = (double)rcut * (double)rcut; P.rc2 = r2; }
    P.rc2_lo = (float)(P.rc2 * (1.0 - 2e-6)); P.rc2_hi = (float)(P.rc2 * (1.0 + 2e-6));
    P.eps_lo = (float)(1e-3 * (1.0 - 2e-6)); P.eps_hi = (float)(1e-3 * (1.0 + 2e-6));
    P.n = n; P.umax = umax; P.maxbins = maxbins; P.ncentre = ncentre; P.cbegin = cbegin; P.is_cart = is_cart ? 1 : 0;
    bool any_open = false;
    long prod = 1;
    for (int k = 0; k < 3; k++) {
        P.per[k] = pbc[k] ? 1 : 0;
        P.dplane[k] = (double)dT[k];
        P.e[k] = pbc[k] ? (int)std::ceil((double)(rcut / dT[k])) : 0;
        AI2B_REQUIRE(P.e[k] < 500, AI2B_ERR_UNSUPPORTED, "cell far smaller than the cutoff (%d images on axis %d)", P.e[k], k);
        if (pbc[k]) {
            const double nb = std::floor(P.dplane[k] / P.rcut_m);
            P.nbh[k] = nb < 1 ? 1 : (nb > maxbins ? maxbins : (int)nb);
        } else {
            any_open = true;
            P.nbh[k] = 1;
        }
        prod *= P.nbh[k];
    }
    // shrink periodic bin counts if the grid would not fit, then hand the rest to the open axes
    while (prod > maxbins) {
        int big = 0;
        for (int k = 1; k < 3; k++) if (P.nbh[k] > P.nbh[big]) big = k;
        prod /= P.nbh[big];
        P.nbh[big] = (P.nbh[big] + 1) / 2;
        prod *= P.nbh[big];
    }
    if (any_open) {
        int nopen = 0;
        for (int k = 0; k < 3; k++) nopen += pbc[k] ? 0 : 1;
        int cap = (int)std::floor(std::pow((double)maxbins / (double)prod, 1.0 / nopen));
        for (int k = 0; k < 3; k++) if (!pbc[k]) P.nbh[k] = cap < 1 ? 1 : cap;
    }
    // The grid is known on the host when every axis is periodic, or when the caller gives the fractional extent
    // of the atoms along the open axes (atoms outside it are clamped into the edge bins, which keeps every
    // pair within reach of the bin search: an extent that is a little off costs time, not pairs).
    NbGrid hg;
    memset(&hg, 0, sizeof(hg));
    const bool host_grid = !any_open || open_ext != nullptr;
    if (host_grid) {
        nb_make_grid(P, open_ext, &hg);
        prod = hg.total;
    }

    unsigned char *w = (unsigned char *)ws;
    NbGrid *grid = (NbGrid *)(w + L.grid);
    unsigned long long *ext = (unsigned long long *)(w + L.ext);
    int2 *ainfo = (int2 *)(w + L.ainfo);
    int *count = (int *)(w + L.count), *start = (int *)(w + L.start);
    auto *spos = (typename Vec4<T>::type *)(w + L.spos);
    int4 *sinfo = (int4 *)(w + L.sinfo);
    float4 *sposw = (float4 *)(w + L.sposw);

    if (reuse_bins) {
        // bins and bin-ordered positions are in the workspace already
    } else if (n <= BINB_MAX_ATOMS) {
        AI2B_CUDA(launch_chained(nb_bin_block_kernel<T>, 1 + side.blocks, BINB_THREADS, 0, st, P, hg, host_grid ? 1 : 0, d_coords, grid, start, spos, sposw,
                                 sinfo, d_status, side));
    } else {
        const int nblk = (n + FILL_THREADS - 1) / FILL_THREADS;
        if (host_grid) {
            AI2B_CUDA(launch_chained(nb_setup_kernel, ((int)prod + 255) / 256, 256, 0, st, hg, grid, count, (int)prod, d_status));
        } else if (n <= SETUP_OPEN_ATOMS) {
            AI2B_CUDA(launch_chained(nb_setup_open_kernel<T>, SETUP_CLUSTER, BINB_THREADS, 0, st, P, d_coords, grid, count, d_status));
        } else {
            nb_init_kernel<<<1, 32, 0, st>>>(ext);
            nb_extent_kernel<T><<<1024, 256, 0, st>>>(P, d_coords, ext);
            nb_grid_kernel<T><<<1, 32, 0, st>>>(P, ext, grid, d_status);
            AI2B_CUDA(cudaMemsetAsync(count, 0, sizeof(int) * ((size_t)maxbins + 1), st));
        }
        AI2B_CUDA(launch_chained(nb_count_kernel<T>, nblk, FILL_THREADS, 0, st, P, grid, d_coords, ainfo, count));
        if ((host_grid ? prod : (long)maxbins) <= FILL_SCAN_BINS) {
            AI2B_CUDA(launch_chained(nb_fill_kernel<T, true>, nblk + side.blocks, FILL_THREADS, 0, st, P, d_coords, ainfo, count, start, spos, sposw, sinfo, grid,
                                     nblk, side));
        } else {
            AI2B_CUDA(launch_chained(nb_scan_kernel, SCAN_CLUSTER, SCAN_BLOCK, 0, st, grid, count, start));
            AI2B_CUDA(launch_chained(nb_fill_kernel<T, false>, nblk + side.blocks, FILL_THREADS, 0, st, P, d_coords, ainfo, count, start, spos, sposw, sinfo, grid,
                                     nblk, side));
        }
    }
    // rows leave as 16-byte stores when they start on 16-byte boundaries and one warp's row fits its share of shared memory
    const int staged = umax % 4 == 0 && (size_t)umax * (sizeof(int) + 3 * sizeof(TO)) <= NBC_STAGE_BYTES &&
                       (reinterpret_cast<size_t>(d_firstneigh) | reinterpret_cast<size_t>(d_rcs)) % 16 == 0;
    const long bins = host_grid ? prod : maxbins;
#define AI2B_ROWS(W, CAP, SPLITS) \
    return launch_rows<T, TO, W, CAP>(P, grid, start, spos, sposw, sinfo, d_numneigh, d_firstneigh, d_rcs, d_status, staged, bins, SPLITS, st)
    // Warps per bin (build times in us; in brackets what a table per atom took, or one lane per atom from 220,000 atoms on):
    //  * small systems: eight, and several blocks share the atoms of a bin until there are about four blocks per SM
    //    (1,000 atoms 9.4 [15.9], 4,913 atoms 15.6 [22.1])
    //  * sparse bins: the table is what costs, so the fewer warps build it the better (18.5 atoms per 1,000 A^3, cutoff 6:
    //    125,000 atoms 134 [138] with two, 1,048,576 atoms 804 [987] with one)
    //  * otherwise four (37 per 1,000 A^3: 13,824 atoms 27.4 [32.3], 64,000 atoms 83 [119], 1,000,000 atoms 907 [1299])
    const double per_bin = host_grid ? (double)n / bins : 8.0;
    if (const char *env = std::getenv("AI2B_NBL_MIN_ATOMS"))     // tuning knob, read per call: systems from this size on take one warp per bin
        if (n >= std::atoi(env)) AI2B_ROWS(1, 192, 1);
    if (n < NBC_SMALL_ATOMS) AI2B_ROWS(8, 448, (int)std::min(4L, std::max(1L, 4L * sm_count() / bins)));
    if (per_bin < 2.5 || (per_bin < 5.5 && n >= 200000)) AI2B_ROWS(1, 192, 1);
    if (per_bin < 5.5) AI2B_ROWS(2, 192, 1);
    AI2B_ROWS(4, 448, 1);
#undef AI2B_ROWS
}


// ---- padded batch of small cells: one launch --------------------------------------------------------
// A training set holds many small periodic structures (tens to hundreds of atoms); the reference's
// dataset builds one list per frame and pads every array to the largest structure
// (ai2pot/data/mlffdataset.py:61-90). For such cells a cell list brings nothing (1-3 bins per axis):
// the (centre, atom, image) triples of the reference's supercell are walked through instead, which is the
// reference's membership rule by construction. One block per (structure, chunk of centres); the
// structure's positions are staged through shared memory in tiles; one warp per centre:
//   1. lanes = images: an image whose atoms (bounding box of the tile) cannot reach the centre is dropped. Of the 27
//      images of a cell of 15 A about six are left at a cutoff of 6 A.
//   2. lanes = atoms of the tile, single precision, |q_j|^2 - 2 q_i q_j < limit for two atoms at a time as in the rows kernel:
//      triples that are certainly outside the cutoff are dropped, the others are queued in order
//   3. lanes = queued triples: the exact predicate, in full warps
// 64 structures of 64 to 256 atoms, 32 warps per SM: 32 us (64 registers, in double precision with 48 bytes of spills); with differences of coordinates, one atom per lane and step,
// image numbers taken apart by divisions and 94 registers (two blocks per SM) 40 us and 2,000 warp instructions per centre; testing
// every triple exactly 275 us.
constexpr int NBB_WARPS = 8;
constexpr int NBB_TILE = 512;       // atoms staged per tile
constexpr int NBB_CPW = 2;          // centres per warp
constexpr int NBB_CPB = NBB_WARPS * NBB_CPW;
constexpr int NBB_MINB = 4;         // blocks per SM
constexpr int NBB_QUEUE = 64;       // queued triples per warp: less than a warp's worth left over + one warp step

template <typename T>
struct NbBatchParams {
    int B, npad, umax, is_cart, per[3], staged;
    T rcut;
    double rc2;
    float rc2_lo, rc2_hi, eps_lo, eps_hi;
};

template <typename T>
__global__ void __launch_bounds__(NBB_WARPS * 32, NBB_MINB)
nb_batch_kernel(NbBatchParams<T> P, const int *__restrict__ binum, const T *__restrict__ cells, const T *__restrict__ coords,
                int *__restrict__ bilist, int *__restrict__ bnumneigh, int *__restrict__ bfirstneigh, T *__restrict__ brcs,
                int *__restrict__ status)
{
    extern __shared__ __align__(16) unsigned char nbb_smem[];     // rows under construction (staged)
    __shared__ T s_pos[NBB_TILE * 3];
    __shared__ ulonglong2 s_cq[NBB_TILE];      // atoms e and e + 32 of every 64, relative to the first: 32 x {x, x', y, y'}, 32 x {z, z', q^2, q'^2}
    __shared__ T s_cell[9];
    __shared__ int s_e[3];
    __shared__ float s_box[NBB_WARPS][7];
    __shared__ int s_queue[NBB_WARPS][NBB_QUEUE], s_img[NBB_WARPS][NBB_QUEUE];
    const int b = blockIdx.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n = min(max(binum[b], 0), P.npad);
    const int c_begin = blockIdx.x * NBB_CPB;
    if (c_begin >= P.npad) return;
    if (c_begin < n && threadIdx.x < 3) {
        // image range per periodic axis: ceil(rcut / interplanar distance), in type T with the operations of
        // source/nblist/include/structure.h:818-843 (no contraction)
        const int k = threadIdx.x;
        T c[9];
        for (int q = 0; q < 9; q++) c[q] = cells[(size_t)b * 9 + q];
        for (int q = 0; q < 3; q++) s_cell[3 * k + q] = c[3 * k + q];
        const T *a = c + 3 * ((k == 0) ? 1 : 0), *bb = c + 3 * ((k == 2) ? 1 : 2);
        const T nx = sub_rn(mul_rn(a[1], bb[2]), mul_rn(a[2], bb[1])), ny = sub_rn(mul_rn(a[2], bb[0]), mul_rn(a[0], bb[2])),
                nz = sub_rn(mul_rn(a[0], bb[1]), mul_rn(a[1], bb[0]));
        const T len = (T)sqrt((double)add_rn(add_rn(mul_rn(nx, nx), mul_rn(ny, ny)), mul_rn(nz, nz)));
        const T ux = nx / len, uy = ny / len, uz = nz / len;
        const T d = (T)fabs((double)add_rn(add_rn(mul_rn(c[3 * k], ux), mul_rn(c[3 * k + 1], uy)), mul_rn(c[3 * k + 2], uz)));
        int e = 0;
        if (P.per[k]) {
            const double q = ceil((double)(P.rcut / d));
            if (!(q < 500.0)) { e = 0; atomicOr(status + 1, 2); }   // degenerate cell: flagged, no images
            else e = (int)q;
        }
        s_e[k] = e;
    }
    __syncthreads();
    const T *cpos = coords + (size_t)b * P.npad * 3;
    auto cart = [&](int j, T &x, T &y, T &z) {
        const T f0 = cpos[3 * j], f1 = cpos[3 * j + 1], f2 = cpos[3 * j + 2];
        if (P.is_cart) { x = f0; y = f1; z = f2; return; }
        x = add_rn(add_rn(mul_rn(f0, s_cell[0]), mul_rn(f1, s_cell[3])), mul_rn(f2, s_cell[6]));
        y = add_rn(add_rn(mul_rn(f0, s_cell[1]), mul_rn(f1, s_cell[4])), mul_rn(f2, s_cell[7]));
        z = add_rn(add_rn(mul_rn(f0, s_cell[2]), mul_rn(f1, s_cell[5])), mul_rn(f2, s_cell[8]));
    };
    const unsigned lt_mask = (1u << lane) - 1u;
    int cnt[NBB_CPW];
#pragma unroll
    for (int q = 0; q < NBB_CPW; q++) cnt[q] = 0;
    // a row is put together in shared memory when one tile holds the structure
    const bool staged = P.staged != 0 && n <= NBB_TILE;
    T *rowp = reinterpret_cast<T *>(nbb_smem) + (size_t)warp * 3 * P.umax;
    int *rowi = reinterpret_cast<int *>(reinterpret_cast<T *>(nbb_smem) + (size_t)NBB_WARPS * 3 * P.umax) + warp * P.umax;
    auto pad_row = [&](int count, int *frow, T *rrow) {
        for (int k = count + lane; k < P.umax; k += 32) {
            frow[k] = -1;
            rrow[3 * k] = T(0); rrow[3 * k + 1] = T(0); rrow[3 * k + 2] = T(0);
        }
    };
    if (c_begin < n) {
        const int e0 = s_e[0], e1 = s_e[1], e2 = s_e[2];
        const int m1 = 2 * e1 + 1, m2 = 2 * e2 + 1, nimg = (2 * e0 + 1) * m1 * m2;
        float c[9];
#pragma unroll
        for (int k = 0; k < 9; k++) c[k] = (float)s_cell[k];
        // image of lane l among the images g0 .. g0 + 31: packed numbers, shift in single precision
        int im_packed = 0;
        float im_x = 0.f, im_y = 0.f, im_z = 0.f;
        auto set_image = [&](int g0) {
            const int im = g0 + lane, i0 = im / (m1 * m2), i1 = (im / m2) % m1, i2 = im % m2;
            const float f0 = (float)(i0 - e0), f1 = (float)(i1 - e1), f2 = (float)(i2 - e2);
            im_packed = i0 | (i1 << 10) | (i2 << 20);      // (at most 2 * 499 + 1 images per axis)
            im_x = f0 * c[0] + f1 * c[3] + f2 * c[6]; im_y = f0 * c[1] + f1 * c[4] + f2 * c[7]; im_z = f0 * c[2] + f1 * c[5] + f2 * c[8];
        };
        set_image(0);
        for (int t0 = 0; t0 < n; t0 += NBB_TILE) {
            const int tn = min(NBB_TILE, n - t0);
            __syncthreads();
            T org[3];
            cart(t0, org[0], org[1], org[2]);
#pragma unroll
            for (int k = 0; k < 3; k++) if (!(fabs((double)org[k]) < 1e15)) org[k] = T(0);      // an atom that has flown off
            float lo[3] = {3e38f, 3e38f, 3e38f}, hi[3] = {-3e38f, -3e38f, -3e38f}, n2max = 0.f;
            for (int s = threadIdx.x; s < ((tn + 63) & ~63) / 2; s += blockDim.x) {
                float q[2][4];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int j = (s & ~31) * 2 + (s & 31) + 32 * h;
                    q[h][0] = q[h][1] = q[h][2] = 0.f; q[h][3] = 3e38f;      // (padding never passes)
                    if (j < tn) {
                        T p[3];
                        cart(t0 + j, p[0], p[1], p[2]);
#pragma unroll
                        for (int k = 0; k < 3; k++) {
                            const float f = (float)(p[k] - org[k]);
                            s_pos[3 * j + k] = p[k]; q[h][k] = f;
                            lo[k] = fminf(lo[k], f); hi[k] = fmaxf(hi[k], f);
                        }
                        q[h][3] = q[h][0] * q[h][0] + q[h][1] * q[h][1] + q[h][2] * q[h][2];
                        n2max = fmaxf(n2max, q[h][3]);      // (an atom without a position is nobody's neighbour)
                    }
                }
                ulonglong2 *dst = s_cq + 2 * (s & ~31) + (s & 31);
                dst[0] = make_ulonglong2(pack2(q[0][0], q[1][0]), pack2(q[0][1], q[1][1]));
                dst[32] = make_ulonglong2(pack2(q[0][2], q[1][2]), pack2(q[0][3], q[1][3]));
            }
#pragma unroll
            for (int k = 0; k < 3; k++) {
#pragma unroll
                for (int o = 16; o >= 1; o >>= 1) {
                    lo[k] = fminf(lo[k], __shfl_xor_sync(FULL_MASK, lo[k], o));
                    hi[k] = fmaxf(hi[k], __shfl_xor_sync(FULL_MASK, hi[k], o));
                }
                if (lane == 0) { s_box[warp][k] = lo[k]; s_box[warp][3 + k] = hi[k]; }
            }
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) n2max = fmaxf(n2max, __shfl_xor_sync(FULL_MASK, n2max, o));
            if (lane == 0) s_box[warp][6] = n2max;
            __syncthreads();
            float reach = 0.f;
#pragma unroll
            for (int k = 0; k < 3; k++) {
                for (int w = 0; w < NBB_WARPS; w++) { lo[k] = fminf(lo[k], s_box[w][k]); hi[k] = fmaxf(hi[k], s_box[w][3 + k]); }
                reach += fmaxf(fabsf(lo[k]), fabsf(hi[k])) + fabsf((float)org[k]) + e0 * fabsf(c[k]) + e1 * fabsf(c[3 + k]) + e2 * fabsf(c[6 + k]);
            }
            for (int w = 0; w < NBB_WARPS; w++) n2max = fmaxf(n2max, s_box[w][6]);
#pragma unroll 1
            for (int q = 0; q < NBB_CPW; q++) {
                const int i = c_begin + warp * NBB_CPW + q;
                if (i >= n) continue;
                T cx, cy, cz;
                cart(i, cx, cy, cz);
                const float fx = (float)(cx - org[0]), fy = (float)(cy - org[1]), fz = (float)(cz - org[2]);
                // d^2 near the cutoff from single-precision coordinates no larger than `reach`: off by less than 64 eps reach rc
                const float rmax = reach + fabsf((float)cx) + fabsf((float)cy) + fabsf((float)cz);
                const float limit = ((float)P.rc2 + 64.f * 6e-8f * rmax * (float)P.rcut) * 1.000002f;
                int *frow = staged ? rowi : bfirstneigh + ((size_t)b * P.npad + i) * P.umax;
                T *rrow = staged ? rowp : brcs + ((size_t)b * P.npad + i) * P.umax * 3;
                int count = cnt[q], queued = 0;
                // exact predicate of the first `m` queued triples
                auto drain = [&](int m) {
                    bool hit = false;
                    int j = 0;
                    T d0 = 0, d1 = 0, d2 = 0;
                    if (lane < m) {
                        j = s_queue[warp][lane];
                        const int img = s_img[warp][lane];
                        const T f0 = T((img & 1023) - e0), f1 = T(((img >> 10) & 1023) - e1), f2 = T((img >> 20) - e2);
                        // this image's shift, applied in the reference's order ((r + a0 n0) + a1 n1) + a2 n2
                        const T ix = add_rn(add_rn(add_rn(s_pos[3 * j], mul_rn(s_cell[0], f0)), mul_rn(s_cell[3], f1)), mul_rn(s_cell[6], f2));
                        const T iy = add_rn(add_rn(add_rn(s_pos[3 * j + 1], mul_rn(s_cell[1], f0)), mul_rn(s_cell[4], f1)), mul_rn(s_cell[7], f2));
                        const T iz = add_rn(add_rn(add_rn(s_pos[3 * j + 2], mul_rn(s_cell[2], f0)), mul_rn(s_cell[5], f1)), mul_rn(s_cell[8], f2));
                        d0 = sub_rn(ix, cx); d1 = sub_rn(iy, cy); d2 = sub_rn(iz, cz);
                        bool undecided = true;
                        if (sizeof(T) == 4) {
                            const float sq = (float)d0 * (float)d0 + (float)d1 * (float)d1 + (float)d2 * (float)d2;
                            hit = sq < P.rc2_lo && sq > P.eps_hi;
                            undecided = !hit && !(sq > P.rc2_hi || sq < P.eps_lo);
                        }
                        if (undecided) {
                            const double dd = add_rn(add_rn(mul_rn((double)d0, (double)d0), mul_rn((double)d1, (double)d1)),
                                                     mul_rn((double)d2, (double)d2));
                            const double ddT = (double)(T)dd;
                            hit = (ddT < P.rc2) && (ddT > 1e-3);
                        }
                    }
                    const unsigned bal = __ballot_sync(FULL_MASK, hit);
                    if (hit) {
                        const int p = count + __popc(bal & lt_mask);
                        if (p < P.umax) {
                            frow[p] = t0 + j;
                            rrow[3 * p] = d0; rrow[3 * p + 1] = d1; rrow[3 * p + 2] = d2;
                        }
                    }
                    count += __popc(bal);
                };
                for (int g0 = 0; g0 < nimg; g0 += 32) {
                    // lanes = images: centre relative to the image, distance to the tile's bounding box
                    if (nimg > 32) set_image(g0);
                    const float qx = fx - im_x, qy = fy - im_y, qz = fz - im_z;
                    const float gx = fmaxf(fmaxf(lo[0] - qx, qx - hi[0]), 0.f), gy = fmaxf(fmaxf(lo[1] - qy, qy - hi[1]), 0.f),
                                gz = fmaxf(fmaxf(lo[2] - qz, qz - hi[2]), 0.f);
                    unsigned near = __ballot_sync(FULL_MASK, g0 + lane < nimg && gx * gx + gy * gy + gz * gz < limit);
                    while (near) {
                        const int l = __ffs(near) - 1;
                        near &= near - 1;
                        const float px = __shfl_sync(FULL_MASK, qx, l), py = __shfl_sync(FULL_MASK, qy, l), pz = __shfl_sync(FULL_MASK, qz, l);
                        const int packed = __shfl_sync(FULL_MASK, im_packed, l);
                        const float p2 = px * px + py * py + pz * pz, size = n2max + p2;
                        unsigned mine = 0;      // bit k: atom 32 k + lane of the tile survives
                        if (size < 1e30f) {
                            // rounding of |q_j|^2 - 2 q_i q_j + |q_i|^2: less than 1e-6 of the squares
                            const float lim = fminf(limit + 2e-6f * size - p2, 1e38f);      // (below the padding)
                            const unsigned long long mx = pack2(-2.f * px, -2.f * px), my = pack2(-2.f * py, -2.f * py), mz = pack2(-2.f * pz, -2.f * pz);
                            const ulonglong2 *cl = s_cq + lane;
#pragma unroll 2
                            for (int k = 0; 32 * k < tn; k += 2, cl += 64) {
                                const ulonglong2 a2 = cl[0], b2 = cl[32];
                                float v0, v1;
                                unpack2(fma2(mx, a2.x, fma2(my, a2.y, fma2(mz, b2.x, b2.y))), v0, v1);
                                if (v0 < lim) mine |= 1u << k;
                                if (v1 < lim) mine |= 2u << k;
                            }
                        } else {                // coordinates whose squares leave the single-precision range, or none: no pre-test
                            for (int k = 0; 32 * k + lane < tn; k++) mine |= 1u << k;
                        }
                        for (unsigned any = __reduce_or_sync(FULL_MASK, mine); any; any &= any - 1) {
                            const int k = __ffs(any) - 1;
                            const bool pass = (mine >> k) & 1u;
                            const unsigned bal = __ballot_sync(FULL_MASK, pass);
                            if (pass) {
                                const int p = queued + __popc(bal & lt_mask);
                                s_queue[warp][p] = 32 * k + lane;
                                s_img[warp][p] = packed;
                            }
                            queued += __popc(bal);
                            __syncwarp();
                            if (queued >= 32) {
                                drain(32);
                                queued -= 32;
                                const int kj = lane < queued ? s_queue[warp][32 + lane] : 0, ki = lane < queued ? s_img[warp][32 + lane] : 0;
                                __syncwarp();
                                if (lane < queued) { s_queue[warp][lane] = kj; s_img[warp][lane] = ki; }
                                __syncwarp();
                            }
                        }
                    }
                }
                if (queued) drain(queued);
                __syncwarp();
                cnt[q] = count;
                if (staged) {
                    pad_row(count, rowi, rowp);
                    __syncwarp();
                    int *fdst = bfirstneigh + ((size_t)b * P.npad + i) * P.umax;
                    T *rdst = brcs + ((size_t)b * P.npad + i) * P.umax * 3;
                    for (int k = lane; k < P.umax / 4; k += 32) reinterpret_cast<int4 *>(fdst)[k] = reinterpret_cast<const int4 *>(rowi)[k];
                    for (int k = lane; k < 3 * P.umax * (int)sizeof(T) / 16; k += 32)
                        reinterpret_cast<int4 *>(rdst)[k] = reinterpret_cast<const int4 *>(rowp)[k];
                    __syncwarp();
                }
            }
        }
    }
    // padding, counts, centre list; rows of padded atom slots (i >= n) are all padding
    int local_max = 0;
#pragma unroll
    for (int q = 0; q < NBB_CPW; q++) {
        const int i = c_begin + warp * NBB_CPW + q;
        if (i >= P.npad) continue;
        const int count = i < n ? cnt[q] : 0;
        if (i >= n || !staged) pad_row(count, bfirstneigh + ((size_t)b * P.npad + i) * P.umax, brcs + ((size_t)b * P.npad + i) * P.umax * 3);
        if (lane == 0) {
            bnumneigh[(size_t)b * P.npad + i] = min(count, P.umax);
            bilist[(size_t)b * P.npad + i] = i < n ? i : 0;
        }
        local_max = max(local_max, count);
    }
    if (lane == 0 && local_max > 0) {
        atomicMax(status, local_max);
        if (local_max > P.umax) atomicOr(status + 1, 1);
    }
}

template <typename T>
static int nblist_build_batch(int B, int npad, const int *d_binum, const T *d_cells, const T *d_coords, int is_cart, double rcut_in,
                              const int *pbc, int umax, int *d_bilist, int *d_bnumneigh, int *d_bfirstneigh, T *d_brcs, int *d_status,
                              cudaStream_t st)
{
    AI2B_REQUIRE(B >= 0 && npad >= 0 && umax >= 0 && rcut_in > 0, AI2B_ERR_INVALID, "ai2b_nblist_build_batch: bad size or cutoff");
    AI2B_REQUIRE(pbc && d_status, AI2B_ERR_INVALID, "ai2b_nblist_build_batch: NULL argument");
    AI2B_CUDA(cudaMemsetAsync(d_status, 0, 2 * sizeof(int), st));
    if (B == 0 || npad == 0) return AI2B_OK;
    AI2B_REQUIRE(d_binum && d_cells && d_coords && d_bilist && d_bnumneigh && d_bfirstneigh && d_brcs, AI2B_ERR_INVALID,
                 "ai2b_nblist_build_batch: NULL argument");
    AI2B_REQUIRE(B <= 65535, AI2B_ERR_UNSUPPORTED, "ai2b_nblist_build_batch: more than 65535 structures in one call");
    NbBatchParams<T> P;
    memset(&P, 0, sizeof(P));
    P.B = B; P.npad = npad; P.umax = umax; P.is_cart = is_cart ? 1 : 0;
    for (int k = 0; k < 3; k++) P.per[k] = pbc[k] ? 1 : 0;
    const T rcut = (T)rcut_in;                 // the float build casts rcut first (nblist_bind.cc:133)
    P.rcut = rcut;
    P.rc2 = (double)rcut * (double)rcut;
    if (sizeof(T) == 8) { volatile double r2 = (double)rcut * (double)rcut; P.rc2 = r2; }
    P.rc2_lo = (float)(P.rc2 * (1.0 - 2e-6)); P.rc2_hi = (float)(P.rc2 * (1.0 + 2e-6));
    P.eps_lo = (float)(1e-3 * (1.0 - 2e-6)); P.eps_hi = (float)(1e-3 * (1.0 + 2e-6));
    const size_t row_bytes = (size_t)umax * (sizeof(int) + 3 * sizeof(T));
    P.staged = umax % 4 == 0 && row_bytes <= 2560 && (reinterpret_cast<size_t>(d_bfirstneigh) | reinterpret_cast<size_t>(d_brcs)) % 16 == 0;
    dim3 grid((unsigned)((npad + NBB_CPB - 1) / NBB_CPB), (unsigned)B);
    nb_batch_kernel<T><<<grid, NBB_WARPS * 32, P.staged ? NBB_WARPS * row_bytes : 0, st>>>(P, d_binum, d_cells, d_coords, d_bilist, d_bnumneigh, d_bfirstneigh, d_brcs,
                                                        d_status);
    AI2B_CUDA(cudaGetLastError());
    return AI2B_OK;
}

// Builds that carry the set-up of the kernel that reads the rows (nep_setup.cuh), as blocks of the last binning launch.
// Rows in single precision from double positions; open_ext: lowest and highest fractional coordinates.
int nblist_build_rows32(int n, int ncentres, const double *h_cell, const double *d_coords, double rcut, const int *h_pbc, const double *open_ext, int umax,
                        int *d_numneigh, int *d_firstneigh, float *d_rcs, int *d_status, void *ws, size_t ws_bytes, cudaStream_t st, const NepSetup &side)
{
    return nblist_build<double, float>(n, ncentres, h_cell, d_coords, 1, rcut, h_pbc, umax, d_numneigh, d_firstneigh, d_rcs, d_status, ws, ws_bytes, st, 0,
                                       false, open_ext, side);
}
template <typename T>
int nblist_build_periodic(int n, const T *h_cell, const T *d_coords, double rcut, int umax, int *d_numneigh, int *d_firstneigh, T *d_rcs, int *d_status,
                          void *ws, size_t ws_bytes, cudaStream_t st, const NepSetup &side)
{
    const int pbc[3] = {1, 1, 1};
    return nblist_build<T>(n, n, h_cell, d_coords, 1, rcut, pbc, umax, d_numneigh, d_firstneigh, d_rcs, d_status, ws, ws_bytes, st, 0, false, nullptr, side);
}
template int nblist_build_periodic<double>(int, const double *, const double *, double, int, int *, int *, double *, int *, void *, size_t, cudaStream_t,
                                           const NepSetup &);
template int nblist_build_periodic<float>(int, const float *, const float *, double, int, int *, int *, float *, int *, void *, size_t, cudaStream_t,
                                          const NepSetup &);

}  // namespace ai2b

using namespace ai2b;

extern "C" int ai2b_nblist_build_batch_f64(int batch_size, int natoms_pad, const int *d_binum, const double *d_cells,
                                           const double *d_coords, int is_cart, double rcut, const int *h_pbc, int umax,
                                           int *d_bilist, int *d_bnumneigh, int *d_bfirstneigh, double *d_brcs, int *d_status,
                                           void *stream)
{
    return nblist_build_batch<double>(batch_size, natoms_pad, d_binum, d_cells, d_coords, is_cart, rcut, h_pbc, umax, d_bilist,
                                      d_bnumneigh, d_bfirstneigh, d_brcs, d_status, (cudaStream_t)stream);
}
extern "C" int ai2b_nblist_build_batch_f32(int batch_size, int natoms_pad, const int *d_binum, const float *d_cells,
                                           const float *d_coords, int is_cart, double rcut, const int *h_pbc, int umax,
                                           int *d_bilist, int *d_bnumneigh, int *d_bfirstneigh, float *d_brcs, int *d_status,
                                           void *stream)
{
    return nblist_build_batch<float>(batch_size, natoms_pad, d_binum, d_cells, d_coords, is_cart, rcut, h_pbc, umax, d_bilist,
                                     d_bnumneigh, d_bfirstneigh, d_brcs, d_status, (cudaStream_t)stream);
}

extern "C" size_t ai2b_nblist_workspace_bytes(int natoms, int is_f64)
{
    return is_f64 ? nb_layout<double>(natoms, nb_maxbins(natoms)).total : nb_layout<float>(natoms, nb_maxbins(natoms)).total;
}

extern "C" int ai2b_nblist_build_launches(int natoms, long long bins)
{
    if (natoms <= 0) return 0;
    return natoms <= BINB_MAX_ATOMS ? 2 : bins <= FILL_SCAN_BINS ? 4 : 5;
}

extern "C" int ai2b_nblist_build_f64(int natoms, const double *h_cell, const double *d_coords, int is_cart, double rcut,
                                     const int *h_pbc, int umax, int *d_numneigh, int *d_firstneigh, double *d_rcs,
                                     int *d_status, void *d_workspace, size_t workspace_bytes, void *stream)
{
    return nblist_build<double>(natoms, natoms, h_cell, d_coords, is_cart, rcut, h_pbc, umax, d_numneigh, d_firstneigh, d_rcs,
                                d_status, d_workspace, workspace_bytes, (cudaStream_t)stream);
}
extern "C" int ai2b_nblist_build_f32(int natoms, const float *h_cell, const float *d_coords, int is_cart, double rcut,
                                     const int *h_pbc, int umax, int *d_numneigh, int *d_firstneigh, float *d_rcs,
                                     int *d_status, void *d_workspace, size_t workspace_bytes, void *stream)
{
    return nblist_build<float>(natoms, natoms, h_cell, d_coords, is_cart, rcut, h_pbc, umax, d_numneigh, d_firstneigh, d_rcs,
                               d_status, d_workspace, workspace_bytes, (cudaStream_t)stream);
}

template <typename T>
static int nblist_sort(int n, int umax, const int *numneigh, int *firstneigh, T *rcs, cudaStream_t st)
{
    AI2B_REQUIRE(n >= 0 && umax >= 0, AI2B_ERR_INVALID, "ai2b_nblist_sort_rows: negative size");
    if (n == 0 || umax == 0) return AI2B_OK;
    AI2B_REQUIRE(numneigh && firstneigh && rcs, AI2B_ERR_INVALID, "ai2b_nblist_sort_rows: NULL argument");
    const int wpb = 4;
    const size_t smem = (size_t)wpb * umax * (4 * sizeof(T) + sizeof(int));
    AI2B_REQUIRE(smem <= 200 * 1024, AI2B_ERR_UNSUPPORTED, "umax %d too large to sort rows in shared memory", umax);
    auto kern = nb_sort_rows_kernel<T>;
    if (smem > 48 * 1024) AI2B_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    long blocks = ((long)n + wpb - 1) / wpb;
    if (blocks > 148 * 8) blocks = 148 * 8;
    kern<<<(unsigned)blocks, wpb * 32, smem, st>>>(n, umax, numneigh, firstneigh, rcs);
    AI2B_CUDA(cudaGetLastError());
    return AI2B_OK;
}
extern "C" int ai2b_nblist_sort_rows_f64(int natoms, int umax, const int *d_numneigh, int *d_firstneigh, double *d_rcs, void *stream)
{
    return nblist_sort<double>(natoms, umax, d_numneigh, d_firstneigh, d_rcs, (cudaStream_t)stream);
}
extern "C" int ai2b_nblist_sort_rows_f32(int natoms, int umax, const int *d_numneigh, int *d_firstneigh, float *d_rcs, void *stream)
{
    return nblist_sort<float>(natoms, umax, d_numneigh, d_firstneigh, d_rcs, (cudaStream_t)stream);
}

// Same build for a local domain with ghost atoms: rows are produced for the first `ncentres`
// atoms only, all `natoms` atoms (centres + ghosts) are candidates. Indices in d_firstneigh are
// positions in d_coords, so ghosts appear as indices >= ncentres (the LAMMPS convention the
// evaluation ops expect with nghost = natoms - ncentres).
extern "C" int ai2b_nblist_build_ghost_f64(int natoms, int ncentres, const double *h_cell, const double *d_coords, int is_cart,
                                           double rcut, const int *h_pbc, int umax, int *d_numneigh, int *d_firstneigh,
                                           double *d_rcs, int *d_status, void *d_workspace, size_t workspace_bytes, void *stream)
{
    return nblist_build<double>(natoms, ncentres, h_cell, d_coords, is_cart, rcut, h_pbc, umax, d_numneigh, d_firstneigh, d_rcs,
                                d_status, d_workspace, workspace_bytes, (cudaStream_t)stream);
}
extern "C" int ai2b_nblist_build_ghost_f32(int natoms, int ncentres, const float *h_cell, const float *d_coords, int is_cart,
                                           double rcut, const int *h_pbc, int umax, int *d_numneigh, int *d_firstneigh,
                                           float *d_rcs, int *d_status, void *d_workspace, size_t workspace_bytes, void *stream)
{
    return nblist_build<float>(natoms, ncentres, h_cell, d_coords, is_cart, rcut, h_pbc, umax, d_numneigh, d_firstneigh, d_rcs,
                               d_status, d_workspace, workspace_bytes, (cudaStream_t)stream);
}
// Rows for the centre range [centre_begin, centre_end) only (row 0 of the outputs = centre_begin), all natoms
// atoms as candidates; with reuse_bins != 0 the binning left in the workspace by an earlier call on the same
// atoms is used again (a domain evaluated in several passes bins once per set of candidates).
extern "C" int ai2b_nblist_build_range_f64(int natoms, int centre_begin, int centre_end, const double *h_cell, const double *d_coords,
                                           int is_cart, double rcut, const int *h_pbc, const double *h_open_extent, int umax,
                                           int reuse_bins, int *d_numneigh,
                                           int *d_firstneigh, double *d_rcs, int *d_status, void *d_workspace, size_t workspace_bytes,
                                           void *stream)
{
    return nblist_build<double>(natoms, centre_end, h_cell, d_coords, is_cart, rcut, h_pbc, umax, d_numneigh, d_firstneigh, d_rcs,
                                d_status, d_workspace, workspace_bytes, (cudaStream_t)stream, centre_begin, reuse_bins != 0, h_open_extent);
}
extern "C" int ai2b_nblist_build_range_f32(int natoms, int centre_begin, int centre_end, const float *h_cell, const float *d_coords,
                                           int is_cart, double rcut, const int *h_pbc, const double *h_open_extent, int umax,
                                           int reuse_bins, int *d_numneigh,
                                           int *d_firstneigh, float *d_rcs, int *d_status, void *d_workspace, size_t workspace_bytes,
                                           void *stream)
{
    return nblist_build<float>(natoms, centre_end, h_cell, d_coords, is_cart, rcut, h_pbc, umax, d_numneigh, d_firstneigh, d_rcs,
                               d_status, d_workspace, workspace_bytes, (cudaStream_t)stream, centre_begin, reuse_bins != 0, h_open_extent);
}
// Double-precision positions, single-precision rows: r_j - r_i is formed in double and rounded once, as
// PairAI2Pot::construct_mlff_input does on the host (interface/lammps/AI2POT/pair_ai2pot.cpp:232-235).
extern "C" int ai2b_nblist_build_ghost_f64_rows32(int natoms, int ncentres, const double *h_cell, const double *d_coords, int is_cart,
                                                  double rcut, const int *h_pbc, int umax, int *d_numneigh, int *d_firstneigh,
                                                  float *d_rcs, int *d_status, void *d_workspace, size_t workspace_bytes,
                                                  void *stream)
{
    return nblist_build<double, float>(natoms, ncentres, h_cell, d_coords, is_cart, rcut, h_pbc, umax, d_numneigh, d_firstneigh, d_rcs,
                                       d_status, d_workspace, workspace_bytes, (cudaStream_t)stream);
}
