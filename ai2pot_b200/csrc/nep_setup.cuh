// Set-up of the specialised NEP kernel (nep_fast.cuh): the model as the kernel reads it, the structures' atom offsets, zeroed
// outputs. It needs nothing of the neighbour rows. A call that builds rows and evaluates (evaluate.cu, md_session.cu) therefore hands
// it to the build, which takes it along as further blocks of its last binning launch: there it is over before the atoms are in their
// bins (the bin set-up in front is shorter than it: 13,824 atoms 54.9 us with the table there, 51.7 here). A launch of its own between
// rows and evaluation costs its two boundaries (13,824 atoms 54.9 us; 1,157 atoms 25.0 -> 20.6).
#pragma once
#include "common.cuh"

namespace ai2b {

constexpr int NEP_NLM = 24;

// padded descriptor count: rows of the network's first layer are 16-byte aligned and an odd
// number of 16-byte chunks long (conflict-free when eight lanes read eight rows)
template <int NMAX>
struct NepFastDims {
    static constexpr int ND = 5 * NMAX;                                   // >= n_r + n_a * l_max
    static constexpr int NDP = ((ND / 4) & 1) ? ND : ND + 4;
    static constexpr int CS = 8;                                          // Chebyshev rows
    static constexpr int TROW = 2 * NMAX * CS + 4;                        // one type pair; rows of different pairs start in different banks
    static constexpr int RS = NMAX + NEP_NLM + (NMAX == 8 ? 4 : 0);       // staging row: g[NMAX] | B_lm[24], conflict-free 16-byte stores
    static constexpr int ESR = NMAX * NEP_NLM + 4;                        // adjoints of an atom's sums, [mu][24]
};
__host__ __device__ inline int nep_r4(int n) { return (n + 3) & ~3; }
__host__ __device__ inline int nep_r32(int n) { return (n + 31) & ~31; }   // neurons per type, padded

// The model as the kernel reads it (elements of T): Chebyshev rows [ti][tj][k][radial | angular], then (unless descriptors
// only) first-layer rows [type][neuron][NDP], biases, second-layer weights, 1 / q_scaler
template <int NMAX>
struct NepTab {
    int w0, b0, w1, iqs, total;
    __host__ __device__ NepTab(int ntypes, int nneu, bool net)
    {
        using D = NepFastDims<NMAX>;
        const int nrow = ntypes * nep_r32(nneu);
        w0 = nep_r4(ntypes * ntypes * D::TROW);
        b0 = w0 + (net ? nrow * D::NDP : 0);
        w1 = b0 + (net ? nrow : 0);
        iqs = w1 + (net ? nrow : 0);
        total = iqs + (net ? nep_r4(D::NDP) : 0);
    }
};

// What the set-up works on; plain pointers, so that the neighbour build can carry it without knowing the model's type
struct NepSetup {
    int blocks = 0;                    // of NEP_SETUP_THREADS threads or more; 0: nothing to do
    int tab_blocks, wide, is_f64;      // wide: NMAX = 8 instead of 4
    int ntypes, n_r, n_a, cs, nneu, nd, net, B;
    const int *binum;
    int *prefix;
    const void *coeffs, *w0, *b0, *w1, *qs;
    void *tab, *z[3];                  // outputs to be zeroed
    size_t nz[3];
};
constexpr int NEP_SETUP_THREADS = 256;

// Row 0 of a function holds 2 c_0 + sum_k c_k (the constant part of sum c_k (T_k + 1)); row k holds s_k c_k with the signs
// s = + + - - + + - -, which turn the recurrences T_k+1 = 2 x T_k - T_k-1 and T'_k+1 = 2 T_k + 2 x T'_k - T'_k-1 into sums.
template <typename T, int NMAX>
__device__ __forceinline__ void nep_setup_block(const NepSetup &S, int block)
{
    using D = NepFastDims<NMAX>;
    if (block < S.tab_blocks) {
        const NepTab<NMAX> L(S.ntypes, S.nneu, S.net != 0);
        const int NP = nep_r32(S.nneu), nfun = S.n_r + S.n_a;
        if (block == 0 && S.B > 1 && threadIdx.x < 32) {      // exclusive sum of the structures' sizes
            int carry = 0;
            for (int b0 = 0; b0 < S.B; b0 += 32) {
                const int b = b0 + threadIdx.x;
                int inc = b < S.B ? S.binum[b] : 0;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(FULL_MASK, inc, o); if ((int)threadIdx.x >= o) inc += v; }
                if (b < S.B) S.prefix[b + 1] = carry + inc;
                carry += __shfl_sync(FULL_MASK, inc, 31);
            }
            if (threadIdx.x == 0) S.prefix[0] = 0;
        }
        const T *coeffs = static_cast<const T *>(S.coeffs), *w0 = static_cast<const T *>(S.w0), *b0 = static_cast<const T *>(S.b0),
                *w1 = static_cast<const T *>(S.w1), *qs = static_cast<const T *>(S.qs);
        T *tab = static_cast<T *>(S.tab);
        for (int i = block * blockDim.x + threadIdx.x; i < L.total; i += S.tab_blocks * blockDim.x) {
            T v = T(0);
            if (i < L.w0) {
                const int pair = i / D::TROW, o = i % D::TROW, k = o / (2 * NMAX), f = o % (2 * NMAX);
                const int row = f < NMAX ? (f < S.n_r ? f : -1) : (f - NMAX < S.n_a ? S.n_r + f - NMAX : -1);
                if (pair < S.ntypes * S.ntypes && k < S.cs && row >= 0) {
                    const T *c = coeffs + ((size_t)pair * nfun + row) * S.cs;
                    if (k == 0) {
                        v = T(2) * c[0];
                        for (int q = 1; q < S.cs; q++) v += c[q];
                    } else {
                        v = (k & 2) ? -c[k] : c[k];
                    }
                }
            } else if (i < L.b0) {
                const int row = (i - L.w0) / D::NDP, k = (i - L.w0) % D::NDP, t = row / NP, p = row % NP;
                if (k < S.nd && p < S.nneu) v = w0[((size_t)t * S.nneu + p) * S.nd + k];
            } else if (i < L.iqs) {
                const int row = (i - L.b0) % (S.ntypes * NP), t = row / NP, p = row % NP;
                if (p < S.nneu) v = (i < L.w1 ? b0 : w1)[t * S.nneu + p];
            } else if (i - L.iqs < S.nd) {
                v = T(1) / qs[i - L.iqs];
            }
            tab[i] = v;
        }
        return;
    }
    const size_t i0 = (size_t)(block - S.tab_blocks) * blockDim.x + threadIdx.x, step = (size_t)(S.blocks - S.tab_blocks) * blockDim.x;
#pragma unroll
    for (int a = 0; a < 3; a++)
        for (size_t i = i0; i < S.nz[a]; i += step) static_cast<T *>(S.z[a])[i] = T(0);
}
// block `block` (all of its threads) of a launch that carries the set-up; after the launch's chain_wait()
__device__ __forceinline__ void nep_setup_any(const NepSetup &S, int block)
{
    if (S.is_f64) {
        if (S.wide) nep_setup_block<double, 8>(S, block);
        else nep_setup_block<double, 4>(S, block);
    } else {
        if (S.wide) nep_setup_block<float, 8>(S, block);
        else nep_setup_block<float, 4>(S, block);
    }
}

// Fills in the set-up that a call of ai2b_nep_efv_* with these arguments would launch. False: that call takes another route (the
// general kernel) or has nothing to evaluate, and does its set-up itself.
template <typename T>
bool nep_plan_setup(T *etot, T *force, T *virial, int cs, int n_r, int n_a, int l_max, int nneu, const T *coeffs, const T *w0, const T *b0,
                    const T *w1, int npad, const int *binum, int ntypes, int umax, int nghost, const T *qs, void *ws, size_t ws_bytes, NepSetup *out);
// ai2b_nep_efv_* for one structure whose set-up has been done by an earlier launch of the chain
template <typename T>
int nep_efv_prepared(T *etot, T *force, T *virial, int cs, int n_r, int n_a, int l_max, int nneu, const T *coeffs, const T *w0, const T *b0,
                     const T *w1, const T *bias, int npad, const int *binum, const int *bilist, const int *numneigh, const int *firstneigh,
                     const T *rcs, const int *types, int ntypes, int umax, int nghost, T rc_r, T rc_a, const T *qs, void *ws, size_t ws_bytes,
                     cudaStream_t st);

}  // namespace ai2b
