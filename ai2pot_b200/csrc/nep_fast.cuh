// NEP energy / force / virial kernel specialised for models with at most NMAX radial and NMAX
// angular functions (NMAX = 4 covers the reference's defaults, ai2pot/models/nep/nep.py:36-40).
// Included by nep_kernels.cu after the shared helpers (NepArgs, NEP_FOR_EACH_LM).
//
// Same math as the general kernel (nep.h:320-529). A warp evaluates 32 / G atoms, G lanes each, and all of its lanes run the
// same trip counts: with loops per group (8 lanes, own neighbour count) the four groups of a warp drift apart and every phase
// is issued up to four times. What bounds it is instruction issue, so every phase is written for few instructions:
//   * set-up (nep_setup.cuh): lays the model out once per call (padded rows, signs and constants folded in) and zeroes the
//     outputs, in a launch of its own or as blocks of a launch of the neighbour build; a block takes the table with a handful
//     of 16-byte copies;
//   * radial pass, lanes = neighbours of the group's atom: Chebyshev sums of all functions and their derivatives in packed
//     pairs, g'_n(r_j) / r_j are kept per neighbour in shared memory;
//   * angular pass, lanes = angular neighbours of all atoms of the warp, back to back: only a fifth of the neighbours are
//     inside the angular cutoff (6.5 of 29, or 2.2 of 17), so lanes that belong to one atom would mostly idle. The harmonics
//     of a neighbour go through shared memory to the lanes that own its atom's sums S[mu][lm];
//   * network: lanes = neurons; up to NMAX = 4 a neuron's row is read once, for its input and for the descriptors' adjoints, with
//     the angular sums parked in shared memory (1,048,576 atoms of a crystal: 950 -> 827 us; with a second walk over the rows,
//     lanes = descriptors, the shared-memory pipe was 82 % busy; without parking the spills made it 1,058 us);
//   * angular forces, lanes as in the angular pass (the neighbour's functions are still in registers): the adjoints are
//     first contracted over the radial functions, sum_mu g_mu e_{mu,lm} and sum_mu g'_mu e_{mu,lm}, which leaves one
//     polynomial and one gradient per neighbour instead of NMAX. The radial force of the neighbour joins here, so every
//     neighbour receives one set of atomics;
//   * radial forces of the other neighbours from the cached derivatives.
// G: 32 lanes per atom when there are few atoms (the chip is filled by atoms x G threads), 8 for many.
// Measured (fp32, whole call, 29 / 6.5 neighbours): see launch_nep_fast.
#pragma once

namespace ai2b {

template <typename T, int N>
__device__ __forceinline__ void load_vec(const T *__restrict__ p, T (&v)[N])
{
    constexpr int PER = 16 / (int)sizeof(T);
    static_assert(N % PER == 0, "row length must be a multiple of 16 bytes");
    if constexpr (sizeof(T) == 4) {
#pragma unroll
        for (int i = 0; i < N / 4; i++) {
            const float4 t = reinterpret_cast<const float4 *>(p)[i];
            v[4 * i] = t.x; v[4 * i + 1] = t.y; v[4 * i + 2] = t.z; v[4 * i + 3] = t.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < N / 2; i++) {
            const double2 t = reinterpret_cast<const double2 *>(p)[i];
            v[2 * i] = t.x; v[2 * i + 1] = t.y;
        }
    }
}
template <typename T, int N>
__device__ __forceinline__ void store_vec(T *__restrict__ p, const T (&v)[N])
{
    if constexpr (sizeof(T) == 4) {
#pragma unroll
        for (int i = 0; i < N / 4; i++)
            reinterpret_cast<float4 *>(p)[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    } else {
#pragma unroll
        for (int i = 0; i < N / 2; i++) reinterpret_cast<double2 *>(p)[i] = make_double2(v[2 * i], v[2 * i + 1]);
    }
}

// Two values that are worked on together: one packed register pair and one instruction in single precision.
template <typename T> struct Pk { T a, b; };
template <> struct Pk<float> { unsigned long long v; };
__device__ __forceinline__ Pk<float> pk(float a, float b) { Pk<float> r; asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ Pk<double> pk(double a, double b) { return {a, b}; }
__device__ __forceinline__ float pk_lo(Pk<float> p) { float a, b; asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p.v)); return a; }
__device__ __forceinline__ float pk_hi(Pk<float> p) { float a, b; asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p.v)); return b; }
__device__ __forceinline__ double pk_lo(Pk<double> p) { return p.a; }
__device__ __forceinline__ double pk_hi(Pk<double> p) { return p.b; }
__device__ __forceinline__ Pk<float> pk_fma(Pk<float> a, Pk<float> b, Pk<float> c)
{
    Pk<float> r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ Pk<double> pk_fma(Pk<double> a, Pk<double> b, Pk<double> c) { return {fma(a.a, b.a, c.a), fma(a.b, b.b, c.b)}; }
__device__ __forceinline__ Pk<float> pk_mul(Pk<float> a, Pk<float> b)
{
    Pk<float> r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ Pk<double> pk_mul(Pk<double> a, Pk<double> b) { return {a.a * b.a, a.b * b.b}; }
template <int N>
__device__ __forceinline__ void load_pk(const float *p, Pk<float> (&v)[N])
{
    static_assert(N % 2 == 0, "16-byte loads");
#pragma unroll
    for (int i = 0; i < N / 2; i++) {
        const ulonglong2 t = reinterpret_cast<const ulonglong2 *>(p)[i];
        v[2 * i].v = t.x; v[2 * i + 1].v = t.y;
    }
}
template <int N>
__device__ __forceinline__ void load_pk(const double *p, Pk<double> (&v)[N])
{
#pragma unroll
    for (int i = 0; i < N; i++) {
        const double2 t = reinterpret_cast<const double2 *>(p)[i];
        v[i].a = t.x; v[i].b = t.y;
    }
}

// 1 / sqrt(v) with a Newton step behind the hardware's estimate in single precision
__device__ __forceinline__ float inv_sqrt(float v) { const float y = rsqrtf(v); return y * fmaf(-0.5f * v * y, y, 1.5f); }
__device__ __forceinline__ double inv_sqrt(double v) { return rsqrt(v); }

// Radial functions g_n (basis.h:300-333,519-530) of one pair, and their derivatives, in pairs of functions. tc: the pair's
// first Chebyshev row (of the radial or the angular functions); t = r / rc.
template <typename T, int NMAX, bool DERIV>
__device__ __forceinline__ void nep_functions(const T *tc, T t, T inv_rc, Pk<T> (&g)[NMAX / 2], Pk<T> (&dg)[NMAX / 2])
{
    constexpr int NP = NMAX / 2, ROW = 2 * NMAX;
    const T s = t - T(1), x = T(2) * s * s - T(1), x2 = T(2) * x;
    const Pk<T> plus = pk(x2, x2), minus = pk(-x2, -x2), p2 = pk(T(2), T(2)), m2 = pk(T(-2), T(-2));
    Pk<T> u0 = pk(T(1), T(1)), u1 = pk(x, x), v0 = pk(T(0), T(0)), v1 = pk(T(1), T(1));
    Pk<T> S[NP], dS[NP], c[NP];
    load_pk<NP>(tc, S);
    load_pk<NP>(tc + ROW, c);
#pragma unroll
    for (int n = 0; n < NP; n++) { S[n] = pk_fma(c[n], u1, S[n]); if (DERIV) dS[n] = c[n]; }
#pragma unroll
    for (int k = 2; k < NepFastDims<NMAX>::CS; k++) {
        const Pk<T> f = (k & 1) ? plus : minus;
        const Pk<T> u2 = pk_fma(f, u1, u0);
        load_pk<NP>(tc + k * ROW, c);
        if (DERIV) {
            const Pk<T> v2 = pk_fma(f, v1, pk_fma((k & 1) ? p2 : m2, u1, v0));
#pragma unroll
            for (int n = 0; n < NP; n++) dS[n] = pk_fma(c[n], v2, dS[n]);
            v0 = v1; v1 = v2;
        }
#pragma unroll
        for (int n = 0; n < NP; n++) S[n] = pk_fma(c[n], u2, S[n]);
        u0 = u1; u1 = u2;
    }
    T sn, cs;
    gsincospi(T(0.5) * t, &sn, &cs);      // (polynomials of t^2 in its place saved 0.6 % of a call at 13,824 atoms, with errors up to 1.8e-7)
    const T fh = T(0.5) * cs * cs;      // half the cutoff function cos^2(pi t / 2)
    const Pk<T> f2 = pk(fh, fh);
#pragma unroll
    for (int n = 0; n < NP; n++) g[n] = pk_mul(f2, S[n]);
    if (DERIV) {
        const T df = T(-0.5 * 3.14159265358979323846) * inv_rc * cs * sn, fx = fh * (T(4) * inv_rc) * s;
        const Pk<T> d2 = pk(df, df), x3 = pk(fx, fx);
#pragma unroll
        for (int n = 0; n < NP; n++) dg[n] = pk_fma(x3, dS[n], pk_mul(d2, S[n]));
    }
}

// N per-lane values (a power of two) summed over the G lanes of every group: lane `sub` of a group returns the total of value
// sub / (G / N) (N <= G). All lanes of the warp take part.
template <typename T, int N, int G>
__device__ __forceinline__ T group_xreduce(T (&v)[N], int lane)
{
    static_assert(N <= G, "one value per lane at most");
    int o = G / 2;
#pragma unroll
    for (int h = N / 2; h >= 1; h >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < h; i++) {
            const T send = up ? v[i] : v[i + h], keep = up ? v[i + h] : v[i];
            v[i] = keep + __shfl_xor_sync(FULL_MASK, send, o);
        }
    }
    T r = v[0];
    for (; o >= 1; o >>= 1) r += __shfl_xor_sync(FULL_MASK, r, o);
    return r;
}

// f[0..2] += (x, y, z): in single precision one 8-byte and one 4-byte atomic (which of the two comes first follows from the
// address: rows of three floats start on 8-byte boundaries or 4 bytes past one)
__device__ __forceinline__ void add3(float *f, float x, float y, float z)
{
    const bool even = (reinterpret_cast<size_t>(f) & 4) == 0;
    float *p2 = even ? f : f + 1, *p1 = even ? f + 2 : f;
    const float a = even ? x : y, b = even ? y : z, c = even ? z : x;
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p2), "f"(a), "f"(b) : "memory");
    atomicAdd(p1, c);
}
__device__ __forceinline__ void add3(double *f, double x, double y, double z) { atomicAdd(f, x); atomicAdd(f + 1, y); atomicAdd(f + 2, z); }

// shared-memory elements (of T) per warp behind the model table; the neighbour lists follow (two bytes per neighbour)
template <int NMAX>
__host__ __device__ inline int nep_fast_warp_elems(int lanes, int nneu, int umax, bool net)
{
    using D = NepFastDims<NMAX>;
    const int AW = 32 / lanes;
    const int stage = 32 * D::RS, es = AW * D::ESR;                 // staging rows, later the adjoints of the sums
    return (stage > es ? stage : es) + AW * 2 * D::NDP +            // descriptors, their adjoints
           (net ? AW * (nep_r32(nneu) + 4) + 96 + AW * umax * NMAX : 0);   // neurons, angular forces, cached derivatives
    // (NMAX = 4 does not write the neurons' part. Without it 13,824 atoms take 56.0 instead of 56.6 us, 1,048,576 atoms 1,600
    // instead of 1,592, and models of 12 species a slower form: it stays.)
}

template <typename T, int G, int MODE, int NMAX, int MINB>
__global__ void __launch_bounds__(NEP_WARPS * 32, MINB) nep_fast_kernel(const NepArgs<T> A, const T *__restrict__ tab, int early_release)
{
    using D = NepFastDims<NMAX>;
    constexpr int AW = 32 / G, NP2 = NMAX / 2, NDP = D::NDP, RS = D::RS, ESR = D::ESR, ROW = 2 * NMAX;
    constexpr int LM = (NEP_NLM + G - 1) / G;            // sums per lane and function
    constexpr int NPL = 32 / G;                          // neurons per lane and round
    constexpr bool PARK = NMAX == 4 && sizeof(T) == 4 && G <= 16;      // the sums wait in shared memory while the network has the registers
    constexpr bool ONEPASS = NMAX == 4;                  // a row of the first layer, the inputs and the adjoints fit in registers
    constexpr bool NET = MODE != NEP_DESC;
    extern __shared__ __align__(16) unsigned char nep_smem[];
    __shared__ T blk_acc[10];
    __shared__ int blk_b;
    __shared__ T fac_s[NEP_NLM];     // (2 - delta_m0) * 2 * C_lm
    __shared__ T c3w_s[NEP_NLM];     // (2 - delta_m0) * C_lm
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sub = lane % G, grp = lane / G;
    if (early_release) chain_release();
    const NepTab<NMAX> L(A.ntypes, A.nneu, NET);
    T *tab_s = reinterpret_cast<T *>(nep_smem);
    const int per_warp = nep_fast_warp_elems<NMAX>(G, A.nneu, A.umax, NET), NP = nep_r32(A.nneu), NPP = NP + 4;
    T *stage = tab_s + L.total + (size_t)warp * per_warp;
    T *es = stage;                                       // [AW][ESR]
    T *q = stage + (32 * RS > AW * ESR ? 32 * RS : AW * ESR) + grp * NDP;
    T *Eq0 = q - grp * NDP + AW * NDP, *Eq = Eq0 + grp * NDP;
    T *act0 = Eq0 + AW * NDP, *act = act0 + (NET ? grp * NPP : 0);
    T *fbuf = act0 + (NET ? AW * NPP : 0);               // [32][3]
    T *dcache0 = fbuf + 96, *dcache = dcache0 + (size_t)grp * A.umax * NMAX;      // [umax][NMAX]: g'_n / r of every neighbour
    unsigned short *alist0 = reinterpret_cast<unsigned short *>(tab_s + L.total + (size_t)NEP_WARPS * per_warp) + (size_t)warp * AW * A.umax;
    unsigned short *alist = alist0 + grp * A.umax;
    const int nlm = A.l_max * A.l_max + 2 * A.l_max;
    const int nq_a = A.l_max > 0 ? A.n_a * A.l_max : 0;
    const T inv_rcr = T(1) / A.rc_r, inv_rca = T(1) / A.rc_a;

    if (threadIdx.x < NEP_NLM) {
        const int lm = threadIdx.x;
        const bool m0 = lm == 0 || lm == 3 || lm == 8 || lm == 15;
        c3w_s[lm] = (m0 ? T(1) : T(2)) * (T)c_C3B[lm];
        fac_s[lm] = (m0 ? T(1) : T(2)) * T(2) * (T)c_C3B[lm];
    }
    // descriptors and their adjoints are read as NDP-long vectors: the padding stays zero
    for (int i = lane; i < AW * 2 * NDP; i += 32) (q - grp * NDP)[i] = T(0);
    chain_wait();        // the table and the offsets come from an earlier launch of the chain (each of its kernels waits)
    for (int i = threadIdx.x; i < L.total * (int)sizeof(T) / 16; i += NEP_WARPS * 32)
        __pipeline_memcpy_async(reinterpret_cast<float4 *>(tab_s) + i, reinterpret_cast<const float4 *>(tab) + i, 16);
    __pipeline_commit();
    const int ntot = A.B == 1 ? A.binum[0] : A.prefix[A.B];
    const int nwarps = gridDim.x * NEP_WARPS;
    __pipeline_wait_prior(0);
    __syncthreads();

    // energy / virial of the atoms this warp has worked on, all of structure `bcur`
    T e_acc = T(0), vir[9];
#pragma unroll
    for (int k = 0; k < 9; k++) vir[k] = T(0);
    int bcur = -1;
    auto flush_to = [&](int b, T *e_dst, T *v_dst) {     // whole warp, one structure
        T r[16];
#pragma unroll
        for (int k = 0; k < 16; k++) r[k] = k == 0 ? e_acc : (MODE == NEP_EFV && k < 10) ? vir[k < 10 ? k - 1 : 0] : T(0);
        const T s = group_xreduce<T, 16, 32>(r, lane);
        const int k = lane >> 1;
        if ((lane & 1) == 0 && (k == 0 || (MODE == NEP_EFV && k < 10))) atomicAdd(k == 0 ? e_dst : v_dst + k - 1, s);
        e_acc = T(0);
#pragma unroll
        for (int k2 = 0; k2 < 9; k2++) vir[k2] = T(0);
    };

    for (int t0 = (blockIdx.x * NEP_WARPS + warp) * AW; t0 < ntot; t0 += nwarps * AW) {
        const int t = t0 + grp;
        const bool valid = t < ntot;
        int b = 0;
        if (valid && A.B > 1) {
            int lo = 0, hi = A.B;
            while (hi - lo > 1) { int mid = (lo + hi) >> 1; if (A.prefix[mid] <= t) lo = mid; else hi = mid; }
            b = lo;
        }
        const int slot = b * A.npad + (valid ? (A.B > 1 ? t - A.prefix[b] : t) : 0);
        const int ci = valid ? A.bilist[slot] : 0;
        const int nn = valid ? min(A.numneigh[slot], A.umax) : 0;
        const size_t tstride = A.npad + (MODE == NEP_DESC ? 0 : A.nghost);
        const int *types = A.types + (size_t)b * tstride;
        const int ti = valid ? types[ci] : 0;
        const int *fn = A.firstneigh + (size_t)slot * A.umax;
        const T *rc = A.rcs + (size_t)slot * A.umax * 3;
        const int nnmax = __reduce_max_sync(FULL_MASK, nn);
        // atoms of one structure accumulate energy and virial in registers; a warp across a boundary adds its own at once
        bool mixed = false;
        if (NET) {
            const int b0 = __shfl_sync(FULL_MASK, b, 0);
            mixed = A.B > 1 && !__all_sync(FULL_MASK, !valid || b == b0);
            if (mixed || b0 != bcur) {
                if (bcur >= 0) flush_to(bcur, A.etot + bcur, A.virial + 9 * bcur);
                bcur = mixed ? -1 : b0;
            }
        }

        // ---- 1. radial pass: q_n, cached g'_n / r, lists of the angular neighbours --------------------
        Pk<T> qa[NP2];
#pragma unroll
        for (int n = 0; n < NP2; n++) qa[n] = pk(T(0), T(0));
        int nang = 0;
        {
            T xn = 0, yn = 0, zn = 0;
            int njn = 0;
            if (sub < nn) { xn = rc[3 * sub]; yn = rc[3 * sub + 1]; zn = rc[3 * sub + 2]; njn = fn[sub]; }
            for (int j0 = 0; j0 < nnmax; j0 += G) {
                const int j = j0 + sub;
                bool on = j < nn;
                const T x = xn, y = yn, z = zn;
                const int tj = on ? types[njn] : 0;
                {   // the next chunk's positions and indices are requested before this chunk is worked on
                    const int jn = j + G;
                    xn = yn = zn = T(0);
                    if (jn < nn) { xn = rc[3 * jn]; yn = rc[3 * jn + 1]; zn = rc[3 * jn + 2]; njn = fn[jn]; }
                }
                const T r2 = x * x + y * y + z * z;
                on = on && r2 > T(0);
                const T rinv = inv_sqrt(on ? r2 : T(1)), r = r2 * rinv;
                const bool ang = on && r <= A.rc_a && A.l_max > 0;
                on = on && r <= A.rc_r;
                Pk<T> g[NP2], dg[NP2];
                nep_functions<T, NMAX, NET>(tab_s + (ti * A.ntypes + tj) * D::TROW, on ? r * inv_rcr : T(1), inv_rcr, g, dg);
                const T w = on ? T(1) : T(0);
                const Pk<T> w2 = pk(w, w);
#pragma unroll
                for (int n = 0; n < NP2; n++) qa[n] = pk_fma(w2, g[n], qa[n]);
                if (NET && j < A.umax) {
                    const T wr = on ? rinv : T(0);
                    T d[NMAX];
#pragma unroll
                    for (int n = 0; n < NP2; n++) { d[2 * n] = wr * pk_lo(dg[n]); d[2 * n + 1] = wr * pk_hi(dg[n]); }
                    store_vec<T, NMAX>(dcache + (size_t)j * NMAX, d);
                }
                const unsigned bal = __ballot_sync(FULL_MASK, ang) >> (G == 32 ? 0 : grp * G) & (G == 32 ? FULL_MASK : (1u << (G & 31)) - 1u);
                // list entry: neighbour slot (10 bits) | neighbour type (4 bits)
                if (ang) alist[nang + __popc(bal & ((1u << sub) - 1u))] = (unsigned short)(j | (tj << 10));
                nang += __popc(bal);
            }
        }
        {
            T v[NMAX];
#pragma unroll
            for (int n = 0; n < NP2; n++) { v[2 * n] = pk_lo(qa[n]); v[2 * n + 1] = pk_hi(qa[n]); }
            if constexpr (NMAX <= G) {
                const T s = group_xreduce<T, NMAX, G>(v, lane);
                if (sub % (G / NMAX) == 0 && sub / (G / NMAX) < A.n_r) q[sub / (G / NMAX)] = s;
            } else {
#pragma unroll
                for (int n = 0; n < NMAX; n++) {
                    T s = v[n];
#pragma unroll
                    for (int o = G / 2; o >= 1; o >>= 1) s += __shfl_xor_sync(FULL_MASK, s, o);
                    if (sub == n % G && n < A.n_r) q[n] = s;
                }
            }
        }
        __syncwarp();

        // ---- 2. angular sums: lane `sub` of a group ends with S[mu][LM sub .. LM sub + LM - 1] of its atom ------
        // the angular neighbours of the warp's atoms in one sequence: group g's are first[g] .. first[g] + nang - 1
        int first = 0, total = 0;
#pragma unroll
        for (int g = 0; g < AW; g++) {
            const int c = __shfl_sync(FULL_MASK, nang, g * G);
            if (g == grp) first = total;
            total += c;
        }
        const bool keep = total <= 32;          // one step: what it computes stays in registers for the force pass
        Pk<T> S[LM][NP2];
#pragma unroll
        for (int i = 0; i < LM; i++)
#pragma unroll
            for (int n = 0; n < NP2; n++) S[i][n] = pk(T(0), T(0));
        // the angular neighbour that this lane works on
        Pk<T> g[NP2], dg[NP2];
        T ux = 0, uy = 0, uz = 0, rinv = 0, rr = 0;
        int pg = 0, pj = 0;
        bool pon = false;
        auto take_pair = [&](int p) {
            pon = p < total;
            int k = p;
            pg = 0;
#pragma unroll
            for (int a = 0; a < AW - 1; a++) {
                const int c = __shfl_sync(FULL_MASK, nang, a * G);
                if (pg == a && k >= c) { k -= c; pg = a + 1; }
            }
            const int pslot = __shfl_sync(FULL_MASK, slot, pg * G), pti = __shfl_sync(FULL_MASK, ti, pg * G);
            T x = T(0), y = T(0), z = A.rc_a;
            int tj = 0;
            pj = 0;
            if (pon) {
                const int ent = alist0[pg * A.umax + k];
                pj = ent & 1023;
                tj = ent >> 10;
                const T *pr = A.rcs + ((size_t)pslot * A.umax + pj) * 3;
                x = pr[0]; y = pr[1]; z = pr[2];
            }
            const T r2 = x * x + y * y + z * z;
            rinv = inv_sqrt(r2);
            rr = r2 * rinv;
            ux = x * rinv; uy = y * rinv; uz = z * rinv;
            nep_functions<T, NMAX, NET>(tab_s + (pti * A.ntypes + tj) * D::TROW + NMAX, rr * inv_rca, inv_rca, g, dg);
        };
        for (int p0 = 0; p0 < total; p0 += 32) {
            take_pair(p0 + lane);
            {
                T row[RS];
#pragma unroll
                for (int n = 0; n < NP2; n++) { row[2 * n] = pk_lo(g[n]); row[2 * n + 1] = pk_hi(g[n]); }
                {
                    NEP_POLY_COMMON(ux, uy, uz)
#define NEP_X(k, val, gx, gy, gz) row[NMAX + k] = (val);
                    NEP_FOR_EACH_LM(NEP_X, ux, uy, uz)
#undef NEP_X
                }
#pragma unroll
                for (int k = NMAX + NEP_NLM; k < RS; k++) row[k] = T(0);
                if (pon) store_vec<T, RS>(stage + lane * RS, row);
            }
            __syncwarp();
            const int k0 = max(first - p0, 0), k1 = min(first + nang - p0, 32);       // this group's rows of the step
            const int steps = __reduce_max_sync(FULL_MASK, k1 - k0);
            for (int k = k0; k < k0 + steps; k++) {
                if (k < k1) {
                    const T *row = stage + k * RS;
                    Pk<T> gj[NP2];
                    load_pk<NP2>(row, gj);
#pragma unroll
                    for (int i = 0; i < LM; i++) {
                        const int lm = LM * sub + i;
                        const T bv = lm < NEP_NLM ? row[NMAX + lm] : T(0);
                        const Pk<T> b2 = pk(bv, bv);
#pragma unroll
                        for (int n = 0; n < NP2; n++) S[i][n] = pk_fma(gj[n], b2, S[i][n]);
                    }
                }
            }
            __syncwarp();
        }

        // ---- 3. angular descriptors q_{mu,l} = sum_m w_m C_lm S^2, network --------------------------------------
        T *tq = es + grp * ESR;
#pragma unroll
        for (int i = 0; i < LM; i++) {
            const int lm = LM * sub + i;
            if (lm < NEP_NLM) {
#pragma unroll
                for (int n = 0; n < NP2; n++) {
                    tq[2 * n * NEP_NLM + lm] = c3w_s[lm] * pk_lo(S[i][n]) * pk_lo(S[i][n]);
                    tq[(2 * n + 1) * NEP_NLM + lm] = c3w_s[lm] * pk_hi(S[i][n]) * pk_hi(S[i][n]);
                }
            }
        }
        __syncwarp();
        for (int p = sub; p < nq_a; p += G) {
            const int mu = p / A.l_max, l = p - mu * A.l_max + 1;
            const T *row = tq + mu * NEP_NLM + l * l - 1;
            T s = row[0] + row[1] + row[2];
            for (int m = 3; m < 2 * l + 1; m += 2) s += row[m] + row[m + 1];
            q[A.n_r + p] = s;
        }
        __syncwarp();
        if constexpr (MODE == NEP_DESC) {
            if (valid)
                for (int k = sub; k < A.nd; k += G) A.desc[(size_t)slot * A.nd + k] = q[k];
            __syncwarp();
        } else {
        for (int k = sub; k < A.nd; k += G) Eq[k] = q[k] * tab_s[L.iqs + k];
        __syncwarp();
        if constexpr (PARK) {      // (the descriptors' terms that lay here have been read)
            static_assert(LM * NP2 * 64 <= 32 * RS, "a lane's sums fit in the staging rows");
#pragma unroll
            for (int i = 0; i < LM; i++)
#pragma unroll
                for (int n = 0; n < NP2; n++) reinterpret_cast<Pk<T> *>(stage)[(i * NP2 + n) * 32 + lane] = S[i][n];
        }
        T e_at = T(0);
        const T *W0t = tab_s + L.w0 + ti * NP * NDP, *B0t = tab_s + L.b0 + ti * NP, *W1t = tab_s + L.w1 + ti * NP;
        if constexpr (ONEPASS) {
            // A neuron's row is read once and used twice, for its input and for its share of the descriptors' adjoints: the
            // shared-memory pipe is what bounds this phase (four wavefronts per 16-byte load, whatever the lanes share).
            Pk<T> e[NDP / 2], a[NDP / 2];
            load_pk<NDP / 2>(Eq, e);
#pragma unroll
            for (int k = 0; k < NDP / 2; k++) a[k] = pk(T(0), T(0));
            for (int p = sub; p < NP; p += G) {
                Pk<T> w[NDP / 2], h0 = pk(B0t[p], T(0)), h1 = pk(T(0), T(0));
                load_pk<NDP / 2>(W0t + p * NDP, w);
#pragma unroll
                for (int k = 0; k < NDP / 2; k += 2) { h0 = pk_fma(w[k], e[k], h0); h1 = pk_fma(w[k + 1], e[k + 1], h1); }
                const T th = gtanh((pk_lo(h0) + pk_hi(h0)) + (pk_lo(h1) + pk_hi(h1)));
                const T w1 = W1t[p];                    // zero for padding neurons
                e_at += w1 * th;
                const T x = w1 * (T(1) - th * th);
                const Pk<T> x2 = pk(x, x);
#pragma unroll
                for (int k = 0; k < NDP / 2; k++) a[k] = pk_fma(x2, w[k], a[k]);
            }
            // over the lanes of the group: two exchanging steps leave a quarter of the descriptors per lane, the rest adds up
            constexpr int H = NDP / 2, Q = NDP / 4;
            T r[H];
            const bool up1 = sub & 1, up2 = sub & 2;
#pragma unroll
            for (int k = 0; k < H; k++) {
                const T lo = (k & 1) ? pk_hi(a[k / 2]) : pk_lo(a[k / 2]), hi = ((k + H) & 1) ? pk_hi(a[(k + H) / 2]) : pk_lo(a[(k + H) / 2]);
                r[k] = (up1 ? hi : lo) + __shfl_xor_sync(FULL_MASK, up1 ? lo : hi, 1);
            }
#pragma unroll
            for (int k = 0; k < Q; k++) {
                r[k] = (up2 ? r[k + Q] : r[k]) + __shfl_xor_sync(FULL_MASK, up2 ? r[k] : r[k + Q], 2);
#pragma unroll
                for (int o = 4; o < G; o <<= 1) r[k] += __shfl_xor_sync(FULL_MASK, r[k], o);
            }
            const int k0 = (up1 ? H : 0) + (up2 ? Q : 0);
            __syncwarp();
            if (sub < 4)
#pragma unroll
                for (int k = 0; k < Q; k++) Eq[k0 + k] = r[k] * tab_s[L.iqs + k0 + k];
        } else {
            for (int p0 = 0; p0 < NP; p0 += NPL * G) {      // lanes = neurons, NPL at a time
                Pk<T> h[NPL];
#pragma unroll
                for (int i = 0; i < NPL; i++) h[i] = pk(T(0), T(0));
#pragma unroll
                for (int c = 0; c < NDP / 4; c++) {
                    Pk<T> e[2];
                    load_pk<2>(Eq + 4 * c, e);
#pragma unroll
                    for (int i = 0; i < NPL; i++) {
                        Pk<T> w[2];
                        load_pk<2>(W0t + (p0 + sub + G * i) * NDP + 4 * c, w);
                        h[i] = pk_fma(w[0], e[0], h[i]);
                        h[i] = pk_fma(w[1], e[1], h[i]);
                    }
                }
#pragma unroll
                for (int i = 0; i < NPL; i++) {
                    const int p = p0 + sub + G * i;
                    const T th = gtanh(pk_lo(h[i]) + pk_hi(h[i]) + B0t[p]);
                    const T w1 = W1t[p];                    // zero for padding neurons
                    e_at += w1 * th;
                    act[p] = w1 * (T(1) - th * th);
                }
            }
            __syncwarp();
            {   // adjoints of the descriptors: lanes = four descriptors each, the neurons in G / 8 parts
                constexpr int PARTS = G >= 8 ? G / 8 : 1, CL = G >= 8 ? 8 : G;
                const int part = sub / CL, pb = part * (NP / PARTS), pe = pb + NP / PARTS;
                for (int c0 = 0; c0 < NDP / 4; c0 += CL) {
                    const int c = c0 + sub % CL;
                    const bool in = c < NDP / 4;
                    const T *wcol = W0t + 4 * (in ? c : 0);
                    Pk<T> a[2][2];
                    a[0][0] = a[0][1] = a[1][0] = a[1][1] = pk(T(0), T(0));
#pragma unroll 2
                    for (int p = pb; p < pe; p += 4) {
                        T x[4];
                        load_vec<T, 4>(act + p, x);
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            Pk<T> w[2];
                            load_pk<2>(wcol + (p + i) * NDP, w);
                            const Pk<T> x2 = pk(x[i], x[i]);
                            a[i & 1][0] = pk_fma(x2, w[0], a[i & 1][0]);
                            a[i & 1][1] = pk_fma(x2, w[1], a[i & 1][1]);
                        }
                    }
                    T r[4] = {pk_lo(a[0][0]) + pk_lo(a[1][0]), pk_hi(a[0][0]) + pk_hi(a[1][0]), pk_lo(a[0][1]) + pk_lo(a[1][1]), pk_hi(a[0][1]) + pk_hi(a[1][1])};
#pragma unroll
                    for (int o = CL; o < G; o <<= 1)
#pragma unroll
                        for (int k = 0; k < 4; k++) r[k] += __shfl_xor_sync(FULL_MASK, r[k], o);
                    if (in && part == 0) {
#pragma unroll
                        for (int k = 0; k < 4; k++) r[k] *= tab_s[L.iqs + 4 * c + k];
                        store_vec<T, 4>(Eq + 4 * c, r);
                    }
                }
            }
            __syncwarp();
        }
        if (valid) e_at += sub == 0 ? A.bias[ti] : T(0);
        else e_at = T(0);
        __syncwarp();
        if constexpr (PARK) {
#pragma unroll
            for (int i = 0; i < LM; i++)
#pragma unroll
                for (int n = 0; n < NP2; n++) S[i][n] = reinterpret_cast<const Pk<T> *>(stage)[(i * NP2 + n) * 32 + lane];
            __syncwarp();
        }
        // adjoints of the sums, [mu][24] (the descriptors' terms that lay there have been read)
#pragma unroll
        for (int i = 0; i < LM; i++) {
            const int lm = LM * sub + i;
            if (lm < NEP_NLM) {
                const int l = lm >= 15 ? 4 : lm >= 8 ? 3 : lm >= 3 ? 2 : 1;
#pragma unroll
                for (int mu = 0; mu < NMAX; mu++) {
                    const T s = (mu & 1) ? pk_hi(S[i][mu / 2]) : pk_lo(S[i][mu / 2]);
                    tq[mu * NEP_NLM + lm] = (lm < nlm && mu < A.n_a) ? fac_s[lm] * Eq[A.n_r + mu * A.l_max + l - 1] * s : T(0);
                }
            }
        }
        __syncwarp();

        // ---- 4. forces and virial --------------------------------------------------------------------------------
        T fx = T(0), fy = T(0), fz = T(0);            // on this group's atom
        auto add_virial = [&](T gx, T gy, T gz, T x, T y, T z) {
            if (MODE == NEP_EFV) {
                vir[0] -= gx * x; vir[1] -= gx * y; vir[2] -= gx * z;
                vir[3] -= gy * x; vir[4] -= gy * y; vir[5] -= gy * z;
                vir[6] -= gz * x; vir[7] -= gz * y; vir[8] -= gz * z;
            }
        };
        for (int p0 = 0; p0 < total; p0 += 32) {       // angular neighbours, with their radial part
            if (!keep) take_pair(p0 + lane);
            const T *ep = es + pg * ESR;
            T V = T(0), U = T(0), Gx = T(0), Gy = T(0), Gz = T(0);     // sum D B, sum l A B, sum A grad B
            Pk<T> gg[NMAX], dd[NMAX];
#pragma unroll
            for (int n = 0; n < NP2; n++) {
                gg[2 * n] = pk(pk_lo(g[n]), pk_lo(g[n])); gg[2 * n + 1] = pk(pk_hi(g[n]), pk_hi(g[n]));
                dd[2 * n] = pk(pk_lo(dg[n]), pk_lo(dg[n])); dd[2 * n + 1] = pk(pk_hi(dg[n]), pk_hi(dg[n]));
            }
            T Av[NEP_NLM], Dv[NEP_NLM];
#pragma unroll
            for (int c = 0; c < NEP_NLM / 4; c++) {
                Pk<T> a[2], d[2];
#pragma unroll
                for (int mu = 0; mu < NMAX; mu++) {
                    Pk<T> e[2];
                    load_pk<2>(ep + mu * NEP_NLM + 4 * c, e);
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        a[h] = mu ? pk_fma(gg[mu], e[h], a[h]) : pk_mul(gg[mu], e[h]);
                        d[h] = mu ? pk_fma(dd[mu], e[h], d[h]) : pk_mul(dd[mu], e[h]);
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    Av[4 * c + 2 * h] = pk_lo(a[h]); Av[4 * c + 2 * h + 1] = pk_hi(a[h]);
                    Dv[4 * c + 2 * h] = pk_lo(d[h]); Dv[4 * c + 2 * h + 1] = pk_hi(d[h]);
                }
            }
            {
                NEP_POLY_COMMON(ux, uy, uz)
#define NEP_X(k, val, gx_, gy_, gz_)                                                      \
    {                                                                                     \
        const T b_ = (val), ab_ = Av[k] * b_;                                             \
        V = fma(Dv[k], b_, V);                                                            \
        U = fma(T((k) >= 15 ? 4 : (k) >= 8 ? 3 : (k) >= 3 ? 2 : 1), ab_, U);              \
        nep_acc1<T>(Av[k], (gx_), Gx);                                                    \
        nep_acc1<T>(Av[k], (gy_), Gy);                                                    \
        nep_acc1<T>(Av[k], (gz_), Gz);                                                    \
    }
                NEP_FOR_EACH_LM(NEP_X, ux, uy, uz)
#undef NEP_X
            }
            // u . grad B_lm = l B_lm: the part of the gradient along u needs no dot product
            const T *Eqp = Eq0 + pg * NDP;
            T *dc = dcache0 + ((size_t)pg * A.umax + pj) * NMAX;
            T d[NMAX], gr = T(0);
            load_vec<T, NMAX>(dc, d);
#pragma unroll
            for (int n = 0; n < NMAX; n++) gr = fma(n < A.n_r ? Eqp[n] : T(0), d[n], gr);
            const T au = V - rinv * U + gr * rr;
            const T gx = pon ? fma(au, ux, rinv * Gx) : T(0), gy = pon ? fma(au, uy, rinv * Gy) : T(0), gz = pon ? fma(au, uz, rinv * Gz) : T(0);
            fbuf[3 * lane] = gx; fbuf[3 * lane + 1] = gy; fbuf[3 * lane + 2] = gz;
            const int pslot = __shfl_sync(FULL_MASK, slot, pg * G), pb = __shfl_sync(FULL_MASK, b, pg * G);
            if (pon) {
                const int nj = A.firstneigh[(size_t)pslot * A.umax + pj];
                add3(A.force + ((size_t)pb * (A.npad + A.nghost) + nj) * 3, -gx, -gy, -gz);
                const T x = ux * rr, y = uy * rr, z = uz * rr;
                if (!mixed) add_virial(gx, gy, gz, x, y, z);
                else if (MODE == NEP_EFV) {
                    T *v = A.virial + 9 * pb;
                    atomicAdd(v, -gx * x); atomicAdd(v + 1, -gx * y); atomicAdd(v + 2, -gx * z);
                    atomicAdd(v + 3, -gy * x); atomicAdd(v + 4, -gy * y); atomicAdd(v + 5, -gy * z);
                    atomicAdd(v + 6, -gz * x); atomicAdd(v + 7, -gz * y); atomicAdd(v + 8, -gz * z);
                }
#pragma unroll
                for (int n = 0; n < NMAX; n++) d[n] = T(0);
                store_vec<T, NMAX>(dc, d);            // done: the radial pass leaves this neighbour out
            }
            __syncwarp();
            const int k1 = min(first + nang - p0, 32);
            for (int k = max(first - p0, 0) + sub; k < k1; k += G) { fx += fbuf[3 * k]; fy += fbuf[3 * k + 1]; fz += fbuf[3 * k + 2]; }
            __syncwarp();
        }
        {
            T eqr[NMAX];
#pragma unroll
            for (int n = 0; n < NMAX; n++) eqr[n] = n < A.n_r ? Eq[n] : T(0);
            T *frc = A.force + (size_t)b * (A.npad + A.nghost) * 3;
            for (int j = sub; j < nn; j += G) {        // radial neighbours
                T d[NMAX], s = T(0);
                load_vec<T, NMAX>(dcache + (size_t)j * NMAX, d);
#pragma unroll
                for (int n = 0; n < NMAX; n++) s = fma(eqr[n], d[n], s);
                if (s != T(0)) {
                    const T x = rc[3 * j], y = rc[3 * j + 1], z = rc[3 * j + 2];
                    const T gx = s * x, gy = s * y, gz = s * z;
                    fx += gx; fy += gy; fz += gz;
                    add3(frc + 3 * (size_t)fn[j], -gx, -gy, -gz);
                    add_virial(gx, gy, gz, x, y, z);
                }
            }
            __syncwarp();
            T f4[4] = {fx, fy, fz, T(0)};
            const T s = group_xreduce<T, 4, G>(f4, lane);
            const int k = sub / (G / 4);
            if (valid && sub % (G / 4) == 0 && k < 3) atomicAdd(frc + 3 * ci + k, s);
        }
        e_acc += e_at;
        if (mixed) {      // per group, straight to the outputs
            T r[10];
            r[0] = e_acc;
#pragma unroll
            for (int k = 0; k < 9; k++) r[1 + k] = vir[k];
#pragma unroll
            for (int k = 0; k < (MODE == NEP_EFV ? 10 : 1); k++) {
#pragma unroll
                for (int o = G / 2; o >= 1; o >>= 1) r[k] += __shfl_xor_sync(FULL_MASK, r[k], o);
                if (valid && sub == 0) atomicAdd(k == 0 ? A.etot + b : A.virial + 9 * b + k - 1, r[k]);
            }
            e_acc = T(0);
#pragma unroll
            for (int k = 0; k < 9; k++) vir[k] = T(0);
        }
        __syncwarp();     // the cached derivatives and lists are rewritten by the next atoms
        }   // MODE != NEP_DESC
    }

    // energy / virial: warps whose atoms belong to the structure of the block's first warp combine in shared memory, the
    // others add to the outputs directly
    if (NET) {
        if (threadIdx.x == 0) blk_b = bcur;
        if (threadIdx.x < 10) blk_acc[threadIdx.x] = T(0);
        __syncthreads();
        if (bcur >= 0) {
            if (bcur == blk_b) flush_to(bcur, &blk_acc[0], &blk_acc[1]);
            else flush_to(bcur, A.etot + bcur, A.virial + 9 * bcur);
        }
        __syncthreads();
        if (threadIdx.x < 10 && blk_b >= 0) {
            const T v = blk_acc[threadIdx.x];
            if (threadIdx.x == 0) atomicAdd(A.etot + blk_b, v);
            else if (MODE == NEP_EFV) atomicAdd(A.virial + 9 * blk_b + threadIdx.x - 1, v);
        }
    }
}

}  // namespace ai2b
