// Row loop of the MTP contractions: products of moments and their adjoints with atoms along the lanes.
//
// Moments of a tile of atoms sit in shared memory as [moment][atom]; a row multiplies two of them and adds the product to a
// third (mtpBasis.h:519-528, linearMtp.h:292-306). What bounds the loop is the shared-memory pipe (two operands of 8 bytes per
// atom and row) and, close behind, instruction issue. So a lane takes 16 bytes of atoms (two in double, four in single
// precision) and a warp works on 32 / GL rows at a time, GL = 16 or 8 lanes each: one record, two operand loads and 2 VEC
// multiply-adds for all of them, 16-byte accesses without bank conflicts and without padding. The tables deal the moments to
// groups of lanes so that the groups of a warp have equally many rows, long moments in pieces (mtp_program.cuh).
// Level 16, fp64: contraction of 13,824 atoms 50 -> 45 us, loss contraction of 9,323 atoms 171 -> 83 us (one 32-lane row at a time
// with 8-byte operands before). What is left is latency: operand loads and the barriers between phases.
#pragma once
#include "mtp_device.cuh"

namespace ai2b {

template <typename T> struct Lane16;      // 16 bytes of atoms
template <> struct Lane16<double> {
    static constexpr int VEC = 2;
    double v[2];
};
template <> struct Lane16<float> {
    static constexpr int VEC = 4;
    float v[4];
};
// explicit ld.shared / st.shared: the loop must not fall back to generic addressing
__device__ __forceinline__ int2 lds_row(unsigned a)
{
    int2 v;
    asm volatile("ld.shared.v2.s32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ void lds16(unsigned a, Lane16<double> &x) { asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(x.v[0]), "=d"(x.v[1]) : "r"(a)); }
__device__ __forceinline__ void lds16(unsigned a, Lane16<float> &x)
{
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x.v[0]), "=f"(x.v[1]), "=f"(x.v[2]), "=f"(x.v[3]) : "r"(a));
}
__device__ __forceinline__ void sts16(unsigned a, const Lane16<double> &x)
{
    asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(x.v[0]), "d"(x.v[1]) : "memory");
}
__device__ __forceinline__ void sts16(unsigned a, const Lane16<float> &x)
{
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(x.v[0]), "f"(x.v[1]), "f"(x.v[2]), "f"(x.v[3]) : "memory");
}
__device__ __forceinline__ double lds_one(unsigned a, double) { double v; asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a)); return v; }
__device__ __forceinline__ float lds_one(unsigned a, float) { float v; asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a)); return v; }

constexpr int PAIR_DONE = 0x7ff;      // low bits of a row's second word: completed moment + 1; MTP_PAIR_WIDE: in pieces, one per group
__device__ __forceinline__ double row_mult(int w, double) { return __hiloint2double(w & ~0xfff, 0); }
__device__ __forceinline__ float row_mult(int w, float) { return __int_as_float(w & ~0xfff); }

// a moment in pieces ends in the same row of all groups of the warp (so the branch is uniform): every group gets the sum
template <typename T, int GL>
__device__ __forceinline__ void sum_groups(Lane16<T> &a)
{
#pragma unroll
    for (int o = GL; o < 32; o <<= 1)
#pragma unroll
        for (int k = 0; k < Lane16<T>::VEC; k++) a.v[k] += __shfl_xor_sync(FULL_MASK, a.v[k], o);
}

// rows of one phase for this lane's group: M[dst] (+ seed) = sum mult X[x] Y[y]; xl, yl, dl: this lane's 16 bytes of row 0 of the
// arrays, rp: the group's first record, n: rows of the warp
template <typename T, int GL, bool SEEDED>
__device__ __forceinline__ void pair_phase(unsigned rp, int n, unsigned xl, unsigned yl, unsigned dl, unsigned seed)
{
    constexpr int VEC = Lane16<T>::VEC, STEP = 8 * (32 / GL), ROW = GL * 16;
    Lane16<T> acc;
#pragma unroll
    for (int k = 0; k < VEC; k++) acc.v[k] = T(0);
    int2 r = lds_row(rp);
#pragma unroll 2
    for (int i = 0; i < n; i++) {
        rp += STEP;
        const int2 nxt = lds_row(rp);       // (the tables end with empty rows)
        Lane16<T> x, y;
        lds16(xl + (unsigned)(r.x & 0xffff) * ROW, x);
        lds16(yl + ((unsigned)r.x >> 16) * ROW, y);
        const T m = row_mult(r.y, T());
#pragma unroll
        for (int k = 0; k < VEC; k++) acc.v[k] = fma(m * x.v[k], y.v[k], acc.v[k]);
        const unsigned done = (unsigned)r.y & PAIR_DONE;
        if (done) {
            if (r.y & MTP_PAIR_WIDE) sum_groups<T, GL>(acc);
            if (SEEDED) {
                const T s = lds_one(seed + (done - 1) * (unsigned)sizeof(T), T());
#pragma unroll
                for (int k = 0; k < VEC; k++) acc.v[k] += s;
            }
            sts16(dl + (done - 1) * ROW, acc);
#pragma unroll
            for (int k = 0; k < VEC; k++) acc.v[k] = T(0);
        }
        r = nxt;
    }
}

// products with their derivative along a direction (linearMtpLoss.h:391-398): M = sum m A B, D = sum m (A' B + A B'); the
// derivatives lie `off` bytes behind the values
template <typename T, int GL>
__device__ __forceinline__ void pair_phase_deriv(unsigned rp, int n, unsigned ml, unsigned off)
{
    constexpr int VEC = Lane16<T>::VEC, STEP = 8 * (32 / GL), ROW = GL * 16;
    Lane16<T> acc, dacc;
#pragma unroll
    for (int k = 0; k < VEC; k++) acc.v[k] = dacc.v[k] = T(0);
    int2 r = lds_row(rp);
    for (int i = 0; i < n; i++) {
        rp += STEP;
        const int2 nxt = lds_row(rp);
        Lane16<T> a, b, da, db;
        const unsigned aa = ml + (unsigned)(r.x & 0xffff) * ROW, ba = ml + ((unsigned)r.x >> 16) * ROW;
        lds16(aa, a);
        lds16(ba, b);
        lds16(aa + off, da);
        lds16(ba + off, db);
        const T m = row_mult(r.y, T());
#pragma unroll
        for (int k = 0; k < VEC; k++) {
            const T mb = m * b.v[k];
            acc.v[k] = fma(a.v[k], mb, acc.v[k]);
            dacc.v[k] = fma(da.v[k], mb, fma(m * a.v[k], db.v[k], dacc.v[k]));
        }
        const unsigned done = (unsigned)r.y & PAIR_DONE;
        if (done) {
            if (r.y & MTP_PAIR_WIDE) { sum_groups<T, GL>(acc); sum_groups<T, GL>(dacc); }
            const unsigned d = ml + (done - 1) * ROW;
            sts16(d, acc);
            sts16(d + off, dacc);
#pragma unroll
            for (int k = 0; k < VEC; k++) acc.v[k] = dacc.v[k] = T(0);
        }
        r = nxt;
    }
}

// adjoints and second-order adjoints (linearMtpLoss.h:400-434): E = seed + sum m E[dst] M[other],
// G = sum m (E[dst] D[other] + G[dst] M[other]); D lies `off` bytes behind M, G behind E
template <typename T, int GL>
__device__ __forceinline__ void pair_phase_second(unsigned rp, int n, unsigned el, unsigned ml, unsigned off, unsigned seed)
{
    constexpr int VEC = Lane16<T>::VEC, STEP = 8 * (32 / GL), ROW = GL * 16;
    Lane16<T> acc, gacc;
#pragma unroll
    for (int k = 0; k < VEC; k++) acc.v[k] = gacc.v[k] = T(0);
    int2 r = lds_row(rp);
    for (int i = 0; i < n; i++) {
        rp += STEP;
        const int2 nxt = lds_row(rp);
        Lane16<T> e, g, m_, d;
        const unsigned ea = el + (unsigned)(r.x & 0xffff) * ROW, ma = ml + ((unsigned)r.x >> 16) * ROW;
        lds16(ea, e);
        lds16(ma, m_);
        lds16(ea + off, g);
        lds16(ma + off, d);
        const T m = row_mult(r.y, T());
#pragma unroll
        for (int k = 0; k < VEC; k++) {
            const T me = m * e.v[k];
            acc.v[k] = fma(me, m_.v[k], acc.v[k]);
            gacc.v[k] = fma(me, d.v[k], fma(m * g.v[k], m_.v[k], gacc.v[k]));
        }
        const unsigned done = (unsigned)r.y & PAIR_DONE;
        if (done) {
            if (r.y & MTP_PAIR_WIDE) { sum_groups<T, GL>(acc); sum_groups<T, GL>(gacc); }
            const T s = lds_one(seed + (done - 1) * (unsigned)sizeof(T), T());
#pragma unroll
            for (int k = 0; k < VEC; k++) acc.v[k] += s;
            const unsigned o = el + (done - 1) * ROW;
            sts16(o, acc);
            sts16(o + off, gacc);
#pragma unroll
            for (int k = 0; k < VEC; k++) acc.v[k] = gacc.v[k] = T(0);
        }
        r = nxt;
    }
}

template <typename T> __device__ __forceinline__ const int2 *stream_rows(const MtpProgramDev::Stream &s) { return sizeof(T) == 8 ? s.row_d : s.row_f; }

}  // namespace ai2b
