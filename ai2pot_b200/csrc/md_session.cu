// Device-resident input path for a molecular-dynamics host (the role of
// PairAI2Pot::construct_mlff_input + compute, interface/lammps/AI2POT/pair_ai2pot.cpp:175-249,383-471).
//
// The reference builds the seven input tensors on the host every step (a loop over the host's
// neighbour list forming r_j - r_i in double and storing float), uploads all of them, runs the
// model and downloads forces. Here a step uploads only the positions (double, as the host keeps
// them) and the model types of the nlocal + nghost atoms; the neighbour rows are built on the
// device (centres = local atoms, candidates = local + ghost atoms, no periodic images: the host's
// ghosts carry the periodicity), the model runs on them, and forces for all nlocal + nghost atoms
// come back for the host's reverse communication, with the energy and the six virial components
// in the host's order. Device and pinned buffers grow when the atom counts grow and are reused
// otherwise, so a steady-state step allocates nothing.
//
// A step's host work: one pass over the positions that copies them into pinned memory and finds their extent (so the
// bin grid is known on the host and the build needs no look at the atoms first), sent off in pieces that travel while the
// next piece is copied; one transfer back of [forces | energy, virial | status]; one pass that adds the forces. 13,824 local
// and 11,415 ghost atoms, NEP: 159 to 178 us per step, by the host, where pageable transfers array by array, a device pass over the extents
// and a scalar loop over the forces took 355 us.
#include "nep_setup.cuh"

#include <cstring>
#if defined(__SSE2__)
#include <emmintrin.h>
#endif

using namespace ai2b;

namespace ai2b {
int nblist_build_rows32(int n, int ncentres, const double *h_cell, const double *d_coords, double rcut, const int *h_pbc, const double *open_ext, int umax,
                        int *d_numneigh, int *d_firstneigh, float *d_rcs, int *d_status, void *ws, size_t ws_bytes, cudaStream_t st, const NepSetup &side);
}

// Positions travel in pieces of this many atoms, MD_SLOTS of which have a place in pinned memory. Pinning costs 0.9 to 2.9 ms per
// 2 MB, of which blocks of less than 1 MB are cut: the ring has a fixed size and is made with the session, and what a
// step brings back comes from the same 2 MB for up to 80,000 atoms. A step of 25,239 atoms takes as long with three slots as with pinned
// memory for all of it (188 and 187 us when the stores still went through the caches; medians, in turn).
constexpr size_t MD_PIECE = 6144;
constexpr int MD_SLOTS = 3;
constexpr size_t MD_RING_BYTES = sizeof(double) * 3 * MD_PIECE * MD_SLOTS;

struct ai2b_md_session {
    int kind = 0;   // 0 = NEP, 1 = linear MTP
    int ntypes = 0, umax = 0;
    double rcut = 0;
    // NEP
    int cs = 0, n_r = 0, n_a = 0, l_max = 0, nneu = 0;
    float rc_r = 0, rc_a = 0;
    float *d_coeffs = nullptr, *d_w0 = nullptr, *d_b0 = nullptr, *d_w1 = nullptr, *d_bias = nullptr, *d_qs = nullptr;
    // MTP
    const ai2b_mtp_program *prog = nullptr;
    float scaling = 0, rmax = 0, rmin = 0;
    float *d_lin = nullptr;
    // per-step buffers
    int cap_all = 0, cap_local = 0;
    unsigned char *d_all = nullptr;                       // one allocation for everything on the device
    unsigned char *d_in = nullptr;                        // [positions | types | nlocal] of the step
    unsigned char *d_out = nullptr;                       // [forces | energy, virial, pad (16) | status (4)]
    double *h_ring = nullptr;                             // pinned: positions on their way to the device, up to MD_SLOTS pieces
    unsigned char *h_out = nullptr, *h_types = nullptr;   // pinned: d_out's copy; types and nlocal (same allocation)
    cudaEvent_t sent[MD_SLOTS] = {};                      // a slot of the ring has been read
    int *d_numneigh = nullptr, *d_firstneigh = nullptr, *d_ilist = nullptr;
    float *d_rcs = nullptr;
    void *d_nbws = nullptr, *d_ws = nullptr;
    size_t nbws = 0, ws = 0;
    cudaStream_t stream = nullptr;
};

namespace {

__global__ void iota_kernel(int *out, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = i;
}

template <typename T>
int upload(T **dst, const T *src, size_t n)
{
    AI2B_CUDA(cudaMalloc((void **)dst, sizeof(T) * (n ? n : 1)));
    if (n) AI2B_CUDA(cudaMemcpy(*dst, src, sizeof(T) * n, cudaMemcpyHostToDevice));
    return AI2B_OK;
}

size_t in_bytes(int nall) { return (size_t)nall * (3 * sizeof(double) + sizeof(int)) + sizeof(int); }
size_t out_bytes(int nall) { return (size_t)nall * 3 * sizeof(float) + 16 * sizeof(float) + 4 * sizeof(int); }

// What a step brings back is copied by a kernel of the chain up to this size: between the last kernel and a copy engine the hand-over
// costs 5 us (900 atoms 68 -> 64 us a step, 25,239 atoms 188 -> 183). The way in stays with the copy engine: there the pieces of a step
// overlap with the host's copying (25,239 atoms 164 us, 176 with kernels).
constexpr size_t MD_KERNEL_COPY = 1 << 20;
int bring_back(void *dst, const void *src, size_t bytes, cudaStream_t st)
{
    if (bytes <= MD_KERNEL_COPY) return ai2b_chained_copy(dst, src, bytes, st);
    AI2B_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st));
    return AI2B_OK;
}

void release_step_buffers(ai2b_md_session *s)
{
    cudaFree(s->d_all);
    cudaFreeHost(s->h_out);
    s->d_all = s->d_in = s->d_out = s->h_out = s->h_types = nullptr;
    s->d_numneigh = s->d_firstneigh = s->d_ilist = nullptr;
    s->d_rcs = nullptr; s->d_nbws = s->d_ws = nullptr;
    // nothing is usable until ensure_capacity has run to its end: a growth that failed half-way (out of
    // memory) must make the next call allocate afresh instead of running on freed or partial buffers
    s->cap_all = s->cap_local = 0;
}

// First step of a session and every growth: one device allocation (0.35 ms; eight of them took 1.3) and one of pinned memory.
int ensure_capacity(ai2b_md_session *s, int nlocal, int nall)
{
    if (nall <= s->cap_all && nlocal <= s->cap_local) return AI2B_OK;
    AI2B_CUDA(cudaStreamSynchronize(s->stream));
    release_step_buffers(s);
    const int call = nall + nall / 5 + 64, cloc = nlocal + nlocal / 5 + 64;   // 20 % head-room against regrowth every step
    s->nbws = ai2b_nblist_workspace_bytes(call, 1);
    s->ws = s->kind == 0 ? ai2b_nep_workspace_bytes(1, s->ntypes, s->n_r, s->n_a, s->cs, 0)
                         : ai2b_mtp_workspace_bytes(s->prog, 1, cloc, s->ntypes);
    size_t total = 0;
    auto take = [&](size_t bytes) { const size_t at = total; total += (bytes + 255) & ~size_t(255); return at; };
    const size_t rows = (size_t)cloc * s->umax;
    const size_t in = take(in_bytes(call)), out = take(out_bytes(call)), numneigh = take(sizeof(int) * cloc), ilist = take(sizeof(int) * cloc),
                 firstneigh = take(sizeof(int) * rows), rcs = take(sizeof(float) * 3 * rows), nbws = take(s->nbws), ws = take(s->ws ? s->ws : 256);
    AI2B_CUDA(cudaMalloc((void **)&s->d_all, total));
    const size_t back = (out_bytes(call) + 255) & ~size_t(255);
    AI2B_CUDA(cudaMallocHost((void **)&s->h_out, back + sizeof(int) * ((size_t)call + 1)));
    s->h_types = s->h_out + back;
    s->d_in = s->d_all + in; s->d_out = s->d_all + out;
    s->d_numneigh = (int *)(s->d_all + numneigh); s->d_ilist = (int *)(s->d_all + ilist); s->d_firstneigh = (int *)(s->d_all + firstneigh);
    s->d_rcs = (float *)(s->d_all + rcs); s->d_nbws = s->d_all + nbws; s->d_ws = s->d_all + ws;
    iota_kernel<<<(cloc + 255) / 256, 256, 0, s->stream>>>(s->d_ilist, cloc);
    AI2B_CUDA(cudaGetLastError());
    s->cap_all = call;
    s->cap_local = cloc;
    return AI2B_OK;
}

int common_init(ai2b_md_session *s)
{
    AI2B_CUDA(cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking));
    AI2B_CUDA(cudaMallocHost((void **)&s->h_ring, MD_RING_BYTES));
    for (cudaEvent_t &e : s->sent) AI2B_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    return AI2B_OK;
}

// dst = src for n positions; the lowest and highest coordinates are folded into lo and hi. dst starts on a 16-byte boundary.
void copy_and_bound(double *dst, const double *src, size_t n, double *lo, double *hi)
{
    size_t i = 0;
#if defined(__SSE2__)
    if (n >= 2) {     // two positions are three pairs: (x y) (z x) (y z). The accumulator comes second: it survives a NaN
        __m128d l[3], h[3];
        for (int k = 0; k < 3; k++) { l[k] = _mm_set1_pd(1e300); h[k] = _mm_set1_pd(-1e300); }
        for (; i + 2 <= n; i += 2)
            for (int k = 0; k < 3; k++) {
                const __m128d v = _mm_loadu_pd(src + 3 * i + 2 * k);
                _mm_stream_pd(dst + 3 * i + 2 * k, v);      // past the caches: the device reads it next (25,239 atoms 183 -> 164 us a step)
                l[k] = _mm_min_pd(v, l[k]);
                h[k] = _mm_max_pd(v, h[k]);
            }
        _mm_sfence();
        for (int k = 0; k < 3; k++) {
            double a[2], b[2];
            _mm_storeu_pd(a, l[k]);
            _mm_storeu_pd(b, h[k]);
            for (int q = 0; q < 2; q++) {
                const int c = (2 * k + q) % 3;
                lo[c] = a[q] < lo[c] ? a[q] : lo[c];
                hi[c] = b[q] > hi[c] ? b[q] : hi[c];
            }
        }
    }
#endif
    for (; i < n; i++)
        for (int c = 0; c < 3; c++) {
            const double v = dst[3 * i + c] = src[3 * i + c];
            lo[c] = v < lo[c] ? v : lo[c];
            hi[c] = v > hi[c] ? v : hi[c];
        }
}

// f (+)= g, single to double precision
template <bool ADD>
void take_forces(double *f, const float *g, size_t n)
{
    size_t i = 0;
#if defined(__SSE2__)
    for (; i + 4 <= n; i += 4) {
        const __m128 v = _mm_loadu_ps(g + i);
        __m128d a = _mm_cvtps_pd(v), b = _mm_cvtps_pd(_mm_movehl_ps(v, v));
        if (ADD) { a = _mm_add_pd(a, _mm_loadu_pd(f + i)); b = _mm_add_pd(b, _mm_loadu_pd(f + i + 2)); }
        _mm_storeu_pd(f + i, a);
        _mm_storeu_pd(f + i + 2, b);
    }
#endif
    for (; i < n; i++) f[i] = ADD ? f[i] + (double)g[i] : (double)g[i];
}

}  // namespace

extern "C" int ai2b_md_session_create_nep(ai2b_md_session **out, int chebyshev_size, int n_radial, int n_angular, int l_max,
                                          int num_neurons, int ntypes, const float *h_coeffs, const float *h_w0, const float *h_b0,
                                          const float *h_w1, const float *h_type_bias, const float *h_q_scaler, float rmax_radial,
                                          float rmax_angular, int umax)
{
    AI2B_REQUIRE(out && h_coeffs && h_w0 && h_b0 && h_w1 && h_type_bias && h_q_scaler, AI2B_ERR_INVALID, "ai2b_md_session_create_nep: NULL argument");
    AI2B_REQUIRE(ntypes >= 1 && umax >= 1 && num_neurons >= 1 && rmax_radial > 0, AI2B_ERR_INVALID, "ai2b_md_session_create_nep: bad size");
    ai2b_md_session *s = new ai2b_md_session();
    s->kind = 0; s->ntypes = ntypes; s->umax = umax; s->rcut = rmax_radial > rmax_angular ? rmax_radial : rmax_angular;
    s->cs = chebyshev_size; s->n_r = n_radial; s->n_a = n_angular; s->l_max = l_max; s->nneu = num_neurons;
    s->rc_r = rmax_radial; s->rc_a = rmax_angular;
    const int nd = l_max == 0 ? n_radial : n_radial + n_angular * l_max;
    int rc = common_init(s);
    if (!rc) rc = upload(&s->d_coeffs, h_coeffs, (size_t)ntypes * ntypes * (n_radial + n_angular) * chebyshev_size);
    if (!rc) rc = upload(&s->d_w0, h_w0, (size_t)ntypes * num_neurons * nd);
    if (!rc) rc = upload(&s->d_b0, h_b0, (size_t)ntypes * num_neurons);
    if (!rc) rc = upload(&s->d_w1, h_w1, (size_t)ntypes * num_neurons);
    if (!rc) rc = upload(&s->d_bias, h_type_bias, (size_t)ntypes);
    if (!rc) rc = upload(&s->d_qs, h_q_scaler, (size_t)nd);
    if (rc) { ai2b_md_session_destroy(s); return rc; }
    *out = s;
    return AI2B_OK;
}

extern "C" int ai2b_md_session_create_mtp(ai2b_md_session **out, const ai2b_mtp_program *prog, int chebyshev_size, float scaling,
                                          int ntypes, int nmus, int alpha_scalar_moments, const float *h_coeffs,
                                          const float *h_linear_coeffs, const float *h_type_bias, const float *h_q_scaler, float rmax,
                                          float rmin, int umax)
{
    AI2B_REQUIRE(out && prog && h_coeffs && h_linear_coeffs && h_type_bias && h_q_scaler, AI2B_ERR_INVALID, "ai2b_md_session_create_mtp: NULL argument");
    AI2B_REQUIRE(ntypes >= 1 && umax >= 1 && nmus >= 1 && alpha_scalar_moments >= 1 && rmax > rmin, AI2B_ERR_INVALID,
                 "ai2b_md_session_create_mtp: bad size");
    ai2b_md_session *s = new ai2b_md_session();
    s->kind = 1; s->ntypes = ntypes; s->umax = umax; s->rcut = rmax; s->prog = prog; s->cs = chebyshev_size; s->scaling = scaling;
    s->rmax = rmax; s->rmin = rmin;
    int rc = common_init(s);
    if (!rc) rc = upload(&s->d_coeffs, h_coeffs, (size_t)ntypes * ntypes * nmus * chebyshev_size);
    if (!rc) rc = upload(&s->d_lin, h_linear_coeffs, (size_t)alpha_scalar_moments);
    if (!rc) rc = upload(&s->d_bias, h_type_bias, (size_t)ntypes);
    if (!rc) rc = upload(&s->d_qs, h_q_scaler, (size_t)alpha_scalar_moments);
    if (rc) { ai2b_md_session_destroy(s); return rc; }
    *out = s;
    return AI2B_OK;
}

extern "C" void ai2b_md_session_destroy(ai2b_md_session *s)
{
    if (!s) return;
    if (s->stream) cudaStreamSynchronize(s->stream);
    release_step_buffers(s);
    cudaFree(s->d_coeffs); cudaFree(s->d_w0); cudaFree(s->d_b0); cudaFree(s->d_w1); cudaFree(s->d_bias); cudaFree(s->d_qs);
    cudaFree(s->d_lin);
    cudaFreeHost(s->h_ring);
    for (cudaEvent_t e : s->sent)
        if (e) cudaEventDestroy(e);
    if (s->stream) cudaStreamDestroy(s->stream);
    delete s;
}

static int session_step(ai2b_md_session *s, int nlocal, int nghost, const double *h_x, const int *h_model_type, int want_virial, bool accumulate,
                        double *h_f, double *h_eng, double *h_virial6, int *h_max_neighbours)
{
    AI2B_REQUIRE(s && h_x && h_model_type && h_f, AI2B_ERR_INVALID, "ai2b_md_session_compute: NULL argument");
    AI2B_REQUIRE(nlocal >= 0 && nghost >= 0, AI2B_ERR_INVALID, "ai2b_md_session_compute: negative atom count");
    const int nall = nlocal + nghost;
    if (nlocal == 0) {
        if (!accumulate) memset(h_f, 0, sizeof(double) * 3 * (size_t)nall);
        return AI2B_OK;
    }
    if (int rc = ensure_capacity(s, nlocal, nall)) return rc;
    cudaStream_t st = s->stream;
    double *d_pos = reinterpret_cast<double *>(s->d_in);
    // types and the atom count travel with the last positions if the ring holds the whole step (a transfer costs 2 us)
    const bool together = in_bytes(nall) <= MD_RING_BYTES;
    const size_t type_bytes = sizeof(int) * ((size_t)nall + 1);
    auto stage_types = [&](void *dst) {
        memcpy(dst, h_model_type, sizeof(int) * nall);
        static_cast<int *>(dst)[nall] = nlocal;
    };
    // positions in pieces: the copy engine takes a piece while the next one is copied and bounded
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    const size_t pieces = ((size_t)nall + MD_PIECE - 1) / MD_PIECE;
    for (size_t k = 0; k < pieces; k++) {
        const size_t i0 = k * MD_PIECE, n = (size_t)nall - i0 < MD_PIECE ? (size_t)nall - i0 : MD_PIECE, slot = k % MD_SLOTS;
        double *h_pos = s->h_ring + 3 * MD_PIECE * slot;
        if (k >= MD_SLOTS) AI2B_CUDA(cudaEventSynchronize(s->sent[slot]));
        copy_and_bound(h_pos, h_x + 3 * i0, n, lo, hi);
        const bool last = k + 1 == pieces;
        if (together && last) stage_types(h_pos + 3 * n);
        AI2B_CUDA(cudaMemcpyAsync(d_pos + 3 * i0, h_pos, sizeof(double) * 3 * n + (together && last ? type_bytes : 0), cudaMemcpyHostToDevice, st));
        if (k + MD_SLOTS < pieces) AI2B_CUDA(cudaEventRecord(s->sent[slot], st));
        if (!together && k == 0) {      // (copied while the first positions travel)
            stage_types(s->h_types);
            AI2B_CUDA(cudaMemcpyAsync(d_pos + 3 * (size_t)nall, s->h_types, type_bytes, cudaMemcpyHostToDevice, st));
        }
    }
    const int *d_types = reinterpret_cast<const int *>(d_pos + 3 * (size_t)nall), *d_binum = d_types + nall;
    float *d_force = reinterpret_cast<float *>(s->d_out), *d_ev = d_force + 3 * (size_t)nall;
    int *d_status = reinterpret_cast<int *>(d_ev + 16);
    const double cell[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};   // no periodic axis: only the extents of the atoms matter
    const int pbc[3] = {0, 0, 0};
    const double ext[6] = {lo[0], lo[1], lo[2], hi[0], hi[1], hi[2]};
    float *d_vir = want_virial ? d_ev + 1 : nullptr;
    // what the evaluation has to set up goes out with a launch of the build
    NepSetup side;
    const bool carried = s->kind == 0 && nep_plan_setup<float>(d_ev, d_force, d_vir, s->cs, s->n_r, s->n_a, s->l_max, s->nneu, s->d_coeffs, s->d_w0, s->d_b0,
                                                               s->d_w1, nlocal, d_binum, s->ntypes, s->umax, nghost, s->d_qs, s->d_ws, s->ws, &side);
    int rc = nblist_build_rows32(nall, nlocal, cell, d_pos, s->rcut, pbc, ext, s->umax, s->d_numneigh, s->d_firstneigh, s->d_rcs, d_status, s->d_nbws,
                                 s->nbws, st, side);
    if (rc) return rc;
    if (carried)
        rc = nep_efv_prepared<float>(d_ev, d_force, d_vir, s->cs, s->n_r, s->n_a, s->l_max, s->nneu, s->d_coeffs, s->d_w0, s->d_b0, s->d_w1, s->d_bias,
                                     nlocal, d_binum, s->d_ilist, s->d_numneigh, s->d_firstneigh, s->d_rcs, d_types, s->ntypes, s->umax, nghost, s->rc_r,
                                     s->rc_a, s->d_qs, s->d_ws, s->ws, st);
    else if (s->kind == 0)
        rc = ai2b_nep_efv_f32(d_ev, d_force, d_vir, s->cs, s->n_r, s->n_a, s->l_max, s->nneu, s->d_coeffs, s->d_w0, s->d_b0, s->d_w1,
                              s->d_bias, 1, nlocal, d_binum, s->d_ilist, s->d_numneigh, s->d_firstneigh, s->d_rcs, d_types, s->ntypes,
                              s->umax, nghost, s->rc_r, s->rc_a, s->d_qs, s->d_ws, s->ws, st);
    else
        rc = ai2b_mtp_efv_f32(s->prog, d_ev, d_force, d_vir, s->cs, s->scaling, s->d_coeffs, s->d_lin, s->d_bias, 1, nlocal,
                              d_binum, s->d_ilist, s->d_numneigh, s->d_firstneigh, s->d_rcs, d_types, s->ntypes, s->umax, nghost,
                              s->rmax, s->rmin, s->d_qs, s->d_ws, s->ws, st);
    if (rc) return rc;
    if ((rc = bring_back(s->h_out, s->d_out, out_bytes(nall), st))) return rc;
    AI2B_CUDA(cudaStreamSynchronize(st));
    const float *h_force = reinterpret_cast<const float *>(s->h_out), *h_ev = h_force + 3 * (size_t)nall;
    const int *status = reinterpret_cast<const int *>(h_ev + 16);
    if (h_max_neighbours) *h_max_neighbours = status[0];
    AI2B_REQUIRE(!status[1], AI2B_ERR_OVERFLOW, "an atom has %d neighbours within the cutoff, umax is %d", status[0], s->umax);
    // pair_ai2pot.cpp:447-468: forces of all nlocal + nghost atoms are added, energy and virial accumulate
    if (accumulate) take_forces<true>(h_f, h_force, 3 * (size_t)nall);
    else take_forces<false>(h_f, h_force, 3 * (size_t)nall);
    if (h_eng) *h_eng += (double)h_ev[0];
    if (want_virial && h_virial6) {
        static const int pick[6] = {0, 4, 8, 1, 2, 5};
        for (int k = 0; k < 6; k++) h_virial6[k] += (double)h_ev[1 + pick[k]];
    }
    return AI2B_OK;
}

extern "C" int ai2b_md_session_compute(ai2b_md_session *s, int nlocal, int nghost, const double *h_x, const int *h_model_type,
                                       int want_virial, double *h_f, double *h_eng, double *h_virial6, int *h_max_neighbours)
{
    return session_step(s, nlocal, nghost, h_x, h_model_type, want_virial, true, h_f, h_eng, h_virial6, h_max_neighbours);
}
extern "C" int ai2b_md_session_forces(ai2b_md_session *s, int nlocal, int nghost, const double *h_x, const int *h_model_type,
                                      int want_virial, double *h_f, double *h_eng, double *h_virial6, int *h_max_neighbours)
{
    return session_step(s, nlocal, nghost, h_x, h_model_type, want_virial, false, h_f, h_eng, h_virial6, h_max_neighbours);
}
