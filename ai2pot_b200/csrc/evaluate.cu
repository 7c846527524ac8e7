// One structure, one model: positions -> neighbour list -> energy, forces, virial in one host call.
//
// The reference's calculators assemble the list and the model's arguments on the host for every call
// (ai2pot/models/potential_utils.py:217-268). Here everything but the positions is described once; a call then is
// the neighbour build and the evaluation back to back, with no argument handling in between: at a few hundred atoms
// the host's share of a call through two separate entry points (50 us) exceeded the device's (31 us).
#include "nep_setup.cuh"

using namespace ai2b;

namespace ai2b {
template <typename T>
int nblist_build_periodic(int n, const T *h_cell, const T *d_coords, double rcut, int umax, int *d_numneigh, int *d_firstneigh, T *d_rcs, int *d_status,
                          void *ws, size_t ws_bytes, cudaStream_t st, const NepSetup &side);
}

static bool apart(const void *a, size_t na, const void *b, size_t nb)
{
    const size_t x = reinterpret_cast<size_t>(a), y = reinterpret_cast<size_t>(b);
    return x + na <= y || y + nb <= x;
}

template <typename T>
static int evaluate_t(const ai2b_evaluation *e, const T *coords, void *stream)
{
    T cell[9];
    for (int k = 0; k < 9; k++) cell[k] = (T)e->cell[k];
    cudaStream_t st = (cudaStream_t)stream;
    T *etot = (T *)e->d_etot, *force = (T *)e->d_force, *virial = (T *)e->d_virial;
    const T *co = (const T *)e->d_coeffs, *bias = (const T *)e->d_type_bias, *qs = (const T *)e->d_q_scaler, *rcs = (const T *)e->d_rcs;
    const T *w0 = (const T *)e->d_w0, *b0 = (const T *)e->d_b0, *w1 = (const T *)e->d_w1;
    // What the evaluation has to set up goes out with a launch of the build, unless it writes to memory that the build still works
    // with (one buffer as the scratch of both, results in the build's scratch, forces that replace the positions, or its status words in
    // the scratch).
    NepSetup side;
    const void *set_up[4] = {e->d_workspace, etot, force, virial};
    const size_t n3 = 3 * sizeof(T) * (size_t)e->natoms, set_up_bytes[4] = {e->workspace_bytes, sizeof(T), n3, 9 * sizeof(T)};
    bool carried = !e->mtp;
    for (int k = 0; k < 4; k++)
        carried = carried && (!set_up[k] || (apart(set_up[k], set_up_bytes[k], e->d_nblist_workspace, e->nblist_workspace_bytes) &&
                                             apart(set_up[k], set_up_bytes[k], coords, n3) &&
                                             apart(set_up[k], set_up_bytes[k], e->d_status, 2 * sizeof(int))));
    carried = carried && nep_plan_setup<T>(etot, force, virial, e->chebyshev_size, e->n_radial, e->n_angular, e->l_max, e->num_neurons, co, w0, b0, w1,
                                           e->natoms, e->d_binum, e->ntypes, e->umax, 0, qs, e->d_workspace, e->workspace_bytes, &side);
    if (int rc = nblist_build_periodic<T>(e->natoms, cell, coords, e->rcut, e->umax, e->d_numneigh, e->d_firstneigh, (T *)e->d_rcs, e->d_status,
                                          e->d_nblist_workspace, e->nblist_workspace_bytes, st, side))
        return rc;
    if (e->mtp) {
        const T *lin = (const T *)e->d_linear_coeffs;
        if constexpr (sizeof(T) == 8)
            return ai2b_mtp_efv_f64(e->mtp, etot, force, virial, e->chebyshev_size, e->scaling, co, lin, bias, 1, e->natoms, e->d_binum, e->d_ilist,
                                    e->d_numneigh, e->d_firstneigh, rcs, e->d_types, e->ntypes, e->umax, 0, e->rmax, e->rmin, qs, e->d_workspace,
                                    e->workspace_bytes, stream);
        else
            return ai2b_mtp_efv_f32(e->mtp, etot, force, virial, e->chebyshev_size, (T)e->scaling, co, lin, bias, 1, e->natoms, e->d_binum, e->d_ilist,
                                    e->d_numneigh, e->d_firstneigh, rcs, e->d_types, e->ntypes, e->umax, 0, (T)e->rmax, (T)e->rmin, qs,
                                    e->d_workspace, e->workspace_bytes, stream);
    }
    if (carried)
        return nep_efv_prepared<T>(etot, force, virial, e->chebyshev_size, e->n_radial, e->n_angular, e->l_max, e->num_neurons, co, w0, b0, w1, bias,
                                   e->natoms, e->d_binum, e->d_ilist, e->d_numneigh, e->d_firstneigh, rcs, e->d_types, e->ntypes, e->umax, 0, (T)e->rmax,
                                   (T)e->rmax_angular, qs, e->d_workspace, e->workspace_bytes, st);
    if constexpr (sizeof(T) == 8)
        return ai2b_nep_efv_f64(etot, force, virial, e->chebyshev_size, e->n_radial, e->n_angular, e->l_max, e->num_neurons, co, w0, b0, w1, bias, 1,
                                e->natoms, e->d_binum, e->d_ilist, e->d_numneigh, e->d_firstneigh, rcs, e->d_types, e->ntypes, e->umax, 0, e->rmax,
                                e->rmax_angular, qs, e->d_workspace, e->workspace_bytes, stream);
    else
        return ai2b_nep_efv_f32(etot, force, virial, e->chebyshev_size, e->n_radial, e->n_angular, e->l_max, e->num_neurons, co, w0, b0, w1, bias, 1,
                                e->natoms, e->d_binum, e->d_ilist, e->d_numneigh, e->d_firstneigh, rcs, e->d_types, e->ntypes, e->umax, 0, (T)e->rmax,
                                (T)e->rmax_angular, qs, e->d_workspace, e->workspace_bytes, stream);
}

extern "C" int ai2b_evaluate(const ai2b_evaluation *e, const void *d_coords, void *stream)
{
    AI2B_REQUIRE(e && (d_coords || e->natoms == 0), AI2B_ERR_INVALID, "ai2b_evaluate: NULL argument");
    return e->is_f64 ? evaluate_t<double>(e, (const double *)d_coords, stream) : evaluate_t<float>(e, (const float *)d_coords, stream);
}

// Copy by a kernel that is part of the chain. Between two kernels a copy engine costs the hand-over there and back, several
// microseconds for a few kilobytes; either side may be pinned host memory.
__global__ void chained_copy_kernel(unsigned char *__restrict__ dst, const unsigned char *__restrict__ src, size_t bytes)
{
    chain_release();
    chain_wait();
    const size_t i0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x, step = (size_t)gridDim.x * blockDim.x;
    size_t done = 0;
    if (((reinterpret_cast<size_t>(dst) | reinterpret_cast<size_t>(src)) & 15) == 0) {
        for (size_t i = i0; i < bytes / 16; i += step) reinterpret_cast<int4 *>(dst)[i] = reinterpret_cast<const int4 *>(src)[i];
        done = bytes & ~size_t(15);
    }
    for (size_t i = done + i0; i < bytes; i += step) dst[i] = src[i];
}

extern "C" int ai2b_chained_copy(void *dst, const void *src, size_t bytes, void *stream)
{
    if (bytes == 0) return AI2B_OK;
    AI2B_REQUIRE(dst && src, AI2B_ERR_INVALID, "ai2b_chained_copy: NULL argument");
    // Few blocks: every SM that takes part has to reach the host's memory first (14 KB in one block of 1,024 threads or in four of
    // 256: a recorded call of 1,157 atoms 27.1 against 28.7 us, and its time depends less on where the blocks land)
    constexpr int THREADS = 1024;
    size_t blocks = (bytes + 16 * THREADS - 1) / (16 * THREADS);
    if (blocks > 148) blocks = 148;
    AI2B_CUDA(launch_chained(chained_copy_kernel, (unsigned)blocks, THREADS, 0, (cudaStream_t)stream, (unsigned char *)dst, (const unsigned char *)src, bytes));
    return AI2B_OK;
}
