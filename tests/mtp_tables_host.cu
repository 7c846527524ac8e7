// Compiles MTP tables into host memory (malloc and memcpy take the place of the device's) and reports, as one line of
// numbers, what the kernels would read of them; with a second argument, what they would read before it is written.
// Input: int32 nm nb nt ns nmus, basic, times, mapping.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "mtp_program.cuh"

template <typename P> static cudaError_t host_malloc(P **p, size_t n) { *p = (P *)malloc(n); return cudaSuccess; }
static cudaError_t host_free(void *p) { free(p); return cudaSuccess; }
static cudaError_t host_device(int *d) { *d = 0; return cudaSuccess; }
static cudaError_t host_copy(void *d, const void *s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
#define cudaMalloc host_malloc
#define cudaFree host_free
#define cudaGetDevice host_device
#define cudaMemcpy host_copy
#include "mtp_program.cu"

struct Watched {      // an array of the tables: remembers how far it was read, and reads nothing
    int *read;
    int2 operator[](int i) const { *read = std::max(*read, i + 1); return make_int2(0, 0); }
};

int main(int argc, char **argv)
{
    std::vector<int> in;
    FILE *f = fopen(argv[1], "rb");
    for (int v; fread(&v, 4, 1, f) == 1;) in.push_back(v);
    fclose(f);
    const int nm = in[0], nb = in[1], nt = in[2], ns = in[3], nmus = in[4];
    ai2b_mtp_program *prog = nullptr;
    if (ai2b_mtp_program_create(nm, nb, &in[5], nt, &in[5 + 4 * nb], ns, &in[5 + 4 * nb + 4 * nt], nmus, &prog)) {
        fprintf(stderr, "%s\n", ai2b_last_error_string());
        return 1;
    }
    const MtpProgramDev &P = prog->dev;
    if (argc > 2) {      // operands of products and of scalars that nothing fills, adjoints that neither a row nor the list of seeds finishes
        std::vector<char> filled(nm, 0), finished(nm, 0);
        for (int m = 0; m < nb; m++) filled[m] = 1;
        for (int i = P.n_adj_const; i < P.n_constant; i++) filled[P.constant[i]] = 1;
        for (int i = 0; i < P.fwd_lev_off[P.nlev]; i++) filled[P.fwd_dst[i].x] = 1;
        for (int i = 0; i < P.n_adj_const; i++) finished[P.constant[i]] = 1;
        for (int i = 0; i < P.rev_lev_off[P.nlev]; i++) finished[P.rev_mom[i].x] = 1;
        int missing = 0;
        for (int i = 0; i < P.nt; i++) missing += !filled[P.fwd_rows[i].x & 0xffff] + !filled[P.fwd_rows[i].x >> 16 & 0xffff];
        for (int s = 0; s < P.ns; s++) missing += !filled[P.map[s]];
        for (int i = 0; i < P.adjoint_rows(); i++) missing += !finished[P.rev_ents[i].x >> 16 & 0xffff];
        printf("%d\n", missing);
        return 0;
    }
    const unsigned char *end = (const unsigned char *)prog->d_blob + prog->blob_bytes;
    std::vector<int2> to(3 * (size_t)nt);      // what the kernels keep for the rows
    const int threads = 1024;
    for (int adjoints = 0; adjoints < 2; adjoints++) {
        int fwd = 0, rev = 0;
        for (int t = 0; t < threads; t++)
            stage_product_rows(P, Watched{&fwd}, Watched{&rev}, adjoints, to.data(), t, threads, ScaledRow<17, true>());
        printf("%d %d ", fwd, rev);
    }
    // adjoint rows that the kernels' loops walk through, the room that rev_flat has, and the phases whose moments do not come with the
    // most rows first
    int unordered = 0;
    auto look = [&](const int4 *q, const int *off) {
        for (int lev = 0; lev < P.nlev; lev++) {
            bool ordered = true;
            for (int i = off[lev] + 1; i < off[lev + 1]; i++) ordered = ordered && q[i].z - q[i].y <= q[i - 1].z - q[i - 1].y;
            unordered += !ordered;
        }
    };
    look(P.fwd_dst, P.fwd_lev_off);
    look(P.rev_mom, P.rev_lev_off);
    printf("%d %ld %d\n", P.rev_lev_row[P.nlev], (long)((end - (const unsigned char *)P.rev_flat) / sizeof(int2)), unordered);
    ai2b_mtp_program_destroy(prog);
}
