// rns_fam_first.cu -- instantiations of the residue transforms' first forward
// pass: radix exponents 5..8, one or two columns per thread, and in parts (two
// columns where a thread has eight rows, one where it has sixteen).
#include "rns_kernels.cuh"

namespace b2m {

template <int LOGR, int V>
static cudaError_t launch(dim3 grid, cudaStream_t s, const RnsArgs& a) {
    using G = RnsCol<LOGR, V>;
    return launch_pdl(a.jobs ? k_rns_first<LOGR, V, true> : k_rns_first<LOGR, V, false>, grid, G::THREADS, G::SMEM * 4,
                      s, a);
}
template <int LOGR, int V>
static cudaError_t parts(dim3 grid, cudaStream_t s, const RnsArgs& a) {
    using G = RnsCol<LOGR, V>;
    return launch_pdl(a.jobs ? k_rns_first_parts<LOGR, V, true> : k_rns_first_parts<LOGR, V, false>, grid, G::THREADS,
                      2 * G::SMEM * 4, s, a);
}

cudaError_t rns_launch_first(int logr, int v, dim3 grid, cudaStream_t s, const RnsArgs& a) {
    switch (16 * (a.q > 1 ? 0 : v) + logr) {
        case 5: return parts<5, 2>(grid, s, a);
        case 6: return parts<6, 2>(grid, s, a);
        case 7: return parts<7, 1>(grid, s, a);
        case 8: return parts<8, 1>(grid, s, a);
        case 21: return launch<5, 1>(grid, s, a);
        case 22: return launch<6, 1>(grid, s, a);
        case 23: return launch<7, 1>(grid, s, a);
        case 24: return launch<8, 1>(grid, s, a);
        case 37: return launch<5, 2>(grid, s, a);
        case 38: return launch<6, 2>(grid, s, a);
        case 39: return launch<7, 2>(grid, s, a);
        case 40: return launch<8, 2>(grid, s, a);
    }
    return cudaErrorInvalidValue;
}

}  // namespace b2m
