// rns_fam_inv.cu -- instantiations of the residue transforms' inverse column
// passes (radix exponents 5..10; the top pass and the others).
#include "rns_kernels.cuh"

namespace b2m {

template <int LOGR, int V>
static cudaError_t launch(bool first, dim3 grid, cudaStream_t s, const RnsArgs& a) {
    using G = RnsCol<LOGR, V>;
    return launch_pdl(first ? k_rns_inv<LOGR, V, true> : k_rns_inv<LOGR, V, false>, grid, G::THREADS, G::SMEM * 4, s,
                      a);
}

cudaError_t rns_launch_inv(int logr, int v, bool first, dim3 grid, cudaStream_t s, const RnsArgs& a) {
    switch (16 * v + logr) {
        case 21: return launch<5, 1>(first, grid, s, a);
        case 22: return launch<6, 1>(first, grid, s, a);
        case 23: return launch<7, 1>(first, grid, s, a);
        case 24: return launch<8, 1>(first, grid, s, a);
        case 25: return launch<9, 1>(first, grid, s, a);
        case 26: return launch<10, 1>(first, grid, s, a);
        case 37: return launch<5, 2>(first, grid, s, a);
        case 38: return launch<6, 2>(first, grid, s, a);
        case 39: return launch<7, 2>(first, grid, s, a);
        case 40: return launch<8, 2>(first, grid, s, a);
    }
    return cudaErrorInvalidValue;
}

}  // namespace b2m
