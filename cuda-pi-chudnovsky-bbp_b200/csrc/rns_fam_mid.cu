// rns_fam_mid.cu -- instantiations of the residue transforms' middle forward
// pass (radix exponents 5..8).
#include "rns_kernels.cuh"

namespace b2m {

template <int LOGR, int V>
static cudaError_t launch(dim3 grid, cudaStream_t s, const RnsArgs& a) {
    return launch_pdl(k_rns_mid<LOGR, V>, grid, RnsCol<LOGR, V>::THREADS, RnsCol<LOGR, V>::SMEM * 4, s, a);
}

cudaError_t rns_launch_mid(int logr, int v, dim3 grid, cudaStream_t s, const RnsArgs& a) {
    switch (16 * v + logr) {
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
