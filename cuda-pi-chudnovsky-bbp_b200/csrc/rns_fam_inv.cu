// rns_fam_inv.cu -- instantiations of the residue transforms' inverse column
// passes (radix exponents 5..10; the top pass and the others).
#include "rns_kernels.cuh"

namespace b2m {

template <int LOGR>
static cudaError_t launch(bool first, dim3 grid, cudaStream_t s, const RnsArgs& a) {
    if (first) k_rns_inv<LOGR, true><<<grid, RnsCol<LOGR>::THREADS, RnsCol<LOGR>::SMEM * 4, s>>>(a);
    else k_rns_inv<LOGR, false><<<grid, RnsCol<LOGR>::THREADS, RnsCol<LOGR>::SMEM * 4, s>>>(a);
    return cudaGetLastError();
}

cudaError_t rns_launch_inv(int logr, bool first, dim3 grid, cudaStream_t s, const RnsArgs& a) {
    switch (logr) {
        case 5: return launch<5>(first, grid, s, a);
        case 6: return launch<6>(first, grid, s, a);
        case 7: return launch<7>(first, grid, s, a);
        case 8: return launch<8>(first, grid, s, a);
        case 9: return launch<9>(first, grid, s, a);
        case 10: return launch<10>(first, grid, s, a);
    }
    return cudaErrorInvalidValue;
}

}  // namespace b2m
