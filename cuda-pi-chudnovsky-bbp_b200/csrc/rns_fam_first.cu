// rns_fam_first.cu -- instantiations of the residue transforms' first forward
// pass (radix exponents 5..10).
#include "rns_kernels.cuh"

namespace b2m {

template <int LOGR>
static cudaError_t launch(dim3 grid, cudaStream_t s, const RnsArgs& a) {
    k_rns_first<LOGR><<<grid, RnsCol<LOGR>::THREADS, RnsCol<LOGR>::SMEM * 4, s>>>(a);
    return cudaGetLastError();
}

cudaError_t rns_launch_first(int logr, dim3 grid, cudaStream_t s, const RnsArgs& a) {
    switch (logr) {
        case 5: return launch<5>(grid, s, a);
        case 6: return launch<6>(grid, s, a);
        case 7: return launch<7>(grid, s, a);
        case 8: return launch<8>(grid, s, a);
        case 9: return launch<9>(grid, s, a);
        case 10: return launch<10>(grid, s, a);
    }
    return cudaErrorInvalidValue;
}

}  // namespace b2m
