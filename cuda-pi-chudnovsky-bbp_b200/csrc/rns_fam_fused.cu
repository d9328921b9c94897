// rns_fam_fused.cu -- instantiations of the residue transforms' last forward
// pass + pointwise product + first inverse pass (radix exponents 6..9).
#include "rns_kernels.cuh"

namespace b2m {

template <int LOGR>
static cudaError_t configure() {
    return cudaFuncSetAttribute(k_rns_fused<LOGR>, cudaFuncAttributeMaxDynamicSharedMemorySize, RnsLast<LOGR>::SMEM * 4);
}
cudaError_t rns_configure() {
    cudaError_t e = configure<6>();
    if (e == cudaSuccess) e = configure<7>();
    if (e == cudaSuccess) e = configure<8>();
    if (e == cudaSuccess) e = configure<9>();
    return e;
}

template <int LOGR>
static cudaError_t launch(dim3 grid, cudaStream_t s, const RnsArgs& a) {
    const u64 per = (u64)RnsLast<LOGR>::SUBS << LOGR;
    grid.x = (unsigned)((a.nt + per - 1) / per);
    return launch_pdl(k_rns_fused<LOGR>, grid, RnsLast<LOGR>::THREADS, RnsLast<LOGR>::SMEM * 4, s, a);
}

cudaError_t rns_launch_fused(int logr, dim3 grid, cudaStream_t s, const RnsArgs& a) {
    switch (logr) {
        case 6: return launch<6>(grid, s, a);
        case 7: return launch<7>(grid, s, a);
        case 8: return launch<8>(grid, s, a);
        case 9: return launch<9>(grid, s, a);
    }
    return cudaErrorInvalidValue;
}

}  // namespace b2m
