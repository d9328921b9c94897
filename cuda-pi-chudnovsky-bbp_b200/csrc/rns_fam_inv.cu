// rns_fam_inv.cu -- instantiations of the residue transforms' inverse column
// passes (radix exponents 5..8; the top pass, the others, and the top pass of
// a transform in parts).
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
        case 37: return launch<5, 2>(first, grid, s, a);
        case 38: return launch<6, 2>(first, grid, s, a);
        case 39: return launch<7, 2>(first, grid, s, a);
        case 40: return launch<8, 2>(first, grid, s, a);
    }
    return cudaErrorInvalidValue;
}

template <int LOGR, int Q>
static cudaError_t parts(dim3 grid, cudaStream_t s, const RnsArgs& a, const RnsCombine& c) {
    using G = RnsCol<LOGR, 1>;
    return launch_pdl(k_rns_inv_parts<LOGR, Q>, grid, G::THREADS, 2 * G::SMEM * 4, s, a, c);
}

// 3 parts at any radix, 5 at 2^6 and below; 2, 4, 6 and 8 have 2^23-point parts.
cudaError_t rns_launch_inv_parts(int logr, dim3 grid, cudaStream_t s, const RnsArgs& a, const RnsCombine& c) {
    switch (16 * a.q + logr) {
        case 39: return parts<7, 2>(grid, s, a, c);
        case 53: return parts<5, 3>(grid, s, a, c);
        case 54: return parts<6, 3>(grid, s, a, c);
        case 55: return parts<7, 3>(grid, s, a, c);
        case 56: return parts<8, 3>(grid, s, a, c);
        case 71: return parts<7, 4>(grid, s, a, c);
        case 85: return parts<5, 5>(grid, s, a, c);
        case 86: return parts<6, 5>(grid, s, a, c);
        case 102: return parts<6, 6>(grid, s, a, c);
        case 134: return parts<6, 8>(grid, s, a, c);
    }
    return cudaErrorInvalidValue;
}

}  // namespace b2m
