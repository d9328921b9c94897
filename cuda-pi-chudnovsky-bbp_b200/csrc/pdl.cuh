// pdl.cuh -- programmatic dependent launch.
//
// The kernels of one product follow each other on a stream and most are a few
// microseconds long at the sizes that trees and Newton steps use, so the gap
// between a kernel's end and the next one's first instruction is a large part
// of the product. launch_pdl lets a kernel's blocks be set up while the
// kernel before it is finishing. Every kernel launched this way calls
// pdl_enter() before it touches memory that an earlier kernel may write or
// read: it returns once all earlier kernels have completed and their writes
// are visible, so nothing is reordered.
//
// "Visible" holds for ordinary loads. Such a kernel is resident while earlier
// ones still write, so what they write is not read-only for its lifetime, and
// it must not promise that: no __ldg (ld.global.nc) and no __restrict__ on
// operands, results, lengths and job tables. A load under either promise is
// outside the guarantee, and the compiler may move it above the wait. The
// resident twiddle tables, complete before any kernel sees them, are the only
// memory read that way.
#pragma once
#include <cuda_runtime.h>

namespace b2m {

__device__ __forceinline__ void pdl_enter() {
#if defined(__CUDA_ARCH__)
    asm volatile("griddepcontrol.launch_dependents;\n\tgriddepcontrol.wait;" ::: "memory");
#endif
}

template <typename... P, typename... A>
cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace b2m
