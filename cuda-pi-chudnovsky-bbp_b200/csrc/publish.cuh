// publish.cuh -- a kernel's result for the host that polls for it.
#pragma once
#include "b2m_internal.h"

namespace b2m {

// host[1] = v and host[2] = w, visible before host[0] = tag.
__device__ __forceinline__ void publish(const HostLen& hl, unsigned long long v, unsigned long long w = 0) {
    volatile unsigned long long* h = hl.host;
    h[1] = v;
    h[2] = w;
    __threadfence_system();
    h[0] = hl.tag;
}

}  // namespace b2m
