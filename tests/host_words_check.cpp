// Host check of HostWords (csrc/b2m_context.h) against a fake of the CUDA
// runtime: a call ends early, its kernel still owes a publication, and the
// next call takes the same slot.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>

// device-only names that the field header mentions
#define __noinline__
static unsigned __funnelshift_l(unsigned, unsigned hi, unsigned) { return hi; }

#include "b2m_context.h"

using namespace b2m;

static HostLen owed;           // a kernel's publication that has not landed yet
static u64 owed_value;
static int syncs = 0;

static void land() {
    if (!owed.host) return;
    owed.host[1] = owed_value;
    owed.host[0] = owed.tag;
    owed = {};
}

extern "C" {
cudaError_t cudaStreamSynchronize(cudaStream_t) {
    ++syncs;
    land();
    return cudaSuccess;
}
cudaError_t cudaStreamQuery(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    *p = calloc(1, n);
    return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFreeHost(void* p) {
    if (owed.host == p) {
        std::puts("freed under a kernel that still writes it");
        std::exit(1);
    }
    free(p);
    return cudaSuccess;
}
}

static int fails = 0;
static void expect(bool ok, const char* what) {
    if (!ok) {
        std::printf("FAILED: %s\n", what);
        ++fails;
    }
}

// A call that launches a publishing kernel and ends without waiting for it.
static u64* abandoned(Context* c, u64 value) {
    HostWords w(c, nullptr);
    owed = w.next();
    owed_value = value;
    return w.words();
}

int main() {
    Context c;
    static u64 slots[64 * 8];
    c.hw = slots;
    u64* slot = abandoned(&c, 1111);
    {
        HostWords w(&c, nullptr);
        expect(w.words() == slot, "the next call takes the slot that was given back");
        const HostLen l = w.next();
        land();  // the late publication, if it is still owed
        expect(w.words()[0] != l.tag, "a late publication has not the next call's tag");
        l.host[1] = 2222;
        l.host[0] = l.tag;
        expect(w.wait() == cudaSuccess && w.words()[1] == 2222, "the next call reads its own value");
    }
    abandoned(&c, 3333);
    {
        HostWords w(&c, nullptr);
        const HostLen l = w.next();
        l.host[1] = 4444;
        l.host[0] = l.tag;
        land();  // after the next call's own
        expect(w.wait() == cudaSuccess && w.words()[1] == 4444, "nothing lands on the next call's words");
    }
    // a call that waited for its last publication gives its slot back at once
    const int before = syncs;
    {
        HostWords w(&c, nullptr);
        w.next();  // launched and not waited for, but a later one is
        const HostLen l = w.next();
        l.host[0] = l.tag;
        expect(w.wait() == cudaSuccess, "wait");
    }
    expect(syncs == before, "no synchronisation after a wait");
    // all slots taken: words of its own
    c.hw_used = ~0ull;
    abandoned(&c, 5555);
    expect(!owed.host, "own words are not freed under a kernel");
    std::puts(fails ? "failed" : "ok");
    return fails != 0;
}
