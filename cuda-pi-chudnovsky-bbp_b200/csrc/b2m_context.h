// b2m_context.h -- the process-wide library context (one device).
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <mutex>
#include <string>
#include <vector>

#include "b2m.h"
#include "b2m_internal.h"

namespace b2m {

struct Context {
    int device = -1;
    int sm_count = 0;
    uint64_t budget = 0;                 // bytes the library may hold on the device
    std::atomic<uint64_t> in_use{0};     // bytes currently reserved against the budget
    u64* d_tables = nullptr;             // dtw | u1 | u2, resident
    RootTables tw{};
    u32* d_err = nullptr;                // sticky device error word (bounded waits)
    cudaStream_t hstream = nullptr;      // stream of the host-buffer entry point
    cudaStream_t hcopy = nullptr;        // its second operand's H2D copy (overlaps operand A's transform)
    cudaEvent_t hev_a = nullptr, hev_b = nullptr;  // operand A / operand B resident
    std::mutex host_mu;                  // serialises b2m_mul_host (shared buffers)
    void* host_dev = nullptr;            // device buffers of b2m_mul_host, grown on demand
    uint64_t host_dev_cap = 0;
    // Pinned host words that kernels publish lengths and carries in
    // (HostWords below): 64 slots of eight words, a bit per slot in use, and
    // the last tag that a slot's users gave out.
    u64* hw = nullptr;
    uint64_t hw_used = 0;
    u64 hw_tag[64] = {};
    std::mutex hw_mu;
    // Inter-pass twiddle tables (twtable_ensure), keyed by (logm, logr).
    struct TwTable {
        int logm, logr;
        u64* fwd;
        u64* inv;
        uint64_t bytes;
        // inv times 2^-logm, for the table's use as pass 0 of a 2^logm-point
        // transform (the inverse pass 0 then applies N^-1 for free); built by
        // twtable_ensure for pass 0, null until then or if the budget is short
        u64* inv0 = nullptr;
        uint64_t inv0_bytes = 0;
    };
    std::mutex twt_mu;
    std::vector<TwTable> twt;
    // Residue-transform tables (rns_launch.cu, under twt_mu): T and its
    // inverses of 2^rns_log entries per prime, small from the start, larger on
    // first need; and the tables of weighted parts, per (q, m).
    uint2* rns_t = nullptr;
    uint2* rns_base = nullptr;
    std::vector<std::pair<uint2*, uint64_t>> rns_grown;  // all but the first, and their bytes
    int rns_log = 0;
    struct RnsWeights {
        int q, m;
        uint2* mem;
        uint64_t bytes;
        const uint2* tree[2];  // forward, inverse
        const uint2* col[2];
    };
    std::vector<RnsWeights> rns_weights;
    // Autotuned plan per transform length (b2m_autotune, batch autotune);
    // used by every product of that length once set.
    std::mutex tune_mu;
    Plan tuned[MAX_LOGN + 1];
    bool has_tuned[MAX_LOGN + 1];
    Context() {
        for (int i = 0; i <= MAX_LOGN; ++i) has_tuned[i] = false;
    }
};

// The plan products of (sub-)transform length 2^logn use: the tuned one if
// any, else the default (three: the radix-3 products' default). need: the
// limbs of the longest product, when known.
inline Plan plan_for(Context* c, int logn, int three = 0, uint64_t need = 0) {
    Plan p;
    {
        std::lock_guard<std::mutex> lk(c->tune_mu);
        p = c->has_tuned[logn] ? c->tuned[logn] : make_plan(logn, three);
    }
    p.three = three;
    p.need = need;
    rns_resolve(c, p, nullptr, false);
    return p;
}
// The plan of an na x nb product: 2^L points, or 3 * 2^(L-2) when that holds
// the 2(na + nb) digits (choose_length), its sub-transform the tuned or
// default plan of that length.
inline Plan product_plan(Context* c, uint64_t na, uint64_t nb) {
    int logn = 0, three = 0;
    choose_length(2 * (na + nb), &logn, &three);
    return plan_for(c, logn, three, na + nb);
}
inline void set_tuned(Context* c, int logn, const Plan& p) {
    std::lock_guard<std::mutex> lk(c->tune_mu);
    c->tuned[logn] = p;
    c->tuned[logn].need = 0;
    c->has_tuned[logn] = true;
}

// A slot of pinned host words for one call on stream s: a kernel writes values
// 1..7, a system-wide fence and then the tag in word 0; the host polls the tag.
// Any number of calls may hold slots; past 64 at a time a call pins its own.
// A slot is given back when no kernel owes it a publication any more: a call
// that ends early, with its last one not waited for, waits for its stream.
// (The words of that publication would land on the next call's, or in freed
// memory.) Tags go on from the slot's last one, so none is ever met twice.
class HostWords {
public:
    HostWords(Context* c, cudaStream_t s) : c_(c), s_(s) {
        std::lock_guard<std::mutex> lk(c->hw_mu);
        for (int i = 0; i < 64 && c->hw; ++i)
            if (!((c->hw_used >> i) & 1)) {
                c->hw_used |= 1ull << i;
                slot_ = i;
                p_ = c->hw + 8 * i;
                tag_ = seen_ = c->hw_tag[i];
                break;
            }
        if (!p_ && cudaHostAlloc(reinterpret_cast<void**>(&p_), 64, cudaHostAllocMapped) != cudaSuccess) p_ = nullptr;
        if (p_) p_[0] = 0;
    }
    ~HostWords() {
        if (seen_ != tag_) cudaStreamSynchronize(s_);
        if (slot_ >= 0) {
            std::lock_guard<std::mutex> lk(c_->hw_mu);
            c_->hw_tag[slot_] = tag_;
            c_->hw_used &= ~(1ull << slot_);
        } else if (p_) {
            cudaFreeHost(p_);
        }
    }
    HostWords(const HostWords&) = delete;
    HostWords& operator=(const HostWords&) = delete;
    u64* words() const { return p_; }  // null: pinning failed
    // The next publication; its kernel gets words() and the tag.
    HostLen next() { return {reinterpret_cast<unsigned long long*>(p_), ++tag_}; }
    // Waits for the last one, and with it for all before it. The stream is
    // asked now and then, so that a failed or finished stream without the tag
    // is an error, not a hang.
    cudaError_t wait() {
        volatile u64* v = p_;
        for (uint32_t n = 1; v[0] != tag_; ++n) {
            if ((n & 0xFFF) == 0) {
                const cudaError_t q = cudaStreamQuery(s_);
                if (q == cudaSuccess && v[0] == tag_) break;
                if (q != cudaErrorNotReady) return q == cudaSuccess ? cudaErrorUnknown : q;
            }
        }
        seen_ = tag_;
        std::atomic_thread_fence(std::memory_order_acquire);
        return cudaSuccess;
    }

private:
    Context* c_;
    cudaStream_t s_;
    int slot_ = -1;
    u64* p_ = nullptr;
    u64 tag_ = 0, seen_ = 0;  // given out, and waited for
};

extern Context* g_ctx;
extern std::mutex g_ctx_mu;

Context* ctx();
void set_error(const std::string& msg);
b2m_status cuda_status(cudaError_t e, const char* what);
int ilog2_pow2(uint64_t n);
uint64_t ntt_length_of(uint64_t na, uint64_t nb);
bool budget_reserve(Context* c, uint64_t bytes);
void budget_release(Context* c, uint64_t bytes);
b2m_status check_sizes(uint64_t na, uint64_t nb, int* logn);

// Reads and clears the device error word (caller has synchronised).
inline b2m_status take_device_error(Context* c) {
    u32 h = 0;
    cudaError_t e = cudaMemcpy(&h, c->d_err, sizeof(u32), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_status(e, "cudaMemcpy(error word)");
    if (h) {
        cudaMemset(c->d_err, 0, sizeof(u32));
        set_error("carry lookback wait exceeded its bound");
        return B2M_ERR_DEVICE_TIMEOUT;
    }
    return B2M_OK;
}

}  // namespace b2m
