// Waits on mbarriers that end: a CTA whose wait has run out of time gives up all its waits, goes on without what it waited for (its outputs are not
// valid) and leaves a word in host memory, which dl_attention_status() tells of.  Loops around waits are finite, so the kernel ends.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

// argument of a kernel that waits (dl_wait_limit)
struct WaitLimit {
    unsigned long long ns;       // from the first wait of a CTA that has failed for some time and behind the kernels ahead of it; 0: no waiting at all
    unsigned* status;            // host memory: the device's word of dl_attention_status()
};
// of a CTA, in shared memory
struct WaitState {
    unsigned long long t0;
    int gave_up;
};
// 0, or -1 where there is no host memory for the status (dl_last_error)
int dl_wait_limit(const char* who, WaitLimit* limit);

#define WAIT_DEADLINE_NS 4000000000ull
#ifndef WAIT_UNIT
#define WAIT_UNIT 0u             // number of the file: the word differs from what any other kernel left
#endif
static __device__ unsigned g_times_given_up;

__device__ __forceinline__ void wait_report(const WaitLimit& l) {
    *(volatile unsigned*)l.status = (WAIT_UNIT << 24) + ((atomicAdd(&g_times_given_up, 1u) + 1u) & 0xFFFFFFu);
    __threadfence_system();
}
// by one thread, ahead of a barrier of the CTA
__device__ __forceinline__ void wait_init(WaitState& w, const WaitLimit& l) {
    w.t0 = 0;
    w.gave_up = l.ns == 0;
    if (l.ns == 0) wait_report(l);
}
__device__ __forceinline__ bool wait_gave_up(const WaitState& w) { return *(const volatile int*)&w.gave_up != 0; }
// asked now and then by a wait that fails: is the CTA's time over?
__device__ __forceinline__ bool wait_over(WaitState& w, const WaitLimit& l) {
    if (wait_gave_up(w)) return true;
    unsigned long long now;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
    const unsigned long long t0 = atomicCAS(&w.t0, 0ull, now);
    if (t0 == 0 || (long long)(now - t0) <= (long long)l.ns) return false;
    if (atomicExch(&w.gave_up, 1) == 0) wait_report(l);
    return true;
}
// CLUSTER: what other CTAs of the cluster did ahead of the phase's end is seen too.  false: given up
template <bool CLUSTER = false>
__device__ __forceinline__ bool wait_phase(uint64_t* bar, uint32_t parity, WaitState& w, const WaitLimit& l) {
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(bar);
    for (unsigned n = 1;; n++) {
        uint32_t ok;
        if (CLUSTER)
            asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(at), "r"(parity) : "memory");
        else
            asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(at), "r"(parity) : "memory");
        if (ok) return true;
        if ((n & 0x3Fu) == 0 && (wait_gave_up(w) || ((n & 0x3FFu) == 0 && wait_over(w, l)))) return false;
    }
}
// ahead of the end of a CTA that gave up: its copies and MMAs in flight end
__device__ __forceinline__ void wait_settle() { __nanosleep(1000000); }
