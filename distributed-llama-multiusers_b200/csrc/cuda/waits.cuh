// Waits on mbarriers that end: a thread whose wait has run out of time goes on without what it waited for, hardly waits any more, frees and fills no stage, and
// leaves a word in host memory, which dl_attention_status() tells of: the outputs are not valid.  Loops around waits are finite, so the kernel ends.
//
// There is no state but the thread's own, and the limit comes last among a kernel's arguments and is read on the slow path alone: what a launch here pays for are
// cold reads and shared stores ahead of its first copies, registers, and arguments themselves (decode attention of 8 rows, launched alone, 7.6 us, 8.2 with 16
// bytes more).  The kernel's parameter has to be a __grid_constant__: a reference to it copies all of it to the stack otherwise.  Kernels that
// stream weights let a warp that only issues copies watch over the other roles' waits (gemv_q40.cu, gemm_q40_tc.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

// argument of a kernel that waits (dl_wait_limit)
struct WaitLimit {
    unsigned long long ns;       // how long (attention_prefill_tc.cu: a CTA in all)
    unsigned* status;            // host memory: the device's word of dl_attention_status()
};
// 0, or -1 where there is no host memory for the status (dl_last_error); dev: the current device where the caller knows it
int dl_wait_limit(const char* who, WaitLimit* limit, int dev = -1);

#define WAIT_DEADLINE_NS 4000000000ull
#ifndef WAIT_UNIT
#define WAIT_UNIT 0u             // number of the file: the word differs from what any other kernel left
#endif
static __device__ unsigned g_times_given_up;

static __device__ __noinline__ void wait_report(const WaitLimit& l) {
    *(volatile unsigned*)l.status = (WAIT_UNIT << 24) + ((atomicAdd(&g_times_given_up, 1u) + 1u) & 0xFFFFFFu);
    __threadfence_system();
}
__device__ __forceinline__ bool wait_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// of a wait that has failed for some time: the time counts from here on, and from the end of the kernels ahead (which this one may have started under);
// a thread that has given up a wait before has none left
static __device__ __noinline__ bool wait_slow(uint32_t bar, uint32_t parity, const WaitLimit& l, bool alive) {
    unsigned long long t0, now;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    do {
        for (int n = 0; n < 256; n++)
            if (wait_try(bar, parity)) return true;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
    } while (alive && now - t0 < l.ns);
    if (alive) wait_report(l);
    return false;
}
// false: given up.  alive: the thread has given up no wait before
__device__ __forceinline__ bool wait_phase(uint64_t* bar, uint32_t parity, const WaitLimit& l, bool alive) {
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(bar);
    for (unsigned n = 0; !wait_try(at, parity);)
        if (++n == 1024) return wait_slow(at, parity, l, alive);
    return true;
}
// ahead of the end of a thread that gave up: copies in flight land
static __device__ __noinline__ void wait_settle() {
    unsigned long long t0, now;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    do {
        __nanosleep(100000);
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
    } while (now - t0 < 1000000);
}
