// mbarriers: arrivals, announced bytes and bounded waits.
#pragma once

#include <cstdint>

namespace tcq {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(uint32_t mbar, uint32_t arrivals) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(arrivals) : "memory");
}
// one arrival that also announces `bytes` of asynchronous stores for the phase in progress
__device__ __forceinline__ void mbar_expect(uint32_t mbar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
}
// One poll (the hardware may park the thread briefly before answering).
__device__ __forceinline__ bool mbar_try_wait(uint32_t mbar, uint32_t parity) {
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(done) : "r"(mbar), "r"(parity) : "memory");
    return done != 0;
}
// Bounded wait: polls until the phase completes or kMbarWaitCycles SM clocks (about a quarter of a
// second) have passed, where a healthy wait takes microseconds.  The caller records the failure
// and stops exchanging metrics, so a counting bug shows up as an error status and invalid codes,
// never as a hang.  (No suspend-time hint on the poll: a hint makes every unsatisfied poll sleep
// for about that long, which cost 7 % of the kernel's throughput.)
//
// `gave_up` is a word in this CTA's shared memory, zero at launch.  The first wait that runs out
// sets it, and from then on no wait of this CTA spins: each polls twice and reports failure, so a
// launch whose protocol broke ends after about one time limit, not one per remaining wait.  The
// flag is looked at on the slow path only and lives in shared memory on purpose: the step loop sits
// at the register limit, and any extra state carried through its fast path (tried: a predicate, a
// second return value) cost 6-7 % of the kernel's throughput.
constexpr long long kMbarWaitCycles = 500000000LL;
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity, volatile unsigned int* gave_up) {
    if (mbar_try_wait(mbar, parity)) return true;
    const long long t0 = clock64();
    const long long limit = *gave_up ? 0 : kMbarWaitCycles;
    while (clock64() - t0 < limit)
        if (mbar_try_wait(mbar, parity)) return true;
    // One more poll after the deadline: a thread that was descheduled across it (time slicing, an attached
    // profiler) must not report a phase that completed meanwhile as lost.
    if (mbar_try_wait(mbar, parity)) return true;
    *gave_up = 1u;
    return false;
}
__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}

}  // namespace tcq
