// How far one group of a CTA's warps has come, told to another group that follows it.
//
// The leader publishes a count, and what it wrote before that is there for whoever has seen the count.  Followers wait with a limit, and
// all of them leave a wait with the same outcome: each has a clock of its own, and if one gave up where another still saw the
// count, the two would go on to different barriers and neither of these would ever be complete.
// (Plain C++ but for the group, so that tests/handoff.cpp runs the same lines with host threads.)
#pragma once

#include <cuda/atomic>

#ifdef __CUDACC__
#define TCQ_HANDOFF __device__ __forceinline__
#else
#define TCQ_HANDOFF inline
#endif

namespace tcq {

TCQ_HANDOFF void handoff_publish(int& word, int count) { cuda::atomic_ref<int, cuda::thread_scope_block>(word).store(count, cuda::memory_order_release); }

// Whether `word` has come to `count`, the same answer in every thread of the group g:
//   g.clock()   this thread's clock, `limit` of which a wait may take
//   g.pause()   between two looks
//   g.all(x)    barrier of the group; whether x holds in all of its threads
template <class Group>
TCQ_HANDOFF bool handoff_wait(Group& g, int& word, int count, long long limit) {
    auto come = [&] { return cuda::atomic_ref<int, cuda::thread_scope_block>(word).load(cuda::memory_order_acquire) >= count; };
    bool there = come();
    if (!there) {
        // (the word is looked at after the clock: a thread that was held up across the limit does not report as missing what has come meanwhile)
        const long long t0 = g.clock();
        for (bool late = false; !(there = come()) && !late; late = g.clock() - t0 >= limit) g.pause();
    }
    return g.all(there);
}

}  // namespace tcq
