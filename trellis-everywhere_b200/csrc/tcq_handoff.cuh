// How far one group of a CTA's warps has come, told to another group that follows it.
//
// The leader publishes a count, and what it wrote before that is there for whoever has seen the count.
// (Plain C++, so that tests/handoff.cpp runs the same lines with host threads.)
#pragma once

#include <cuda/atomic>

#ifdef __CUDACC__
#define TCQ_HANDOFF __device__ __forceinline__
#else
#define TCQ_HANDOFF inline
#endif

namespace tcq {

TCQ_HANDOFF void handoff_publish(int& word, int count) { cuda::atomic_ref<int, cuda::thread_scope_block>(word).store(count, cuda::memory_order_release); }

TCQ_HANDOFF int handoff_count(int& word) { return cuda::atomic_ref<int, cuda::thread_scope_block>(word).load(cuda::memory_order_acquire); }

}  // namespace tcq
