// A wait that may give up, and that a group of threads acts on together. (No CUDA in here: the tests
// compile it for the host too.)
#pragma once

#ifdef __CUDACC__
#define MOE_AGREE_FN __device__ __forceinline__
#else
#define MOE_AGREE_FN inline
#endif

namespace moe {

// The leader looks (it may wait, and read what others write at any time), the group follows: every
// thread of the barrier gets the leader's answer. A thread must not look for itself behind the
// barrier: with a write in between, some would leave and the others wait for them at the next one,
// for good. The leader alone writes *answer; a barrier of the group lies between two calls.
template <typename Look, typename Barrier>
MOE_AGREE_FN bool agree(bool leader, volatile int* answer, Look look, Barrier barrier) {
  if (leader) *answer = look() ? 1 : 0;
  barrier();
  return *answer != 0;
}

}  // namespace moe
