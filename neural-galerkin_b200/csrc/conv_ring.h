// The ring of shared-memory stages of the convolution's tile kernels, as a producer warp walks it.  Plain C++: the
// kernels run it on the device, tests on the host.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define NGS_RING_FN __host__ __device__ __forceinline__
#else
#define NGS_RING_FN inline
#endif

// Steps whose copies may be in flight when the walk ends: first .. last - 1, step r in stage r % stages, its full
// barrier's phase of parity (r / stages) & 1.
struct RingSpan {
  int first, last;
};

// One step a stage, in order, until next() has no more valid elements (a step of its own, without copies: the end
// marker).  acquire(stage, parity, fresh) waits until the stage's step of the round before is consumed -- which its
// copies have landed for; there is none in a fresh stage -- and false gives up; issue(stage, valid) hands the stage its
// copies, or the marker (valid 0).
// Where the walk gives up, or the marker is the step that waited, copies of the steps before are still on their way:
// all issued ones but those that a later step of the same stage waited for.
template <typename Next, typename Acquire, typename Issue>
NGS_RING_FN RingSpan ring_walk(int stages, Next&& next, Acquire&& acquire, Issue&& issue) {
  int st = 0, begun = 0, copies = 0;
  uint32_t parity = 1u;                        // of the round before this one
  for (bool more = true; more;) {
    const int valid = next();
    more = valid > 0;
    if (!acquire(st, parity, begun < stages)) break;
    issue(st, valid);
    begun++;
    if (more) copies++;
    if (++st == stages) {
      st = 0;
      parity ^= 1u;
    }
  }
  return {begun > stages ? begun - stages : 0, copies};
}
