// The waits that one of several issuing warps makes before it forms the products of k block kb from a ring of stages into a ring of
// sums.  Plain C++, so that tests can walk the order on the host as the kernel does (tests/test_issue_turns.py).
//
// A wait names a parity, and a parity two uses old looks like the present one: a wait for a use is right only if the use before it is
// known to be over.  The warp that takes block kb has not seen block kb - stages of the same stage where that was another warp's, and
// planes that TMA brings for two blocks may land in either order.  So it first waits until the stage has been given back by block
// kb - stages: that its use before was over is known from the warp's own last block, whose splitting warps had to see it, while there
// are no more warps than stages.  What was given back had been full, so the wait for `full` cannot take the old use for the new one.
// The sums are drained in order, by warps that the warp's own last block waited for, so one wait does for them.
#pragma once

#ifdef __CUDACC__
#define RING_HD __device__ __forceinline__
#else
#define RING_HD inline
#endif

enum RingBarrier { RING_STAGE_EMPTY = 0, RING_STAGE_FULL = 1, RING_SUM_EMPTY = 2 };

// `wait(barrier, index, parity)` returns false when it gave up; so does this, at once.
template <class Wait>
RING_HD bool ring_issue_turn(int kb, int stages, int sums, Wait wait) {
  const int s = kb % stages, buf = kb % sums;
  const unsigned use = (unsigned)(kb / stages) & 1u, sum_use = (unsigned)(kb / sums) & 1u;
  return wait(RING_STAGE_EMPTY, s, use ^ 1u) && wait(RING_STAGE_FULL, s, use) && wait(RING_SUM_EMPTY, buf, sum_use ^ 1u);
}
