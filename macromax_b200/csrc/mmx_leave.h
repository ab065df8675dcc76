// How the CTAs leave a launch in which they wait for one another (k_loop).  Plain C++: also compiled for the host.
#pragma once

#if defined(__CUDACC__)
#define MMX_LEAVE_FN __host__ __device__ __forceinline__
#else
#define MMX_LEAVE_FN inline
#endif

// Words shared by the CTAs of a launch, all 0 between launches.
enum : int { LEAVE_ARRIVED = 0, LEAVE_LEFT = 1, LEAVE_GAVE_UP = 2, LEAVE_WORDS = 3 };

struct LeaveResult {
  bool last;     // this CTA is the last one to leave: it writes the launch's results and clears the words
  bool stalled;  // (last) some CTA gave up a wait
};

// One CTA leaves.  add(word, v) adds to a word and returns what was there before, in order with everything that the CTA
// does before and after it.  A CTA that gave up says so before it is counted, so that the last one to be counted sees it,
// in whichever order they leave; the results have one writer, which writes after every other CTA has left.
template <class Add> MMX_LEAVE_FN LeaveResult leave_launch(unsigned ctas, bool gave_up, Add&& add) {
  if (gave_up) add(LEAVE_GAVE_UP, 1u);
  LeaveResult r;
  r.last = add(LEAVE_LEFT, 1u) == ctas - 1;
  r.stalled = r.last && add(LEAVE_GAVE_UP, 0u) != 0;
  return r;
}
