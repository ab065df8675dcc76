// How the CTAs leave a launch in which they wait for one another (k_loop).  Plain C++: also compiled for the host.
#pragma once

#if defined(__CUDACC__)
#define MMX_LEAVE_FN __host__ __device__ __forceinline__
#else
#define MMX_LEAVE_FN inline
#endif

// Words shared by the CTAs of a launch, all 0 between launches: arrivals at the barrier; CTAs that have left, and those of
// them that gave up in the upper half (so at most 65535 CTAs).
enum : int { LEAVE_ARRIVED = 0, LEAVE_LEFT = 1, LEAVE_WORDS = 2 };
constexpr unsigned kLeaveGaveUp = 1u << 16;

struct LeaveResult {
  bool last;     // this CTA is the last one to leave: it writes the launch's results and clears the words
  bool stalled;  // (last) some CTA gave up a wait
};

// One CTA leaves.  add(word, v) adds to a word, after everything that the CTA did, and returns what was there before.  A CTA
// that gave up says so as it is counted, so that the last one sees it in whichever order they leave; the results have one
// writer, which writes after every other CTA has left.
template <class Add> MMX_LEAVE_FN LeaveResult leave_launch(unsigned ctas, bool gave_up, Add&& add) {
  const unsigned before = add(LEAVE_LEFT, gave_up ? kLeaveGaveUp + 1u : 1u);
  LeaveResult r;
  r.last = (before & (kLeaveGaveUp - 1u)) == ctas - 1;
  r.stalled = r.last && (gave_up || before >= kLeaveGaveUp);
  return r;
}
