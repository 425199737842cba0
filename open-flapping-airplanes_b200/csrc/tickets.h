// Where a ticket of a job lies. Plain C++, so that it is tested on the host.
#pragma once
#ifdef __CUDACC__
#define OFA_HD __host__ __device__ __forceinline__
#else
#define OFA_HD inline
#endif

namespace ofa {

// The place of ticket g within its step, for a block whose last ticket was of step `step`, the first ticket of which is `first`; both move on. A block's
// tickets grow by little, but one that gets its place on an SM late may find its first ticket anywhere in a launch (up to 4.0e9 of them): a difference of
// tickets does not fit an int, and the steps passed by are not walked.
OFA_HD unsigned place_ticket(unsigned g, unsigned per_step, int& step, unsigned& first) {
  unsigned r = g - first;
  if (r >= per_step) {
    unsigned n = 1;
    r -= per_step;
    if (r >= per_step) { const unsigned q = r / per_step; n += q; r -= q * per_step; }
    step += (int)n;
    first += n * per_step;
  }
  return r;
}

}  // namespace ofa
