// A wait that ends the same way for every lane of a warp.  A bounded wait can
// succeed in one lane and run out in its neighbour, and a lane can read the
// abort flag a moment before or after it is set; lanes that decided alone would
// then part -- some at the warp's next barrier, some at the CTA's -- and wait
// for one another without limit.  So the lanes vote: all go on, or all leave.
#pragma once

#ifdef __CUDACC__
#define GX_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define GX_HOST_DEVICE inline
#endif

namespace gx {

// wait: this lane's bounded wait (true: it succeeded); aborted: this lane's view
// of the abort flag, read after the wait; all: true in every lane if every
// lane's argument is.
template <class Wait, class Aborted, class All>
GX_HOST_DEVICE bool warp_agrees(Wait wait, Aborted aborted, All all)
{
  const bool good = wait() && !aborted();
  return all(good);
}

}  // namespace gx
