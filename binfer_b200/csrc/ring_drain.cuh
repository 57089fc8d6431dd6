// Copies in flight when a kernel gives up a wait: the parities to wait for.
#pragma once

#ifdef __CUDACC__
#define BF_HOST_DEVICE __host__ __device__
#else
#define BF_HOST_DEVICE
#endif

// A thread fills the stages of a ring in turn, with `phase` flipping from round to round, and left with
// `stage` and `phase` those of the next fill.  landed(s, parity) for every stage with the parity of its last
// fill, which an mbarrier of that stage passes once that fill is complete; one that was never filled passes
// at once.  (Either parity will not do: of the two one is always passed.)
template <class Landed>
BF_HOST_DEVICE inline void ring_drain(int stages, int stage, unsigned phase, Landed landed) {
  for (int s = 0; s < stages; ++s) landed(s, s < stage ? phase : phase ^ 1u);
}
