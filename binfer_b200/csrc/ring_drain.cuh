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

// One place that a thread fills again and again, each time once the copy before has landed.  Where a wait for
// one gave up, that copy is still on its way: no other may be asked for (its barrier's phase is open, its
// place is in use), and the thread waits for it at the end.
struct OnePlace {
  unsigned asked = 0;
  template <class Ask>
  BF_HOST_DEVICE void fill(bool gave_up, Ask ask) {
    if (gave_up) return;
    ask();
    ++asked;
  }
  template <class Landed>
  BF_HOST_DEVICE void drain(Landed landed) const {
    ring_drain(1, 0, asked & 1u, landed);
  }
};
