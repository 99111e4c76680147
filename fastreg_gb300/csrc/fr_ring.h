// fr_ring.h -- the order of a staging ring's fills, and the wait that ends them.
//
// Header-only, plain C++ outside nvcc: the TMA-staged kernels include it through fr_tma.cuh, and a
// CPU test compiles it on its own against a model of the slots' barriers.
#pragma once

#ifdef __CUDACC__
#define FR_RING_FN __device__ __forceinline__
#else
#define FR_RING_FN inline
#endif

namespace frg {

// A ring of `S` slots filled in order by one producer thread: fill n of the block's
// stream of fills goes to slot n % S, and the k-th fill of a slot completes phase k of its
// barrier (parity k & 1).
template <int S>
struct SliceRing {
    FR_RING_FN static int slot(unsigned n) { return (int)(n % S); }
    FR_RING_FN static unsigned parity(unsigned n) { return (n / S) & 1u; }
};

// Waits, by wait(slot, parity), for every copy that may be in flight after `issued` fills: the last
// fill of each slot (a slot is filled again only after its fill before has landed).  A block that gives up
// calls it before its shared memory goes.  It needs the number of fills issued and
// nothing else: which of them the block has waited for, and whether one of those waits failed, does
// not matter, since waiting again for a phase that has completed returns at once.
template <int S, typename Wait>
FR_RING_FN void drain_fills(unsigned issued, Wait wait) {
    for (unsigned n = issued > (unsigned)S ? issued - (unsigned)S : 0u; n < issued; ++n)
        wait(SliceRing<S>::slot(n), SliceRing<S>::parity(n));
}

}  // namespace frg
