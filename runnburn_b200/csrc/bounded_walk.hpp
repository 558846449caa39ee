// Control flow around waits that may give up, apart from the kernels that use it so that it also compiles for the host.
#pragma once

#ifdef __CUDACC__
#define RNB_WALK __device__ __forceinline__
#else
#define RNB_WALK inline
#endif

namespace rnb {

// The tiles first, first + step, ... below `tiles`, taken in turn by warps that meet at barriers inside `body`.  `wait(i)` waits
// for the i-th of them with a limit and may give up in one warp while it succeeds in another; `agree` makes the outcome
// common (true if all warps pass true), so that nobody goes on to a barrier that another warp has left.  False: some warp gave up.
template <class Wait, class Agree, class Body>
RNB_WALK bool walk_tiles(int first, int step, int tiles, Wait &&wait, Agree &&agree, Body &&body) {
    int count = 0;
    for (int tile = first; tile < tiles; tile += step, count++) {
        if (!agree(wait(count))) return false;
        body(tile);
    }
    return true;
}

// What a thread that fills a ring of `ring` slots does before it leaves, whatever came of its own waits: it waits for the last
// fill of every slot (wait(slot, parity)), so that no copy is still under way when the memory is used for something else or given
// back.  Another role may have given up although this one has not.
template <class Wait>
RNB_WALK void drain_ring(unsigned issued, unsigned ring, Wait &&wait) {
    for (unsigned i = issued > ring ? issued - ring : 0; i < issued; i++) wait(i % ring, (i / ring) & 1u);
}

}  // namespace rnb
