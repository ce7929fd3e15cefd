// pair_loop.h -- the loop in which two warps take groups together (the batched group walk on
// two warps per group).  Apart from the kernels so that a host program can run it.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define GSIM_PAIR_FN __device__ __forceinline__
#else
#define GSIM_PAIR_FN inline
#endif

namespace gsim {

// Shared by the two warps; failed is zero before the loop.
struct PairTurn {
    uint32_t unit;    // the group of this turn
    uint32_t failed;  // a wait of one of the warps ran out
};

// Runs walk(unit) on both warps for the units that the leading one takes, until one is not
// below `total` or a walk returns false (a bounded wait on the other warp ran out).  One side
// may give up where the other, only slow, finishes its walk and comes back for the next unit,
// so neither leaves the loop alone: the one that failed says so and both leave after the next
// barrier, which therefore always has both.  sync: a barrier of the two warps that also orders
// their shared memory.
template <class Take, class Sync, class Walk>
GSIM_PAIR_FN void pair_loop(PairTurn& turn, bool lead, uint32_t total, Take&& take, Sync&& sync, Walk&& walk) {
    for (bool ok = true;;) {
        if (!ok) turn.failed = 1u;
        if (lead) turn.unit = take();
        sync();
        const uint32_t u = turn.failed ? total : turn.unit;
        sync();  // read by both before either writes the next turn
        if (u >= total) return;
        ok = walk(u);
    }
}

}  // namespace gsim
