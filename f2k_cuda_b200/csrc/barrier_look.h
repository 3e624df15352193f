// A converged warp's looks at mbarriers ahead of the point where it needs them.
//
// The warp issues its MMAs from one elected lane. Having seen a barrier complete orders only the lane that
// saw it behind what the barrier covers, and a vote passes on a truth value but no memory order: every lane
// therefore looks at every barrier itself, so whichever lane is elected has acquired all of them.
// (Half of the lanes on either barrier and a __syncwarp behind the vote is as good and takes the same time:
// fused call at 4608 tokens x 32 heads 330.7 us that way, 330.2 us this way.)
//
// Ops: test(bar_a, par_a, bar_b, par_b)  this lane's look at one barrier (bar_a == bar_b) or two, no waiting
//      all(pred)                         vote over the warp
//      wait(bar, par)                    bounded wait by every lane; false on expiry, the same in every lane
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define F2K_WARP_FN __device__ __forceinline__
#else
#define F2K_WARP_FN inline
#endif

namespace f2k {

struct Look {
    uint32_t bar_a, par_a, bar_b, par_b;
    bool seen;
};

template <class Ops>
F2K_WARP_FN Look look_at(const Ops& ops, uint32_t bar_a, uint32_t par_a, uint32_t bar_b, uint32_t par_b) {
    return Look{bar_a, par_a, bar_b, par_b, ops.test(bar_a, par_a, bar_b, par_b)};
}
template <class Ops>
F2K_WARP_FN Look look_at(const Ops& ops, uint32_t bar, uint32_t par) {
    return look_at(ops, bar, par, bar, par);
}

// True once every lane is ordered behind both barriers of the look; false when a wait ran out.
template <class Ops>
F2K_WARP_FN bool finish(const Ops& ops, const Look& l) {
    if (ops.all(l.seen)) return true;
    return ops.wait(l.bar_a, l.par_a) && (l.bar_b == l.bar_a || ops.wait(l.bar_b, l.par_b));
}

}  // namespace f2k
