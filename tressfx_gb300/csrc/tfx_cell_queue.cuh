// The queue in which a construct warp collects the cells it has to evaluate: 64 entries of shared memory, to which
// the lanes that keep a cell add theirs, and from which the warp takes 32 at a time.  Plain C++ but for its warp
// (ballot, sync) and its entries, so that the order of its accesses can be checked off the device.
//
// An entry is touched by different lanes from one use to the next, so every such pair of accesses has a sync()
// between them; a ballot brings the lanes together but orders no memory.
#pragma once
#include <cuda_runtime.h>

#if defined(__CUDACC__)
#define TFX_LANE_FN __device__ __forceinline__
#else
#define TFX_LANE_FN inline
#endif

namespace tfx {

#if defined(__CUDACC__)
struct DeviceWarp {
    TFX_LANE_FN static unsigned ballot(bool p) { return __ballot_sync(0xffffffffu, p); }
    TFX_LANE_FN static void sync() { __syncwarp(); }
    TFX_LANE_FN static int count(unsigned m) { return __popc(m); }
};
#endif

// One lane's hold of the queue, a ring.  `entries`: what entries[i] reads and writes.
template <class Warp, class Entries>
struct CellQueue {
    Entries entries;
    int lane;
    unsigned head = 0, held = 0;   // the first entry (0 or 32) and how many there are, the same in every lane

    // All lanes call it; those with `keep` add `e`.  At most 31 entries are held before it.
    TFX_LANE_FN void add(bool keep, uint2 e) {
        const unsigned m = Warp::ballot(keep);
        if (keep) entries[(head + held + Warp::count(m & ((1u << lane) - 1u))) & 63u] = e;
        held += Warp::count(m);
    }
    TFX_LANE_FN bool full() const { return held >= 32; }
    // All lanes call it when full(): a lane's own of the first 32 entries.
    TFX_LANE_FN uint2 take() {
        Warp::sync();
        const uint2 e = entries[head + lane];
        Warp::sync();   // what is added next may go into these entries
        head ^= 32u;
        held -= 32;
        return e;
    }
    // All lanes call it at the end: whether the lane has one of the remaining entries.
    TFX_LANE_FN bool last(uint2& e) {
        Warp::sync();
        const bool mine = (unsigned)lane < held;
        if (mine) e = entries[head + lane];
        Warp::sync();
        return mine;
    }
};

}  // namespace tfx
