// dataflow_queue.h -- the queue of the 3D dataflow sweep kernel: counters of missing dependencies, the
// ring of ready items, and what a completion does to them.  Device code; the CPU check
// tests/native/dataflow_order_check.cpp compiles it with g++ over a memory that tracks which writes
// are ordered before which reads.
//
// Who sees what.  The words of the queue are accessed by relaxed atomics, so what orders a tile's field
// and lock words before the tiles that read them are fences (M::fence, acquire and release at once):
//   a warp that processed a tile      writes, fence, decrements the dependents' counters;
//   a lane whose decrement is the last  fence (it has seen all decrements: acquire; what it pushes or
//                                     goes on with is ordered behind them: release);
//   a lane that takes an item from the ring   takes, fence.
// Without the second one the taker sees the writes of the last completer, but of the other tiles
// the item waited for only what that completer had seen before its own decrement.
#pragma once

#include "dataflow3.h"

#ifdef __CUDACC__
#define PFAST_QUEUE __device__ __forceinline__
#else
#define PFAST_QUEUE inline
#endif

namespace pfast {

constexpr unsigned kSlotEmpty = 0xffffffffu;

struct alignas(16) DataflowShared {
    unsigned head, tail;   // ring positions: next to take / next to fill
    int done;              // items completed in this outer iteration
    int abort;
    int item;
    int flags[2];          // clusters, by iteration parity: bit 0 some tile moved, bit 1 some tile due
};

// The queue words of a block or cluster: the counters, the ring and its state (cluster: in the shared
// memory of its first block, reached through distributed shared memory).
struct DataflowQueue {
    unsigned* cnt;
    unsigned* slots;
    unsigned qmask;
    DataflowShared* sh;
};

// Puts a ready item into the ring (the caller is ordered behind what made it ready, see above).
template <class M>
PFAST_QUEUE void df_push(const M& m, const DataflowQueue& Q, unsigned e) {
    const unsigned p = m.add(&Q.sh->tail, 1u);
    unsigned* slot = Q.slots + (p & Q.qmask);
    // a slot still holds an earlier round's item only while that item's taker is about to
    // exchange it out (at most ntiles <= ring size items are outstanding): wait for it
    for (int spin = 0; m.cas(slot, kSlotEmpty, e) != kSlotEmpty; ++spin)
        if (spin > (1 << 22) || m.stopped(Q)) { m.stop(Q); return; }
}

// The k-th possible dependent of item (o, x), k < 13 (dataflow3.h: dependents()): -1, or the item
// that has one missing dependency fewer.
PFAST_QUEUE int df_dependent(const TileGrid3& g, int o, int x, int k) {
    if (k == 0) return o < 7 ? (x << 3) | (o + 1) : -1;
    const int a = (k - 1) >> 2, s = ((k - 1) >> 1) & 1, later = (k - 1) & 1;
    const int y = tile_neighbour(g, x, a, s);
    if (y < 0) return -1;
    if (!later) return side_upstream(o, a, 1 - s) ? (y << 3) | o : -1;
    return o < 7 && !side_upstream(o + 1, a, 1 - s) ? (y << 3) | (o + 1) : -1;
}

// Item e has one missing dependency fewer; returns its count before.  A block keeps two 4-bit
// counters per tile, four tiles per word; a cluster (CL), whose completions would wait for the
// re-arming of one, all eight orders' counters, one word per tile.
template <bool CL, class M>
PFAST_QUEUE unsigned df_notify(const M& m, const DataflowQueue& Q, int e) {
    const int y = e >> 3;
    const unsigned shf = CL ? 4u * (unsigned)(e & 7) : 8u * (unsigned)(y & 3) + 4u * (unsigned)(e & 1);
    return (m.sub(Q.cnt + (CL ? y : y >> 2), 1u << shf) >> shf) & 15u;
}

// Re-arm x's counter of parity o for order o + 2 (it is zero: it fired for (o, x), and no
// dependency of (o + 2, x) completes before (o, x) did).
template <class M>
PFAST_QUEUE void df_rearm(const M& m, const TileGrid3& g, const DataflowQueue& Q, int o, int x) {
    if (o + 2 < 8)
        m.add(Q.cnt + (x >> 2), (unsigned)dep_count(g, o + 2, x) << (8u * (unsigned)(x & 3) + 4u * (unsigned)(o & 1)));
}

// Completion of item (o, x) by one lane: re-arm, then notify the dependents (the notifications
// are all in flight together).  Of the items that become ready, one is returned for the lane to
// go on with; the others join the ring.
template <bool CL, class M>
PFAST_QUEUE unsigned df_complete(const M& m, const TileGrid3& g, const DataflowQueue& Q, int o, int x) {
    if constexpr (!CL) {
        df_rearm(m, g, Q, o, x);
        m.fence();
    }
    int dep[13];
    unsigned old[13];
    bool ready = false;
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int k = 0; k < 13; ++k) {
        dep[k] = df_dependent(g, o, x, k);
        old[k] = dep[k] >= 0 ? df_notify<CL>(m, Q, dep[k]) : 2u;
    }
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int k = 0; k < 13; ++k) ready |= old[k] == 1u;
    if (ready) m.fence();
    unsigned keep = kSlotEmpty;
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int k = 0; k < 13; ++k) {
        if (old[k] == 1u) {
            if (keep == kSlotEmpty) keep = (unsigned)dep[k];
            else df_push(m, Q, (unsigned)dep[k]);
        } else if (old[k] == 0u) {
            m.stop(Q);   // more completions than dependencies: stop
        }
    }
    return keep;
}

// Lane `lane`'s part of a completion by a whole warp, one dependent per lane: returns its dependent if
// that became ready.  What the warp wrote is behind a warp barrier.
template <bool CL, class M>
PFAST_QUEUE unsigned df_complete_lane(const M& m, const TileGrid3& g, const DataflowQueue& Q, int o, int x, int lane) {
    const int dep = lane < 13 ? df_dependent(g, o, x, lane) : -1;
    if (dep < 0) return kSlotEmpty;
    m.fence();
    const unsigned old = df_notify<CL>(m, Q, dep);
    if (old == 0u) m.stop(Q);
    if (old != 1u) return kSlotEmpty;
    m.fence();
    return (unsigned)dep;
}

}  // namespace pfast
