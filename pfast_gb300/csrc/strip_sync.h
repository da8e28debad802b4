// strip_sync.h -- how the warps of the 2D strips schedule hand over tiles to one another.  Device code;
// the CPU check tests/native/strip_sync_check.cpp compiles it with g++ over a memory that tracks
// which accesses are ordered before which.
//
// Every lane of a warp stores field values that lanes of other warps read (the rows facing the next
// strip), while one lane stores and one lane polls the progress words.  A shuffle or a reduction
// between lanes orders no memory, so a warp barrier stands between the lanes' accesses and the
// fence of the lane that publishes, and between the fence of the lane that polled and the lanes' accesses.
#pragma once

#ifdef __CUDACC__
#define PFAST_STRIP __device__ __forceinline__
#else
#define PFAST_STRIP inline
#endif

namespace pfast {

// *word = value, behind every access of the warp's lanes so far.  W: the calling lane's view of its warp.
template <class W>
PFAST_STRIP void strip_publish(const W& w, volatile int* word, int value) {
    w.barrier();
    if (w.leader()) {
        w.fence();
        w.store(word, value);
    }
}

// Waits until *word >= want, in front of every later access of the warp's lanes; false: given up.
template <class W>
PFAST_STRIP bool strip_wait(const W& w, volatile int* word, int want) {
    int ok = 1;
    if (w.leader()) {
        ok = w.poll(word, want);
        w.fence();
    }
    ok = w.broadcast(ok);
    w.barrier();
    return ok != 0;
}

}  // namespace pfast
