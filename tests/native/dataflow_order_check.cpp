// Checks on the CPU that the queue of the 3D dataflow sweeps (pfast_gb300/csrc/dataflow_queue.h) orders
// what a tile's processing wrote before every processing that reads it.  The queue's functions run
// over a memory with vector clocks: relaxed atomics, of which a read-modify-write continues the release
// sequence of its word; fences that acquire what the lane's atomics have read and release what the lane
// has seen; warp barriers.  Lanes of several warps run the kernel's loop (take, complete locked
// items, process one, complete it by the whole warp) in random turns; a lane that starts on tile x must
// have seen the last writes to x and to its face neighbours by every lane that made them.
// Prints "ok <mode> <grid>" per grid, or "FAIL ..." and exits 1.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <random>
#include <vector>

#include "dataflow_queue.h"

using namespace pfast;

static const int kLanes = 13, kWarps = 6, kN = kLanes * kWarps;
typedef std::vector<unsigned> Clock;
static void join(Clock& a, const Clock& b) { for (int i = 0; i < kN; ++i) a[i] = std::max(a[i], b[i]); }

struct Machine {
    std::map<const void*, Clock> word;          // what the last value of a word carries
    std::vector<Clock> seen, released, read;    // per lane: seen, released by its last fence, read since
    bool stop = false;
    Machine() : seen(kN, Clock(kN, 0)), released(seen), read(seen) {
        for (int l = 0; l < kN; ++l) seen[l][l] = 1;
    }
    Clock& at(const void* p) { auto& c = word[p]; if (c.empty()) c.assign(kN, 0); return c; }
    void rmw(int l, const void* p) { Clock& w = at(p); join(read[l], w); join(w, released[l]); }
    void fence(int l) { join(seen[l], read[l]); released[l] = seen[l]; }
    void warp_barrier(int warp) {
        Clock c(kN, 0);
        for (int l = 0; l < kLanes; ++l) join(c, seen[warp * kLanes + l]);
        for (int l = 0; l < kLanes; ++l) seen[warp * kLanes + l] = c;
    }
};

struct Memory {   // one lane's
    Machine* m;
    int l;
    unsigned add(unsigned* p, unsigned v) const { m->rmw(l, p); const unsigned o = *p; *p += v; return o; }
    unsigned sub(unsigned* p, unsigned v) const { m->rmw(l, p); const unsigned o = *p; *p -= v; return o; }
    unsigned cas(unsigned* p, unsigned want, unsigned v) const {
        if (*p == want) { m->rmw(l, p); *p = v; return want; }
        join(m->read[l], m->at(p));
        return *p;
    }
    unsigned exch(unsigned* p, unsigned v) const { m->rmw(l, p); const unsigned o = *p; *p = v; return o; }
    void fence() const { m->fence(l); }
    bool stopped(const DataflowQueue&) const { return m->stop; }
    void stop(const DataflowQueue&) const { m->stop = true; }
};

struct Write { int lane; unsigned when; };

template <bool CL>
static int run(const TileGrid3& g, unsigned seed) {
    std::mt19937 rng(seed);
    const int n = tile_count(g);
    Machine M;
    int qcap = 1;
    while (qcap < n) qcap <<= 1;
    std::vector<unsigned> cnt(CL ? n : (n + 3) / 4, 0), slots(qcap, kSlotEmpty);
    DataflowShared sh = {};
    DataflowQueue Q{cnt.data(), slots.data(), (unsigned)qcap - 1, &sh};
    for (int x = 0; x < n; ++x) {
        if (CL) cnt[x] = dep_counts(g, x);
        else cnt[x >> 2] |= (unsigned)(dep_count(g, 0, x) | (dep_count(g, 1, x) << 4)) << (8 * (x & 3));
    }
    slots[0] = (unsigned)first_tile(g) << 3;
    sh.tail = 1;
    std::vector<std::vector<Write>> last(n);   // the last processing's writes of every tile
    std::vector<int> done(8 * n, 0);
    std::vector<unsigned> e(kN, kSlotEmpty);
    int completed = 0;
    auto sees = [&](int lane, int x) {
        auto one = [&](int y) {
            for (const Write& w : last[y]) if (M.seen[lane][w.lane] < w.when) return false;
            return true;
        };
        if (!one(x)) return false;
        for (int a = 0; a < 3; ++a)
            for (int s = 0; s < 2; ++s) {
                const int y = tile_neighbour(g, x, a, s);
                if (y >= 0 && !one(y)) return false;
            }
        return true;
    };
    auto fail = [&](const char* what, int x) {
        std::printf("FAIL %s %s grid %dx%dx%d tile %d\n", CL ? "cluster" : "block", what, g.nbk, g.nbi, g.nbj, x);
        return 1;
    };
    for (long step = 0; completed < 8 * n; ++step) {
        if (step > 4000000L || M.stop) return fail("stalled", -1);
        const int w = rng() % kWarps, l0 = w * kLanes;
        bool holding = false;
        for (int l = 0; l < kLanes; ++l) holding |= e[l0 + l] != kSlotEmpty;
        if (!holding) {   // take some of the ready items
            const int avail = (int)(sh.tail - sh.head);
            if (avail <= 0) continue;
            const int take = std::min(kLanes, std::max(1, avail / (int)(1 + rng() % kWarps)));
            const unsigned h = sh.head;
            sh.head += take;
            for (int l = 0; l < take; ++l) {
                const Memory m{&M, l0 + l};
                e[l0 + l] = m.exch(slots.data() + ((h + l) & Q.qmask), kSlotEmpty);
                m.fence();
            }
        }
        int mine = -1;
        std::vector<unsigned> next(kLanes, kSlotEmpty);
        std::vector<char> due(kLanes, 0);
        for (int l = 0; l < kLanes; ++l) {
            const unsigned it = e[l0 + l];
            if (it == kSlotEmpty) continue;
            if (!sees(l0 + l, (int)(it >> 3))) return fail("lock word read before its writes are seen", (int)(it >> 3));
            due[l] = rng() % 2;
            if (due[l] && mine < 0) mine = l;
        }
        for (int l = 0; l < kLanes; ++l) {
            const unsigned it = e[l0 + l];
            if (it == kSlotEmpty || due[l]) continue;
            if (done[(it & 7) * n + (it >> 3)]++) return fail("item twice", (int)(it >> 3));
            ++completed;
            next[l] = df_complete<CL>(Memory{&M, l0 + l}, g, Q, (int)(it & 7), (int)(it >> 3));
        }
        if (mine >= 0) {
            for (int l = 0; l < kLanes; ++l) {
                if (due[l] && l != mine) next[l] = e[l0 + l];
                if (next[l] != kSlotEmpty) df_push(Memory{&M, l0 + l}, Q, next[l]);
            }
            const int x = (int)(e[l0 + mine] >> 3), o = (int)(e[l0 + mine] & 7);
            M.warp_barrier(w);
            for (int l = 0; l < kLanes; ++l)
                if (!sees(l0 + l, x)) return fail("tile processed before its inputs are seen", x);
            last[x].clear();
            for (int l = 0; l < kLanes; ++l) last[x].push_back(Write{l0 + l, ++M.seen[l0 + l][l0 + l]});
            if (done[o * n + x]++) return fail("item twice", x);
            ++completed;
            if (!CL) df_rearm(Memory{&M, l0}, g, Q, o, x);
            M.warp_barrier(w);
            for (int l = 0; l < kLanes; ++l) next[l] = df_complete_lane<CL>(Memory{&M, l0 + l}, g, Q, o, x, l);
            M.warp_barrier(w);
        }
        for (int l = 0; l < kLanes; ++l) {
            if (!CL && next[l] != kSlotEmpty) { df_push(Memory{&M, l0 + l}, Q, next[l]); next[l] = kSlotEmpty; }
            e[l0 + l] = next[l];
        }
    }
    return 0;
}

int main() {
    const int grids[][3] = {{1, 1, 3}, {2, 2, 2}, {3, 4, 2}, {1, 5, 6}, {4, 4, 4}, {2, 7, 1}};
    for (const auto& gd : grids) {
        const TileGrid3 g{gd[0], gd[1], gd[2]};
        for (unsigned seed = 1; seed <= 40; ++seed)
            if (run<true>(g, seed) || run<false>(g, seed)) return 1;
        std::printf("ok %dx%dx%d\n", gd[0], gd[1], gd[2]);
    }
    return 0;
}
