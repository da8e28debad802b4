// tune_policy.h -- the 3D sweep autotuner's choice of (schedule, tile shape) for one phase
// (host code; the CPU check tests/native/tune_policy_check.cpp compiles it with g++).
//
// Candidates c = 2 * schedule + shape: schedule 0 one launch per tile diagonal, 1 dataflow
// (one launch per phase), 2 hybrid (first outer iteration per diagonal, then dataflow); shape
// 0 = 4x8x32 tiles, 1 = 8x4x32.  pfast_survey3d_autotune records each candidate's phase times
// per (device, sweep kind, grid, active instances); a phase then takes the fastest allowed one.
// A dataflow or hybrid time belongs to the cluster size it was measured with (below), which depends
// on the evaluations under way beside it.
#pragma once

#include <array>
#include <map>
#include <mutex>
#include <tuple>

namespace pfast {

constexpr int kTuneCandidates = 6;

struct TuneEntry {
    double ms[kTuneCandidates] = {};   // summed phase times
    int n[kTuneCandidates] = {};       // phases timed
};

// The candidates a phase may use: schedule_opt and shape_opt as pfast_options (0 automatic,
// else schedule 1..3 / shape 1..2); dataflow_fits[s]: the grid's tiles of shape s fit the
// dataflow kernel's shared memory.  Dataflow or hybrid asked for on a grid that does not fit:
// per diagonal.
inline unsigned tune_allowed(int schedule_opt, int shape_opt, const bool dataflow_fits[2]) {
    unsigned allowed = 0;
    for (int shape = 0; shape < 2; ++shape) {
        if (shape_opt != 0 && shape_opt - 1 != shape) continue;
        if (schedule_opt == 0 || schedule_opt == 1) allowed |= 1u << shape;
        if ((schedule_opt == 0 || schedule_opt == 2) && dataflow_fits[shape]) allowed |= 4u << shape;
        if ((schedule_opt == 0 || schedule_opt == 3) && dataflow_fits[shape]) allowed |= 16u << shape;
    }
    if (!allowed) allowed = shape_opt == 0 ? 1u : 1u << (shape_opt - 1);
    return allowed;
}

// The candidate of a phase once every allowed candidate has been timed: the one with the smallest
// mean phase time (the first of equal ones).  Before that (which no sweep asks: they take untuned_pick
// below until TuneTable has every time) the dataflow kernel with 4x8x32 tiles from two active
// instances per SM, else one launch per tile diagonal, else the lowest allowed candidate.
inline int tune_pick(const TuneEntry* e, unsigned allowed, int nact, int sms) {
    if (e) {
        int best = -1;
        bool all = true;
        for (int c = 0; c < kTuneCandidates; ++c) {
            if (!(allowed >> c & 1)) continue;
            if (e->n[c] == 0) { all = false; break; }
            if (best < 0 || e->ms[c] / e->n[c] < e->ms[best] / e->n[best]) best = c;
        }
        if (all && best >= 0) return best;
    }
    const int first = nact >= 2 * sms && (allowed & 0xcu) ? 2 : 0;
    for (int c = first; c < kTuneCandidates; ++c)
        if (allowed >> c & 1) return c;
    for (int c = 0; c < kTuneCandidates; ++c)
        if (allowed >> c & 1) return c;
    return 0;
}

// The dataflow kernel solves an instance with one block, or with a cluster of cs = 2..16 blocks that
// share its queue, where the instances alone would leave SMs idle.  A cluster size is wanted
// while the clusters need about one block per SM (the hardware packs the blocks of a cluster
// densely, so beyond that some SMs hold several and others none) and the grid has tiles for them.
// Measured (gradients on smooth random models, ms, blocks per source in brackets; runs differ by up to 7 %
// with where the hardware places the clusters): mixed, 128 x 128 x 64 nodes: 64 sources 82 (1), 65 (2); 40
// sources 57 (2), 51 (3), 59 (4); plain, 96 x 96 x 48: 16 sources 494 (1), 327 (2), 186 (4), 137 (8);
// 40 sources 338 (2), 239 (3), 236 (4).
// Any size, not powers of two alone, which left up to half of the SMs idle just above a step
// (plain, 128 x 128 x 100: 21 sources 640 ms (4), 409 (7); 96 x 96 x 48: 42 sources 321 (2), 228 (3)).
// Sizes of 9 to 15 only on grids of 100 tiles a block: 12 sources of 96 x 96 x 48 (432 tiles) 130 (8), 145 (12).
constexpr int kMaxCluster = 16;

inline bool cluster_wanted(int cs, bool plain, int nact, int ntiles, int sms) {
    return 10LL * nact * cs <= (plain ? 11LL : 13LL) * sms && ntiles >= (cs > 8 && cs < kMaxCluster ? 100 : 8) * cs;
}

// Warps per block of a cluster.  Few: the ready tiles of a source are few as well, and what
// bounds them is the latency of one tile, so they should lie on different SM sub-partitions, and
// idle warps only poll the queue.  The plain kinds saturate a sub-partition's FP64 pipe with one warp.
// Measured (ms, warps per block in brackets): one shot of 128 x 128 x 64 nodes, plain, 16 blocks: 88 (2),
// 67 (4), 73 (6), 119 (11, all that fit); 16 sources of 96 x 96 x 48, plain gradient, 8 blocks: 179 (2),
// 138 (4), 194 (6); 24 sources of 155 x 75 x 101, mixed forward, 6 blocks: 49 (2), 32 (4), 35 (6); 9 sources
// of 90 x 71 x 53, mixed gradient, 16 blocks: 22 (2), 25 (4), 25 (6); 30 sources of 128 x 128 x 64, mixed
// gradient, 5 blocks: 61 (4), 55 (6); 64 sources, 2 blocks: 109 (4), 89 (6), 75 (8), 64 (12).
inline int cluster_warps(int cs, bool plain) {
    if (plain || cs >= 8) return 4;
    return cs >= 4 ? 6 : 12;
}

// The candidate of a phase that has not been timed, among `allowed` (tune_allowed): the dataflow
// kernel, except where one launch per tile diagonal is ahead (the tile counts of both lines are those
// measured on 152 SMs):
// - the plain kinds, whose FP64 pipe needs one warp per SM sub-partition only, with at most three
//   blocks per instance that leave SMs idle, where a diagonal holds enough tiles for all SMs.
//   Gradients, ms per diagonal / dataflow (tiles a diagonal): 84 sources of 96 x 96 x 48 404 / 562
//   (1450), 61 of 226 x 35 x 68 744 / 953 (1480), 49 of 100 x 171 x 47 758 / 787 (1440), 64 of
//   96 x 96 x 48 362 / 342 (1110), 84 of 64 x 64 x 32 170 / 154 (670); one block each from three
//   quarters of the SMs on: 119 of 67 x 137 x 26 517 / 433 (1730), 123 of 104 x 125 x 25 593 / 500
//   (2200); two or three each from all SMs on: forward of 79 of 37 x 126 x 108 320 / 291 (1590).  On
//   rough models (every node at random) the per-diagonal launches stay ahead a little longer;
// - the FP32 bulk kinds with one block per instance where a diagonal holds many tiles (256 sources,
//   forward and adjoint ms per diagonal / dataflow: 256 x 256 x 128, 30,000 tiles a diagonal, 172 / 184 and
//   245 / 250; 200 x 200 x 100, 20,400: 94 / 91, 127 / 127; 176 x 176 x 100, 16,600: 71 / 66, 90 / 85;
//   128 x 128 x 64, 7,700: 24 / 20, 33 / 29).  The line lies at 16,384, a little below where the two meet.
// cluster: blocks per instance of the dataflow kernel; plain / fp32: the phase's kind (neither: polish).
inline int untuned_pick(unsigned allowed, bool plain, bool fp32, int cluster, int nact, long long ntiles, int ndiag,
                        int sms) {
    bool dataflow = true;
    if (plain)
        dataflow = cluster > 3 || 4 * nact * cluster >= (cluster > 1 ? 4 : 3) * sms || ntiles * nact < 1200LL * ndiag;
    if (fp32 && cluster <= 1) dataflow = ntiles * nact < 16384LL * ndiag;
    const int order[2][kTuneCandidates] = {{0, 1, 2, 3, 4, 5}, {2, 3, 4, 5, 0, 1}};
    for (int c : order[dataflow])
        if (allowed >> c & 1) return c;
    return 0;
}

// Whether every allowed candidate has been timed (tune_pick then takes the fastest).
inline bool tune_complete(const TuneEntry* e, unsigned allowed) {
    if (!e) return false;
    for (int c = 0; c < kTuneCandidates; ++c)
        if ((allowed >> c & 1) && e->n[c] == 0) return false;
    return true;
}

// The phase times of all candidates, from every thread.  With 16 blocks per source for 9 sources alone and
// one when eight threads evaluate side by side, the time of a dataflow candidate says nothing about
// the other case: a phase asks for the times of the cluster sizes it would launch with, measured as
// it runs (alone or beside other evaluations) or else in the other way.
class TuneTable {
public:
    using Phase = std::array<int, 6>;   // device, sweep kind, nz, nr, nc, active instances

    void record(const Phase& p, bool alone, int c, const int cluster[2], double ms) {
        if (!(ms > 0.0)) return;
        std::lock_guard<std::mutex> g(mu_);
        Time& t = times_[std::make_tuple(p, alone, c, blocks(c, cluster))];
        t.ms += ms;
        t.n += 1;
    }

    // The fastest allowed candidate once all are timed with these cluster sizes; -1 before that.
    int pick(const Phase& p, bool alone, unsigned allowed, const int cluster[2], int sms) const {
        std::lock_guard<std::mutex> g(mu_);
        for (const bool how : {alone, !alone}) {
            TuneEntry e;
            for (int c = 0; c < kTuneCandidates; ++c) {
                auto it = times_.find(std::make_tuple(p, how, c, blocks(c, cluster)));
                if (it == times_.end()) continue;
                e.ms[c] = it->second.ms;
                e.n[c] = it->second.n;
            }
            if (tune_complete(&e, allowed)) return tune_pick(&e, allowed, p[5], sms);
        }
        return -1;
    }

private:
    struct Time { double ms = 0.0; int n = 0; };
    static int blocks(int c, const int cluster[2]) { return c < 2 ? 0 : cluster[c & 1]; }   // per diagonal: none
    mutable std::mutex mu_;
    std::map<std::tuple<Phase, bool, int, int>, Time> times_;
};

}  // namespace pfast
