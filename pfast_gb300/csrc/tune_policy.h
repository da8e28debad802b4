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
// Measured (ms of a mixed gradient of 128 x 128 x 64 nodes, blocks per source): 64 sources 95 (1), 81
// (2); 40 sources 71 (2), 70 (4); 100 sources 99 (1), 103 (2); plain, 96 x 96 x 48: 16 sources 602
// (1), 331 (2), 202 (4), 175 (8), 287 (16); 40 sources 331 (2), 299 (4).
// Any size, not powers of two alone, which left up to half of the SMs idle just above a step
// (plain gradient of 128 x 128 x 100: 21 sources 628 ms with 4 blocks, 395 with 7; 96 x 96 x 48: 42
// sources 314 (2), 223 (3); mixed, 128 x 128 x 100: 13 sources 53 (8), 46 (15)).  Sizes of 9 to 15 only on
// grids of 100 tiles a block: 12 sources of 96 x 96 x 48 (432 tiles) took 126 ms with 8 blocks, 162 with 13.
constexpr int kMaxCluster = 16;

inline bool cluster_wanted(int cs, bool plain, int nact, int ntiles, int sms) {
    return 10LL * nact * cs <= (plain ? 11LL : 13LL) * sms && ntiles >= (cs > 8 && cs < kMaxCluster ? 100 : 8) * cs;
}

// Warps per block of a cluster.  Few: the ready tiles of a source are few as well, and what
// bounds them is the latency of one tile, so they should lie on different SM sub-partitions, and
// idle warps only poll the queue.  The plain kinds saturate a sub-partition's FP64 pipe with one warp.
// Measured (ms; warps per block): one shot of 128 x 128 x 64 nodes, plain, 16 blocks: 117 (2),
// 88 (4), 102 (6), 171 (11, all that fit); 16 sources of 96 x 96 x 48, plain gradient, 8 blocks: 208
// (2), 175 (4), 235 (6), 361 (11); 24 sources of 155 x 75 x 101, mixed forward, 8 blocks: 72 (2),
// 49 (4), 48 (6), 54 (8); 9 sources of 90 x 71 x 53, mixed gradient, 16 blocks: 40.1 (2), 39.9 (4),
// 41.3 (6); 64 sources of 128 x 128 x 64, mixed gradient, 2 blocks: 97 (8), 83 (12), 81 (24).
inline int cluster_warps(int cs, bool plain) {
    if (plain || cs >= 8) return 4;
    return cs >= 4 ? 6 : 12;
}

// The candidate of a phase that has not been timed, among `allowed` (tune_allowed): the dataflow
// kernel, except where one launch per tile diagonal is ahead:
// - the plain kinds, whose FP64 pipe needs one warp per SM sub-partition only, with at most three
//   blocks per instance that leave SMs idle, where a diagonal holds enough tiles for all SMs.
//   Gradients, ms per diagonal / dataflow (tiles a diagonal): 84 sources of 96 x 96 x 48 393 / 552
//   (1450), 61 of 226 x 35 x 68 723 / 924 (1480), 49 of 100 x 171 x 47 738 / 790-880 (1440), 64 of
//   96 x 96 x 48 352 / 333 (1110), 84 of 64 x 64 x 32 165 / 151 (670); one block each from three
//   quarters of the SMs on: 119 of 67 x 137 x 26 504 / 427 (2100), 123 of 104 x 125 x 25 579 / 493
//   (2200); two or three each from all SMs on: forward of 79 of 37 x 126 x 108 575 / 472 (1590);
// - the FP32 bulk kinds with one block per instance where a diagonal holds many tiles (256 sources
//   of 256 x 256 x 128, 30,000 tiles a diagonal: forward 165 / 176, adjoint 242 / 250; 256
//   sources of 96 x 96 x 48, 4,400: 12.3 / 8.8, 14.6 / 11.6).
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
