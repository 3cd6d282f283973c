// sc_team.cuh — the levels of a Leiden pass that are too small for a launch per
// step: one thread-block cluster (or one block) runs them all (sc_team.cu).
#pragma once

#include "sc_internal.cuh"

namespace sc {

// Largest level the team takes: its node count bounds the block's dense
// accumulators and scans in shared memory, its entry count the share of the
// chip (16 of 148 SMs) that still beats a launch and a read-back per step.
constexpr uint32_t TEAM_MAX_NODES = 8192;
constexpr uint64_t TEAM_MAX_ENTRIES = uint64_t(1) << 20;

// Device memory the team works in: sized for a level of n nodes and E entries,
// kept by the caller for the passes of one run.
struct TeamSpace {
    DBuf<unsigned char> mem;
    uint32_t n = 0;
    uint64_t E = 0;
};

// What the team left: the pass is finished (labels written), or it stopped
// before `level` because that level's graph left the exact regime.
struct TeamResult {
    bool finished = false;
    uint64_t level = 0;        // levels counted from the pass's first
    uint64_t n_clusters = 0;   // finished: communities of the final labels
    double improvement = 0.0;  // the pass's, with what the caller had before
    uint64_t sweeps = 0, moves = 0, levels = 0;
    double ms_local_move = 0, ms_refine = 0, ms_aggregate = 0;
    double alg_bytes_local_move = 0, alg_bytes_aggregate = 0;
    // not finished: the level's graph and membership (ids < C, in the caller's memb)
    std::unique_ptr<DevGraph> graph;
    uint64_t C = 0;
};

// Blocks of the largest team that the device can place: 16, 8 or 0 (asked once per
// context, not above its team_most). With 0 every level goes a launch per step.
uint32_t team_offer(Ctx& c);

// Whether the team may take g under cfg.
bool team_takes(Ctx& c, const DevGraph& g, const sc_leiden_config& cfg);

// Runs the pass from `level` on g (memb: ids < C) to its end. node_map (g.n
// words): finished, the final label of each of g's nodes; else its node in the
// level reached, whose membership is then in memb.
void team_run(Ctx& c, const DevGraph& g, uint32_t* memb, uint64_t C, const sc_leiden_config& cfg, uint64_t pass_seed,
              uint64_t level, double improvement, TeamSpace& space, uint32_t* node_map, TeamResult& out);

// The last sweeps of a larger level's local moving: once a sweep has at most
// tail_limit active nodes (0: the team cannot take this level), the team runs on
// until the level is done or a sweep outgrows it.
uint32_t tail_limit(Ctx& c, const DevGraph& g, const sc_leiden_config& cfg);
struct TailResult {
    bool done = false;
    bool swapped = false;  // not done: the next sweep's list is lists[1], its count counts[1]
    uint32_t sweep = 0;    // not done: the sweep to go on with
    uint32_t epoch = 0, swept = 0;
    uint64_t moves_before = 0;
};
// params: the level's Params (sc_move.cuh), its counters and gains running on.
// first: the list of sweep `sweep` (lists[0], or null for all n nodes).
TailResult tail_run(Ctx& c, const void* params, uint32_t n, const uint32_t* first, uint32_t* const lists[2],
                    uint32_t* const counts[2], uint32_t* stamp, uint32_t sweep, uint32_t epoch, uint64_t moves_before,
                    uint64_t budget);

}  // namespace sc
