// walk_launch.h -- launching the walk.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "walk.cuh"

namespace gfsm {

constexpr int kWalkThreads = 128;
// A limited walk (Engine::run_walk) is a few passes: a warp that has taken a
// pass's rounds writes what is left in its queues to a list, and the next
// pass deals the list to all warps.  What the last one leaves is not walked.
constexpr int kWalkPasses = 4;
constexpr uint32_t kWalkRounds[kWalkPasses] = {16, 24, 32, 96};
constexpr uint32_t kWalkListed = 1u << 18;  // units a list holds

constexpr int kWalkTotals = 32;

struct WalkResult {
    unsigned long long unit;  // units handed out so far
    uint32_t done;     // CTAs of the last pass that have finished
    uint32_t gave_up;  // the last pass left work: the counts are not complete
    uint32_t listed[kWalkPasses];  // work units each pass left to the next ...
    uint32_t taken[kWalkPasses];   // ... and how many of them that one has handed out
    // candidates, expansions, algorithmic bytes and the bytes of the partial
    // mappings extended (what whole levels would hold), in parts
    unsigned long long total[kWalkTotals][4];
};

struct WalkArgs {
    WalkGraph g;
    const WNode *__restrict__ nodes;
    const WSfx *__restrict__ sfx;
    const WAgain *__restrict__ again;
    const uint32_t *__restrict__ root_lo;
    const unsigned long long *__restrict__ root_off;  // [roots + 1]
    uint32_t roots, core, node_count, sfxs;
    unsigned long long units;  // root_off[roots]
    unsigned long long *counts;  // per slot
    WalkResult *result;          // the counts follow it
    // Where the last CTA of the call copies result and counts (pinned host
    // memory; null: the caller copies them): a copy of a few hundred bytes is
    // 6 us in a stream.
    uint4 *host;
    uint32_t host_words;         // in 16 bytes
    uint32_t last;               // this pass is the call's last (set by launch_walk)
    // mappings of a lone query (null: counts only): up to max_rows rows of k
    // original vertex ids, tuple position i in column col[i]
    uint32_t *rows;
    uint32_t *rows_ctr;
    const uint32_t *order;
    unsigned long long max_rows;
    uint8_t col[MAXQ];
    Chunk *queues;            // walk_queue_bytes(core, sms) of scratch
    // limited walks only: this pass, its rounds, what the one before left,
    // where it leaves its own
    uint32_t pass, max_rounds;
    const Chunk *list_in;
    Chunk *list_out;
    uint32_t chunk, warp_chunks;  // set by launch_walk
};

// Bytes of the warps' queues for tuples of up to `core` vertices.
uint64_t walk_queue_bytes(uint32_t core, int sms);
// Bytes of the two lists of a limited walk.
uint64_t walk_list_bytes(uint32_t core);
// limited: kWalkPasses passes, with `lists` for what they leave one another.
cudaError_t launch_walk(const WalkArgs &args, bool lab, bool limited, Chunk *lists, int sms, cudaStream_t st);

}  // namespace gfsm
