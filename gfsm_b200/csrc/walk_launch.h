// walk_launch.h -- launching the walk.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "walk.cuh"

namespace gfsm {

constexpr int kWalkThreads = 128;

struct WalkResult {
    unsigned long long unit;  // units handed out so far
    unsigned long long candidates, expansions, alg_bytes;
    unsigned long long frontier_bytes;  // of the partial mappings extended: what whole levels would hold
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
    WalkResult *result;
    Chunk *queues;            // walk_queue_bytes(core, sms) of scratch
    uint32_t chunk, warp_chunks;  // set by launch_walk
};

// Bytes of the warps' queues for tuples of up to `core` vertices.
uint64_t walk_queue_bytes(uint32_t core, int sms);
cudaError_t launch_walk(const WalkArgs &args, bool lab, int sms, cudaStream_t st);

}  // namespace gfsm
