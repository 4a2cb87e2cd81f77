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
#ifndef GFSM_WALK_LISTED  // (set by a test that fills a list)
#define GFSM_WALK_LISTED (1u << 18)
#endif
constexpr uint32_t kWalkListed = GFSM_WALK_LISTED;  // units a list holds
// A whole walk: every so many times 32 rounds a warp looks whether there is
// work left to take; once there is not, it leaves what it has queued to the
// next pass, whose warps share it (k_split).  Rounds take 1-2 us (of suffixes
// up to 8, they count as 4), a pass costs about 25.
constexpr uint32_t kWalkLookFew = 1;   // fewer units than warps: a warp may hold a whole tree
constexpr uint32_t kWalkLookMany = 8;

constexpr int kWalkTotals = 32;

struct WalkResult {
    unsigned long long unit;  // units handed out so far
    uint32_t done;     // CTAs of the last pass that have finished
    uint32_t gave_up;  // the last pass left work: the counts are not complete
    struct List {
        uint32_t listed, taken;  // work units a pass left to the next, how many of them that one has handed out
        uint32_t refused;        // (k_split) listed > kWalkListed: where the list ends
    } list[kWalkPasses];         // limited: one a pass; whole walks use the first
    uint32_t kept;               // warps of a whole walk's pass that left work
    // candidates, expansions, algorithmic bytes and the bytes of the partial
    // mappings extended (what whole levels would hold), in parts
    unsigned long long total[kWalkTotals][4];
};

// A warp of a whole walk between two passes: entries and candidates of its
// queues (lane d: depth d), the suffix queue's entries and pairs, units it has
// taken and not begun.
struct WalkState {
    uint32_t ents[32], left[32];
    unsigned long long u_next, u_end;
    uint32_t open, sents, spairs, pad;
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
    uint32_t last;               // this pass may be the call's last (set by walk_pass)
    // mappings of a lone query (null: counts only): up to max_rows rows of k
    // original vertex ids, tuple position i in column col[i]
    uint32_t *rows;
    uint32_t *rows_ctr;
    const uint32_t *order;
    unsigned long long max_rows;
    uint8_t col[MAXQ];
    Chunk *queues;            // walk_queue_bytes(core, sms) of scratch
    // set by walk_pass: a limited pass' rounds, a whole walk's rounds between
    // looks (in 32; 0: none), and the CTAs that have finished before one hands
    // its work on; the list that the pass before left
    // (null: the first), and where this one, or k_split, leaves its own (null:
    // nowhere); whole walks: the warps' states, those the pass before had, and
    // the units that k_split makes of one
    uint32_t max_rounds, look, most;
    const Chunk *list_in;
    Chunk *list_out;
    WalkResult::List *in, *out;
    WalkState *state_in, *state_out;
    uint32_t state_warps, share;
    uint32_t chunk, warp_chunks, ctas;
};

// Bytes of the warps' queues for tuples of up to `core` vertices.
uint64_t walk_queue_bytes(uint32_t core, int sms);
// Bytes of the lists of a call with several passes.
uint64_t walk_list_bytes(uint32_t core);
// Pass p of a call: a limited walk has kWalkPasses, a whole one goes on while
// warps of its last pass have kept work (`kept`: how many; lists null: one pass).
cudaError_t launch_walk(const WalkArgs &args, bool lab, bool limited, Chunk *lists, int p, uint32_t kept, int sms,
                        cudaStream_t st);

}  // namespace gfsm
