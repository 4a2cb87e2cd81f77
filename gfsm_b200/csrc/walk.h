// walk.h -- the walk: a call's whole search as one kernel, each lane running
// its own depth-first enumeration (device code in walk_kernel.cuh, host tables
// in walk_plan.cpp).  Compiled by the host compiler too (tests of the tables).
#pragma once
#include <cstdint>
#include <memory>
#include <vector>

#include "gfsm_internal.h"

#ifdef __CUDACC__
#define GFSM_HD __host__ __device__ __forceinline__
#else
#define GFSM_HD inline
#endif

namespace gfsm {

constexpr int kWalkReqs = 8;   // requirement rows a node holds beyond its anchor
constexpr uint32_t kNoGroup = 15;
constexpr int kSfxGroups = 7;  // groups of equal leaves a suffix holds

// A node of the trie of a call's plans: the queries that agree on everything
// the search does down to one depth.  A tuple (partial mapping) belongs to a
// node; a node's children are consecutive, and all take their candidates from
// the same slice of one row.
struct alignas(16) WNode {
    uint32_t child;             // first child node
    uint16_t nchild, nsfx;      // children, and suffixes counted at this node
    uint32_t sfx;               // first suffix
    uint32_t slot;              // count slot of a query that ends here (final_)
    uint32_t next_lo, next_hi;  // id window of the children's candidates
    uint16_t next_lb, next_ub;  // symmetry breaking: the children's candidate exceeds / stays below
                                // the vertices at these tuple positions
    uint8_t next_anchor;        // tuple position whose row the children take candidates from
    uint8_t next_grp;           // label group of the window
    uint8_t next_trim;          // the window is narrower than its group by enough to matter
    uint8_t final_;             // a query's last vertex
    uint64_t need;              // entries its row must have, a byte per label group (WalkGraph::nlf)
    uint8_t nreq;               // the check of a candidate of this node: requirements (bits 0-3) and
                                // the label group it comes from (4-7; kNoGroup: not within one)
    uint8_t anchor, anchor_lab, anchor_check;
    uint32_t again;             // (first << 8 | number): WAgain entries, more needs of earlier vertices
    uint8_t req_pos[kWalkReqs], req_lab[kWalkReqs];
};
static_assert(sizeof(WNode) == 64, "WNode layout");

// A node that many queries share can ask of a vertex's row only what all of
// them need; the rest is asked here, at the node where they part.
struct WAgain {
    uint64_t need;
    uint32_t pos, pad;
};

// Leaves of a query with the same anchor and window.  A leaf is a query
// vertex whose only requirement is the edge to its anchor.
struct alignas(16) WSfxGroup {
    uint32_t lo, hi;   // id window
    uint16_t lb, ub;   // symmetry breaking against core positions
    uint8_t anchor;    // core position
    uint8_t lab;       // edge label of the anchor edge
    uint8_t grp;       // label group of the window
    uint8_t form;      // bits 0-3 leaves in the group, 4-5 groups from here on whose windows meet
                       // (0: counted with the one before), 6 the window is narrower than its group
};
// The trailing leaves of a query, counted together at the last core vertex:
// the number of ways to place them all, on distinct vertices outside the core.
struct alignas(16) WSfx {
    uint32_t slot;
    uint8_t ng, nleaf;
    uint8_t pad[10];
    WSfxGroup g[kSfxGroups];
};
static_assert(sizeof(WSfx) == 128, "WSfx layout");

struct WalkScratch;
struct WalkTables {
    std::shared_ptr<WalkScratch> scratch;
    std::vector<WNode> nodes;           // root nodes first
    std::vector<WSfx> sfx;
    std::vector<WAgain> again;
    std::vector<uint32_t> root_lo;      // per root node: first id of its window
    std::vector<unsigned long long> root_off;  // [roots + 1] exclusive prefix of the root windows
    std::vector<uint32_t> slot;         // per query: its count slot
    std::vector<uint64_t> mult;         // per query: what its count is multiplied by
    uint32_t nslots = 0;
    uint32_t core = 0;                  // deepest core (tuple columns)
};

struct WalkQuery {
    const DQuery *dq;
    const Plan *plan;
    uint32_t lo, hi;  // root window
    bool sym;         // symmetry breaking applies
};

// Tables of a call against g (its host fields).  share: queries with equal prefixes share nodes.
// leaves: count trailing leaves together (data without repeated entries).
// cross: leaves on different anchors may share a window (their rows are
// intersected by one lane: only where rows are short).  desc: symmetry
// conditions keep the embedding whose earlier vertex has the larger id.
// False when a plan does not fit the tables (the level steps take it then).
bool build_walk(const std::vector<WalkQuery> &qs, const DeviceGraph &g, bool share, bool leaves, bool cross, bool desc,
                WalkTables &out);
// Memory build_walk works in, kept by the tables for the next call; drops it
// where a very large batch has grown it.
void trim_walk(WalkTables &t);

}  // namespace gfsm
