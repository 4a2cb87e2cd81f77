// walk_kernel.cuh -- a call's whole search as one kernel.
//
// The level steps (engine.cu) write every partial mapping of a level to HBM
// and read it back at the next, find a candidate's parent by binary search,
// and pay several launches per level.  Where rows are short (road-like and
// bounded-degree graphs) a parent has about one candidate, and that work is
// several times the check itself: 23 warp instructions per candidate.  Here
// every warp searches depth first over its own small queues, one per depth,
// and nothing leaves the chip's caches but counts.  Prefixes are shared
// through the same trie as in the level steps; trailing leaves are counted
// without being enumerated (walk.cuh); a batch's vertices are filtered by
// their neighbours' labels.
//
// Bound: instruction issue and the latency of a round's dependent loads
// (queue entry, row entry, row pointers by label group); ncu on
// 64 grid queries, cold caches: 48% issue active with 22 of 32 lanes, 8.7
// long-scoreboard stalls an issue, DRAM 0.62 TB/s.
// Before (level steps) and after, whole calls: one 5-vertex query on 2,000
// vertices 208 -> 40 us, one 7-vertex query on the 1,400 x 1,400 grid 294 ->
// 84-102 us, 64 such queries of 4-10 vertices 3.4 -> 1.36-1.46 ms, 4,096 of
// them from edge lists 102 -> 55 ms.  One lane per search (no queues) left 9
// of 32 lanes active: 4,096 queries took 507 ms.
//
// Work is shared by passes.  A warp keeps the trees below its roots, and most
// calls end so.  Where a few warps hold most of the work, they stop, k_split
// cuts their queues into units, and all warps of the next pass take those: ten
// roots on rows of 30, a path of six vertices, 24.5 -> 0.95 ms; a clique of 48
// in a grid, a path of five, 9.1 -> 1.9 ms.  (The level steps take 0.5 and 0.3
// ms there: their tiles split any row evenly.)  No warp waits for another.
//
// Compiled by the host compiler too, with 32-lane stand-ins for the warp
// intrinsics (the test that runs every lane of it in a random order).
#pragma once
#include "walk_launch.h"

namespace gfsm {

namespace {

#ifdef __CUDACC__
#define GFSM_DYN_SHARED(x) extern __shared__ __align__(16) uint32_t x[]
#endif

constexpr uint32_t kFull = 0xffffffffu;
constexpr uint32_t kWarps = kWalkThreads / 32;
// CTAs an SM runs: 32 warps at 64 registers.  40 warps (48 registers) hide
// more latency but cost instructions (before the loops were rolled, walk.cuh):
// 4,096 grid queries 57.4 against 58.4 ms, but one 67 against 63 us, 32 edge-labelled queries 215 against 197 us.
constexpr uint32_t kCtas = 8;

// A word read back from a queue or a list is clamped to the array it indexes
// before it is used (within() and vertex() in walk.cuh, place() here), at no
// cost that could be measured: no access leaves its array whatever a queue
// holds.  The host test of this kernel asserts that no clamp ever acts.
//
// A queue holds the partial mappings of one depth whose candidates are still
// to be checked.  A round takes 32 candidates of the deepest depth that has
// so many, so every deeper queue holds fewer than 32 entries (each has a
// candidate at least) and takes the round's up to 32 children: 63 at most.
constexpr uint32_t kQueue = 64;
// An entry is 16-byte chunks (each kQueue apart): a header -- the children's
// first node, slice start, slice length, candidates left -- and the tuple.
// Tuples whose suffixes are still to be counted have a queue of their own,
// emptied down to 31 pairs before any other round (header: first suffix,
// tuple length, -, suffixes left).
__host__ __device__ constexpr uint32_t tuple_chunks(uint32_t n) { return (n + 3) / 4; }
// An entry's place in its queue (63 entries at most, see above).
__device__ __forceinline__ uint32_t place(uint32_t e) {
    GFSM_CLAMPED(e >= kQueue);
    return e % kQueue;
}
// Chunks before depth d's queue (d >= 1; its entries have d vertices).
__host__ __device__ constexpr uint32_t queue_base(uint32_t d) {
    // sum over x < d of 1 + ceil(x / 4): four depths to each chunk count
    const uint32_t f = (d - 1) / 4, r = (d - 1) % 4;
    return kQueue * ((d - 1) + 2 * f * (f + 1) + r * (f + 1));
}
static_assert(queue_base(1) == 0 && queue_base(2) == 2 * kQueue && queue_base(6) == 11 * kQueue, "queue layout");
// Chunks of one warp's queues: depths 1 .. core - 1, then the suffix queue.
__host__ __device__ constexpr uint32_t queue_chunks(uint32_t core) {
    return queue_base(core) + kQueue * (1 + tuple_chunks(core));
}

__device__ __forceinline__ unsigned long long warp_total(unsigned long long x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(kFull, x, o);
    return x;
}

// Deals 32 items to 32 lanes: lane i brings n items, lane l gets item `local`
// of lane `from` (the first 32 items in lane order).  incl: running total.
// The lanes that bring any come before those that bring none.
__device__ __forceinline__ void deal(uint32_t n, uint32_t lane, uint32_t &incl, uint32_t &total, uint32_t &from,
                                     uint32_t &local) {
    incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, incl, o);
        if (lane >= (uint32_t)o) incl += y;
    }
    total = __shfl_sync(kFull, incl, 31);
    const uint32_t excl = incl - n;
    // the bits where a lane's items start; from = how many started before
    const uint32_t first = __reduce_or_sync(kFull, n && excl < 32 ? 1u << excl : 0u);
    from = (__popc(first & (kFull >> (31 - lane))) - 1) & 31;
    local = lane - __shfl_sync(kFull, excl, from);
}

// Bits of a lane's total from which it is added to the call's.
#ifndef GFSM_SPILL_BITS  // (set by a test)
#define GFSM_SPILL_BITS 30
#endif
constexpr uint32_t kSpillBits = GFSM_SPILL_BITS;

// Candidates in a unit that a limited pass leaves, at least: few, since the
// search below each can be long and there are far more warps than units.
constexpr uint32_t kUnit = 8;

// The unit of a queue entry (header h) that starts at its candidate `at`:
// children whole in groups where the slice is short, else parts of one slice.
__device__ __forceinline__ Chunk unit_at(const Chunk &h, uint32_t at, uint32_t size) {
    const uint32_t len = max(h.z, 1u), j = at / len, i = at - j * len;
    Chunk u{h.x + j, h.y + i, min(min(len - i, size), h.w - at), 0};
    u.w = u.z;
    if (i == 0 && u.z == len) u.w = len * min(max(1u, size / len), (h.w - at) / len);
    return u;  // (one candidate at least)
}

// Units in a list of which `listed` were asked for.
__host__ __device__ inline uint32_t list_units(uint32_t listed, uint32_t refused) {
    return listed <= kWalkListed ? listed : min(refused, kWalkListed);
}

// MODE: a whole walk's first pass, a pass of a limited walk, or a whole walk's
// later pass (as run-time switches they cost the first pass 5-12%).
// ROWS: mappings are written (their tables have no suffixes).
enum WalkMode { kWhole, kLimited, kLater };
template <bool LAB, WalkMode MODE, bool ROWS>
__global__ void __launch_bounds__(kWalkThreads, kCtas) k_walk(const WalkArgs a) {
    constexpr bool LIM = MODE == kLimited;
    GFSM_DYN_SHARED(sh);  // walk_smem() bytes
    __shared__ unsigned long long cta_sum[kWarps][4];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, below = (1u << lane) - 1u;
    const Tuple t{sh + (warp * tuple_chunks(a.core) * 32 + lane) * 4, 128};  // this lane's candidate's tuple
    Chunk *const queues = a.queues + (size_t)(blockIdx.x * kWarps + warp) * a.warp_chunks;
    Chunk *const squeue = queues + queue_base(a.core);
    uint32_t sents = 0, spairs = 0;  // the suffix queue's entries and (tuple, suffix) pairs
    uint32_t ents = 0, left = 0;     // lane d: entries and candidates of depth d's queue,
    const uint32_t base = queue_base(max(lane, 1u));  // and where it starts
    uint32_t fslot = 0, cand = 0, kept = 0, bytes = 0, front = 0;
    unsigned long long fcount = 0;
    unsigned long long u_next = 0, u_end = 0;  // this warp's units
    bool more = true;
    uint32_t rounds = 0;
    if (MODE == kLater && blockIdx.x * kWarps + warp < a.state_warps) {  // what this warp kept
        const WalkState &st = a.state_in[blockIdx.x * kWarps + warp];
        if (st.open) {
            ents = within(st.ents[lane], kQueue - 1);
            left = st.left[lane];
            sents = within(st.sents, kQueue - 1);
            spairs = st.spairs;
            u_next = st.u_next;
            u_end = min(st.u_end, a.units);
        }
    }
    // units of the list (l_end == 0: none left), dealt a few at a time
    const uint32_t l_count = MODE != kWhole && a.list_in ? list_units(__ldcg(&a.in->listed), __ldcg(&a.in->refused)) : 0u;
    const uint32_t l_chunk = max(1u, min(32u, l_count / (gridDim.x * kWarps)));
    uint32_t l_next = 1, l_end = l_count ? 1u : 0u;
    const uint32_t unit_chunks = 1 + tuple_chunks(a.core) + 1;
    // n units, a lane each, into the queues of their depths
    auto take_units = [&](uint32_t first, uint32_t n) {
        const Chunk *const u = a.list_in + (size_t)(first + lane) * unit_chunks;
        const bool has = lane < n;
        Chunk h{0, 0, 0, 0};
        uint32_t d = 0;
        if (has) {
            h = u[0];
            d = max(within(u[1].x, a.core - 1), 1u);
        }
        for (uint32_t rest = __ballot_sync(kFull, has); rest;) {
            const uint32_t depth = __shfl_sync(kFull, d, __ffs(rest) - 1);
            const uint32_t same = __ballot_sync(kFull, has && d == depth);
            const uint32_t e0 = __shfl_sync(kFull, ents, depth);
            Chunk *const q = queues + __shfl_sync(kFull, base, depth);
            const bool mine = has && d == depth;
            if (mine) {
                const uint32_t e = place(e0 + __popc(same & below));
                q[e] = h;
                for (uint32_t x = 0; x * 4 < depth; ++x) q[(1 + x) * kQueue + e] = u[2 + x];
            }
            const uint32_t got = __reduce_add_sync(kFull, mine ? h.w : 0u);
            if (lane == depth) {
                ents = e0 + __popc(same);
                left += got;
            }
            rest &= ~same;
        }
        __syncwarp();
    };
    auto add = [&](uint32_t slot, unsigned long long n) {
        if (fslot != slot && fcount) {
            atomicAdd(a.counts + fslot, fcount);
            fcount = 0;
        }
        fslot = slot;
        fcount += n;
    };
    // A lane's totals have 32 bits: they are added to the call's before they
    // can wrap (a round adds under 2^27 to each, several rounds 2^30 at most).
    auto spill = [&] {
        if (__any_sync(kFull, (bytes | front) >> kSpillBits)) {
            unsigned long long *const to = a.result->total[blockIdx.x % kWalkTotals];
            atomicAdd(to, (unsigned long long)cand);
            atomicAdd(to + 1, (unsigned long long)kept);
            atomicAdd(to + 2, (unsigned long long)bytes);
            atomicAdd(to + 3, (unsigned long long)front);
            cand = kept = bytes = front = 0;
        }
    };
    for (;;) {
        // ---- this round's work: suffixes once there are 32 pairs; else the
        // deepest depth with 32 candidates; else new roots; else (no more
        // roots) the shallowest depth with any; at last the rest of the pairs
        // (there is no queue of depth 0: in a whole walk lane 0's `left` counts
        // rounds, those of suffixes several times)
        const uint32_t full = __ballot_sync(kFull, left >= 32), any = __ballot_sync(kFull, left != 0) & ~1u;
        uint32_t d = 0;
        bool sfx = spairs >= 32;
        const bool closing = LIM && ++rounds > a.max_rounds;
        if (closing && !sfx) {
            if (!spairs) break;
            sfx = true;
        }
        if (!LIM && lane == 0) left += sfx ? 4 : 1;
        if (!sfx) {
            if (!LIM && (full & 1u)) {
                // A whole walk's warp looks now and then: once there is nothing
                // left to take in this pass and most of the chip is idle, what it
                // has queued goes to the next one, and to all warps.
                spill();
                bool end = false;
                if (lane == 0) {
                    left = 0;
                    ++ents;
                    end = a.look && !(ents & (a.look - 1)) && full > 1 && __ldcg(&a.result->done) >= a.most &&
                          __ldcg(&a.result->unit) >= a.units &&
                          (MODE == kWhole || !l_count || __ldcg(&a.in->taken) >= l_count);
                }
                if (__any_sync(kFull, end)) break;
            }
            if (full > 1) {
                d = 31 - __clz(full);
            } else {
                if (MODE != kWhole && l_end) {  // units that the pass before left come first
                    if (l_next >= l_end) {
                        uint32_t u = 0;
                        if (lane == 0) {
                            u = __ldcg(&a.in->taken);
                            if (u < l_count) u = atomicAdd(&a.in->taken, l_chunk);
                        }
                        l_next = __shfl_sync(kFull, u, 0);
                        l_end = min(l_next + l_chunk, l_count);
                        if (l_next >= l_count) l_next = l_end = 0;
                    }
                    if (l_end) {
                        take_units(l_next, min(l_end - l_next, 32u));
                        l_next += 32;
                        continue;
                    }
                }
                if (more && u_next >= u_end) {
                    // (a warp's first take goes straight to the counter; later it
                    // looks whether any are left: all warps adding to one
                    // word just to find out took 20 us, with 40 warps an SM)
                    unsigned long long u = 0;
                    if (lane == 0) {
                        if (u_end || (MODE != kWhole && a.list_in)) u = __ldcg(&a.result->unit);
                        if (u < a.units) u = atomicAdd(&a.result->unit, (unsigned long long)a.chunk);
                    }
                    u_next = __shfl_sync(kFull, u, 0);
                    u_end = min(u_next + a.chunk, a.units);
                    more = u_next < a.units;
                }
                if (!more) {
                    if (any) d = __ffs(any) - 1;
                    else if (spairs) sfx = true;
                    else break;
                }
            }
        }
        uint32_t c = 0, v = 0, idx = 0;
        bool act = false;
        if (sfx || d) {
            // ---- 32 items from the top of a queue, dealt to the lanes
            const uint32_t qd = __shfl_sync(kFull, base, d);
            Chunk *const q = sfx ? squeue : queues + qd;
            const uint32_t nd = __shfl_sync(kFull, ents, d), n = within(sfx ? sents : nd, kQueue);
            const uint32_t rem = lane < n ? q[n - 1 - lane].w : 0;
            uint32_t incl, total, from, local;
            deal(rem, lane, incl, total, from, local);
            const uint32_t take = min(total, 32u), e = n - 1 - from;
            const uint32_t frem = __shfl_sync(kFull, rem, from);
            act = lane < take;
            Chunk h{0, 0, 0, 0};
            if (act) {
                h = q[e];
                const uint32_t nc = sfx ? within(h.y, a.core) : d;
                for (uint32_t x = 0; x * 4 < nc; ++x) t.chunk(x) = q[(1 + x) * kQueue + e];
            }
            const uint32_t gone = __popc(__ballot_sync(kFull, rem && incl <= take));
            if (rem && incl > take && incl - rem < take) q[n - 1 - lane].w = incl - take;
            // from the end of what the entry had left: brought along by shuffle,
            // since the word in memory changes above (another lane's store)
            uint32_t i = frem - 1 - local;
            if (sfx) {
                sents = n - gone;
                spairs -= take;
                if (act) {
                    const WSfx *sx = a.sfx + within(h.x + i, a.sfxs - 1);
                    const uint32_t nc = within(h.y, a.core);
                    uint32_t first = 0;
                    const unsigned long long ways = suffix_count<LAB>(a.g, sx, t, nc, bytes, first);
                    if (ways) add(__ldg(&sx->slot), ways);
                    const uint32_t nleaf = __ldg(&sx->nleaf);
                    if (nleaf > 1 && first) front += (uint32_t)tuple_bytes(nc - 1);
                    if (nleaf > 2) front += first * (uint32_t)tuple_bytes(nc);
                }
                spill();  // (a hub's row is added for each of its suffixes)
                __syncwarp();
                continue;
            }
            if (lane == d) {
                ents = n - gone;
                left -= take;
            }
            if (act) {
                c = h.x;
                if (i >= h.z) {  // (child node, slice entry); the quotient is exact after one correction
                    uint32_t j = (uint32_t)__fdividef((float)i, (float)h.z);
                    if (j * h.z > i) --j;
                    if (i - j * h.z >= h.z) ++j;
                    c += j;
                    i -= j * h.z;
                }
                c = within(c, a.node_count - 1);
                idx = within(h.y + i, a.g.m - 1);
                v = __ldg(a.g.adj + idx);
            }
        } else {
            const unsigned long long u = u_next + lane;
            act = u < u_end;
            if (act) {
                uint32_t lo = 0, hi = a.roots;  // largest p with root_off[p] <= u
                while (hi - lo > 1) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (__ldg(a.root_off + mid) <= u) lo = mid; else hi = mid;
                }
                c = lo;
                v = __ldg(a.root_lo + lo) + (uint32_t)(u - __ldg(a.root_off + lo));
                bytes += 4;
            }
            u_next = min(u_next + 32, u_end);
        }
        // ---- check (the node's words are fetched along with the candidate)
        const WNode *const w = a.nodes + c;
        uint4 w0 = __ldg(reinterpret_cast<const uint4 *>(w)), w1 = __ldg(reinterpret_cast<const uint4 *>(w) + 1);
        const bool go = act && walk_check<LAB>(a.g, w, a.again, t, d, v, idx, bytes);
        cand += act;
        kept += go;
        if (go) {
            t.append(d, v);
            if (w1.w >> 24) {
                add(w0.w, 1);
                if constexpr (ROWS) {
                    const uint32_t slot = atomicAdd(a.rows_ctr, 1u);
                    if (slot < a.max_rows)
                        for (uint32_t x = 0; x <= d; ++x)
                            a.rows[(size_t)slot * (d + 1) + a.col[x]] = __ldg(a.order + vertex(a.g, t[x]));
                }
            }
        } else {
            w0.y = 0;
        }
        // ---- a tuple with suffixes joins the suffix queue
        const uint32_t nsfx = w0.y >> 16;
        const uint32_t sput = __ballot_sync(kFull, nsfx);
        if (sput) {
            if (nsfx) {
                const uint32_t e = place(sents + __popc(sput & below));
                squeue[e] = Chunk{w0.z, d + 1, 0, nsfx};
                for (uint32_t x = 0; x * 4 <= d; ++x) squeue[(1 + x) * kQueue + e] = t.chunk(x);
            }
            sents += __popc(sput);
            spairs += __reduce_add_sync(kFull, nsfx);
        }
        // ---- its children's slice; what has candidates joins the next queue
        // (a node's depth is its entry's: none below the last queue has children)
        GFSM_CLAMPED(d + 1 >= a.core && (w0.y & 0xffffu));
        const uint32_t nkid = d + 1 < a.core ? w0.y & 0xffffu : 0u;
        uint32_t s = 0, len = 0;
        if (nkid) walk_slice(a.g, Chunk{w1.x, w1.y, w1.z, w1.w}, t, s, len, bytes);
        const uint32_t put = __ballot_sync(kFull, len != 0);
        if (put) {
            Chunk *const q = queues + __shfl_sync(kFull, base, d + 1);
            const uint32_t n = __shfl_sync(kFull, ents, d + 1);
            if (len) {
                const uint32_t e = place(n + __popc(put & below));
                q[e] = Chunk{w0.x, s, len, len * nkid};
                for (uint32_t x = 0; x * 4 <= d; ++x) q[(1 + x) * kQueue + e] = t.chunk(x);
                front += (uint32_t)tuple_bytes(d);
                bytes += 4 * (d + 1);
            }
            const uint32_t got = __reduce_add_sync(kFull, len * nkid);
            if (lane == d + 1) {
                ents = n + __popc(put);
                left += got;
            }
        }
        __syncwarp();  // queue entries are read by other lanes next
    }
    // ---- what a pass of a whole walk leaves stays in its queues (k_split)
    bool open = false;
    if (!LIM && a.state_out) {
        if (lane == 0) ents = left = 0;
        open = __any_sync(kFull, left != 0);
        if (open && lane == 0) atomicAdd(&a.result->kept, 1u);
    }
    // ---- what a limited pass leaves: every queue entry as units of kUnit
    // candidates or more (about 64 to an entry at most), whole children or parts of one slice
    if (LIM && __any_sync(kFull, left != 0)) {
        if (!a.list_out) {
            if (lane == 0) a.result->gave_up = 1;
        } else {
            for (uint32_t d = 1; d < a.core; ++d) {
                const Chunk *const q = queues + __shfl_sync(kFull, base, d);
                const uint32_t n = within(__shfl_sync(kFull, ents, d), kQueue);
                for (uint32_t e = lane; e < n; e += 32) {
                    const Chunk h = q[e];
                    const uint32_t size = max(kUnit, (h.w + 63) / 64);
                    for (uint32_t at = 0; at < h.w;) {
                        const Chunk u = unit_at(h, at, size);
                        at += u.w;
                        const uint32_t slot = atomicAdd(&a.out->listed, 1u);
                        if (slot >= kWalkListed) {
                            a.result->gave_up = 1;
                            break;
                        }
                        Chunk *const o = a.list_out + (size_t)slot * unit_chunks;
                        o[0] = u;
                        o[1] = Chunk{d, 0, 0, 0};
                        for (uint32_t x = 0; x * 4 < d; ++x) o[2 + x] = q[(1 + x) * kQueue + e];
                    }
                }
            }
        }
    }
    // ---- counts and totals.  All warps adding to the same words one by one
    // took 25 us (with 40 warps an SM): a warp whose lanes hold one slot's count adds once, a CTA its
    // totals once, to one of kWalkTotals places.
    const uint32_t hold = __ballot_sync(kFull, fcount != 0);
    if (hold) {
        const uint32_t slot = __shfl_sync(kFull, fslot, __ffs(hold) - 1);
        if (__all_sync(kFull, fcount == 0 || fslot == slot)) {
            const unsigned long long n = warp_total(fcount);
            if (lane == 0) atomicAdd(a.counts + slot, n);
        } else if (fcount) {
            atomicAdd(a.counts + fslot, fcount);
        }
    }
    const unsigned long long sum[4] = {warp_total(cand), warp_total(kept), warp_total(bytes), warp_total(front)};
    if (lane < 4) cta_sum[warp][lane] = lane < 2 ? (lane ? sum[1] : sum[0]) : (lane == 3 ? sum[3] : sum[2]);
    __syncthreads();
    if (threadIdx.x < 4) {
        unsigned long long n = 0;
        for (uint32_t w = 0; w < kWarps; ++w) n += cta_sum[w][threadIdx.x];
        if (n) atomicAdd(&a.result->total[blockIdx.x % kWalkTotals][threadIdx.x], n);
    }
    if (!LIM && a.state_out) {
        WalkState &st = a.state_out[blockIdx.x * kWarps + warp];
        if (lane == 0) st.open = open;
        if (open) {
            st.ents[lane] = ents;
            st.left[lane] = left;
            if (lane == 0) {
                st.sents = sents;
                st.spairs = spairs;
                st.u_next = u_next;
                st.u_end = u_end;
            }
        }
    }
    // ---- the last CTA to get here hands the call's results to the host
    if (a.last) {
        __shared__ bool mine;
        __threadfence();  // this thread's adds, before its CTA is counted
        __syncthreads();
        if (threadIdx.x == 0) mine = atomicAdd(&a.result->done, 1u) == gridDim.x - 1;
        __syncthreads();
        if (mine) {
            __threadfence();
            const uint4 *const from = reinterpret_cast<const uint4 *>(a.result);
            for (uint32_t i = threadIdx.x; a.host && i < a.host_words; i += kWalkThreads) a.host[i] = __ldcg(from + i);
            if (threadIdx.x == 0) a.result->done = 0;  // for the next pass
        }
    }
}

// Between two passes of a whole walk: what the warps that closed have queued
// becomes units for all warps of the next, a warp each, shallowest depths (the
// largest trees) first, about `share` units a warp and one depth at least.
// Where the list has no room, the work stays with its warp.
__global__ void __launch_bounds__(kWalkThreads) k_split(const WalkArgs a) {
    const uint32_t lane = threadIdx.x & 31u, w = blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (w >= a.state_warps || !a.state_in[w].open) return;
    WalkState &st = a.state_in[w];
    const uint32_t ents = st.ents[lane], left = st.left[lane], unit_chunks = 1 + tuple_chunks(a.core) + 1;
    const Chunk *const queues = a.queues + (size_t)w * a.warp_chunks;
    uint32_t depths = 0, total = 0, mine = 0, at0 = 0;
    for (uint32_t pass = 0; pass < 2; ++pass) {  // count, then write
        for (uint32_t d = 1; d < a.core; ++d) {
            const uint32_t all = __shfl_sync(kFull, left, d), n = within(__shfl_sync(kFull, ents, d), kQueue);
            if (pass ? !(depths >> d & 1u) : !all || total >= a.share) continue;
            const Chunk *const q = queues + queue_base(d);
            const uint32_t size = max(kUnit, (all + a.share - 1) / a.share);
            for (uint32_t e = lane; e < n; e += 32) {
                const Chunk h = q[e];
                for (uint32_t at = 0; at < h.w;) {
                    const Chunk u = unit_at(h, at, size);
                    at += u.w;
                    if (pass) {
                        Chunk *const o = a.list_out + (size_t)at0++ * unit_chunks;
                        o[0] = u;
                        o[1] = Chunk{d, 0, 0, 0};
                        for (uint32_t x = 0; x * 4 < d; ++x) o[2 + x] = q[(1 + x) * kQueue + e];
                    } else {
                        ++mine;
                    }
                }
            }
            if (!pass) {
                depths |= 1u << d;
                total = __reduce_add_sync(kFull, mine);
            }
        }
        if (!pass) {  // room for all of them, or none is listed
            uint32_t incl = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFull, incl, o);
                if (lane >= (uint32_t)o) incl += y;
            }
            uint32_t first = 0;
            if (lane == 0) {
                first = atomicAdd(&a.out->listed, total);
                // the first warp without room: the list ends where it would have begun
                if (first <= kWalkListed && first + total > kWalkListed) a.out->refused = first;
            }
            first = __shfl_sync(kFull, first, 0);
            if (first + total > kWalkListed) return;
            at0 = first + incl - mine;
        }
    }
    if (depths >> lane & 1u) st.ents[lane] = st.left[lane] = 0;
}

// Bytes of dynamic shared memory: every lane's tuple.
inline uint32_t walk_smem(uint32_t core) { return tuple_chunks(core) * 32 * 16 * kWarps; }

// The units a warp takes at a time and the CTAs of the first pass.
struct WalkShape {
    uint32_t chunk, ctas;
};
inline WalkShape walk_shape(unsigned long long units, uint32_t roots, bool limited, int sms) {
    const unsigned long long warps = (unsigned long long)sms * kCtas * kWarps;
    // A warp takes 32 units at a time, up to 256 where each warp has many.
    // With fewer than that each takes its share at once, so that a small
    // call's roots spread over the whole chip; up to 128 under one root node
    // (3.2 takes a warp of 32 left some of them a fourth: one grid query 66
    // -> 57 us).  Under several, whose trees differ, each takes eight times,
    // 8 units at least (a take costs about 10 ns of the counter): against 32
    // or its share at once, kernel times of 32 edge-labelled queries 207 ->
    // 179 us, 275 on a small grid 200 -> 143 us, 1,179 on a larger one 1.35
    // -> 1.12 ms; one at a time three to twelve times as long.
    unsigned long long chunk = units / (warps * 16) / 32 * 32;
    chunk = std::min<unsigned long long>(limited ? 32 : 256, std::max<unsigned long long>(chunk, 32));
    const unsigned long long share = std::max<unsigned long long>(1, (units + warps - 1) / warps);
    if (!limited && roots > 1) {
        if (share < 256) chunk = std::min(share, std::max<unsigned long long>(8, share / 8));
    } else if (units < warps * (limited ? 32 : 128)) {
        chunk = share;
    }
    const unsigned long long need = (units + chunk - 1) / chunk;
    const uint32_t all = (uint32_t)sms * kCtas;
    return {(uint32_t)chunk,
            (uint32_t)std::max<unsigned long long>(1, std::min<unsigned long long>(all, (need + kWarps - 1) / kWarps))};
}

inline void (*walk_kernel(const WalkArgs &a, bool lab, WalkMode mode))(const WalkArgs) {
    if (a.rows && mode == kLater) return lab ? k_walk<true, kLater, true> : k_walk<false, kLater, true>;
    if (a.rows) return lab ? k_walk<true, kWhole, true> : k_walk<false, kWhole, true>;
    if (mode == kLater) return lab ? k_walk<true, kLater, false> : k_walk<false, kLater, false>;
    if (mode == kLimited) return lab ? k_walk<true, kLimited, false> : k_walk<false, kLimited, false>;
    return lab ? k_walk<true, kWhole, false> : k_walk<false, kWhole, false>;
}

// The arguments of pass p (see launch_walk); for a whole walk's p > 0 those of
// the k_split before it as well.
inline WalkArgs walk_pass(const WalkArgs &args, bool limited, Chunk *lists, int p, uint32_t kept, int sms) {
    WalkArgs a = args;
    a.warp_chunks = queue_chunks(a.core);
    const WalkShape shape = walk_shape(a.units, a.roots, limited, sms);
    a.chunk = shape.chunk;
    const uint32_t all = (uint32_t)sms * kCtas;
    a.ctas = p ? all : shape.ctas;
    Chunk *const list[2] = {lists, lists + (size_t)kWalkListed * (2 + tuple_chunks(a.core))};
    a.last = !limited || p + 1 == kWalkPasses;
    if (limited) {
        a.max_rounds = kWalkRounds[p];
        a.list_in = p ? list[(p - 1) & 1] : nullptr;
        a.list_out = a.last ? nullptr : list[p & 1];
        a.in = p ? a.result->list + (p - 1) : nullptr;
        a.out = a.result->list + p;
    } else if (lists) {
        // one list (k_split's output, the next pass' input) and the warps' states
        a.state_out = reinterpret_cast<WalkState *>(list[1]);
        if (p) {
            a.list_in = a.list_out = list[0];
            a.in = a.out = a.result->list;
            a.state_in = a.state_out;
            a.state_warps = (p > 1 ? all : shape.ctas) * kWarps;
            a.share = std::max(64u, kWalkListed / std::max(1u, kept));
        }
        a.most = a.ctas - std::min(a.ctas, all / 4);
        a.look = (p ? kept * 64ull : a.units) < (unsigned long long)all * kWarps ? kWalkLookFew : kWalkLookMany;
    }
    return a;
}

}  // namespace

}  // namespace gfsm
