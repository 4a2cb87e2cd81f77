// walk_plan.cpp -- host tables of the walk: the trie of a call's plans and
// the suffixes of trailing leaves.
#include <algorithm>
#include <cstring>
#include <memory>
#include <thread>

#include "walk.h"

namespace gfsm {

namespace {

// Everything that makes two queries the same at one depth: how a candidate is
// checked, and which slice the next depth's candidates come from.
struct Step {
    uint8_t check[24];   // nreq, anchor, anchor_lab, anchor_check, 0, requirements (WNode's last words)
    uint32_t lo, hi;     // the next depth's window
    uint16_t lb, ub;
    uint8_t anchor, grp, trim;
    uint8_t kind;        // 0: more core vertices, 1: the suffix follows, 2: the query ends here
};
static_assert(sizeof(Step) == 40, "no padding in a key");

struct Query {
    uint32_t core = 0;
    Step st[MAXQ];
    uint64_t need[MAXQ];  // WNode::need of each core depth
    WSfx sfx;
    uint64_t mult = 1;
};


typedef uint8_t Bytes8 __attribute__((vector_size(8)));
uint64_t bytes_min(uint64_t a, uint64_t b) {
    Bytes8 x, y;
    std::memcpy(&x, &a, 8);
    std::memcpy(&y, &b, 8);
    x = x < y ? x : y;
    std::memcpy(&a, &x, 8);
    return a;
}

uint64_t hash_bytes(const void *p, size_t n, uint64_t h) {
    const char *c = static_cast<const char *>(p);
    for (; n >= 8; n -= 8, c += 8) {
        uint64_t x;
        std::memcpy(&x, c, 8);
        h = (h ^ x) * 0xff51afd7ed558ccdull;
        h ^= h >> 32;
    }
    return h;
}

// Open-addressing set of item ids; the caller compares.
struct IdTable {
    std::vector<uint32_t> cell;
    uint32_t mask;
    void reset(size_t n) {
        size_t c = 2;
        while (c < 2 * n) c *= 2;
        cell.assign(c, ~0u);
        mask = (uint32_t)(c - 1);
    }
    template <class Eq>
    uint32_t find_or_add(uint64_t h, uint32_t id, Eq eq) {  // the equal item's id, or id itself (added)
        for (uint32_t i = (uint32_t)(h ^ (h >> 29)) & mask;; i = (i + 1) & mask) {
            if (cell[i] == ~0u) {
                cell[i] = id;
                return id;
            }
            if (eq(cell[i])) return cell[i];
        }
    }
};

// Can the placements of these leaves be counted without enumerating them?
// Groups whose windows meet may take the same vertex: one such group alone is
// a falling factorial, two have a closed form over their intersection
// (suffix_count in walk.cuh), three or more are left to the search.
bool classify(WSfx &s, bool cross) {
    // order the groups so that classes of meeting windows are consecutive
    uint8_t cls[kSfxGroups];
    for (int i = 0; i < s.ng; ++i) cls[i] = (uint8_t)i;
    for (int pass = 0; pass < s.ng; ++pass)
        for (int i = 0; i < s.ng; ++i)
            for (int j = 0; j < s.ng; ++j)
                if (std::max(s.g[i].lo, s.g[j].lo) < std::min(s.g[i].hi, s.g[j].hi))
                    cls[i] = cls[j] = std::min(cls[i], cls[j]);
    WSfxGroup out[kSfxGroups];
    int n = 0;
    for (int c = 0; c < s.ng; ++c) {
        const int first = n;
        bool same_anchor = true;
        for (int i = 0; i < s.ng; ++i)
            if (cls[i] == c) {
                out[n] = s.g[i];
                same_anchor = same_anchor && out[n].anchor == out[first].anchor;
                ++n;
            }
        const int sz = n - first;
        if (!sz) continue;
        if (sz > 2 || (sz == 2 && !same_anchor && !cross)) return false;
        out[first].form |= (uint8_t)(sz << 4);
    }
    std::copy(out, out + n, s.g);
    return true;
}

// A window, its label group, and whether it leaves out enough of the group to
// be worth applying.  A window's upper end is the degree filter, which never
// changes a count: where the vertices it leaves out hold under 1 / kTrimShare
// of the group's entries, the whole group is taken.  Its part of a row needs
// no search then (WalkGraph::rowgrp), and queries that differ in a vertex's
// degree alone share their nodes.
struct Window {
    uint32_t lo, hi;
    uint8_t grp, trim;  // group 255: none (no row pointers by group then)
};
constexpr uint64_t kTrimShare = 4;
Window window_of(const DeviceGraph &g, uint32_t lo, uint32_t hi) {
    const auto it = std::upper_bound(g.group_start.begin(), g.group_start.end(), lo);
    const size_t gi = it == g.group_start.begin() ? 0 : (size_t)(it - g.group_start.begin()) - 1;
    if (gi + 1 >= g.group_start.size() || gi >= 255 || lo >= hi) return {lo, hi, 255, 1};
    const uint32_t a = g.group_start[gi], b = g.group_start[gi + 1];
    const uint64_t all = g.h_rowptr[b] - g.h_rowptr[a], cut = g.h_rowptr[b] - g.h_rowptr[std::min(hi, b)];
    if (lo != a || hi > b || cut * kTrimShare > all) return {lo, hi, (uint8_t)gi, 1};
    return {a, b, (uint8_t)gi, 0};
}

// Turns the leaves [s, k) of a query into a suffix; false if it cannot be.
bool make_suffix(const DQuery &dq, const DeviceGraph &dg, uint32_t s, const uint16_t *lb, const uint16_t *ub, bool cross, WSfx &out) {
    std::memset(&out, 0, sizeof(out));
    out.nleaf = (uint8_t)(dq.k - s);
    for (uint32_t d = s; d < dq.k; ++d) {
        const DLevel &L = dq.lv[d];
        if (L.nreq || L.anchor_check || L.anchor >= s) return false;
        const Window w = window_of(dg, L.lo, L.hi);
        WSfxGroup g{w.lo, w.hi, lb[d], ub[d], L.anchor, L.anchor_lab, w.grp, (uint8_t)(1u | w.trim << 6)};
        int i = 0;
        for (; i < out.ng; ++i) {
            WSfxGroup &o = out.g[i];
            if (o.lo == g.lo && o.hi == g.hi && o.lb == g.lb && o.ub == g.ub && o.anchor == g.anchor &&
                o.lab == g.lab) {
                ++o.form;
                break;
            }
        }
        if (i < out.ng) continue;
        if (out.ng == kSfxGroups) return false;
        out.g[out.ng++] = g;
    }
    return classify(out, cross);
}

bool make_query(const WalkQuery &w, const DeviceGraph &g, bool leaves, bool cross, bool desc, Query &q) {
    const DQuery &dq = *w.dq;
    const uint32_t k = dq.k;
    uint32_t depth[MAXQ] = {};
    for (uint32_t d = 0; d < k; ++d) depth[w.plan->qvid[d]] = d;
    // A condition (a, b), a placed before b, bounds b by a.  With the core
    // cut at s, the conditions whose a is a leaf are dropped: the leaves are
    // then counted in every order, the product of those a's orbits too often.
    auto bounds = [&](uint32_t s, uint16_t *lb, uint16_t *ub, uint64_t &mult) {
        std::fill(lb, lb + MAXQ, (uint16_t)0);
        std::fill(ub, ub + MAXQ, (uint16_t)0);
        mult = w.sym ? w.plan->aut : 1;
        if (!w.sym) return;
        uint64_t orbit[MAXQ];
        std::fill(orbit, orbit + MAXQ, 1);
        for (const auto &c : w.plan->sym_cond) {
            const uint32_t a = depth[c.first], b = depth[c.second];
            if (a >= s) ++orbit[a];
            else (desc ? ub : lb)[b] |= (uint16_t)(1u << a);
        }
        for (uint32_t d = s; d < k; ++d) mult /= orbit[d];
    };
    uint16_t lb[MAXQ], ub[MAXQ];
    uint32_t s = k;
    if (leaves && k >= 2) {
        uint32_t n = 0;  // trailing levels without a requirement
        while (n + 1 < k && !dq.lv[k - 1 - n].nreq && !dq.lv[k - 1 - n].anchor_check) ++n;
        for (; n; --n) {
            bounds(k - n, lb, ub, q.mult);
            if (make_suffix(dq, g, k - n, lb, ub, cross, q.sfx)) {
                s = k - n;
                break;
            }
        }
    }
    if (s == k) bounds(k, lb, ub, q.mult);
    q.core = s;
    // Neighbours the vertex of each depth has in the query: the later ones
    // are looked for in its row, and so are the earlier ones where the data
    // is symmetric.
    uint8_t need[MAXQ][8] = {};
    uint8_t grp[MAXQ];
    for (uint32_t d = 0; d < k; ++d) {
        const DLevel &L = dq.lv[d];
        grp[d] = window_of(g, L.lo, L.hi).grp;
        uint32_t back = d ? 1u << L.anchor : 0u;
        for (uint32_t r = 0; r < L.nreq; ++r)
            if (L.req_pos[r] != REQ_SELF) back |= 1u << L.req_pos[r];
        for (uint32_t p = 0; p < d; ++p)
            if (back >> p & 1u) {
                if (grp[d] < 8) ++need[p][grp[d]];
                if (g.symmetric && grp[p] < 8) ++need[d][grp[p]];
            }
    }
    for (uint32_t d = 0; d < s; ++d) {
        std::memcpy(&q.need[d], need[d], 8);
        const DLevel &L = dq.lv[d];
        if (L.nreq > kWalkReqs) return false;
        Step &t = q.st[d];
        std::memset(&t, 0, sizeof(t));
        const Window own = window_of(g, L.lo, L.hi);
        t.check[0] = (uint8_t)(L.nreq | (own.grp < kNoGroup ? own.grp : kNoGroup) << 4);
        t.check[1] = L.anchor;
        t.check[2] = L.anchor_lab;
        t.check[3] = L.anchor_check;
        std::memcpy(t.check + 8, L.req_pos, kWalkReqs);
        std::memcpy(t.check + 8 + kWalkReqs, L.req_lab, kWalkReqs);
        t.kind = d + 1 < s ? 0 : s < k ? 1 : 2;
        if (t.kind == 0) {
            const DLevel &N = dq.lv[d + 1];
            t.anchor = N.anchor;
            const Window win = window_of(g, N.lo, N.hi);
            t.lo = win.lo;
            t.hi = win.hi;
            t.grp = win.grp;
            t.trim = win.trim;
            t.lb = lb[d + 1];
            t.ub = ub[d + 1];
        }
    }
    return true;
}

struct Kid {
    uint32_t parent, rep;
};
struct Needs {
    uint64_t of[MAXQ];
};

}  // namespace

// Kept between calls: fresh pages for a few MB cost as much as the work.
struct WalkScratch {
    RawVec<Query> qs;
    std::vector<std::pair<uint32_t, uint32_t>> root;
    std::vector<uint32_t> alive, parent, made, order, place, next;
    std::vector<Kid> kids;
    std::vector<Needs> needs, asked;
    std::vector<std::pair<uint32_t, uint32_t>> sfx_of;
    IdTable full, checks, seen;
};

void trim_walk(WalkTables &t) {
    if (t.scratch && t.scratch->qs.size() > (1u << 16)) t = WalkTables();
}

bool build_walk(const std::vector<WalkQuery> &ws, const DeviceGraph &g, bool share, bool leaves, bool cross, bool desc,
                WalkTables &out) {
    const uint32_t nq = (uint32_t)ws.size();
    if (!out.scratch) out.scratch = std::make_shared<WalkScratch>();
    WalkScratch &m = *out.scratch;
    RawVec<Query> &qs = m.qs;
    qs.resize(nq);
    // root windows: whole groups as well, except where the window is part of
    // the result (one part of a partition, a query of one vertex)
    std::vector<std::pair<uint32_t, uint32_t>> &root = m.root;
    root.resize(nq);
    for (uint32_t i = 0; i < nq; ++i) {
        root[i] = {ws[i].lo, ws[i].hi};
        const DLevel &L = ws[i].dq->lv[0];
        if (L.lo != ws[i].lo || L.hi != ws[i].hi || ws[i].dq->k < 2) continue;
        const Window w = window_of(g, L.lo, L.hi);
        root[i] = {w.lo, w.hi};
    }
    // the queries one by one: a few host threads for a large batch
    const int nt = std::max(1, std::min<int>(host_threads(), (int)(nq / 128)));
    std::vector<char> fits(nt, 1);
    auto work = [&](int t) {
        for (uint32_t i = (uint32_t)t; i < nq; i += (uint32_t)nt)
            fits[t] = fits[t] && make_query(ws[i], g, leaves, cross, desc, qs[i]);
    };
    std::vector<std::thread> pool;
    for (int t = 1; t < nt; ++t) {
        try {
            pool.emplace_back(work, t);
        } catch (...) {  // no thread to be had: this one does its share
            work(t);
        }
    }
    work(0);
    for (std::thread &th : pool) th.join();
    for (char f : fits)
        if (!f) return false;
    uint32_t core = 0;
    for (uint32_t i = 0; i < nq; ++i) core = std::max(core, qs[i].core);
    out.core = core;
    out.slot.assign(nq, 0);
    out.mult.resize(nq);
    for (uint32_t i = 0; i < nq; ++i) out.mult[i] = qs[i].mult;
    out.nodes.clear();
    out.sfx.clear();
    out.again.clear();
    out.nodes.reserve(4 * nq);
    out.nslots = 0;

    // level by level: the queries still alive, each at its parent's node
    std::vector<uint32_t> &alive = m.alive, &parent = m.parent, &made = m.made, &order = m.order, &place = m.place,
                          &next = m.next;
    alive.resize(nq);
    parent.resize(nq);
    made.resize(nq);
    for (uint32_t i = 0; i < nq; ++i) {
        alive[i] = i;
        parent[i] = share ? 0u : i;
    }
    std::vector<Kid> &kids = m.kids;
    std::vector<Needs> &needs = m.needs, &asked = m.asked;  // per node of this level and of the one before
    uint32_t parent_base = 0;
    std::vector<std::pair<uint32_t, uint32_t>> &sfx_of = m.sfx_of;  // (node, query), this level's suffixes
    for (uint32_t d = 0; !alive.empty(); ++d) {
        const uint32_t base = (uint32_t)out.nodes.size();
        kids.clear();
        IdTable &full = m.full, &checks = m.checks;
        full.reset(alive.size());
        checks.reset(alive.size());
        auto root_same = [&](uint32_t a, uint32_t b) { return d || root[a] == root[b]; };
        auto head = [&](uint32_t i) {
            uint64_t h = 0x9e3779b97f4a7c15ull * (parent[i] + 1);
            if (!d) h ^= ((uint64_t)root[i].first << 32 | root[i].second) * 0xc4ceb9fe1a85ec53ull;
            return h;
        };
        // queries that go on first: one whose suffix follows joins any node
        // that checks its candidates the same way
        for (int pass = 0; pass < 2; ++pass)
            for (const uint32_t i : alive) {
                const Step &t = qs[i].st[d];
                if ((t.kind == 1) != (pass == 1)) continue;
                const uint32_t id = (uint32_t)kids.size();
                uint32_t k = id;
                const uint64_t hc = hash_bytes(t.check, sizeof(t.check), head(i));
                auto same_check = [&](uint32_t x) {
                    const uint32_t r = kids[x].rep;
                    return kids[x].parent == parent[i] && root_same(r, i) &&
                           !std::memcmp(qs[r].st[d].check, t.check, sizeof(t.check));
                };
                if (pass == 0)
                    k = full.find_or_add(hash_bytes(&t, sizeof(t), head(i)), id, [&](uint32_t x) {
                        const uint32_t r = kids[x].rep;
                        return kids[x].parent == parent[i] && root_same(r, i) &&
                               !std::memcmp(&qs[r].st[d], &t, sizeof(t));
                    });
                if (k == id) {
                    const uint32_t c = checks.find_or_add(hc, id, same_check);
                    if (pass == 1) k = c;
                }
                if (k == id) kids.push_back({parent[i], i});
                made[i] = k;
            }
        // number this level's nodes by parent, so that siblings are consecutive
        const uint32_t pb = d ? parent_base : 0u, np = d ? base - parent_base : share ? 1u : nq;
        place.assign(np + 1, 0);  // (a counting sort: first where each parent's children start)
        for (const Kid &k : kids) ++place[k.parent - pb + 1];
        for (uint32_t x = 0; x < np; ++x) place[x + 1] += place[x];
        order.resize(kids.size());
        for (uint32_t x = 0; x < kids.size(); ++x) order[place[kids[x].parent - pb]++] = x;
        place.resize(kids.size());
        for (uint32_t x = 0; x < order.size(); ++x) {
            const Kid &kd = kids[order[x]];
            place[order[x]] = base + x;
            out.nodes.emplace_back();
            WNode &n = out.nodes.back();
            std::memset(&n, 0, sizeof(n));
            const Step &t = qs[kd.rep].st[d];
            std::memcpy(&n.nreq, t.check, sizeof(t.check));
            n.next_lo = t.lo;
            n.next_hi = t.hi;
            n.next_lb = t.lb;
            n.next_ub = t.ub;
            n.next_anchor = t.anchor;
            n.next_grp = t.grp;
            n.next_trim = t.trim;
            if (d) {
                WNode &p = out.nodes[kd.parent];
                if (p.nchild == 0xffff) return false;
                if (!p.nchild++) p.child = base + x;
            }
        }
        // what the rows of a node's vertices need: what all its queries do.
        // For its own vertex that is part of the check; for the earlier ones
        // what their nodes, shared by more queries, could not ask yet.
        needs.resize(kids.size());
        for (Needs &n : needs) std::fill(n.of, n.of + d + 1, ~0ull);
        for (const uint32_t i : alive)
            for (uint32_t t = 0; t <= d; ++t) {
                uint64_t &a = needs[place[made[i]] - base].of[t];
                a = bytes_min(a, qs[i].need[t]);
            }
        for (uint32_t x = 0; x < order.size(); ++x) {
            WNode &n = out.nodes[base + x];
            n.need = needs[x].of[d];
            const uint32_t first = (uint32_t)out.again.size();
            for (uint32_t t = 0; t < d; ++t) {
                const uint64_t had = asked[kids[order[x]].parent - parent_base].of[t], now = needs[x].of[t];
                if (bytes_min(had, now) != now) out.again.push_back({now, t, 0});
            }
            n.again = first << 8 | (uint32_t)(out.again.size() - first);
        }
        if (out.again.size() >= (1u << 24)) return false;
        asked.swap(needs);
        parent_base = base;
        // queries that end here, and suffixes (equal ones once per node)
        next.clear();
        sfx_of.clear();
        for (const uint32_t i : alive) {
            const uint32_t node = place[made[i]];
            const Step &t = qs[i].st[d];
            if (t.kind == 0) {
                parent[i] = node;
                next.push_back(i);
            } else if (t.kind == 1) {
                sfx_of.push_back({node, i});
            } else {
                WNode &n = out.nodes[node];
                if (!n.final_) {
                    n.final_ = 1;
                    n.slot = out.nslots++;
                }
                out.slot[i] = n.slot;
            }
        }
        std::stable_sort(sfx_of.begin(), sfx_of.end(),
                         [](const std::pair<uint32_t, uint32_t> &a, const std::pair<uint32_t, uint32_t> &b) {
                             return a.first < b.first;
                         });
        for (size_t a = 0; a < sfx_of.size();) {
            size_t b = a;
            WNode &n = out.nodes[sfx_of[a].first];
            n.sfx = (uint32_t)out.sfx.size();
            size_t end = a;
            while (end < sfx_of.size() && sfx_of[end].first == sfx_of[a].first) ++end;
            IdTable &seen = m.seen;
            seen.reset(end - a);
            for (; b < sfx_of.size() && sfx_of[b].first == sfx_of[a].first; ++b) {
                const uint32_t i = sfx_of[b].second;
                WSfx &s = qs[i].sfx;
                const uint32_t id = (uint32_t)out.sfx.size();
                const uint32_t got = seen.find_or_add(hash_bytes(&s.ng, sizeof(WSfx) - 4, 1), id, [&](uint32_t x) {
                    return !std::memcmp(&out.sfx[x].ng, &s.ng, sizeof(WSfx) - 4);
                });
                if (got == id) {
                    if (n.nsfx == 0xffff) return false;
                    ++n.nsfx;
                    s.slot = out.nslots++;
                    out.sfx.push_back(s);
                }
                out.slot[i] = out.sfx[got].slot;
            }
            a = b;
        }
        if (d == 0) {  // the root windows
            out.root_lo.clear();
            out.root_off.assign(1, 0);
            for (uint32_t x = 0; x < order.size(); ++x) {
                const auto &w = root[kids[order[x]].rep];
                out.root_lo.push_back(w.first);
                out.root_off.push_back(out.root_off.back() + (w.second - w.first));
            }
        }
        alive.swap(next);
    }
    return true;
}

}  // namespace gfsm
