// walk.cuh -- what one lane of the walk does: check a candidate, find a
// slice, count a suffix.  Host code too, so that a plain loop over the same
// functions can be compared with the oracle where there is no GPU.
#pragma once
#include "walk.h"

namespace gfsm {

#ifdef __CUDA_ARCH__
template <class T>
GFSM_HD T wld(const T *p) { return __ldg(p); }
#else
template <class T>
GFSM_HD T wld(const T *p) { return *p; }
#endif

struct WalkGraph {
    const uint32_t *__restrict__ rowptr;
    const uint32_t *__restrict__ adj;
    const uint8_t *__restrict__ elab;  // LAB instantiations: may be null (repeated entries, one label)
    // Row pointers by label group: row u's entries of group x are
    // adj[rowgrp[u * groups + x], rowgrp[u * groups + x + 1]).  Null: not
    // built (many groups), rows are searched.
    const uint32_t *__restrict__ rowgrp;
    // Entries of every row by label group, a byte each (at most 255); null
    // with more than 8 groups.
    const uint64_t *__restrict__ nlf;
    uint32_t groups;
    uint32_t single_label;
    uint32_t n, m;
};

// The tuple of one lane, in 16-byte chunks of four vertices; the chunks lie
// `step` words apart.  Words past the last vertex of its chunk hold kNoVertex.
constexpr uint32_t kNoVertex = 0xffffffffu;
struct alignas(16) Chunk {
    uint32_t x, y, z, w;
};
struct Tuple {
    uint32_t *m;
    uint32_t step;
    GFSM_HD uint32_t operator[](uint32_t i) const { return m[(i >> 2) * step + (i & 3u)]; }
    GFSM_HD Chunk &chunk(uint32_t c) const { return *reinterpret_cast<Chunk *>(m + c * step); }
    GFSM_HD void append(uint32_t n, uint32_t v) const {  // vertex n, behind vertices 0 .. n-1
        if (n & 3u) m[(n >> 2) * step + (n & 3u)] = v;
        else chunk(n >> 2) = Chunk{v, kNoVertex, kNoVertex, kNoVertex};
    }
    GFSM_HD bool has(uint32_t n, uint32_t v) const {
        bool f = false;
#pragma unroll 1
        for (uint32_t c = 0; c * 4 < n; ++c) {
            const Chunk k = chunk(c);
            f = f || k.x == v || k.y == v || k.z == v || k.w == v;
        }
        return f;
    }
};

// Told whether a clamp acts, which none should: the host test of the kernel
// counts them.
#ifndef GFSM_CLAMPED
#define GFSM_CLAMPED(acts)
#endif

// A word read back from a queue, kept inside the array it indexes whatever
// the queue holds.
GFSM_HD uint32_t within(uint32_t x, uint32_t last) {
    GFSM_CLAMPED(x > last);
    return x < last ? x : last;
}
// A vertex of a tuple read back from a queue.
GFSM_HD uint32_t vertex(const WalkGraph &g, uint32_t u) {
    GFSM_CLAMPED(u >= g.n);
    return u < g.n ? u : 0u;
}

// Rows of up to kWalkScan entries are trimmed from their ends; longer ones are
// searched.
constexpr uint32_t kWalkScan = 8;

// Loops of a few turns are kept rolled (unroll 1): the kernel's loop has to
// stay in the instruction cache.  4,096 grid queries, whole calls 67.3 ms with
// them unrolled, 55.4 ms rolled; 64 of them 1.37 and 1.34 ms.

// Entries below lo and below hi of the row adj[rs, re).
GFSM_HD void row_window(const WalkGraph &g, uint32_t rs, uint32_t re, uint32_t lo, uint32_t hi, uint32_t &s,
                        uint32_t &e) {
    // (one loop for both ends: less code in the kernel)
    uint32_t key = lo, first = rs;
    for (uint32_t end = 0; end < 2; ++end) {
        uint32_t a = first, b = re;
        if (key == 0) b = a;
        if (key >= g.n) a = b;
#pragma unroll 1
        while (a < b) {
            const uint32_t mid = a + ((b - a) >> 1);
            if (wld(g.adj + mid) < key) a = mid + 1; else b = mid;
        }
        if (!end) s = first = a;
        else e = a;
        key = hi;
    }
}

// reqExists (HnGPU.cu:34-52): does adj[rs, re) hold v (LAB: under label lab)?
template <bool LAB>
GFSM_HD bool row_has(const WalkGraph &g, uint32_t rs, uint32_t re, uint32_t v, uint32_t lab) {
    if constexpr (LAB) {
        if (g.elab) {
            uint32_t a = rs, b = re;
#pragma unroll 1
        while (a < b) {
                const uint32_t mid = a + ((b - a) >> 1);
                if (wld(g.adj + mid) < v) a = mid + 1; else b = mid;
            }
            for (; a < re && wld(g.adj + a) == v; ++a)
                if (wld(g.elab + a) == lab) return true;
            return false;
        }
    }
    if (lab != g.single_label) return false;
#pragma unroll 1
    while (re - rs > 4) {  // a label group's part of a row mostly is no longer
        const uint32_t mid = rs + ((re - rs) >> 1);
        if (wld(g.adj + mid) < v) rs = mid + 1; else re = mid + 1;
    }
    bool f = false;
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i)
        if (rs + i < re && wld(g.adj + rs + i) == v) f = true;
    return f;
}

// Is every byte of a at least that of b?
GFSM_HD bool bytes_at_least(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
    return !(__vsubus4((uint32_t)b, (uint32_t)a) | __vsubus4((uint32_t)(b >> 32), (uint32_t)(a >> 32)));
#else
    for (int i = 0; i < 64; i += 8)
        if ((a >> i & 255u) < (b >> i & 255u)) return false;
    return true;
#endif
}

// A candidate v (entry idx of its row; d = 0: a root, no row) of node w,
// behind the d vertices of t: injectivity (HnGPU.cu:223-236), the anchor
// edge's label, the other requirements (:243-252).
template <bool LAB>
GFSM_HD bool walk_check(const WalkGraph &g, const WNode *w, const WAgain *again, const Tuple &t, uint32_t d, uint32_t v,
                        uint32_t idx, uint32_t &bytes) {
    const uint32_t head = wld(reinterpret_cast<const uint32_t *>(&w->nreq));  // nreq and group, anchor, its label, its check
    const uint32_t more = wld(&w->again);
    bool ok = !t.has(d, v);
    // a neighbour for each of the query vertex's, by label; and for each of
    // the earlier vertices', where this node's queries part from others
    ok = ok && (!g.nlf || bytes_at_least(wld(g.nlf + v), wld(&w->need)));
    for (uint32_t i = 0; ok && g.nlf && i < (more & 255u); ++i) {
        const WAgain *q = again + (more >> 8) + i;
        ok = bytes_at_least(wld(g.nlf + vertex(g, t[wld(&q->pos)])), wld(&q->need));
    }
    if (LAB && ok && d) {
        const uint32_t lab = (head >> 16) & 255u;
        if (head >> 24) {
            const uint32_t u = vertex(g, t[(head >> 8) & 255u]);
            ok = row_has<LAB>(g, wld(g.rowptr + u), wld(g.rowptr + u + 1), v, lab);
        } else if (g.elab) {
            ok = wld(g.elab + idx) == lab;
        }
    }
    // a row's entries of v's own label group are enough (the whole row of a
    // self-loop requirement at a root, whose group a partition may cut)
    const uint32_t grp = head >> 4 & 15u;
    for (uint32_t r = 0; ok && r < (head & 15u); ++r) {
        const uint32_t pos = wld(&w->req_pos[r]);
        const uint32_t u = vertex(g, pos == REQ_SELF ? v : t[pos]);
        const bool part = g.rowgrp && grp != kNoGroup;
        const uint32_t *p = part ? g.rowgrp + (size_t)u * g.groups + grp : g.rowptr + u;
        const uint32_t rs = wld(p), re = wld(p + 1);
        bytes += 4 * (re - rs + 1);
        ok = row_has<LAB>(g, rs, re, v, wld(&w->req_lab[r]));
    }
    return ok;
}

// A window narrowed by symmetry breaking (bits 0-15: the positions it
// exceeds, 16-31: those it stays below).
GFSM_HD void narrow(const Tuple &t, uint32_t masks, uint32_t &lo, uint32_t &hi) {
    while (masks) {
#ifdef __CUDA_ARCH__
        const uint32_t i = __ffs(masks) - 1;
#else
        const uint32_t i = (uint32_t)__builtin_ctz(masks);
#endif
        masks &= masks - 1;
        const uint32_t x = t[i & 15u];
        if (i < 16) lo = lo > x + 1 ? lo : x + 1;
        else hi = hi < x ? hi : x;
    }
}

// The part adj[s, e) of u's row in a window: its label group's entries,
// searched only where the window leaves some of the group out.
GFSM_HD void slice_of(const WalkGraph &g, uint32_t u, uint32_t grp, bool trim, uint32_t lo, uint32_t hi, uint32_t &s,
                      uint32_t &e) {
    u = vertex(g, u);
    if (g.rowgrp) {
        const uint32_t *p = g.rowgrp + (size_t)u * g.groups + grp;
        s = wld(p);
        e = wld(p + 1);
    } else {
        s = wld(g.rowptr + u);
        e = wld(g.rowptr + u + 1);
        trim = true;
    }
    if (trim) {
        if (e - s > kWalkScan) {
            if (lo < hi) row_window(g, s, e, lo, hi, s, e);
            else e = s;
        } else {  // one or two entries usually
#pragma unroll 1
            while (s < e && wld(g.adj + e - 1) >= hi) --e;
#pragma unroll 1
            while (s < e && wld(g.adj + s) < lo) ++s;
        }
    }
}

// A leaf group at hand: its window (narrowed by the tuple) in its anchor's row.
struct Leaf {
    uint32_t lo, hi, s, e, lab, mult;
};
GFSM_HD Leaf leaf_slice(const WalkGraph &g, const Tuple &t, const WSfxGroup *q, uint32_t &bytes) {
    Leaf l;
    l.lo = wld(&q->lo);
    l.hi = wld(&q->hi);
    const uint32_t masks = wld(reinterpret_cast<const uint32_t *>(&q->lb));
    const uint32_t rest = wld(reinterpret_cast<const uint32_t *>(&q->anchor));  // anchor, label, group, form
    if (masks) narrow(t, masks, l.lo, l.hi);
    l.lab = (rest >> 8) & 255u;
    l.mult = (rest >> 24) & 15u;
    slice_of(g, t[rest & 255u], (rest >> 16) & 255u, masks || (rest >> 30 & 1u), l.lo, l.hi, l.s, l.e);
    bytes += 4 * (l.e - l.s + 2);
    return l;
}

// Vertices of a leaf's slice that are not among the nc core vertices.
template <bool LAB>
GFSM_HD uint32_t leaf_set(const WalkGraph &g, const Tuple &t, uint32_t nc, const Leaf &l) {
    const uint32_t n = l.e - l.s;
    uint32_t k = 0;
    if ((LAB && g.elab) || n <= 2 * kWalkScan) {
#pragma unroll 1
        for (uint32_t i = l.s; i < l.e; ++i) {
            bool ok = !t.has(nc, wld(g.adj + i));
            if (LAB && g.elab) ok = ok && wld(g.elab + i) == l.lab;
            k += ok ? 1u : 0u;
        }
        return k;
    }
    k = n;
#pragma unroll 1
    for (uint32_t i = 0; i < nc; ++i) {
        const uint32_t x = t[i];
        if (x >= l.lo && x < l.hi && row_has<false>(g, l.s, l.e, x, g.single_label)) --k;
    }
    return k;
}

// Vertices outside the core that two leaves' slices share.
template <bool LAB>
GFSM_HD uint32_t leaf_meet(const WalkGraph &g, const Tuple &t, uint32_t nc, const Leaf &a, const Leaf &b) {
    uint32_t k = 0;
#pragma unroll 1
    for (uint32_t i = a.s; i < a.e; ++i) {
        const uint32_t x = wld(g.adj + i);
        bool ok = x >= b.lo && x < b.hi && !t.has(nc, x);
        if (LAB && g.elab) ok = ok && wld(g.elab + i) == a.lab;
        ok = ok && row_has<LAB>(g, b.s, b.e, x, (LAB && g.elab) ? b.lab : g.single_label);
        k += ok ? 1u : 0u;
    }
    return k;
}

GFSM_HD uint64_t falling(uint64_t n, uint32_t c) {  // n (n-1) ... (n-c+1)
    uint64_t r = 1;
#pragma unroll 1
    for (uint32_t i = 0; i < c; ++i) r = n > i ? r * (n - i) : 0;
    return r;
}

// Ways to place the leaves of suffix x behind the nc core vertices of t,
// all on distinct vertices.  first: vertices the first group can take.
template <bool LAB>
GFSM_HD uint64_t suffix_count(const WalkGraph &g, const WSfx *x, const Tuple &t, uint32_t nc, uint32_t &bytes,
                              uint32_t &first) {
    uint64_t total = 1;
    const uint32_t ng = wld(&x->ng);
    Leaf a{};
    uint32_t na = 0;  // the group before, when this one's window meets its
    for (uint32_t i = 0; i < ng; ++i) {
        const Leaf l = leaf_slice(g, t, &x->g[i], bytes);
        const uint32_t n = leaf_set<LAB>(g, t, nc, l);
        if (i == 0) first = n;
        if (n < l.mult) return 0;
        const uint32_t groups = wld(&x->g[i].form) >> 4 & 3u;
        if (groups == 2) {
            a = l;
            na = n;
        } else if (groups == 0) {
            // j of a's leaves on the m vertices both can take, the others
            // outside them, then this group's on what is left of its own
            const uint64_t m = leaf_meet<LAB>(g, t, nc, a, l);
            uint64_t sum = 0, choose = 1;
            for (uint32_t j = 0; j <= a.mult && j <= m; ++j) {
                if (n >= j) sum += choose * falling(m, j) * falling(na - m, a.mult - j) * falling(n - j, l.mult);
                choose = choose * (a.mult - j) / (j + 1);
            }
            total *= sum;
        } else {
            total *= falling(n, l.mult);
        }
        if (!total) return 0;
    }
    return total;
}

// The children's candidates behind the tuple t of a node (words 4-7 of it:
// window, masks, anchor | group | trim | final).
GFSM_HD void walk_slice(const WalkGraph &g, const Chunk &w, const Tuple &t, uint32_t &s, uint32_t &len,
                        uint32_t &bytes) {
    uint32_t lo = w.x, hi = w.y, e;
    if (w.z) narrow(t, w.z, lo, hi);
    slice_of(g, t[w.w & 255u], (w.w >> 8) & 255u, w.z || (w.w >> 16 & 255u), lo, hi, s, e);
    len = e - s;
    bytes += 4 * (len + 2);
}

}  // namespace gfsm
