// The walk's tables and per-candidate functions on the host: a plain
// depth-first loop over them, for tests without a GPU.
//   walk_host <vertex labels> <share> <leaves> <cross> <desc> <data> <query>...
// prints each query's count (one line each), then "core <c> nodes <n> sfx <s>".
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <numeric>

#include "../gfsm_b200/csrc/walk.cuh"

using namespace gfsm;

// The device CCSR's host-side fields and arrays, as build_device_graph
// leaves them.
static void host_ccsr(const HostGraph &h, bool vl, DeviceGraph &g, std::vector<uint32_t> &adj, std::vector<uint8_t> &lab) {
    const uint32_t n = h.n;
    const uint64_t m = h.src.size();
    std::vector<uint32_t> deg(n, 0), order(n), inv(n);
    for (uint32_t s : h.src) deg[s]++;
    std::iota(order.begin(), order.end(), 0u);
    std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) {
        if (vl && h.vlabel[a] != h.vlabel[b]) return h.vlabel[a] < h.vlabel[b];
        return deg[a] > deg[b];
    });
    for (uint32_t i = 0; i < n; ++i) inv[order[i]] = i;
    std::vector<uint64_t> key(m);
    std::iota(key.begin(), key.end(), 0ull);
    std::stable_sort(key.begin(), key.end(), [&](uint64_t a, uint64_t b) {
        return std::make_pair(inv[h.src[a]], inv[h.dst[a]]) < std::make_pair(inv[h.src[b]], inv[h.dst[b]]);
    });
    g.n = n;
    g.m = m;
    g.h_rowptr.assign(n + 1, 0);
    g.vl_grouped = vl;
    adj.resize(m);
    lab.resize(m);
    for (uint64_t i = 0; i < m; ++i) {
        adj[i] = inv[h.dst[key[i]]];
        lab[i] = h.lab[key[i]];
        g.h_rowptr[inv[h.src[key[i]]] + 1]++;
        g.multi = g.multi || (i && adj[i] == adj[i - 1] && h.src[key[i]] == h.src[key[i - 1]]);
    }
    for (uint32_t i = 0; i < n; ++i) {
        g.max_degree = std::max(g.max_degree, g.h_rowptr[i + 1]);
        g.h_rowptr[i + 1] += g.h_rowptr[i];
    }
    bool one = true;
    for (uint8_t l : lab) one = one && l == lab[0];
    g.elab = one ? nullptr : lab.data();
    g.single_label = m ? lab[0] : 0;
    g.symmetric = true;
    for (uint32_t u = 0; u < n && g.symmetric; ++u)
        for (uint32_t i = g.h_rowptr[u]; i < g.h_rowptr[u + 1]; ++i) {
            const uint32_t v = adj[i];
            g.symmetric = g.symmetric && std::binary_search(adj.begin() + g.h_rowptr[v], adj.begin() + g.h_rowptr[v + 1], u);
        }
    g.group_value = {0};
    g.group_start = {0, n};
    if (vl) {
        g.group_value.clear();
        g.group_start.clear();
        for (uint32_t i = 0; i < n; ++i)
            if (!i || h.vlabel[order[i]] != h.vlabel[order[i - 1]]) {
                g.group_value.push_back(h.vlabel[order[i]]);
                g.group_start.push_back(i);
            }
        g.group_start.push_back(n);
    }
}

template <bool LAB>
static void dfs(const WalkGraph &g, const WalkTables &w, uint32_t node, const Tuple &t, uint32_t d, uint32_t v, uint32_t idx,
                std::vector<uint64_t> &cnt) {
    uint32_t bytes = 0;
    const WNode &n = w.nodes[node];
    for (uint32_t x = d; x & 3u; ++x) t.m[(x >> 2) * t.step + (x & 3u)] = kNoVertex;  // what a deeper call left
    if (!walk_check<LAB>(g, &n, w.again.data(), t, d, v, idx, bytes)) return;
    t.append(d, v);
    if (n.final_) ++cnt[n.slot];
    for (uint32_t x = 0; x < n.nsfx; ++x) {
        uint32_t first = 0;
        cnt[w.sfx[n.sfx + x].slot] += suffix_count<LAB>(g, &w.sfx[n.sfx + x], t, d + 1, bytes, first);
    }
    if (!n.nchild) return;
    uint32_t s = 0, len = 0;
    walk_slice(g, reinterpret_cast<const Chunk *>(&n)[1], t, s, len, bytes);
    for (uint32_t j = 0; j < n.nchild; ++j)
        for (uint32_t i = 0; i < len; ++i) dfs<LAB>(g, w, n.child + j, t, d + 1, g.adj[s + i], s + i, cnt);
}

int main(int argc, char **argv) {
    if (argc < 8) return 2;
    const bool vl = atoi(argv[1]), share = atoi(argv[2]), leaves = atoi(argv[3]), cross = atoi(argv[4]), desc = atoi(argv[5]);
    gfsm_limits lim;
    gfsm_limits_default(&lim);
    lim.vertex_labels = vl;
    gfsm_ctx *ctx = nullptr;
    if (gfsm_init(&ctx, &lim, -1)) return 3;
    gfsm_graph *data = nullptr;
    if (gfsm_graph_load_text(ctx, argv[6], &data)) return 4;
    DeviceGraph g;
    std::vector<uint32_t> adj;
    std::vector<uint8_t> lab;
    host_ccsr(data->h, vl, g, adj, lab);
    const bool sym_ok = g.symmetric && !g.multi && !g.elab;
    const int nq = argc - 7;
    std::vector<DQuery> dq(nq);
    std::vector<gfsm_plan *> plans(nq);
    std::vector<WalkQuery> ws;
    std::vector<int> at(nq, -1);
    for (int i = 0; i < nq; ++i) {
        gfsm_graph *q = nullptr;
        if (gfsm_graph_load_text(ctx, argv[7 + i], &q) || gfsm_query_prepare(ctx, q, &plans[i])) return 5;
        uint32_t lo = 0, hi = 0;
        bool never = false;
        if (build_dquery(plans[i]->p, g, lim, dq[i], lo, hi, never)) return 6;
        if (never) continue;
        at[i] = (int)ws.size();
        ws.push_back({&dq[i], &plans[i]->p, lo, hi, sym_ok && plans[i]->p.aut > 1 && plans[i]->p.sym_vl == vl});
        gfsm_graph_destroy(q);
    }
    WalkTables w;
    if (!build_walk(ws, g, share, leaves && !g.multi, cross, desc, w)) return 7;
    std::vector<uint32_t> grp;
    const uint32_t ng = (uint32_t)g.group_value.size();
    for (uint32_t u = 0; u < g.n; ++u)
        for (uint32_t x = 0; x < ng; ++x)
            grp.push_back((uint32_t)(std::lower_bound(adj.begin() + g.h_rowptr[u], adj.begin() + g.h_rowptr[u + 1],
                                                      g.group_start[x]) - adj.begin()));
    grp.push_back((uint32_t)g.m);
    std::vector<uint64_t> nlf(g.n, 0);
    for (uint32_t u = 0; u < g.n; ++u)
        for (uint32_t x = 0; x < ng && x < 8; ++x)
            nlf[u] |= (uint64_t)std::min(255u, grp[u * ng + x + 1] - grp[u * ng + x]) << (8 * x);
    // (share = 0 also runs without the row pointers by group)
    WalkGraph wg{g.h_rowptr.data(), adj.data(), g.elab, share ? grp.data() : nullptr, share ? nlf.data() : nullptr, ng, g.single_label, g.n, (uint32_t)g.m};
    std::vector<uint64_t> cnt(w.nslots, 0);
    std::vector<Chunk> col(w.core / 4 + 1);
    const Tuple t{&col[0].x, 4};
    for (size_t p = 0; p < w.root_lo.size(); ++p)
        for (unsigned long long u = w.root_off[p]; u < w.root_off[p + 1]; ++u) {
            const uint32_t v = w.root_lo[p] + (uint32_t)(u - w.root_off[p]);
            if (g.elab || g.multi) dfs<true>(wg, w, (uint32_t)p, t, 0, v, 0, cnt);
            else dfs<false>(wg, w, (uint32_t)p, t, 0, v, 0, cnt);
        }
    for (int i = 0; i < nq; ++i)
        printf("%llu\n", at[i] < 0 ? 0ull : (unsigned long long)(cnt[w.slot[at[i]]] * w.mult[at[i]]));
    printf("core %u nodes %zu sfx %zu\n", w.core, w.nodes.size(), w.sfx.size());
    return 0;
}
