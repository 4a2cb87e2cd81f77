// The walk's kernel itself on the host (tests without a GPU): every lane is a
// fiber, the lanes of a warp meet at each warp intrinsic -- all 32 at the same
// line, or it is an error -- and run in a random order in between, so that an
// access that needs another lane's store without a meeting in between sees the
// old word in some order.  Each array ends at an unmapped page, and a clamp of
// the kernel that changes an index is counted.
//   walk_emu <vertex labels> <share> <leaves> <cross> <desc> <form> <seed> <data> <query>...
// form: walk, limited, or poison (limited, with a depth out of range in every
// list unit).  Prints each query's count (one line each), then
// "passes <p> listed <l> unfinished <0|1> clamped <c> candidates <n> kept <n>
// bytes <n> front <n>".
#include <setjmp.h>
#include <sys/mman.h>
#include <ucontext.h>
#include <unistd.h>

#include <cmath>
#include <cstring>
#include <random>

static uint64_t g_clamped = 0;
#define GFSM_CLAMPED(acts) (g_clamped += (acts) ? 1 : 0)

#define main walk_host_main
#include "walk_host.cpp"
#undef main
#include "../gfsm_b200/csrc/walk_launch.h"

// ---- fibers: one CTA at a time
namespace emu {
constexpr int kThreadsMax = 128;
struct Fiber {
    ucontext_t first;
    jmp_buf at;
    bool started = false, done = false, waiting = false;
    int line = 0;            // the meeting it waits at
    bool cta = false;        // of the whole CTA
    uint64_t val = 0;
};
Fiber fib[kThreadsMax];
uint64_t snap[kThreadsMax];  // each warp's values at its last meeting
jmp_buf sched;
int cur = 0;
uint32_t tid, bid, gdim;
std::mt19937_64 rng;
void (*body)();

void entry() {
    body();
    fib[cur].done = true;
    _longjmp(sched, 1);
}
void wait_at(int line, bool cta, uint64_t val) {
    Fiber &f = fib[cur];
    f.line = line;
    f.cta = cta;
    f.val = val;
    f.waiting = true;
    if (!_setjmp(f.at)) _longjmp(sched, 1);
}
[[noreturn]] void fail(const char *what, int line) {
    fprintf(stderr, "%s (line %d)\n", what, line);
    exit(9);
}
void run_cta(uint32_t b, uint32_t grid) {
    static char *stacks = static_cast<char *>(mmap(nullptr, kThreadsMax << 17, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
    bid = b;
    gdim = grid;
    for (int i = 0; i < kThreadsMax; ++i) {
        Fiber &f = fib[i];
        f.started = f.done = f.waiting = false;
        getcontext(&f.first);
        f.first.uc_stack.ss_sp = stacks + ((size_t)i << 17);
        f.first.uc_stack.ss_size = 1 << 17;
        f.first.uc_link = nullptr;
        makecontext(&f.first, entry, 0);
    }
    for (;;) {
        // a random runnable lane, until there is none
        int order[kThreadsMax], n = 0;
        for (int i = 0; i < kThreadsMax; ++i)
            if (!fib[i].done && !fib[i].waiting) order[n++] = i;
        std::shuffle(order, order + n, rng);
        for (int x = 0; x < n; ++x) {
            cur = order[x];
            tid = (uint32_t)cur;
            if (!_setjmp(sched)) {
                if (fib[cur].started) _longjmp(fib[cur].at, 1);
                fib[cur].started = true;
                setcontext(&fib[cur].first);
            }
        }
        int done = 0, at_cta = 0;
        for (int i = 0; i < kThreadsMax; ++i) {
            done += fib[i].done;
            at_cta += !fib[i].done && fib[i].cta;
        }
        if (done == kThreadsMax) return;
        if (at_cta == kThreadsMax) {
            for (int i = 0; i < kThreadsMax; ++i) fib[i].waiting = false, fib[i].cta = false;
            continue;
        }
        bool moved = false;
        for (int w = 0; w < kThreadsMax; w += 32) {
            int same = 0, warp_done = 0;
            for (int i = w; i < w + 32; ++i) {
                warp_done += fib[i].done;
                same += fib[i].waiting && !fib[i].cta && fib[i].line == fib[w].line;
            }
            if (warp_done == 32 || fib[w].cta) continue;
            if (same != 32) fail("a warp's lanes wait at different places", fib[w].line);
            for (int i = w; i < w + 32; ++i) snap[i] = fib[i].val, fib[i].waiting = false;
            moved = true;
        }
        if (!moved) fail("a CTA's warps wait at different places", fib[0].line);
    }
}
uint64_t meet(int line, uint64_t v) {  // returns this warp's first lane
    wait_at(line, false, v);
    return (uint64_t)(cur & ~31);
}
template <class T>
T as(uint64_t x) {
    T r;
    std::memcpy(&r, &x, sizeof(T));
    return r;
}
template <class T>
uint64_t bits(T x) {
    uint64_t r = 0;
    std::memcpy(&r, &x, sizeof(T));
    return r;
}
template <class T>
T shfl(int line, T v, uint32_t from) {
    const uint64_t w = meet(line, bits(v));
    return as<T>(snap[w + (from & 31u)]);
}
template <class T>
T shfl_up(int line, T v, uint32_t by) {
    const uint32_t lane = (uint32_t)cur & 31u;
    const uint64_t w = meet(line, bits(v));
    return as<T>(snap[w + (lane >= by ? lane - by : lane)]);
}
template <class T>
T shfl_xor(int line, T v, uint32_t by) {
    const uint32_t lane = (uint32_t)cur & 31u;
    const uint64_t w = meet(line, bits(v));
    return as<T>(snap[w + (lane ^ by)]);
}
uint32_t ballot(int line, bool p) {
    const uint64_t w = meet(line, p);
    uint32_t r = 0;
    for (int i = 0; i < 32; ++i) r |= (uint32_t)snap[w + i] << i;
    return r;
}
uint32_t reduce_add(int line, uint32_t v) {
    const uint64_t w = meet(line, v);
    uint32_t r = 0;
    for (int i = 0; i < 32; ++i) r += (uint32_t)snap[w + i];
    return r;
}
uint32_t reduce_or(int line, uint32_t v) {
    const uint64_t w = meet(line, v);
    uint32_t r = 0;
    for (int i = 0; i < 32; ++i) r |= (uint32_t)snap[w + i];
    return r;
}
struct Dim {
    uint32_t x;
};
alignas(16) uint32_t shared[1 << 16];

// an array that ends at an unmapped page
template <class T>
T *guarded(size_t count) {
    const size_t page = (size_t)sysconf(_SC_PAGESIZE), len = std::max<size_t>(16, (count * sizeof(T) + 15) & ~(size_t)15);
    const size_t whole = (len + page - 1) / page * page;
    char *p = static_cast<char *>(mmap(nullptr, whole + page, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
    mprotect(p + whole, page, PROT_NONE);
    return reinterpret_cast<T *>(p + whole - len);
}
template <class T>
T *guarded(const std::vector<T> &v) {
    T *p = guarded<T>(v.size());
    if (!v.empty()) std::memcpy(static_cast<void *>(p), v.data(), v.size() * sizeof(T));
    return p;
}
}  // namespace emu

#undef __global__
#undef __device__
#undef __host__
#undef __forceinline__
#undef __noinline__
#undef __launch_bounds__
#undef __shared__
#define __global__ static
#define __device__
#define __host__
#define __forceinline__ inline
#define __noinline__
#define __launch_bounds__(...)
#define __shared__ static
#define GFSM_DYN_SHARED(x) uint32_t *const x = emu::shared
#define threadIdx (emu::Dim{(uint32_t)emu::cur})
#define blockIdx (emu::Dim{emu::bid})
#define gridDim (emu::Dim{emu::gdim})
#define __shfl_sync(m, v, l) emu::shfl(__LINE__, v, l)
#define __shfl_up_sync(m, v, l) emu::shfl_up(__LINE__, v, l)
#define __shfl_xor_sync(m, v, l) emu::shfl_xor(__LINE__, v, l)
#define __ballot_sync(m, p) emu::ballot(__LINE__, (p) ? true : false)
#define __any_sync(m, p) (emu::ballot(__LINE__, (p) ? true : false) != 0u)
#define __all_sync(m, p) (emu::ballot(__LINE__, (p) ? true : false) == 0xffffffffu)
#define __reduce_add_sync(m, v) emu::reduce_add(__LINE__, v)
#define __reduce_or_sync(m, v) emu::reduce_or(__LINE__, v)
#define __syncwarp() emu::meet(__LINE__, 0)
#define __syncthreads()                       \
    do {                                      \
        emu::wait_at(__LINE__, true, 0);      \
    } while (0)
#define __threadfence() ((void)0)
#define __popc(x) ((uint32_t)__builtin_popcount(x))
#define __ffs(x) ((int)__builtin_ffs((int)(x)))
#define __clz(x) ((x) ? __builtin_clz(x) : 32)
#define __fdividef(a, b) ((a) / (b))
template <class T>
static T __ldg(const T *p) { return *p; }
template <class T>
static T __ldcg(const T *p) { return *p; }
template <class T, class U>
static T atomicAdd(T *p, U v) {
    const T old = *p;
    *p += (T)v;
    return old;
}
using std::max;
using std::min;

#include "../gfsm_b200/csrc/walk_kernel.cuh"

static WalkArgs g_args;
static void (*g_kernel)(const WalkArgs);

int main(int argc, char **argv) {
    if (argc < 10) return 2;
    const bool vl = atoi(argv[1]), share = atoi(argv[2]), leaves = atoi(argv[3]), cross = atoi(argv[4]), desc = atoi(argv[5]);
    const std::string form = argv[6];
    const bool limited = form == "limited" || form == "poison";
    emu::rng.seed((uint64_t)atoll(argv[7]));
    gfsm_limits lim;
    gfsm_limits_default(&lim);
    lim.vertex_labels = vl;
    gfsm_ctx *ctx = nullptr;
    if (gfsm_init(&ctx, &lim, -1)) return 3;
    gfsm_graph *data = nullptr;
    if (gfsm_graph_load_text(ctx, argv[8], &data)) return 4;
    DeviceGraph g;
    std::vector<uint32_t> adj;
    std::vector<uint8_t> lab;
    host_ccsr(data->h, vl, g, adj, lab);
    const bool sym_ok = g.symmetric && !g.multi && !g.elab;
    const int nq = argc - 9;
    std::vector<DQuery> dq(nq);
    std::vector<gfsm_plan *> plans(nq);
    std::vector<WalkQuery> ws;
    std::vector<int> at(nq, -1);
    for (int i = 0; i < nq; ++i) {
        gfsm_graph *q = nullptr;
        if (gfsm_graph_load_text(ctx, argv[9 + i], &q) || gfsm_query_prepare(ctx, q, &plans[i])) return 5;
        uint32_t lo = 0, hi = 0;
        bool never = false;
        if (build_dquery(plans[i]->p, g, lim, dq[i], lo, hi, never)) return 6;
        if (!never) {
            at[i] = (int)ws.size();
            ws.push_back({&dq[i], &plans[i]->p, lo, hi, sym_ok && plans[i]->p.aut > 1 && plans[i]->p.sym_vl == vl});
        }
        gfsm_graph_destroy(q);
    }
    WalkTables w;
    if (!build_walk(ws, g, share, leaves && !g.multi, cross, desc, w)) return 7;
    const uint32_t ng = (uint32_t)g.group_value.size();
    std::vector<uint32_t> grp;
    for (uint32_t u = 0; u < g.n; ++u)
        for (uint32_t x = 0; x < ng; ++x)
            grp.push_back((uint32_t)(std::lower_bound(adj.begin() + g.h_rowptr[u], adj.begin() + g.h_rowptr[u + 1],
                                                      g.group_start[x]) - adj.begin()));
    grp.push_back((uint32_t)g.m);
    std::vector<uint64_t> nlf(g.n, 0);
    for (uint32_t u = 0; u < g.n; ++u)
        for (uint32_t x = 0; x < ng && x < 8; ++x)
            nlf[u] |= (uint64_t)std::min(255u, grp[u * ng + x + 1] - grp[u * ng + x]) << (8 * x);
    const int sms = 1;  // a chip of 32 warps
    WalkArgs a{};
    a.g = {emu::guarded(std::vector<uint32_t>(g.h_rowptr.begin(), g.h_rowptr.end())), emu::guarded(adj),
           g.elab ? emu::guarded(lab) : nullptr, share ? emu::guarded(grp) : nullptr, share ? emu::guarded(nlf) : nullptr, ng,
           g.single_label, g.n, (uint32_t)g.m};
    a.nodes = emu::guarded(w.nodes);
    a.sfx = emu::guarded(w.sfx);
    a.again = emu::guarded(w.again);
    a.root_lo = emu::guarded(w.root_lo);
    a.root_off = emu::guarded(w.root_off);
    a.roots = (uint32_t)w.root_lo.size();
    a.core = w.core;
    a.node_count = (uint32_t)w.nodes.size();
    a.sfxs = (uint32_t)w.sfx.size();
    a.units = w.root_off[a.roots];
    a.counts = emu::guarded<unsigned long long>(w.nslots);
    a.result = emu::guarded<WalkResult>(1);
    a.queues = emu::guarded<Chunk>((size_t)sms * kCtas * kWarps * queue_chunks(w.core));
    a.warp_chunks = queue_chunks(w.core);
    const size_t list_chunks = (size_t)kWalkListed * (2 + tuple_chunks(w.core));
    Chunk *const list[2] = {emu::guarded<Chunk>(list_chunks), emu::guarded<Chunk>(list_chunks)};
    WalkState *const state = emu::guarded<WalkState>((size_t)sms * kCtas * kWarps);
    const bool labelled = g.elab || g.multi;
    emu::body = [] { g_kernel(g_args); };
    WalkResult *r = a.result;
    uint32_t passes = 0, listed = 0, kept = 0;
    bool rest = false;
    for (int p = 0; p < (limited ? kWalkPasses : 1 << 20); ++p) {
        g_args = walk_pass(a, limited, list[0], p, kept, sms);
        if (limited) {  // (each list at its own pages)
            if (g_args.list_in) g_args.list_in = list[(p - 1) & 1];
            if (g_args.list_out) g_args.list_out = list[p & 1];
        } else {
            g_args.state_out = state;
            if (p) {
                g_args.state_in = state;
                *g_args.out = {};
                r->kept = 0;
                g_kernel = k_split;
                const uint32_t ctas = (g_args.state_warps + kWarps - 1) / kWarps;
                for (uint32_t b = 0; b < ctas; ++b) emu::run_cta(b, ctas);
                listed += list_units(g_args.out->listed, g_args.out->refused);
            }
        }
        g_kernel = walk_kernel(g_args, labelled, limited ? kLimited : p ? kLater : kWhole);
        for (uint32_t b = 0; b < g_args.ctas; ++b) emu::run_cta(b, g_args.ctas);
        if (p) rest = rest || g_args.in->taken < list_units(g_args.in->listed, g_args.in->refused);
        const uint32_t units = limited && g_args.list_out ? std::min(g_args.out->listed, kWalkListed) : 0;
        listed += units;
        passes += units || !passes || !limited;
        if (form == "poison")
            for (uint32_t u = 0; u < units; ++u)
                list[p & 1][(size_t)u * (2 + tuple_chunks(w.core)) + 1].x = 0xfffffff0u + u;
        kept = r->kept;
        if (!limited && !kept) break;
    }
    rest = rest || r->gave_up != 0 || r->unit < a.units;
    for (int i = 0; i < nq; ++i)
        printf("%llu\n", at[i] < 0 ? 0ull : (unsigned long long)(a.counts[w.slot[at[i]]] * w.mult[at[i]]));
    unsigned long long total[4] = {};
    for (const auto &t : r->total)
        for (int i = 0; i < 4; ++i) total[i] += t[i];
    printf("passes %u listed %u unfinished %d clamped %llu candidates %llu kept %llu bytes %llu front %llu\n", passes, listed,
           (int)rest, (unsigned long long)g_clamped, total[0], total[1], total[2], total[3]);
    return 0;
}
