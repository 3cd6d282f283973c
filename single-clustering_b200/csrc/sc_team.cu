// sc_team.cu — a pass's small levels in one launch.
//
// A level of some hundred nodes takes microseconds of work, but as a launch per
// step it took 60 launches and half a dozen read-backs: 0.11 ms of local moving,
// 0.13 ms of refinement and 0.30 ms of aggregation, whatever its size, and a
// pass ends with three to six such levels. Here a team (one cluster of blocks, or
// one block for the smallest) keeps going from level to level on the device:
// local moving to its last sweep, refinement, the renumberings, the contraction
// and the new graph's statistics, with the cluster's hardware barrier between
// steps and one read-back at the end. A team of several blocks sheds all but one
// of them once a level is small enough for one.
//
// Every step decides and sums exactly as the kernels of sc_leiden.cu and
// sc_graph.cu do: the same hashes, gains, tie and conflict rules, fixed-point or
// exact sums that do not depend on the order. It takes graphs inside the exact
// summation regime with bitwise symmetric weights only, and hands back to the
// caller a level that leaves that regime.
#include "sc_move.cuh"
#include "sc_team.cuh"

namespace sc {

namespace {

constexpr int TEAM_THREADS = 512;
constexpr int TEAM_WARPS = TEAM_THREADS / 32;
// Blocks of a team (8 beside other instances' work). Measured on a 300-node run
// (18 + 4 sweeps, 8 levels): 1.38 ms of kernel time in one block, 0.94 with 4
// blocks, 0.81 with 8, 0.74 with 16; on levels of 6,475 nodes and 452k entries
// 6.1, 3.9 and 2.6 ms with 4, 8 and 16.
constexpr uint32_t TEAM_CLUSTER = 16;
// A level one block runs alone: with a node or two a warp, barriers inside the
// block cost less than the cluster's (64 against 16: 0.74 and 0.78 ms there).
constexpr uint32_t SOLO_NODES = 64;
constexpr uint64_t SOLO_ENTRIES = 4096;
// Active nodes a block, up to which the last sweeps are the team's. With 192 / 384 /
// 768: CPM at 200k nodes 20.4 / 20.5 / 21.3 ms, 96 uneven graphs 28.2 / 28.4 / 29.4, a
// sweep of resolutions over 200k nodes 72.4 / 71.9 / 70.9, RB at 4M 106.3 / 106.1 / 106.0.
constexpr uint32_t TAIL_NODES_PER_BLOCK = 384;
constexpr uint32_t TEAM_BIG = TEAM_MAX_NODES / 8;  // rows past a warp's table, per block (8 blocks at least, or one of SOLO_NODES)
constexpr uint32_t GROUPS = 4;  // nodes a block decides side by side (decide_group)
constexpr uint32_t SLOTS_MAX = 2 * TEAM_MAX_NODES;  // community ids of a level: the partition's and one fresh per node
static_assert(SOLO_NODES <= TEAM_BIG, "one block's nodes fit its list");
static_assert(SLOTS_MAX / 32 <= TEAM_THREADS, "the id bitmaps are scanned one word a thread");

// One graph of the two a pass alternates between.
struct TeamBuf {
    uint64_t* ptr;
    uint32_t* nbr;
    float* w;
    double *strength, *node_w, *self_loop;
};

struct TeamCtl {
    // per level
    unsigned long long moves;
    long long gain;
    unsigned long long ctr[3];     // entries, candidates, nodes scored by local moving
    unsigned acount[2];            // active nodes of this sweep and the next
    int e0_w, e0_nw;               // the coarse graph: lowest set bits,
    unsigned max_deg, loops;       // largest degree, any self-loop,
    unsigned long long ecount;     // entries with row <= neighbour,
    double strength, nw, upper;    // Σ strength, Σ node weight, Σ of those entries' weights
    // results
    unsigned state;                // 1: finished, 2: stopped before `level`
    unsigned buf;                  // stopped: which TeamBuf holds the level's graph
    unsigned memb2;                // stopped: the membership is in the second array
    unsigned n;
    unsigned long long E, C, level, sweeps, total_moves, levels;
    double improvement, alg_lm, alg_agg;
    double total_weight;
    unsigned long long edge_count;
    unsigned long long t_lm, t_rf, t_ag;  // ns
};

struct TeamArgs {
    TeamBuf in, buf[2];
    uint32_t n;
    uint64_t E, C;
    double total_weight;
    uint64_t edge_count;
    int e0_w, e0_nw;
    uint32_t *memb, *memb2;
    long long *Kf, *Wf;
    uint32_t* csize;
    uint32_t *tgt, *hint, *from, *epoch, *moved, *stamp, *list0, *list1, *refined;
    long long* dgain;
    uint32_t *grp, *node_at, *members, *gcnt, *gcap, *gcur, *cnt, *bits;
    double* loops;
    uint32_t* tnbr;
    float* tw;
    TeamCtl* ctl;
    unsigned long long* refine_ctr;
    uint32_t* status;
    int objective, refine, need_nc;
    double gamma, randomness, improvement;
    uint64_t pass_seed, level, max_levels;
};

struct WarpTable {
    long long vals[WCAP];
    uint32_t keys[WCAP];
    uint32_t list[WARP_DEGREE];
};
struct WarpRow {  // contraction
    long long vals[WCAP];
    uint32_t keys[WCAP];
    uint32_t lk[WARP_DEGREE];
    float lw[WARP_DEGREE];
};
struct TeamSmem {
    union {
        WarpTable table[TEAM_WARPS];
        WarpRow row[TEAM_WARPS];
        long long dense[SLOTS_MAX];
    };
    union {
        struct {
            uint32_t start[TEAM_MAX_NODES + 1];
            uint32_t cap[TEAM_MAX_NODES + 1];
        };
        struct {
            uint32_t word[2][SLOTS_MAX / 32];  // id bitmaps and the ids before each word
            uint32_t before[2][SLOTS_MAX / 32];
        };
    };
    uint32_t big[TEAM_BIG];
    uint4 item[TEAM_BIG];  // node, row start, degree, community
    uint32_t nbig, bigmax, nitem, next;
    uint32_t wcnt[TEAM_WARPS];
    unsigned long long wsum[TEAM_WARPS];
    unsigned long long total;
    double red_g[32];
    uint32_t red_c[32];
    uint32_t target[GROUPS], member[GROUPS];
};

struct Team {
    uint32_t rank, size;
    __device__ void sync() const {
        if (size == 1) {
            __syncthreads();
        } else {
            __syncwarp();  // the barrier takes a warp's arrival as one: its lanes come together first
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        }
    }
};

__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// Exclusive prefix of x over the block; the block's sum in s.total.
__device__ __forceinline__ unsigned long long block_prefix(TeamSmem& s, unsigned long long x) {
    const unsigned lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    unsigned long long incl = x;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if ((int)lane >= o) incl += t;
    }
    if (lane == 31) s.wsum[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        unsigned long long v = lane < TEAM_WARPS ? s.wsum[lane] : 0ull;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long t = __shfl_up_sync(0xFFFFFFFFu, v, o);
            if ((int)lane >= o) v += t;
        }
        if (lane < TEAM_WARPS) s.wsum[lane] = v;
        if (lane == 31) s.total = v;
    }
    __syncthreads();
    const unsigned long long before = (wid ? s.wsum[wid - 1] : 0ull) + incl - x;
    __syncthreads();  // wsum is free again
    return before;
}

// Exclusive prefix of a[0 .. m) into out[0 .. m], m <= TEAM_MAX_NODES, by every block for itself.
__device__ __forceinline__ uint32_t block_scan(TeamSmem& s, const uint32_t* a, uint32_t m, uint32_t* out) {
    constexpr uint32_t PER = TEAM_MAX_NODES / TEAM_THREADS;
    uint32_t x[PER], sum = 0;
    const uint32_t per = (m + TEAM_THREADS - 1) / TEAM_THREADS;
#pragma unroll
    for (uint32_t t = 0; t < PER; ++t) {
        const uint32_t i = threadIdx.x * per + t;
        x[t] = t < per && i < m ? a[i] : 0u;
        sum += x[t];
    }
    uint32_t run = (uint32_t)block_prefix(s, sum);
    const uint32_t total = (uint32_t)s.total;
#pragma unroll
    for (uint32_t t = 0; t < PER; ++t) {
        const uint32_t i = threadIdx.x * per + t;
        if (t < per && i < m) out[i] = run;
        run += x[t];
    }
    if (threadIdx.x == 0) out[m] = total;
    __syncthreads();
    return total;
}

// What a node's choice needs besides its neighbour communities.
struct NodeSide {
    long long kf, af;
    double k, a, sl;
    bool fresh;  // its own empty community is a candidate (local_move.rs:92-100)
};
template <bool REFINE>
__device__ __forceinline__ NodeSide node_side(const Params& p, uint32_t v, uint32_t own) {
    NodeSide s;
    s.kf = to_fix(p.strength[v], p.inv_scale);
    s.af = to_fix(p.node_w[v], p.inv_nscale);
    s.k = from_fix(s.kf, p.scale);
    s.a = from_fix(s.af, p.nscale);
    s.sl = p.self_loop[v];
    const uint32_t f = (uint32_t)(p.S0 + v);
    s.fresh = !REFINE && f != own && p.csize[own] > 1 && p.csize[f] == 0;
    return s;
}

// The gain of joining a community: its own one without it (OWN), the fresh
// empty one (FRESH) or another (JOIN). Lanes of a warp evaluate all kinds in one
// go: the division that each takes is most of a decision's latency.
enum Kind { OWN, FRESH, JOIN };
__device__ __forceinline__ double gain_as(const Params& p, const NodeCfg& q, const NodeSide& s, Kind kind, uint32_t c,
                                          long long acc) {
    double kc = 0.0, nc = 0.0;
    if (kind != FRESH) {
        kc = from_fix(p.Kf[c] - (kind == OWN ? s.kf : 0ll), p.scale);
        if (p.need_nc) nc = from_fix(p.Wf[c] - (kind == OWN ? s.af : 0ll), p.nscale);
    }
    return gain_of(p, q, kind == FRESH ? 0.0 : from_fix(acc, p.scale), s.sl, s.k, kc, s.a, nc);
}

// A candidate's key from its gain: the gain itself, or refinement's draw (-inf:
// no candidate; `>=` takes ties, refine.rs:91-95).
template <bool REFINE>
__device__ __forceinline__ double key_of(const Params& p, const NodeCfg& q, uint32_t v, uint32_t cu, double gain,
                                         double base) {
    if (!REFINE) return gain;
    const double rel = __dsub_rn(gain, base);
    return rel >= 0.0 ? refine_key(p, q, rel, v - q.base, cu - q.base) : -INFINITY;
}

// The choice from the best candidate (g, c): the target, or NONE32; *gain its
// improvement in fixed point.
template <bool REFINE>
__device__ __forceinline__ uint32_t choose(const Params& p, const NodeCfg& q, const NodeSide& s, uint32_t v,
                                           uint32_t own, double base, double ge, double g, uint32_t c,
                                           long long* gain) {
    *gain = 0;
    if (REFINE) return c;
    uint32_t best = own;
    double bg = base;
    if (c != NONE32 && better(g, c, bg, best)) {
        best = c;
        bg = g;
    }
    if (s.fresh && better(ge, (uint32_t)(p.S0 + v), bg, best)) {
        best = (uint32_t)(p.S0 + v);
        bg = ge;
    }
    const double d = __dsub_rn(bg, base);
    if (best == own || !(d > q.thr)) return NONE32;
    *gain = to_fix(d, p.inv_scale);
    return best;
}

// One warp decides node v (row at b, deg <= WARP_DEGREE). Returns the number of
// candidate communities (the same in every lane).
template <bool REFINE, bool MULTI>
__device__ uint32_t decide_warp(const Params& p, uint32_t v, uint64_t b, uint32_t deg, uint32_t own, WarpTable& t,
                                uint32_t* s_cnt) {
    const unsigned FULL = 0xFFFFFFFFu;
    const unsigned lane = threadIdx.x & 31u;
    const NodeCfg q = node_cfg<MULTI>(p, v);
    const uint32_t cv = REFINE ? p.constraint[v] : 0u;
    double g = -INFINITY;
    uint32_t c = NONE32, ncand;
    uint32_t u0 = 0, cu0 = NONE32;  // the first chunk's entry of this lane
    bool ok0 = false;
    const NodeSide side = node_side<REFINE>(p, v, own);
    double base, ge = 0.0;
    if (deg <= 32) {
        // one chunk: the lowest lane of each community's entries holds its sum
        long long x = 0;
        if (lane < deg) {
            u0 = p.nbr[b + lane];
            x = to_fix((double)p.w[b + lane], p.inv_scale);
            ok0 = u0 != v && (!REFINE || p.constraint[u0] == cv);
            if (ok0) cu0 = p.memb[u0];
        }
        const unsigned peers = peers_of(cu0, ok0);
        const long long acc = peer_sum(peers, ok0 ? x : 0ll);
        const bool lead = ok0 && __ffs(peers) - 1 == (int)lane;
        const unsigned ob = __ballot_sync(FULL, lead && cu0 == own);
        long long wof = __shfl_sync(FULL, acc, ob ? __ffs(ob) - 1 : 0);
        if (!ob) wof = 0;
        const bool cand = lead && cu0 != own;
        const unsigned cands = __ballot_sync(FULL, cand);
        ncand = __popc(cands);
        // two lanes without a candidate take the own and the fresh community
        const unsigned idle = ~cands, idle2 = idle & (idle - 1);
        if (idle2) {  // warp-uniform
            const int ol = __ffs(idle) - 1, fl = __ffs(idle2) - 1;
            double gg = 0.0;
            if (cand) gg = gain_as(p, q, side, JOIN, cu0, acc);
            else if ((int)lane == ol) gg = gain_as(p, q, side, OWN, own, wof);
            else if ((int)lane == fl) gg = gain_as(p, q, side, FRESH, 0, 0);
            base = __shfl_sync(FULL, gg, ol);
            ge = __shfl_sync(FULL, gg, fl);
            if (cand) g = key_of<REFINE>(p, q, v, cu0, gg, base);
        } else {
            base = gain_as(p, q, side, OWN, own, wof);
            ge = gain_as(p, q, side, FRESH, 0, 0);
            if (cand) g = key_of<REFINE>(p, q, v, cu0, gain_as(p, q, side, JOIN, cu0, acc), base);
        }
        if (g != -INFINITY) c = cu0;
    } else {
        uint32_t cap = 64;
        while (cap < 2 * deg) cap <<= 1;
        const uint32_t mask = cap - 1;
        for (uint32_t i = lane; i < cap; i += 32) {
            t.keys[i] = EMPTYK;
            t.vals[i] = 0;
        }
        if (lane == 0) *s_cnt = 0;
        __syncwarp();
        // four chunks' gathers in flight before any of them enters the table
        for (uint32_t base0 = 0; base0 < deg; base0 += 128) {
            uint32_t u[4], cu[4];
            float w[4];
            bool ok[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t j = base0 + 32 * k + lane;
                ok[k] = j < deg;
                u[k] = ok[k] ? p.nbr[b + j] : v;
                w[k] = ok[k] ? p.w[b + j] : 0.0f;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                ok[k] = ok[k] && u[k] != v;
                if (REFINE && ok[k]) ok[k] = p.constraint[u[k]] == cv;
                cu[k] = ok[k] ? p.memb[u[k]] : 0u;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (base0 + 32 * k >= deg) break;  // warp-uniform
                const unsigned peers = peers_of(cu[k], ok[k]);
                const long long x = peer_sum(peers, ok[k] ? to_fix((double)w[k], p.inv_scale) : 0ll);
                if (ok[k] && __ffs(peers) - 1 == (int)lane)
                    hinsert_listed(t.keys, t.vals, mask, cu[k], x, p.status, t.list, s_cnt, WARP_DEGREE);
            }
        }
        __syncwarp();
        const uint32_t ndist = min(*s_cnt, WARP_DEGREE);
        const long long wof = hlookup(t.keys, t.vals, mask, own);
        // items: the own community, the fresh one, then the distinct neighbour communities
        uint32_t mine = 0;
        for (uint32_t i0 = 0; i0 < ndist + 2; i0 += 32) {
            const uint32_t i = i0 + lane;
            const uint32_t slot = i >= 2 && i < ndist + 2 ? t.list[i - 2] : 0u;
            const uint32_t cu = i >= 2 && i < ndist + 2 ? t.keys[slot] : own;
            const bool cand = i >= 2 && cu != own;
            double gg = 0.0;
            if (cand || i < 2)
                gg = gain_as(p, q, side, i == 0 ? OWN : i == 1 ? FRESH : JOIN, cu, i == 0 ? wof : t.vals[slot]);
            if (i0 == 0) {
                base = __shfl_sync(FULL, gg, 0);
                ge = __shfl_sync(FULL, gg, 1);
            }
            if (cand) {
                ++mine;
                gg = key_of<REFINE>(p, q, v, cu, gg, base);
                if (gg != -INFINITY && better(gg, cu, g, c)) {
                    g = gg;
                    c = cu;
                }
            }
        }
        for (int o = 16; o; o >>= 1) mine += __shfl_xor_sync(FULL, mine, o);
        ncand = mine;
    }
    warp_best(g, c);
    long long gain;
    const uint32_t target = choose<REFINE>(p, q, side, v, own, base, ge, g, c, &gain);
    // the member of a singleton target, for conflict detection
    uint32_t member = NONE32;
    if (target != NONE32 && p.csize[target] == 1) {
        if (deg <= 32) {
            if (ok0 && cu0 == target) member = u0;
        } else {
            for (uint32_t base = 0; base < deg; base += 32) {
                const uint32_t j = base + lane;
                const uint32_t u = j < deg ? p.nbr[b + j] : v;
                const bool hit = u != v && p.memb[u] == target;
                if (hit) member = u;
                if (__ballot_sync(FULL, hit)) break;
            }
        }
        for (int o = 16; o; o >>= 1) member = min(member, __shfl_xor_sync(FULL, member, o));
    }
    if (lane == 0 && target != NONE32) {
        p.tgt[v] = target;
        p.from[v] = own;
        p.dgain[v] = gain;
        p.hint[v] = member;
        p.epoch[v] = p.cur;
    }
    __syncwarp();
    return ncand;
}

// A group of warps decides node v (longer rows than a warp takes): a quarter of
// the block, so that four nodes' latencies overlap, or the whole block. With
// DENSE it keeps one accumulator per community id (ids < slots): no probing, no
// table size to fit, and stored weights are positive, so a zero sum means no
// entry; a quarter of the block holds a quarter of the ids. Without (the ids of
// a large level) a hash table twice the degree.
struct Group {
    uint32_t id, threads;  // named barrier 1 + id; threads of the group
    __device__ uint32_t tid() const { return threadIdx.x % threads; }
    __device__ void sync() const {
        __syncwarp();  // as in Team::sync
        asm volatile("bar.sync %0, %1;" ::"r"(1 + id), "r"(threads) : "memory");
    }
};
constexpr uint32_t GROUP_BYTES = SLOTS_MAX / GROUPS * sizeof(long long);
constexpr uint32_t GROUP_DEGREE = 1024;  // longest row of a quarter's table, and of the block's
constexpr uint32_t BLOCK_DEGREE = 4096;
static_assert(2 * GROUP_DEGREE * 12 <= GROUP_BYTES && 2 * BLOCK_DEGREE * 12 <= GROUPS * GROUP_BYTES,
              "a table of twice the degree fits the accumulators' memory");

template <bool REFINE, bool MULTI, bool DENSE>
__device__ uint32_t decide_group(const Params& p, uint32_t v, uint32_t slots, TeamSmem& s, const Group& grp) {
    const unsigned FULL = 0xFFFFFFFFu;
    const unsigned lane = threadIdx.x & 31u;
    const uint32_t tid = grp.tid(), warps = grp.threads / 32;
    double* red_g = s.red_g + grp.id * (32 / GROUPS);  // a group of the whole block has id 0
    uint32_t* red_c = s.red_c + grp.id * (32 / GROUPS);
    const uint64_t b = p.ptr[v], e = p.ptr[v + 1];
    const uint32_t own = p.memb[v];
    const NodeCfg q = node_cfg<MULTI>(p, v);
    const NodeSide side = node_side<REFINE>(p, v, own);
    const uint32_t cv = REFINE ? p.constraint[v] : 0u;
    if (!DENSE) {
        slots = 64;
        while (slots < 2 * (uint32_t)(e - b)) slots <<= 1;
    }
    long long* sums = s.dense + grp.id * (SLOTS_MAX / GROUPS);
    uint32_t* keys = reinterpret_cast<uint32_t*>(sums + slots);  // !DENSE only
    for (uint32_t i = tid; i < slots; i += grp.threads) {
        sums[i] = 0;
        if (!DENSE) keys[i] = EMPTYK;
    }
    if (tid == 0) s.member[grp.id] = NONE32;
    grp.sync();
    // four chunks' gathers in flight, as in decide_warp
    for (uint64_t j0 = b + (tid & ~31u); j0 < e; j0 += 4 * grp.threads) {  // warp-uniform
        uint32_t u[4], cu[4];
        float w[4];
        bool ok[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint64_t j = j0 + k * grp.threads + lane;
            ok[k] = j < e;
            u[k] = ok[k] ? p.nbr[j] : v;
            w[k] = ok[k] ? p.w[j] : 0.0f;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            ok[k] = ok[k] && u[k] != v;
            if (REFINE && ok[k]) ok[k] = p.constraint[u[k]] == cv;
            cu[k] = ok[k] ? p.memb[u[k]] : 0u;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (j0 + k * grp.threads >= e) break;  // warp-uniform
            const unsigned peers = peers_of(cu[k], ok[k]);
            const long long x = peer_sum(peers, ok[k] ? to_fix((double)w[k], p.inv_scale) : 0ll);
            if (!ok[k] || __ffs(peers) - 1 != (int)lane) continue;
            if (DENSE) atomicAdd((unsigned long long*)(sums + cu[k]), (unsigned long long)x);
            else hinsert(keys, sums, slots - 1, cu[k], x, p.status);
        }
    }
    grp.sync();
    double g = -INFINITY, base = 0.0, ge = 0.0;
    uint32_t c = NONE32, mine = 0;
    const long long wof = DENSE ? sums[own] : hlookup(keys, sums, slots - 1, own);
    if (lane < 2) base = gain_as(p, q, side, lane == 0 ? OWN : FRESH, own, wof);
    ge = __shfl_sync(FULL, base, 1);
    base = __shfl_sync(FULL, base, 0);
    for (uint32_t i = tid; i < slots; i += grp.threads) {
        const uint32_t cu = DENSE ? i : keys[i];
        const long long acc = sums[i];
        if ((DENSE ? acc == 0 : cu == EMPTYK) || cu == own) continue;
        ++mine;
        const double gg = key_of<REFINE>(p, q, v, cu, gain_as(p, q, side, JOIN, cu, acc), base);
        if (gg != -INFINITY && better(gg, cu, g, c)) {
            g = gg;
            c = cu;
        }
    }
    warp_best(g, c);
    if (lane == 0) {
        red_g[tid / 32] = g;
        red_c[tid / 32] = c;
    }
    grp.sync();
    if (tid < 32) {
        g = lane < warps ? red_g[lane] : -INFINITY;
        c = lane < warps ? red_c[lane] : NONE32;
        warp_best(g, c);
        long long gain;
        const uint32_t target = choose<REFINE>(p, q, side, v, own, base, ge, g, c, &gain);
        if (tid == 0) {
            s.target[grp.id] = target;
            if (target != NONE32) {
                p.tgt[v] = target;
                p.from[v] = own;
                p.dgain[v] = gain;
                p.epoch[v] = p.cur;
            }
        }
    }
    grp.sync();
    const uint32_t target = s.target[grp.id];
    if (target != NONE32 && p.csize[target] == 1) {
        for (uint64_t j = b + tid; j < e; j += grp.threads) {
            const uint32_t u = p.nbr[j];
            if (u != v && p.memb[u] == target) s.member[grp.id] = u;  // one member: one writer
        }
    }
    grp.sync();
    if (tid == 0 && target != NONE32) p.hint[v] = s.member[grp.id];
    grp.sync();
    return mine;  // this thread's share of the candidates
}

struct Tally {
    unsigned long long deg, cand, nodes;
};

// The block's share of list[0 .. m) (null: all of [0, m)): the items at its rank
// and every team.size-th after it. pick(v, &item) says whether node v takes part
// and fills its item. The nodes that do are gathered into s.item, and f(item)
// runs for each, a warp at a time, first come first served: a hash batch is a
// random eighth or half of the nodes, and dealt out beforehand the warps' shares
// differ by a factor of two to three.
template <class P, class F>
__device__ __forceinline__ void for_picked(const Team& team, TeamSmem& s, const uint32_t* list, uint32_t m, P pick,
                                           F f) {
    const unsigned FULL = 0xFFFFFFFFu;
    const unsigned lane = threadIdx.x & 31u;
    for (uint32_t i0 = team.rank; i0 < m; i0 += team.size * TEAM_THREADS) {  // block-uniform
        const uint32_t i = i0 + team.size * threadIdx.x;
        uint4 it = make_uint4(0, 0, 0, 0);
        const bool mine = i < m && pick(list ? list[i] : i, it);
        const unsigned bal = __ballot_sync(FULL, mine);
        if (bal) {
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(&s.nitem, (uint32_t)__popc(bal));
            at = __shfl_sync(FULL, at, 0) + __popc(bal & ((1u << lane) - 1u));
            if (mine) s.item[at] = it;  // at most TEAM_BIG items a block
        }
    }
    __syncthreads();
    const uint32_t count = s.nitem;
    for (;;) {
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(&s.next, 1u);
        at = __shfl_sync(FULL, at, 0);
        if (at >= count) break;
        f(s.item[at]);
    }
    __syncthreads();
    if (threadIdx.x == 0) s.nitem = s.next = 0;
    __syncthreads();
}

// Decisions of the nodes of one batch among list[0 .. m): those whose hash batch is b.
template <bool REFINE, bool MULTI, bool DENSE>
__device__ void decide_batch(const Params& p, const Team& team, TeamSmem& s, const uint32_t* list, uint32_t m,
                             uint32_t sweep, int B, int b, uint32_t slots, Tally& tally) {
    const unsigned lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    for_picked(
        team, s, list, m,
        [&](uint32_t v, uint4& it) {
            if (batch_of<MULTI>(p.seed, sweep, v, B, p.inst, p.icfg) != b) return false;
            const uint32_t own = p.memb[v];
            if (REFINE && p.csize[own] != 1) return false;  // refine.rs:60-62
            const uint64_t rb = p.ptr[v];
            it = make_uint4(v, (uint32_t)rb, (uint32_t)(p.ptr[v + 1] - rb), own);
            if (it.z <= WARP_DEGREE) return true;
            const uint32_t at = atomicAdd(&s.nbig, 1u);
            if (at < TEAM_BIG) s.big[at] = v;
            else atomicOr(p.status, DEV_OVERFLOW);
            if (!DENSE) atomicMax(&s.bigmax, it.z);
            return false;
        },
        [&](const uint4& it) {
            const uint32_t nc = decide_warp<REFINE, MULTI>(p, it.x, it.y, it.z, it.w, s.table[wid], &s.wcnt[wid]);
            if (lane == 0) {
                tally.deg += it.z;
                tally.cand += nc;
                tally.nodes += 1;
            }
        });
    const uint32_t nbig = min(s.nbig, TEAM_BIG);
    const bool quarters = DENSE ? slots <= SLOTS_MAX / GROUPS : s.bigmax <= GROUP_DEGREE;
    const uint32_t parts = quarters ? GROUPS : 1u;
    const Group grp{threadIdx.x / (TEAM_THREADS / parts), TEAM_THREADS / parts};
    for (uint32_t i = grp.id; i < nbig; i += parts) {
        const uint32_t v = s.big[i];
        tally.cand += decide_group<REFINE, MULTI, DENSE>(p, v, slots, s, grp);
        if (grp.tid() == 0) {
            tally.deg += p.ptr[v + 1] - p.ptr[v];
            tally.nodes += 1;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) s.nbig = s.bigmax = 0;
}

// Commits the decisions of epoch p.cur among list[0 .. m).
template <bool REFINE, bool MULTI>
__device__ void apply_batch(const Params& p, const Team& team, const uint32_t* list, uint32_t m,
                            unsigned long long* moves, long long* gain) {
    unsigned long long nmoves = 0;
    long long gsum = 0;
    for (uint32_t i0 = team.rank * TEAM_THREADS; i0 < m; i0 += team.size * TEAM_THREADS) {
        const uint32_t i = i0 + threadIdx.x;
        if (i >= m) continue;
        const uint32_t v = list ? list[i] : i;
        if (p.epoch[v] != p.cur || cancelled<MULTI>(p, v)) continue;
        const uint32_t t = p.tgt[v], old = p.from[v];
        const long long kf = to_fix(p.strength[v], p.inv_scale);
        p.memb[v] = t;
        atomicAdd((unsigned long long*)(p.Kf + old), (unsigned long long)(-kf));
        atomicAdd((unsigned long long*)(p.Kf + t), (unsigned long long)kf);
        if (p.need_nc) {
            const long long af = to_fix(p.node_w[v], p.inv_nscale);
            atomicAdd((unsigned long long*)(p.Wf + old), (unsigned long long)(-af));
            atomicAdd((unsigned long long*)(p.Wf + t), (unsigned long long)af);
        }
        atomicSub(p.csize + old, 1u);
        atomicAdd(p.csize + t, 1u);
        if (!REFINE) {
            nmoves++;
            if (MULTI) {
                if (p.dgain[v])
                    atomicAdd((unsigned long long*)(p.gain_inst + p.inst[v]), (unsigned long long)p.dgain[v]);
            } else {
                gsum += p.dgain[v];
            }
            p.moved[v] = p.cur;
        }
    }
    if (REFINE) return;
    warp_add(moves, nmoves);
    if (!MULTI) warp_add((unsigned long long*)gain, (unsigned long long)gsum);
}

// Queues the neighbours of the nodes that moved in epoch p.cur and now sit in
// another community (k_activate), a warp per moved node.
__device__ void activate_batch(const Params& p, const Team& team, TeamSmem& s, const uint32_t* list, uint32_t m,
                               uint32_t* stamp, uint32_t mark, uint32_t* next, unsigned* ncount) {
    const unsigned FULL = 0xFFFFFFFFu;
    const unsigned lane = threadIdx.x & 31u;
    for_picked(
        team, s, list, m,
        [&](uint32_t v, uint4& it) {
            if (p.moved[v] != p.cur) return false;
            const uint64_t rb = p.ptr[v];
            it = make_uint4(v, (uint32_t)rb, (uint32_t)(p.ptr[v + 1] - rb), p.memb[v]);
            return true;
        },
        [&](const uint4& it) {
            for (uint32_t j0 = 0; j0 < it.z; j0 += 32) {
                uint32_t u = 0;
                bool add = false;
                if (j0 + lane < it.z) {
                    u = p.nbr[it.y + j0 + lane];
                    add = u != it.x && p.memb[u] != it.w && stamp[u] < mark && atomicMax(stamp + u, mark) < mark;
                }
                const unsigned bal = __ballot_sync(FULL, add);
                if (!bal) continue;
                const int lead = __ffs(bal) - 1;
                uint32_t at = 0;
                if ((int)lane == lead) at = atomicAdd(ncount, (unsigned)__popc(bal));
                at = __shfl_sync(FULL, at, lead);
                if (add) next[at + __popc(bal & ((1u << lane) - 1u))] = u;
            }
        });
}

// Rank of id among the set bits of bitmap k (TeamSmem::word / before).
__device__ __forceinline__ uint32_t rank_of(const TeamSmem& s, int k, uint32_t id) {
    return s.before[k][id >> 5] + __popc(s.word[k][id >> 5] & ((1u << (id & 31)) - 1u));
}

__device__ __forceinline__ float pair_value(uint32_t g, uint32_t h, double acc, const double* loops, bool* keep) {
    const float val = h == g ? __double2float_rn(__dmul_rn(0.5, __dadd_rn(acc, loops[g]))) : __double2float_rn(acc);
    *keep = acc > 0.0 && (double)val != 0.0;
    return val;
}

// Coarse row g from its members' entries (at most WARP_DEGREE of them): one
// warp, sums per neighbour group in a hash, kept entries in ascending order.
__device__ void contract_warp(const Params& p, const TeamArgs& a, const TeamSmem& s, uint32_t g, WarpRow& t) {
    const unsigned FULL = 0xFFFFFFFFu;
    const unsigned lane = threadIdx.x & 31u;
    const uint32_t cap = s.cap[g + 1] - s.cap[g];
    uint32_t size = 64;
    while (size < 2 * cap) size <<= 1;
    for (uint32_t i = lane; i < size; i += 32) {
        t.keys[i] = EMPTYK;
        t.vals[i] = 0;
    }
    __syncwarp();
    for (uint32_t m0 = s.start[g]; m0 < s.start[g + 1]; m0 += 32) {
        uint64_t b = 0;
        uint32_t d = 0;
        if (m0 + lane < s.start[g + 1]) {
            const uint32_t v = a.members[m0 + lane];
            b = p.ptr[v];
            d = (uint32_t)(p.ptr[v + 1] - b);
        }
        uint32_t incl = d;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(FULL, incl, o);
            if ((int)lane >= o) incl += x;
        }
        const uint32_t excl = incl - d, total = __shfl_sync(FULL, incl, 31);
        for (uint32_t base = 0; base < total; base += 32) {
            const uint32_t i = base + lane;
            int L = 0;  // the member holding flattened entry i
            for (int step = 16; step; step >>= 1) {
                const uint32_t e = __shfl_sync(FULL, excl, L + step);
                if (e <= i) L += step;
            }
            const uint32_t eL = __shfl_sync(FULL, excl, L);
            const uint64_t bL = __shfl_sync(FULL, b, L);
            const bool ok = i < total;
            uint32_t h = 0;
            long long x = 0;
            if (ok) {
                const uint64_t j = bL + (i - eL);
                h = a.grp[p.nbr[j]];
                x = to_fix((double)p.w[j], p.inv_scale);
            }
            const unsigned peers = peers_of(h, ok);
            const long long acc = peer_sum(peers, x);
            if (ok && __ffs(peers) - 1 == (int)lane) hinsert(t.keys, t.vals, size - 1, h, acc, a.status);
        }
    }
    __syncwarp();
    uint32_t nk = 0;
    for (uint32_t i0 = 0; i0 < size; i0 += 32) {
        const uint32_t h = t.keys[i0 + lane];
        bool keep = false;
        float val = 0.0f;
        if (h != EMPTYK) val = pair_value(g, h, from_fix(t.vals[i0 + lane], p.scale), a.loops, &keep);
        const unsigned bal = __ballot_sync(FULL, keep);
        if (keep) {
            const uint32_t at = nk + __popc(bal & ((1u << lane) - 1u));
            t.lk[at] = h;
            t.lw[at] = val;
        }
        nk += __popc(bal);
    }
    __syncwarp();
    for (uint32_t i = lane; i < nk; i += 32) {
        const uint32_t h = t.lk[i];
        uint32_t r = 0;
        for (uint32_t j = 0; j < nk; ++j) r += t.lk[j] < h;
        a.tnbr[s.cap[g] + r] = h;
        a.tw[s.cap[g] + r] = t.lw[i];
    }
    if (lane == 0) a.cnt[g] = nk;
    __syncwarp();
}

// Coarse row g of any size: the block, one accumulator per group (G of them),
// read back in ascending order.
__device__ void contract_block(const Params& p, const TeamArgs& a, TeamSmem& s, uint32_t g, uint32_t G) {
    const unsigned FULL = 0xFFFFFFFFu;
    const unsigned lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    for (uint32_t i = threadIdx.x; i < G; i += TEAM_THREADS) s.dense[i] = 0;
    __syncthreads();
    for (uint32_t m = s.start[g] + wid; m < s.start[g + 1]; m += TEAM_WARPS) {
        const uint32_t v = a.members[m];
        const uint64_t b = p.ptr[v], e = p.ptr[v + 1];
        for (uint64_t j0 = b; j0 < e; j0 += 128) {  // four chunks' gathers in flight
            uint32_t h[4];
            float w[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint64_t j = j0 + 32 * k + lane;
                h[k] = j < e ? p.nbr[j] : NONE32;
                w[k] = j < e ? p.w[j] : 0.0f;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (h[k] != NONE32) h[k] = a.grp[h[k]];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (j0 + 32 * k >= e) break;  // warp-uniform
                const bool ok = h[k] != NONE32;
                const unsigned peers = peers_of(h[k], ok);
                const long long x = peer_sum(peers, ok ? to_fix((double)w[k], p.inv_scale) : 0ll);
                if (ok && __ffs(peers) - 1 == (int)lane)
                    atomicAdd((unsigned long long*)(s.dense + h[k]), (unsigned long long)x);
            }
        }
    }
    __syncthreads();
    uint32_t done = 0;
    for (uint32_t h0 = 0; h0 < G; h0 += TEAM_THREADS) {
        const uint32_t h = h0 + threadIdx.x;
        bool keep = false;
        float val = 0.0f;
        if (h < G && s.dense[h] != 0) val = pair_value(g, h, from_fix(s.dense[h], p.scale), a.loops, &keep);
        const uint32_t at = done + (uint32_t)block_prefix(s, keep ? 1ull : 0ull);
        if (keep) {
            a.tnbr[s.cap[g] + at] = h;
            a.tw[s.cap[g] + at] = val;
        }
        done += (uint32_t)s.total;
        __syncthreads();  // s.total is read before the next prefix
    }
    if (threadIdx.x == 0) a.cnt[g] = done;
    __syncthreads();
}

__global__ void __launch_bounds__(TEAM_THREADS, 1) k_team(const __grid_constant__ TeamArgs a) {
    extern __shared__ __align__(16) unsigned char raw[];
    TeamSmem& s = *reinterpret_cast<TeamSmem*>(raw);
    const unsigned lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    Team team{blockIdx.x, gridDim.x};  // the grid is one cluster
    TeamCtl* ctl = a.ctl;
    if (threadIdx.x == 0) s.nbig = s.bigmax = s.nitem = s.next = 0;
    __syncthreads();

    TeamBuf cur = a.in;
    uint32_t n = a.n, next_buf = 0, memb_at = 0;
    uint64_t E = a.E, C = a.C, level = a.level;
    double total_weight = a.total_weight, improvement = a.improvement;
    uint64_t edge_count = a.edge_count, sweeps = 0, total_moves = 0, levels = 0;
    int e0_w = a.e0_w, e0_nw = a.e0_nw;
    double alg_lm = 0.0, alg_agg = 0.0;
    unsigned long long t_lm = 0, t_rf = 0, t_ag = 0;
    unsigned state = 0;
    uint32_t K = 0;

    Params p{};
    p.tgt = a.tgt;
    p.hint = a.hint;
    p.from = a.from;
    p.dgain = a.dgain;
    p.epoch = a.epoch;
    p.moved = a.moved;
    p.status = a.status;
    p.objective = a.objective;
    p.gamma = a.gamma;
    p.need_nc = a.need_nc;
    p.Kf = a.Kf;
    p.Wf = a.Wf;
    p.csize = a.csize;

    for (uint32_t x = team.rank * TEAM_THREADS + threadIdx.x; x < a.n; x += team.size * TEAM_THREADS) a.node_at[x] = x;

    for (;; ++level) {
        if (team.size > 1 && n <= SOLO_NODES && E <= SOLO_ENTRIES) {
            team.sync();
            if (team.rank) return;
            team.size = 1;
        }
        const uint32_t g0 = team.rank * TEAM_THREADS + threadIdx.x, gstep = team.size * TEAM_THREADS;
        uint32_t* memb = memb_at ? a.memb2 : a.memb;
        uint32_t* memb_next = memb_at ? a.memb : a.memb2;
        const uint32_t slots = (uint32_t)(C + n);
        if (level >= a.max_levels) {  // the last level's membership, renumbered
            for (uint32_t i = g0; i < SLOTS_MAX / 32; i += gstep) a.bits[SLOTS_MAX / 32 + i] = 0;
            team.sync();
            for (uint32_t v = g0; v < n; v += gstep) atomicOr(a.bits + SLOTS_MAX / 32 + (memb[v] >> 5), 1u << (memb[v] & 31));
            team.sync();
            const uint32_t wv = a.bits[SLOTS_MAX / 32 + threadIdx.x];
            s.word[1][threadIdx.x] = wv;
            s.before[1][threadIdx.x] = (uint32_t)block_prefix(s, (unsigned long long)__popc(wv));
            K = (uint32_t)s.total;
            __syncthreads();
            for (uint32_t x = g0; x < a.n; x += gstep) a.node_at[x] = rank_of(s, 1, memb[a.node_at[x]]);
            state = 1;
            break;
        }
        const uint64_t lvl_seed = hash3(a.pass_seed, level, 0x1eafull);
        unsigned long long t0 = now_ns();
        p.ptr = cur.ptr;
        p.nbr = cur.nbr;
        p.w = cur.w;
        p.strength = cur.strength;
        p.node_w = cur.node_w;
        p.self_loop = cur.self_loop;
        p.memb = memb;
        p.constraint = nullptr;
        p.S0 = C;
        p.four_m = 4.0 * total_weight;
        p.thr = 1e-12 * fmax(fabs(total_weight), 1.0);  // local_move.rs:26-28
        const int F = e0_w == 0x7FFFFFFF ? 0 : e0_w, Fn = e0_nw == 0x7FFFFFFF ? 0 : e0_nw;
        p.scale = ldexp(1.0, F);
        p.inv_scale = ldexp(1.0, -F);
        p.nscale = ldexp(1.0, Fn);
        p.inv_nscale = ldexp(1.0, -Fn);
        p.theta = 0.0;
        p.seed = lvl_seed;
        TeamBuf out = a.buf[next_buf];
        // ---- a clean level
        for (uint32_t i = g0; i < slots; i += gstep) {
            a.Kf[i] = 0;
            if (a.need_nc) a.Wf[i] = 0;
            a.csize[i] = 0;
        }
        for (uint32_t v = g0; v < n; v += gstep) {
            a.epoch[v] = a.moved[v] = a.stamp[v] = a.hint[v] = 0;
            a.gcnt[v] = a.gcap[v] = a.gcur[v] = 0;
            a.loops[v] = 0.0;
            out.node_w[v] = 0.0;
        }
        for (uint32_t i = g0; i < 2 * (SLOTS_MAX / 32); i += gstep) a.bits[i] = 0;
        if (g0 == 0) {
            ctl->moves = 0;
            ctl->gain = 0;
            ctl->ctr[0] = ctl->ctr[1] = ctl->ctr[2] = 0;
            ctl->acount[0] = n;
            ctl->acount[1] = 0;
            ctl->e0_w = ctl->e0_nw = 0x7FFFFFFF;
            ctl->max_deg = ctl->loops = 0;
            ctl->ecount = 0;
            ctl->strength = ctl->nw = ctl->upper = 0.0;
        }
        team.sync();
        for (uint32_t v = g0; v < n; v += gstep) {
            const uint32_t c = memb[v];
            atomicAdd((unsigned long long*)(a.Kf + c), (unsigned long long)to_fix(cur.strength[v], p.inv_scale));
            if (a.need_nc)
                atomicAdd((unsigned long long*)(a.Wf + c), (unsigned long long)to_fix(cur.node_w[v], p.inv_nscale));
            atomicAdd(a.csize + c, 1u);
        }
        team.sync();
        // ---- local moving (local_move in sc_leiden.cu, step for step)
        Tally tally{0, 0, 0};
        const unsigned long long budget = (unsigned long long)n * 100;  // MAX_MOVES_PER_NODE, local_move.rs:32
        unsigned long long moves_before = 0;
        uint32_t epoch = 0, did = 0;
        for (uint32_t sweep = 0; sweep < (uint32_t)MAX_SWEEPS; ++sweep) {
            const uint32_t m = ctl->acount[sweep & 1];
            const unsigned long long moves = ctl->moves;
            if (sweep > 0 && moves == moves_before) break;
            if (moves >= budget || m == 0) break;
            moves_before = moves;
            const uint32_t* list = sweep ? (sweep & 1 ? a.list1 : a.list0) : nullptr;
            uint32_t* next = sweep & 1 ? a.list0 : a.list1;
            unsigned* ncount = &ctl->acount[(sweep + 1) & 1];
            for (int b = 0; b < LM_BATCHES; ++b) {
                p.cur = ++epoch;
                decide_batch<false, false, true>(p, team, s, list, m, sweep, LM_BATCHES, b, slots, tally);
                team.sync();
                if (b == 0 && g0 == 0) *ncount = 0;  // last read a sweep ago; first written after the next barrier
                apply_batch<false, false>(p, team, list, m, &ctl->moves, &ctl->gain);
                team.sync();
                // beside the next batch's decisions: it writes only the next sweep's list
                activate_batch(p, team, s, list, m, a.stamp, sweep + 2, next, ncount);
            }
            team.sync();
            ++did;
        }
        sweeps += did;
        {
            warp_add(ctl->ctr + 0, tally.deg);
            warp_add(ctl->ctr + 1, tally.cand);
            warp_add(ctl->ctr + 2, tally.nodes);
        }
        if (g0 == 0) {
            const unsigned long long t1 = now_ns();
            t_lm += t1 - t0;
            t0 = t1;
        }
        // ---- refinement (refine in sc_leiden.cu)
        const uint32_t* collapse = memb;
        if (a.refine) {
            team.sync();  // the last commits are read, and the aggregates below replaced
            for (uint32_t v = g0; v < n; v += gstep) {
                a.refined[v] = v;
                a.Kf[v] = to_fix(cur.strength[v], p.inv_scale);
                if (a.need_nc) a.Wf[v] = to_fix(cur.node_w[v], p.inv_nscale);
                a.csize[v] = 1;
                a.epoch[v] = 0;
            }
            p.memb = a.refined;
            p.constraint = memb;
            p.S0 = n;
            p.thr = 0.0;
            p.theta = a.randomness * (edge_count > 0 ? total_weight / (double)edge_count : 1.0);  // refine.rs:44-50
            p.seed = hash3(lvl_seed, 0x7e71eull, 1);
            Tally rt{0, 0, 0};
            team.sync();
            for (int b = 0; b < RF_BATCHES; ++b) {
                p.cur = (uint32_t)(b + 1);
                decide_batch<true, false, true>(p, team, s, nullptr, n, 0xFFFFFFFFu, RF_BATCHES, b, n, rt);
                team.sync();
                apply_batch<true, false>(p, team, nullptr, n, nullptr, nullptr);
                team.sync();
            }
            warp_add(a.refine_ctr + 0, rt.nodes);
            warp_add(a.refine_ctr + 1, rt.deg);
            warp_add(a.refine_ctr + 2, rt.cand);
            collapse = a.refined;
        } else {
            team.sync();
        }
        if (g0 == 0) {
            const unsigned long long t1 = now_ns();
            t_rf += t1 - t0;
            t0 = t1;
        }
        // ---- ascending ranks of the groups and of the partition's ids
        for (uint32_t v = g0; v < n; v += gstep) {
            const uint32_t r = collapse[v], c = memb[v];
            atomicOr(a.bits + (r >> 5), 1u << (r & 31));
            atomicOr(a.bits + SLOTS_MAX / 32 + (c >> 5), 1u << (c & 31));
        }
        team.sync();
        improvement += (double)ctl->gain * p.scale;
        total_moves += ctl->moves;
        alg_lm += 16.0 * (double)ctl->ctr[2] + 12.0 * (double)ctl->ctr[0] + 8.0 * (double)ctl->ctr[1];
        ++levels;
        {
            const uint32_t wa = a.bits[threadIdx.x], wb = a.bits[SLOTS_MAX / 32 + threadIdx.x];
            s.word[0][threadIdx.x] = wa;
            s.word[1][threadIdx.x] = wb;
            const unsigned long long pre =
                block_prefix(s, (unsigned long long)__popc(wa) | ((unsigned long long)__popc(wb) << 32));
            s.before[0][threadIdx.x] = (uint32_t)pre;
            s.before[1][threadIdx.x] = (uint32_t)(pre >> 32);
        }
        const uint32_t G = (uint32_t)s.total, C2 = (uint32_t)(s.total >> 32);
        __syncthreads();
        if (G >= n) {  // the graph no longer shrinks (mod.rs:263-265): the partition's ranks are the labels
            for (uint32_t x = g0; x < a.n; x += gstep) a.node_at[x] = rank_of(s, 1, memb[a.node_at[x]]);
            K = C2;
            state = 1;
            break;
        }
        // ---- groups: sizes, entries, node weights, self-loops, the coarse membership
        for (uint32_t v = g0; v < n; v += gstep) {
            const uint32_t g = rank_of(s, 0, collapse[v]);
            a.grp[v] = g;
            atomicAdd(a.gcnt + g, 1u);
            atomicAdd(a.gcap + g, (uint32_t)(cur.ptr[v + 1] - cur.ptr[v]));
            atomicAdd(out.node_w + g, cur.node_w[v]);  // exact in any order
            const double sl = cur.self_loop[v];
            if (sl != 0.0) atomicAdd(a.loops + g, sl);
            memb_next[g] = rank_of(s, 1, memb[v]);  // the same for every member (mod.rs:269-272)
        }
        for (uint32_t x = g0; x < a.n; x += gstep) a.node_at[x] = rank_of(s, 0, collapse[a.node_at[x]]);
        team.sync();
        block_scan(s, a.gcnt, G, s.start);
        block_scan(s, a.gcap, G, s.cap);
        for (uint32_t v = g0; v < n; v += gstep) {
            const uint32_t g = a.grp[v];
            a.members[s.start[g] + atomicAdd(a.gcur + g, 1u)] = v;
        }
        team.sync();
        // ---- contraction: small rows a warp each, larger ones the block
        {
            for_picked(
                team, s, nullptr, G,
                [&](uint32_t g, uint4& it) {
                    it.x = g;
                    if (s.cap[g + 1] - s.cap[g] <= WARP_DEGREE) return true;
                    const uint32_t at = atomicAdd(&s.nbig, 1u);
                    if (at < TEAM_BIG) s.big[at] = g;
                    else atomicOr(a.status, DEV_OVERFLOW);
                    return false;
                },
                [&](const uint4& it) { contract_warp(p, a, s, it.x, s.row[wid]); });
            const uint32_t nbig = min(s.nbig, TEAM_BIG);
            for (uint32_t i = 0; i < nbig; ++i) contract_block(p, a, s, s.big[i], G);
            __syncthreads();
            if (threadIdx.x == 0) s.nbig = 0;
        }
        team.sync();
        // ---- the coarse graph and its statistics (finalize in sc_graph.cu)
        const uint64_t E2 = block_scan(s, a.cnt, G, s.start);
        {
            int low = 0x7FFFFFFF, low_nw = 0x7FFFFFFF;
            unsigned loop = 0, mdeg = 0;
            unsigned long long ups = 0;
            double sum_s = 0.0, sum_nw = 0.0, sum_up = 0.0;
            const uint32_t warps = TEAM_WARPS * team.size;
            for (uint32_t g = wid * team.size + team.rank; g < G; g += warps) {
                const uint32_t o = s.start[g], len = s.start[g + 1] - o, src = s.cap[g];
                double acc = 0.0, sl = 0.0;
                for (uint32_t j = lane; j < len; j += 32) {
                    const uint32_t h = a.tnbr[src + j];
                    const float w = a.tw[src + j];
                    out.nbr[o + j] = h;
                    out.w[o + j] = w;
                    low = min(low, lowbit_exp_f32(w));
                    acc += h == g ? 2.0 * (double)w : (double)w;
                    if (h == g) {
                        sl = (double)w;
                        loop = 1;
                    }
                    if (h >= g) {
                        ++ups;
                        sum_up += (double)w;
                    }
                }
                for (int d = 16; d; d >>= 1) {
                    acc += __shfl_xor_sync(0xFFFFFFFFu, acc, d);
                    sl = fmax(sl, __shfl_xor_sync(0xFFFFFFFFu, sl, d));
                }
                if (lane == 0) {
                    out.ptr[g] = o;
                    out.strength[g] = acc;
                    out.self_loop[g] = sl;
                    const double nw = out.node_w[g];
                    low_nw = min(low_nw, lowbit_exp_f64(nw));
                    sum_s += acc;
                    sum_nw += nw;
                    mdeg = max(mdeg, len);
                }
            }
            for (int d = 16; d; d >>= 1) {
                low = min(low, __shfl_xor_sync(0xFFFFFFFFu, low, d));
                loop |= __shfl_xor_sync(0xFFFFFFFFu, loop, d);
                ups += __shfl_xor_sync(0xFFFFFFFFu, ups, d);
                sum_up += __shfl_xor_sync(0xFFFFFFFFu, sum_up, d);
            }
            if (lane == 0) {
                if (low != 0x7FFFFFFF) atomicMin(&ctl->e0_w, low);
                if (low_nw != 0x7FFFFFFF) atomicMin(&ctl->e0_nw, low_nw);
                if (loop) atomicOr(&ctl->loops, 1u);
                if (mdeg) atomicMax(&ctl->max_deg, mdeg);
                if (ups) atomicAdd(&ctl->ecount, ups);
                atomicAdd(&ctl->strength, sum_s);
                atomicAdd(&ctl->nw, sum_nw);
                atomicAdd(&ctl->upper, sum_up);
            }
            if (g0 == 0) out.ptr[G] = E2;
        }
        team.sync();
        alg_agg += 12.0 * (double)E + 12.0 * (double)n + 8.0 * (double)E2 + 24.0 * (double)G;
        e0_w = ctl->e0_w;
        e0_nw = ctl->e0_nw;
        total_weight = ctl->upper;
        edge_count = ctl->ecount;
        const bool exact = (e0_w == 0x7FFFFFFF || ctl->strength < ldexp(1.0, 52 + e0_w)) &&
                           (e0_nw == 0x7FFFFFFF || ctl->nw < ldexp(1.0, 52 + e0_nw));
        n = G;
        E = E2;
        C = C2;
        memb_at ^= 1u;
        cur = out;
        next_buf ^= 1u;
        if (g0 == 0) {
            const unsigned long long t1 = now_ns();
            t_ag += t1 - t0;
            t0 = t1;
        }
        if (!exact) {
            ++level;
            state = 2;
            break;
        }
        team.sync();  // the statistics are read before the next level clears them
    }
    if (team.rank == 0 && threadIdx.x == 0) {
        ctl->state = state;
        ctl->buf = next_buf ^ 1u;
        ctl->memb2 = memb_at;
        ctl->n = n;
        ctl->E = E;
        ctl->C = state == 1 ? K : C;
        ctl->level = level;
        ctl->sweeps = sweeps;
        ctl->total_moves = total_moves;
        ctl->levels = levels;
        ctl->improvement = improvement;
        ctl->alg_lm = alg_lm;
        ctl->alg_agg = alg_agg;
        ctl->total_weight = total_weight;
        ctl->edge_count = edge_count;
        ctl->t_lm = t_lm;
        ctl->t_rf = t_rf;
        ctl->t_ag = t_ag;
    }
}

// ------------------------------------------------------------ the last sweeps of a larger level
struct TailCtl {
    unsigned done, which, sweep, epoch, swept, pad;
    unsigned long long moves_before;
};
struct TailArgs {
    Params p;
    const uint32_t* first;  // the first sweep's list (null: all of [0, n))
    uint32_t* list[2];      // later lists: sweep k of this launch reads list[k & 1]
    unsigned* count[2];
    uint32_t* stamp;
    uint32_t n, sweep, epoch, limit;
    unsigned long long moves_before, budget;
    TailCtl* ctl;
};

// Local moving from sweep a.sweep on, whose list the host has counted, until
// the level is done or a sweep has more than a.limit active nodes.
template <bool MULTI>
__global__ void __launch_bounds__(TEAM_THREADS, 1) k_move_tail(const __grid_constant__ TailArgs a) {
    extern __shared__ __align__(16) unsigned char raw[];
    TeamSmem& s = *reinterpret_cast<TeamSmem*>(raw);
    const Team team{blockIdx.x, gridDim.x};
    const bool lead = team.rank == 0 && threadIdx.x == 0;
    if (threadIdx.x == 0) s.nbig = s.bigmax = s.nitem = s.next = 0;
    __syncthreads();
    Params p = a.p;
    Tally tally{0, 0, 0};
    uint32_t sweep = a.sweep, epoch = a.epoch, swept = 0, which = 0;
    unsigned long long moves_before = a.moves_before;
    bool done = true;
    for (; sweep < (uint32_t)MAX_SWEEPS; ++sweep) {
        const uint32_t* list = swept || !a.first ? a.list[which] : a.first;
        if (!swept && !a.first) list = nullptr;
        const uint32_t m = swept || a.first ? *a.count[which] : a.n;
        const unsigned long long moves = p.counters[0];
        if (swept) {  // the host has checked the first sweep
            if (moves == moves_before || moves >= a.budget || m == 0) break;
            if (m > a.limit) {
                done = false;
                break;
            }
            moves_before = moves;
        }
        unsigned* ncount = a.count[which ^ 1];
        uint32_t* next = a.list[which ^ 1];
        for (int b = 0; b < LM_BATCHES; ++b) {
            p.cur = ++epoch;
            decide_batch<false, MULTI, false>(p, team, s, list, m, sweep, LM_BATCHES, b, 0, tally);
            team.sync();
            if (b == 0 && lead) *ncount = 0;
            apply_batch<false, MULTI>(p, team, list, m, p.counters, p.gain_acc);
            team.sync();
            activate_batch(p, team, s, list, m, a.stamp, sweep + 2, next, ncount);
        }
        team.sync();
        which ^= 1u;
        ++swept;
    }
    warp_add(p.counters + 1, tally.deg);
    warp_add(p.counters + 2, tally.cand);
    warp_add(p.counters + 3, tally.nodes);
    if (lead) {
        a.ctl->done = done;
        a.ctl->which = which;
        a.ctl->sweep = sweep;
        a.ctl->epoch = epoch;
        a.ctl->swept = swept;
        a.ctl->moves_before = moves_before;
    }
}

// A launch of one cluster of `blocks` blocks with the team's shared memory.
struct TeamLaunch {
    cudaLaunchConfig_t config{};
    cudaLaunchAttribute cluster{};
    template <class K>
    TeamLaunch(Ctx& c, K kernel, uint32_t blocks) {
        SC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TeamSmem)));
        SC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        config.gridDim = dim3(blocks);
        config.blockDim = dim3(TEAM_THREADS);
        config.dynamicSmemBytes = sizeof(TeamSmem);
        config.stream = c.stream;
        cluster.id = cudaLaunchAttributeClusterDimension;
        cluster.val.clusterDim.x = blocks;
        cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
        config.attrs = &cluster;
        config.numAttrs = 1;
    }
    TeamLaunch(const TeamLaunch&) = delete;
    TeamLaunch& operator=(const TeamLaunch&) = delete;
};

template <class K, class A>
void launch_team(Ctx& c, K kernel, uint32_t blocks, const A& args) {
    TeamLaunch l(c, kernel, blocks);
    SC_CUDA(cudaLaunchKernelEx(&l.config, kernel, args));
    c.launches++;
}

// Half a team beside other instances' work.
uint32_t team_blocks(Ctx& c) { return c.side[0] ? team_offer(c) : std::min(team_offer(c), TEAM_CLUSTER / 2); }

}  // namespace

// A cluster of 16 blocks, each with most of an SM's shared memory, needs 16 free SMs
// that the hardware lets share one: more than the 8 every device promises, and not
// there on every part or partition of a GPU. All of the team's kernels have the
// same threads and shared memory (and one block an SM), so k_team answers for them.
uint32_t team_offer(Ctx& c) {
    if (c.team_offered < 0) {
        c.team_offered = 0;
        if (c.smem_optin < sizeof(TeamSmem)) return 0;
        for (uint32_t blocks = TEAM_CLUSTER; blocks >= TEAM_CLUSTER / 2 && !c.team_offered; blocks /= 2) {
            TeamLaunch l(c, k_team, blocks);
            int clusters = 0;
            if (cudaOccupancyMaxActiveClusters(&clusters, k_team, &l.config) != cudaSuccess) {
                cudaGetLastError();  // a cluster size that the device does not have
                clusters = 0;
            }
            if (clusters > 0) c.team_offered = (int32_t)blocks;
        }
    }
    return std::min((uint32_t)c.team_offered, c.team_most);
}

bool team_takes(Ctx& c, const DevGraph& g, const sc_leiden_config& cfg) {
    return team_offer(c) && g.n > 0 && g.n <= TEAM_MAX_NODES && g.E <= TEAM_MAX_ENTRIES && !cfg.has_max_community_weight && g.exact_w &&
           g.exact_nw && g.part_max_2m == 0.0 && g.part_max_nw == 0.0 && graph_bitwise_symmetric(c, g);
}

void team_run(Ctx& c, const DevGraph& g, uint32_t* memb, uint64_t C, const sc_leiden_config& cfg, uint64_t pass_seed,
              uint64_t level, double improvement, TeamSpace& space, uint32_t* node_map, TeamResult& out) {
    const uint32_t n = (uint32_t)g.n;
    const uint64_t E = g.E;
    if (C > n) fail(SC_E_INTERNAL, "more community ids than nodes");
    TeamArgs a{};
    // one allocation, carved in 16-byte steps
    size_t total = 0;
    auto carve = [&](unsigned char* base) {
        size_t off = 0;
        auto take = [&](auto*& p, size_t count) {
            using T = std::remove_reference_t<decltype(*p)>;
            p = base ? reinterpret_cast<T*>(base + off) : nullptr;
            off += (count * sizeof(T) + 15) & ~size_t(15);
        };
        for (TeamBuf& b : a.buf) {
            take(b.ptr, (size_t)n + 1);
            take(b.nbr, E);
            take(b.w, E);
            take(b.strength, n);
            take(b.node_w, n);
            take(b.self_loop, n);
        }
        take(a.memb2, n);
        take(a.Kf, 2 * (size_t)n);
        take(a.Wf, 2 * (size_t)n);
        take(a.csize, 2 * (size_t)n);
        for (uint32_t** p : {&a.tgt, &a.hint, &a.from, &a.epoch, &a.moved, &a.stamp, &a.list0, &a.list1, &a.refined,
                             &a.grp, &a.members, &a.gcnt, &a.gcap, &a.gcur, &a.cnt})
            take(*p, n);
        take(a.dgain, n);
        take(a.loops, n);
        take(a.bits, 2 * (SLOTS_MAX / 32));
        take(a.tnbr, E);
        take(a.tw, E);
        take(a.ctl, 1);
        total = off;
    };
    carve(nullptr);
    if (space.n < n || space.E < E || !space.mem.get()) {
        space.mem.alloc(c, total);
        space.n = n;
        space.E = E;
    }
    carve(space.mem.get());
    a.in = TeamBuf{g.ptr, g.nbr, g.w, g.strength, g.node_w, g.self_loop};
    a.n = n;
    a.E = E;
    a.C = C;
    a.total_weight = g.total_weight;
    a.edge_count = g.edge_count;
    a.e0_w = g.e0_w;
    a.e0_nw = g.e0_nw;
    a.memb = memb;
    a.node_at = node_map;
    a.refine_ctr = c.d_refine_ctr;
    a.status = c.d_status;
    a.objective = cfg.objective;
    a.refine = cfg.refine;
    a.need_nc = cfg.objective == SC_OBJECTIVE_CPM;
    a.gamma = cfg.resolution;
    a.randomness = cfg.refine_randomness;
    a.improvement = improvement;
    a.pass_seed = pass_seed;
    a.level = level;
    a.max_levels = cfg.max_levels;

    const bool solo = n <= SOLO_NODES && E <= SOLO_ENTRIES;
    const uint32_t blocks = solo ? 1u : team_blocks(c);
    launch_team(c, k_team, blocks, a);

    TeamCtl r;
    {
        Mailbox mb(c);
        const TeamCtl* h = mb.get(a.ctl, 1);
        mb.wait();
        r = *h;
    }
    out.finished = r.state == 1;
    if (!out.finished && r.state != 2) {
        check_device_status(c);
        fail(SC_E_INTERNAL, "the small-level kernel ended without a result");
    }
    out.level = r.level;
    out.improvement = r.improvement;
    out.sweeps = r.sweeps;
    out.moves = r.total_moves;
    out.levels = r.levels;
    out.ms_local_move = 1e-6 * (double)r.t_lm;
    out.ms_refine = 1e-6 * (double)r.t_rf;
    out.ms_aggregate = 1e-6 * (double)r.t_ag;
    out.alg_bytes_local_move = r.alg_lm;
    out.alg_bytes_aggregate = r.alg_agg;
    if (out.finished) {
        out.n_clusters = r.C;
        return;
    }
    out.C = r.C;
    if (r.memb2) d2d(c, memb, a.memb2, r.n);
    const TeamBuf& b = a.buf[r.buf];
    out.graph.reset(graph_from_contraction(c, r.n, r.E, b.ptr, b.nbr, b.w, b.node_w));
}

uint32_t tail_limit(Ctx& c, const DevGraph& g, const sc_leiden_config& cfg) {
    if (cfg.has_max_community_weight || g.max_degree > BLOCK_DEGREE || g.E > 0xFFFFFFFFull) return 0;
    return team_blocks(c) * TAIL_NODES_PER_BLOCK;
}

TailResult tail_run(Ctx& c, const void* params, uint32_t n, const uint32_t* first, uint32_t* const lists[2],
                    uint32_t* const counts[2], uint32_t* stamp, uint32_t sweep, uint32_t epoch, uint64_t moves_before,
                    uint64_t budget) {
    DBuf<TailCtl> ctl(c, 1);
    TailArgs a{};
    a.p = *static_cast<const Params*>(params);
    a.first = first;
    a.list[0] = lists[0];
    a.list[1] = lists[1];
    a.count[0] = counts[0];
    a.count[1] = counts[1];
    a.stamp = stamp;
    a.n = n;
    a.sweep = sweep;
    a.epoch = epoch;
    a.limit = std::min<uint32_t>(TEAM_MAX_NODES, 2 * team_blocks(c) * TAIL_NODES_PER_BLOCK);
    a.moves_before = moves_before;
    a.budget = budget;
    a.ctl = ctl.get();
    if (a.p.inst) launch_team(c, k_move_tail<true>, team_blocks(c), a);
    else launch_team(c, k_move_tail<false>, team_blocks(c), a);
    const TailCtl r = to_host(c, ctl.get());
    TailResult t;
    t.done = r.done != 0;
    t.swapped = r.which != 0;
    t.sweep = r.sweep;
    t.epoch = r.epoch;
    t.swept = r.swept;
    t.moves_before = r.moves_before;
    return t;
}

}  // namespace sc
