// sc_move.cuh — what every kernel that scores or commits moves shares: the
// parameters of a level, the objectives' gains in the reference's operation
// order, the conflict rule and the hash tables of neighbour communities.
#pragma once

#include "sc_prims.cuh"

namespace sc {

namespace {

constexpr unsigned TB = 256;
constexpr int NBUCKET = 6;          // G8, G16, G32, warp (shared hash), block (shared hash), hub (global hash)
constexpr uint32_t WARP_DEGREE = 256;  // largest degree of the warp-per-node bucket
constexpr int WCAP = 2 * WARP_DEGREE;  // per-warp shared hash entries
constexpr int WARPS_PER_BLOCK = 4;
constexpr int HCAP_SMEM = 2 * HUB_DEGREE;  // shared hash entries per block (u32 key + i64 val): 24 KB
constexpr int LM_BATCHES = 2;
constexpr int RF_BATCHES = 8;
constexpr int MAX_SLOTS = 64;  // (batch, bucket) counters, cursors and offsets are sized for this
static_assert(LM_BATCHES * NBUCKET <= MAX_SLOTS && RF_BATCHES * NBUCKET <= MAX_SLOTS,
              "batch x bucket slots exceed the fixed counter arrays");
constexpr int MAX_SWEEPS = 100;
constexpr uint32_t EMPTYK = 0xFFFFFFFFu;

struct Params {
    // graph
    const uint64_t* ptr;
    const uint32_t* nbr;
    const float* w;
    const double* strength;
    const double* node_w;
    const double* self_loop;
    // partition being changed (working partition or refined partition)
    uint32_t* memb;
    long long* Kf;
    long long* Wf;
    uint32_t* csize;
    // refinement only: the constraint (working membership)
    const uint32_t* constraint;
    // decisions
    uint32_t* tgt;
    uint32_t* hint;
    uint32_t* from;
    long long* dgain;
    uint32_t* epoch;
    uint32_t cur;
    uint64_t S0;           // fresh-community id base (local moving)
    // objective
    int objective;
    double gamma, four_m, thr;
    double scale, inv_scale;    // 2^F, 2^-F for edge-weight quantities
    double nscale, inv_nscale;  // same for node weights
    int has_limit;
    double limit;
    int need_nc;                // community node weights are read (CPM, or a weight cap)
    double theta;               // refinement randomness (<= 0: argmax)
    uint64_t seed;
    uint32_t* status;
    unsigned long long* counters;  // [0] moves, [1] Σdeg, [2] Σcand, [3] nodes
    long long* gain_acc;
    // max_community_weight: one joiner per target community per batch (the
    // highest claim key wins), so a community never passes the cap
    unsigned long long* claim;
    uint32_t* moved;  // epoch in which the node last committed a move
    // batched runs over a disjoint union of instances (nullptr: one instance,
    // the scalars above): each node's instance, the instances' settings, and
    // each instance's gain accumulator
    const uint32_t* inst;
    const struct InstCfg* icfg;
    long long* gain_inst;
};

// Settings of one instance of a batched run, for the current level.
struct InstCfg {
    double gamma, four_m, thr, theta;
    uint64_t seed;    // the instance's seed for this level (local moving or refinement)
    uint32_t base;    // the instance's first node id in the union at this level
    uint32_t frozen;  // 1: the instance takes no decisions (it stopped, as its own run would)
};

// What a node's decisions read: the run's scalars, or its instance's. Hashes
// and tie rules see instance-local ids (node id - base), so a node of a batched
// run draws exactly what it draws in its instance's own run.
struct NodeCfg {
    double gamma, four_m, thr, theta;
    uint64_t seed;
    uint32_t base;
};

template <bool MULTI>
__device__ __forceinline__ NodeCfg node_cfg(const Params& p, uint32_t v) {
    if (!MULTI) return NodeCfg{p.gamma, p.four_m, p.thr, p.theta, p.seed, 0u};
    const InstCfg& c = p.icfg[p.inst[v]];
    return NodeCfg{c.gamma, c.four_m, c.thr, c.theta, c.seed, c.base};
}

__device__ __forceinline__ long long to_fix(double x, double inv) { return __double2ll_rn(__dmul_rn(x, inv)); }
__device__ __forceinline__ double from_fix(long long q, double s) { return __dmul_rn(__ll2double_rn(q), s); }

// Rb::delta_insert (objective.rs:91-106) / Cpm::delta_insert (:158-169)
__device__ __forceinline__ double gain_of(const Params& p, const NodeCfg& q, double wto, double sl, double k,
                                          double kc, double a, double nc) {
    if (p.objective == SC_OBJECTIVE_RB) {
        if (q.four_m == 0.0) return 0.0;
        return __dsub_rn(__dadd_rn(wto, sl),
                         __ddiv_rn(__dmul_rn(__dmul_rn(q.gamma, k), __dadd_rn(__dmul_rn(2.0, kc), k)),
                                   q.four_m));
    }
    return __dsub_rn(__dadd_rn(wto, sl),
                     __dmul_rn(__dmul_rn(__dmul_rn(q.gamma, a),
                                         __dsub_rn(__dadd_rn(__dmul_rn(2.0, nc), a), 1.0)),
                               0.5));  // x / 2, exactly
}

__device__ __forceinline__ bool better(double g, uint32_t c, double bg, uint32_t bc) {
    return g > bg || (g == bg && c < bc);
}

// The best (g, c) of a warp, or of each half, by `better`: the largest key, then
// the lowest id. Integer reductions of the key's two words in the doubles' order
// (zeros made positive: they are equal): four rounds of shuffles and double
// comparisons are a chain of 16 dependent shuffles. A NaN is no candidate.
__device__ __forceinline__ uint64_t order_key(double g) {
    const uint64_t b = (uint64_t)__double_as_longlong(g == g ? __dadd_rn(g, 0.0) : -INFINITY);
    return b ^ ((b >> 63) ? ~0ull : 1ull << 63);
}
__device__ __forceinline__ double key_order(uint64_t k) {
    return __longlong_as_double((long long)(k ^ ((k >> 63) ? 1ull << 63 : ~0ull)));
}

__device__ __forceinline__ void warp_best(double& g, uint32_t& c) {
    const unsigned FULL = 0xFFFFFFFFu;
    const uint64_t k = order_key(g);
    const uint32_t hi = __reduce_max_sync(FULL, (uint32_t)(k >> 32));
    bool top = (uint32_t)(k >> 32) == hi;
    const uint32_t lo = __reduce_max_sync(FULL, top ? (uint32_t)k : 0u);
    top = top && (uint32_t)k == lo;
    c = __reduce_min_sync(FULL, top ? c : 0xFFFFFFFFu);
    g = key_order((uint64_t)hi << 32 | lo);
}

// The same for the groups of G lanes of a warp, with what the best one's lane
// holds in m.
template <int G>
__device__ __forceinline__ void group_best(double& g, uint32_t& c, uint32_t& m) {
    const unsigned FULL = 0xFFFFFFFFu;
    if constexpr (G >= 16) {
        const bool up = G == 16 && (threadIdx.x & 16u);
        auto max_of = [&](uint32_t x) {
            if (G == 32) return __reduce_max_sync(FULL, x);
            const uint32_t a = __reduce_max_sync(FULL, up ? 0u : x), b = __reduce_max_sync(FULL, up ? x : 0u);
            return up ? b : a;
        };
        const uint64_t k = order_key(g);
        const uint32_t hi = max_of((uint32_t)(k >> 32));
        bool top = (uint32_t)(k >> 32) == hi;
        const uint32_t lo = max_of(top ? (uint32_t)k : 0u);
        top = top && (uint32_t)k == lo;
        const uint32_t best = ~max_of(top ? ~c : 0u);
        const unsigned at = __ballot_sync(FULL, top && c == best) & (G == 32 ? FULL : up ? 0xFFFF0000u : 0xFFFFu);
        m = __shfl_sync(FULL, m, __ffs(at) - 1);
        c = best;
        g = key_order((uint64_t)hi << 32 | lo);
    } else {
#pragma unroll
        for (int o = G / 2; o; o >>= 1) {
            const double og = __shfl_xor_sync(FULL, g, o);
            const uint32_t oc = __shfl_xor_sync(FULL, c, o), om = __shfl_xor_sync(FULL, m, o);
            if (better(og, oc, g, c)) {
                g = og;
                c = oc;
                m = om;
            }
        }
    }
}

__device__ __forceinline__ uint64_t prio(uint64_t seed, uint32_t ep, uint32_t v) {
    return hash3(seed ^ 0xA5A5A5A5DEADBEEFull, ep, v);
}

// Whether node x's move (decided in epoch p.cur) is cancelled. x and the
// member h of its target are nodes of the same instance.
template <bool MULTI>
__device__ __forceinline__ bool cancelled(const Params& p, uint32_t x) {
    uint32_t h = p.hint[x];
    if (h == NONE32) return false;
    if (p.epoch[h] != p.cur) return false;  // the target's member is not moving
    if (p.hint[h] == x) {                   // mutual: the lower priority yields
        const NodeCfg q = node_cfg<MULTI>(p, x);
        uint64_t px = prio(q.seed, p.cur, x - q.base), ph = prio(q.seed, p.cur, h - q.base);
        return px < ph || (px == ph && x < h);
    }
    return true;
}

template <bool MULTI>
__device__ __forceinline__ unsigned long long claim_key(const Params& p, uint32_t v) {
    const NodeCfg q = node_cfg<MULTI>(p, v);
    return ((unsigned long long)p.cur << 40) | ((prio(q.seed ^ 0x77ull, p.cur, v - q.base) & 0xFFull) << 32) | v;
}

// Whether node x's move is dropped: cancelled, or beaten to a capped community.
template <bool MULTI>
__device__ __forceinline__ bool lost(const Params& p, uint32_t x) {
    if (cancelled<MULTI>(p, x)) return true;
    return p.has_limit && p.claim[p.tgt[x]] != claim_key<MULTI>(p, x);
}

// Refinement's randomised choice (refine.rs:110-153) draws candidate c with
// probability exp(rel_c / theta) / sum. Gumbel-max draws from the same
// distribution: argmax_c rel_c / theta + G_c with G_c = -log(-log U_c), U_c
// uniform in (0, 1) from a hash of (seed, epoch, node, c). The result does not
// depend on the order candidates are visited in, so no candidate list or sort
// is needed. theta <= 0 is the deterministic argmax (ties to the lower id).
// v and c are instance-local ids (refined community ids are node ids).
__device__ __forceinline__ double refine_key(const Params& p, const NodeCfg& q, double rel, uint32_t v,
                                             uint32_t c) {
    if (q.theta <= 0.0) return rel;
    uint64_t h = hash3(q.seed ^ 0x5151515151515151ull, ((uint64_t)p.cur << 32) | v, c);
    double u = ((double)(h >> 11) + 0.5) * 0x1.0p-53;
    return __dadd_rn(__ddiv_rn(rel, q.theta), -log(-log(u)));
}

// The hash batch of node v in a sweep, or -1 for a node of a frozen instance.
template <bool MULTI>
__device__ __forceinline__ int batch_of(uint64_t seed, uint32_t sweep, uint64_t v, int B, const uint32_t* inst,
                                        const InstCfg* icfg) {
    if (!MULTI) return (int)(hash3(seed, sweep, v) % (uint64_t)B);
    const InstCfg& c = icfg[inst[v]];
    if (c.frozen) return -1;
    return (int)(hash3(c.seed, sweep, v - c.base) % (uint64_t)B);
}

// Read-only load (ld.global.nc): the decide kernels never write the graph, the
// membership or the community aggregates they read; only the commit kernels do.
template <class T>
__device__ __forceinline__ T ro(const T* a) {
    return __ldg(a);
}

// Warp-aggregated counter add.
__device__ __forceinline__ void warp_add(unsigned long long* ctr, unsigned long long x) {
    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xFFFFFFFFu, x, o);
    if ((threadIdx.x & 31) == 0 && x) atomicAdd(ctr, x);
}

// ------------------------------------------------------------ large-degree decide
__device__ __forceinline__ uint32_t hslot(uint32_t c, uint32_t mask) {
    return (c * 0x9E3779B1u) & mask;
}

__device__ bool hinsert(uint32_t* keys, long long* vals, uint32_t mask, uint32_t c, long long x,
                        uint32_t* status) {
    uint32_t h = hslot(c, mask);
    for (uint32_t probe = 0; probe <= mask; ++probe) {
        uint32_t k = keys[h];
        if (k == c) {
            atomicAdd((unsigned long long*)(vals + h), (unsigned long long)x);
            return true;
        }
        if (k == EMPTYK) {
            uint32_t prev = atomicCAS(keys + h, EMPTYK, c);
            if (prev == EMPTYK || prev == c) {
                atomicAdd((unsigned long long*)(vals + h), (unsigned long long)x);
                return true;
            }
        }
        h = (h + 1) & mask;
    }
    atomicOr(status, DEV_OVERFLOW);
    return false;
}

// hinsert that also appends every slot it claims to `list` (the distinct keys,
// in no particular order; the caller sized `list` for all of them).
__device__ void hinsert_listed(uint32_t* keys, long long* vals, uint32_t mask, uint32_t c, long long x,
                               uint32_t* status, uint32_t* list, uint32_t* count, uint32_t list_cap) {
    uint32_t h = hslot(c, mask);
    for (uint32_t probe = 0; probe <= mask; ++probe) {
        uint32_t k = keys[h];
        if (k == EMPTYK) {
            const uint32_t prev = atomicCAS(keys + h, EMPTYK, c);
            if (prev == EMPTYK) {
                const uint32_t i = atomicAdd(count, 1u);
                if (i < list_cap) list[i] = h;
                else atomicOr(status, DEV_OVERFLOW);
            }
            k = prev == EMPTYK ? c : prev;
        }
        if (k == c) {
            atomicAdd((unsigned long long*)(vals + h), (unsigned long long)x);
            return;
        }
        h = (h + 1) & mask;
    }
    atomicOr(status, DEV_OVERFLOW);
}

__device__ long long hlookup(const uint32_t* keys, const long long* vals, uint32_t mask, uint32_t c) {
    uint32_t h = hslot(c, mask);
    for (uint32_t probe = 0; probe <= mask; ++probe) {
        uint32_t k = keys[h];
        if (k == c) return vals[h];
        if (k == EMPTYK) return 0;
        h = (h + 1) & mask;
    }
    return 0;
}

// Block-wide argmax of (g, c) with ties to the lower id.
__device__ void block_argmax(double& g, uint32_t& c, double* sg, uint32_t* sc) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int o = 16; o; o >>= 1) {
        double og = __shfl_xor_sync(0xFFFFFFFFu, g, o);
        uint32_t oc = __shfl_xor_sync(0xFFFFFFFFu, c, o);
        if (better(og, oc, g, c)) {
            g = og;
            c = oc;
        }
    }
    if (lane == 0) {
        sg[wid] = g;
        sc[wid] = c;
    }
    __syncthreads();
    if (wid == 0) {
        int nw = blockDim.x >> 5;
        g = lane < nw ? sg[lane] : -INFINITY;
        c = lane < nw ? sc[lane] : NONE32;
        for (int o = 16; o; o >>= 1) {
            double og = __shfl_xor_sync(0xFFFFFFFFu, g, o);
            uint32_t oc = __shfl_xor_sync(0xFFFFFFFFu, c, o);
            if (better(og, oc, g, c)) {
                g = og;
                c = oc;
            }
        }
        if (lane == 0) {
            sg[0] = g;
            sc[0] = c;
        }
    }
    __syncthreads();
    g = sg[0];
    c = sc[0];
    __syncthreads();
}

}  // namespace

}  // namespace sc
