// sc_knn.cu — Gaussian kNN graph builder (src/neighborhood/mod.rs) on sm_100a.
//
// 1. k_knn_prep       X (f32) -> A = [-2x, 1, 1, 0..] and B = [x, |x|^2 hi, |x|^2 lo, 0..]
//                     in 16 bits, KA = 32 (D <= 30) or 64 (D <= 62) columns: f16,
//                     scaled by a power of two, where the points' range allows it,
//                     BF16 otherwise (f16_exp).
//                     A . B = |c|^2 - 2 q.c = |q - c|^2 - |q|^2: the row-constant
//                     |q|^2 does not change a row's ranking, so the contraction
//                     yields ranking scores directly.
//    k_knn_prep_f8    the FP8 (e4m3) operands, 64 one-byte columns (D <= 61): B =
//                     [x / S, three e4m3 terms of |x|^2 / S_n, 0..] with one scale
//                     for the point set, A = f_q [-2 x S / S_n, 1, 1, 1, 0..] with a
//                     power-of-two scale f_q per query row. A . B = (f_q / S_n) (|c|^2
//                     - 2 q.c): a positive factor per row, so the ranking is kept
//                     (a per-point scale on B would rescale columns and break it).
//                     64-byte rows: the tile geometry, swizzle and descriptors of the
//                     BF16 KA = 32 path; each K step is one kind::f8f6f4 MMA of K = 32.
// 2. k_knn_tc         persistent tcgen05 kernel, one CTA per SM. A group of 256
//                     queries (two M = 128 tiles) stays in shared memory; every
//                     128-candidate tile of B streams in by TMA (no multicast)
//                     through a STAGES-deep ring; one thread issues
//                     tcgen05.mma (M=128, N=128, K=16, 16 bit -> FP32) into a
//                     double-buffered TMEM accumulator (2 x 2 x 128 columns);
//                     16 epilogue warps read it with tcgen05.ld and keep scores
//                     in shared memory. A first scan keeps minima that bound each
//                     query's (k+1)-th distance, a second one starts from that
//                     bound and keeps each (query, half)'s 32 best candidates.
// 3. k_knn_rerank     exact FP32 distances sum (q_d - c_d)^2 of the R candidates
//                     (no norm expansion, so no cancellation), sorted by
//                     (distance, self first, index); the first k+1 are kept.
// 4. k_knn_sigma / k_knn_pairs / CSR: sigma (median of the positive distances,
//                     neighborhood/mod.rs:105-124, or the k-th distance), the
//                     Gaussian weight of :139-163, lower-id or union emission,
//                     sorted into a CSR that from_csr_parts then finishes.
//
// Every wait on an mbarrier is bounded: on timeout the CTA records
// DEV_TIMEOUT, drains the copies it issued (again bounded), frees its TMEM and
// returns; the host turns the status into SC_E_TIMEOUT.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cudaTypedefs.h>

#include "sc_prims.cuh"

namespace sc {

namespace {

constexpr int QT = 2;              // query tiles of 128 per CTA group
constexpr int TILE = 128;          // rows per tile (M and N of the MMA)
constexpr int HALVES = 2;          // each accumulator row is read as two 64-column halves
constexpr int RCAND = 32;          // candidates kept per (query, half) before the exact re-rank
constexpr int RTOTAL = RCAND * HALVES;  // candidates per query handed to the re-rank
constexpr int NUM_EPI_WARPS = 4 * QT * HALVES;  // a full set of 4 TMEM lane quarters per (tile, half)
constexpr int KNN_THREADS = 32 * (2 + NUM_EPI_WARPS);
template <int KA>
constexpr int stages_for() { return KA == 32 ? 6 : 3; }  // B ring depth within 227 KB
constexpr uint32_t WAIT_LIMIT = DEFAULT_WAIT_LIMIT;  // drain waits: copies / MMAs already issued
constexpr uint32_t TMEM_COLS = 512;

// ------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

// Bounded wait for the phase with the given parity to complete: at most
// `limit` try_wait attempts, false when they ran out.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint32_t limit = WAIT_LIMIT) {
    const uint32_t addr = smem_u32(bar);
    for (uint32_t it = 0; it < limit; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(addr), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
            smem_u32(dst)),
        "l"((uint64_t)map), "r"(smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// One lane of a converged warp, the same one each time.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xFFFFFFFF;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(p));
    return p != 0;
}

// Shared-memory matrix descriptor, K-major, swizzled rows of KA * 2 bytes:
// start >> 4 at [0,14), stride between 8-row groups >> 4 at [32,46),
// version 1 at [46,48), layout at [61,64) (4 = 64B swizzle, 2 = 128B swizzle).
template <int KA>
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    constexpr uint64_t row_bytes = KA * 2;
    constexpr uint64_t sbo = 8 * row_bytes;
    constexpr uint64_t layout = (KA == 32) ? 4ull : 2ull;
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFF);
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= 1ull << 46;
    d |= layout << 61;
    return d;
}

// Instruction descriptor, kind::f16: D f32, A and B both f16 (format 0) or both
// bf16 (format 1), both K-major, N = 128, M = 128.
__host__ __device__ constexpr uint32_t idesc_16bit_128x128(bool f16) {
    return (1u << 4) | (f16 ? 0u : (1u << 7) | (1u << 10)) | ((uint32_t)(TILE >> 3) << 17) |
           ((uint32_t)(TILE >> 4) << 24);
}

__device__ __forceinline__ void mma_16bit(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Instruction descriptor, kind::f8f6f4: D f32, A/B e4m3 (format 0), both K-major, N = 128, M = 128.
__host__ __device__ constexpr uint32_t idesc_e4m3_128x128() {
    return (1u << 4) | ((uint32_t)(TILE >> 3) << 17) | ((uint32_t)(TILE >> 4) << 24);
}

__device__ __forceinline__ void mma_e4m3(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// 64 accumulator columns of this lane's row. The wait stands in the same
// statement, so no use of the values can be moved before it.
__device__ __forceinline__ void tmem_ld64(uint32_t taddr, float (&v)[64]) {
    uint32_t r[64];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x64.b32 {"
        "%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,"
        "%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47,"
        "%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63}, [%64];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]),
          "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]),
          "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]),
          "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]),
          "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 64; ++i) v[i] = __uint_as_float(r[i]);
}

// 8 accumulator columns of this lane's row.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// A (query, half)'s candidates: CAND_SLOTS slots of shared memory, filled in
// order; when a row of the warp has no room for the next, all rows are cut back
// to their RCAND best together, equal ones by their order. Every lane of the warp
// calls it. A row of `cnt` keeps min(cnt, RCAND), in the first slots. Returns the score
// from which on nothing is a candidate any more: the worst kept of a full row,
// else cap. Near tiles bring a row's candidates in a burst, 95 a query at
// 1M x 50; a search for the worst of a full row at each of them (a call for one
// or two rows at a time, while all warps of the block wait) held up every warp by
// 290 cycles a tile, this by 60.
constexpr uint32_t SLOT_STRIDE = QT * HALVES * TILE;  // (tile, half, row) owners: one column per owner
constexpr int CAND_SLOTS = RCAND + 4;
__device__ __noinline__ float cand_cut(float* cs, uint32_t* ci, uint32_t owner, uint32_t cnt, float cap) {
    constexpr int TOP = CAND_SLOTS - RCAND + 1;
    float top[TOP];  // the row's largest, descending
#pragma unroll
    for (int i = 0; i < TOP; ++i) top[i] = -INFINITY;
#pragma unroll 4
    for (uint32_t s = 0; s < (uint32_t)CAND_SLOTS; ++s) {
        float v = s < cnt ? cs[s * SLOT_STRIDE + owner] : -INFINITY;
#pragma unroll
        for (int i = 0; i < TOP; ++i) {
            const float hi = fmaxf(top[i], v);
            v = fminf(top[i], v);
            top[i] = hi;
        }
    }
    if (cnt < (uint32_t)RCAND) return cap;
    const uint32_t drop = cnt - RCAND;  // of the largest: the worst kept is top[drop]
    float worst = top[0];
    uint32_t ties = 0;  // dropped ones that equal the worst kept
#pragma unroll
    for (int i = 1; i < TOP; ++i)
        if ((uint32_t)i <= drop) {
            ties = top[i] == worst ? ties + 1 : 0;
            worst = top[i];
        }
    if (drop) {
        // of the entries that equal the worst kept the first ones stay: slots fill
        // in the order of the points, and ties go to the lower index
        uint32_t room = 0xFFFFFFFFu;
        if (ties) {
            room = 0;
            for (uint32_t s = 0; s < cnt; ++s) room += cs[s * SLOT_STRIDE + owner] == worst ? 1u : 0u;
            room -= ties;
        }
        uint32_t w = owner;
#pragma unroll 4
        for (uint32_t s = 0; s < cnt; ++s) {
            const float v = cs[s * SLOT_STRIDE + owner];
            const uint32_t id = ci[s * SLOT_STRIDE + owner];
            bool keep = v <= worst;
            if (v == worst) {
                keep = room > 0;
                room -= keep ? 1u : 0u;
            }
            if (keep) {
                cs[w] = v;
                ci[w] = id;
                w += SLOT_STRIDE;
            }
        }
    }
    return fminf(worst, cap);
}

// A bounding scan keeps scores alone: BOUND_SLOTS per (query, half), cut back to
// the BOUND_KEEP smallest (ascending, in the first slots) when a row of the warp
// is nearly full. Returns the largest kept of a row that holds BOUND_KEEP or
// more, +inf for one that holds fewer. Every lane of the warp calls it.
//
// Its time counts for every warp of the block: with one tile of slack, all wait
// for the one that cuts. Each value moved up through the list in turn took 15,800
// cycles a cut (15 cuts a warp in 1750 tiles of 1M x 50 points), 16 values at a
// time through a sorting network 10,400; the scan went from 7.3 to 5.8 ms.
constexpr int BOUND_KEEP = 16;
constexpr int BOUND_SLOTS = 2 * RCAND;  // the candidates' scores and ids in one

__device__ __forceinline__ void order2(float& a, float& b) {
    const float lo = fminf(a, b);
    b = fmaxf(a, b);
    a = lo;
}

__device__ __noinline__ float bound_cut(float* cs, uint32_t owner, uint32_t cnt) {
    static_assert(BOUND_KEEP == 16 && BOUND_SLOTS % 16 == 0, "blocks of 16 slots");
    float best[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) best[i] = INFINITY;
#pragma unroll 1
    for (uint32_t s = 0; s < (uint32_t)BOUND_SLOTS; s += 16) {
        if (!__any_sync(0xFFFFFFFFu, s < cnt)) break;
        float v[16];
#pragma unroll
        for (uint32_t i = 0; i < 16; ++i) v[i] = s + i < cnt ? cs[(s + i) * SLOT_STRIDE + owner] : INFINITY;
        // Batcher's odd-even merge sort, ascending
#pragma unroll
        for (int p = 1; p < 16; p <<= 1)
#pragma unroll
            for (int k = p; k >= 1; k >>= 1)
#pragma unroll
                for (int j = k % p; j + k < 16; j += 2 * k)
#pragma unroll
                    for (int i = 0; i < k; ++i)
                        if (i + j + k < 16 && (i + j) / (2 * p) == (i + j + k) / (2 * p)) order2(v[i + j], v[i + j + k]);
        // the 16 smallest of both lists, a bitonic sequence, then in order
#pragma unroll
        for (int i = 0; i < 16; ++i) best[i] = fminf(best[i], v[15 - i]);
#pragma unroll
        for (int k = 8; k >= 1; k >>= 1)
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if ((i & k) == 0) order2(best[i], best[i + k]);
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) cs[i * SLOT_STRIDE + owner] = best[i];
    return best[15];
}

// ------------------------------------------------------------ prep
// What the operand kernels know of the point set (device words, zeroed first;
// non-negative floats order like their bit patterns, so integer atomics find
// the largest).
struct KnnScale {
    unsigned maxabs;   // max |x_ij|
    unsigned maxnorm;  // max |x_i|^2
    unsigned minrow;   // ~bits of the smallest max_j |x_ij| of a point that is not all zeros (atomicMax of ~bits)
    unsigned rho;      // max |x_i - x^_i| / |x_i|, x^ the 16-bit operand (k_knn_prep)
};

// The 16-bit operands are f16 where the points' range allows it, BF16 otherwise:
// both run at the same rate, f16 rounds 8 times finer (11 significant bits), so
// the score bounds that the scans start from are that much tighter and fewer
// scores pass them. f16 needs a common power-of-two scale that brings the
// largest coordinate to [64, 128); a point whose largest coordinate is then
// 2^-6 or more keeps |x - x^| <= (2^-11 + 2^-16) |x| although its small
// coordinates may fall below f16's normal range. Points of a wider range (an
// outlier 2^12 times the rest) keep BF16's relative rounding. Returns the
// scale's exponent, or INT32_MIN for BF16.
__device__ __forceinline__ int f16_exp(const KnnScale* k) {
    const float ma = __uint_as_float(k->maxabs), mr = __uint_as_float(~k->minrow);
    if (!(ma > 0x1.0p-40f) || !(ma < 0x1.0p40f) || k->minrow == 0u || !(mr * 0x1.0p12f >= ma)) return INT32_MIN;
    return 6 - ilogbf(ma);
}

// Rows of X as the contraction's operands, a warp per row (lane j holds columns
// j and j + 32): A = [-2 x^, c1, c2, 0..], B = [x^, hi, lo, 0..], with c1 hi +
// c2 lo = |x|^2 to 22 bits in f16 (c1 = 32 and c2 = 2^-5 keep both terms in its
// range) and to 16 bits in BF16 (c1 = c2 = 1). Also each row's norm and the
// norm of its rounding error, both rounded up: with the largest relative one
// (rho) they bound every score's error (score_margin).
template <int KA>
__global__ void k_knn_prep(const float* __restrict__ X, uint64_t n, uint32_t d, KnnScale* sc, uint16_t* A,
                           uint16_t* B, float* __restrict__ nx, float* __restrict__ rx) {
    const unsigned FULL = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const int e = f16_exp(sc);
    const bool f16 = e != INT32_MIN;
    const float s = f16 ? ldexpf(1.0f, e) : 1.0f, inv = f16 ? ldexpf(1.0f, -e) : 1.0f;
    float rho = 0.0f;
    for (uint64_t i = warp; i < n; i += nwarps) {
        float x[KA / 32], nrm = 0.0f, res = 0.0f;
        uint16_t a[KA / 32], b[KA / 32];
#pragma unroll
        for (int t = 0; t < KA / 32; ++t) {
            const uint32_t j = lane + 32 * t;
            x[t] = j < d ? X[i * d + j] : 0.0f;
            nrm = __fmaf_rn(x[t], x[t], nrm);
            float back;  // the operand's value, in the points' units
            if (f16) {
                const __half h = __float2half_rn(x[t] * s);
                back = __half2float(h) * inv;
                b[t] = __half_as_ushort(h);
                a[t] = __half_as_ushort(__float2half_rn(-2.0f * __half2float(h)));
            } else {
                const __nv_bfloat16 h = __float2bfloat16_rn(x[t]);
                back = __bfloat162float(h);
                b[t] = __bfloat16_as_ushort(h);
                a[t] = __bfloat16_as_ushort(__float2bfloat16_rn(-2.0f * back));
            }
            const float df = x[t] - back;
            res = __fmaf_rn(df, df, res);
        }
        for (int o = 16; o; o >>= 1) {
            nrm += __shfl_xor_sync(FULL, nrm, o);
            res += __shfl_xor_sync(FULL, res, o);
        }
        uint16_t hi, lo, c1, c2;
        if (f16) {
            const float v = nrm * s * s * (1.0f / 32.0f);
            const __half h = __float2half_rn(v);
            hi = __half_as_ushort(h);
            lo = __half_as_ushort(__float2half_rn((v - __half2float(h)) * 1024.0f));
            c1 = __half_as_ushort(__float2half_rn(32.0f));
            c2 = __half_as_ushort(__float2half_rn(0x1.0p-5f));
        } else {
            const __nv_bfloat16 h = __float2bfloat16_rn(nrm);
            hi = __bfloat16_as_ushort(h);
            lo = __bfloat16_as_ushort(__float2bfloat16_rn(nrm - __bfloat162float(h)));
            c1 = c2 = __bfloat16_as_ushort(__float2bfloat16_rn(1.0f));
        }
#pragma unroll
        for (int t = 0; t < KA / 32; ++t) {
            const uint32_t j = lane + 32 * t;
            if (j == d) {
                a[t] = c1;
                b[t] = hi;
            } else if (j == d + 1) {
                a[t] = c2;
                b[t] = lo;
            } else if (j > d + 1) {
                a[t] = b[t] = 0;
            }
            A[i * KA + j] = a[t];
            B[i * KA + j] = b[t];
        }
        // FP32 sums of squares of at most 62 terms: 2^-17 covers their rounding
        const float up = 1.0f + 0x1.0p-16f;
        if (lane == 0) {
            nx[i] = sqrtf(nrm) * up;
            rx[i] = sqrtf(res) * up;
        }
        if (nrm > 0.0f) rho = fmaxf(rho, sqrtf(res) / sqrtf(nrm) * (up * up));
    }
    if (lane == 0 && rho > 0.0f) atomicMax(&sc->rho, __float_as_uint(rho));
}

// The point set's ranges (KnnScale).
__global__ void k_knn_scales(const float* __restrict__ X, uint64_t n, uint32_t d, KnnScale* sc) {
    float ma = 0.0f, mn = 0.0f, mr = INFINITY;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const float* x = X + i * d;
        float nrm = 0.0f, row = 0.0f;
        for (uint32_t j = 0; j < d; ++j) {
            row = fmaxf(row, fabsf(x[j]));
            nrm = __fmaf_rn(x[j], x[j], nrm);
        }
        ma = fmaxf(ma, row);
        if (row > 0.0f) mr = fminf(mr, row);
        mn = fmaxf(mn, nrm);
    }
    for (int o = 16; o; o >>= 1) {
        ma = fmaxf(ma, __shfl_xor_sync(0xFFFFFFFFu, ma, o));
        mn = fmaxf(mn, __shfl_xor_sync(0xFFFFFFFFu, mn, o));
        mr = fminf(mr, __shfl_xor_sync(0xFFFFFFFFu, mr, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&sc->maxabs, __float_as_uint(ma));
        atomicMax(&sc->maxnorm, __float_as_uint(mn));
        if (mr < INFINITY) atomicMax(&sc->minrow, ~__float_as_uint(mr));
    }
}

__device__ __forceinline__ uint8_t to_e4m3(float x) { return (uint8_t)__nv_cvt_float_to_fp8(x, __NV_SATFINITE, __NV_E4M3); }

__device__ __forceinline__ float from_e4m3(uint8_t b) {
    __nv_fp8_e4m3 v;
    v.__x = (__nv_fp8_storage_t)b;
    return (float)v;
}

// FP8 operands (64 one-byte columns, D <= 61): see the file comment.
__global__ void k_knn_prep_f8(const float* __restrict__ X, uint64_t n, uint32_t d, const KnnScale* __restrict__ sc,
                              uint8_t* A, uint8_t* B) {
    constexpr uint32_t W = 64;
    const float ma = __uint_as_float(sc->maxabs), mn = __uint_as_float(sc->maxnorm);
    const float S = ma > 0.0f ? ma / 256.0f : 1.0f;
    const float Sn = mn > 0.0f ? mn / 256.0f : 1.0f;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const float* x = X + i * d;
        uint8_t* a = A + i * W;
        uint8_t* b = B + i * W;
        float nrm = 0.0f, m = 0.0f;
        for (uint32_t j = 0; j < d; ++j) {
            nrm = __fmaf_rn(x[j], x[j], nrm);
            m = fmaxf(m, fabsf(2.0f * x[j] * S / Sn));
        }
        // power-of-two row factor f with m f <= 448, f in [2^-9, 2^8] (both e4m3-exact)
        int e = 8;
        if (m > 0.0f) {
            e = (int)floorf(log2f(448.0f / m));
            e = e < -9 ? -9 : (e > 8 ? 8 : e);
        }
        const float f = ldexpf(1.0f, e);
        for (uint32_t j = 0; j < d; ++j) {
            a[j] = to_e4m3(-2.0f * x[j] * S / Sn * f);
            b[j] = to_e4m3(x[j] / S);
        }
        // |x|^2 / S_n as three e4m3 terms (each takes the remainder of the last)
        float v = nrm / Sn;
        for (uint32_t t = 0; t < 3; ++t) {
            const uint8_t q = to_e4m3(v);
            b[d + t] = q;
            a[d + t] = to_e4m3(f);
            v -= from_e4m3(q);
        }
        for (uint32_t j = d + 3; j < W; ++j) {
            a[j] = 0;
            b[j] = 0;
        }
    }
}

// ------------------------------------------------------------ tensor-core candidate search
template <int KA>
struct KnnSmem {
    static constexpr int STAGES = stages_for<KA>();
    static constexpr uint32_t TILE_BYTES = TILE * KA * 2;
    static constexpr uint32_t SLOTS = QT * HALVES * TILE;                       // (tile, half, row) owners
    static constexpr uint32_t A_OFF = 0;
    static constexpr uint32_t B_OFF = A_OFF + QT * TILE_BYTES;
    static constexpr uint32_t C_OFF = B_OFF + STAGES * TILE_BYTES;               // candidate scores
    static constexpr uint32_t I_OFF = C_OFF + CAND_SLOTS * SLOTS * 4;            // candidate ids (or more scores)
    static constexpr uint32_t BAR_OFF = I_OFF + CAND_SLOTS * SLOTS * 4;
    static constexpr uint32_t NBAR = 2 * STAGES + 2 * 2 * QT + 2;
    static constexpr uint32_t MISC_OFF = BAR_OFF + NBAR * 8;
    static constexpr uint32_t BYTES = MISC_OFF + 64 + 1024;  // + alignment slack
    static_assert(BYTES <= 227 * 1024, "shared memory of the kNN kernel exceeds 227 KB");
    static_assert(SLOTS == SLOT_STRIDE, "one candidate column per (tile, half, row)");
};

// The point tiles a query group scans, in order: every tile, or (a pruned
// search) the group's ranges of (first tile, tile count), which never overlap.
// The next range is in registers before the current one ends: the loads of
// a range list of single tiles stood in every tile's way.
struct TileWalk {
    const uint2* r;
    uint32_t nr, ri, off, all;
    uint2 cur, nxt;
    __device__ uint2 at(uint32_t i) const { return r && i < nr ? r[i] : make_uint2(0u, 0u); }
    __device__ TileWalk(const uint32_t* rptr, const uint2* rngs, uint32_t g, uint32_t ntiles)
        : r(rptr ? rngs + rptr[g] : nullptr), nr(rptr ? rptr[g + 1] - rptr[g] : 0), ri(0), off(0), all(ntiles) {
        cur = at(0);
        nxt = at(1);
    }
    __device__ uint32_t count() const {
        if (!r) return all;
        uint32_t c = 0;
        for (uint32_t i = 0; i < nr; ++i) c += r[i].y;
        return c;
    }
    __device__ uint32_t next() {  // called count() times at most
        if (!r) return off++;
        while (off >= cur.y) {
            cur = nxt;
            ++ri;
            nxt = at(ri + 1);
            off = 0;
        }
        return cur.x + off++;
    }
};

// min of three in one instruction; a NaN gives way to a number, like fminf.
__device__ __forceinline__ float fmin3(float a, float b, float c) {
    float m;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
    return m;
}

// F8: the operands are e4m3 bytes with the row size of BF16 KA columns.
// rptr / rngs (nullable): the tile ranges of each query group (pruned search).
// qcap (nullable): per query, a score no kept candidate reaches (a proven
// bound from an earlier pass); the rows start from it instead of +inf, so far
// points are never candidates.
// gorder (nullable): the groups in descending order of their tile counts; the
// CTAs take them forwards and backwards in turn, so the sums of their counts
// stay close (200k x 50 points: 782 groups of 90 to 500 tiles; taken as they
// come, an SM idled 29 to 36% of the kernel).
// BOUND: the scan only bounds each query's (k+1)-th score: bound[q] receives the
// BOUND_KEEP smallest 8-column minima of either half, ascending. k+1 minima are
// k+1 points, so their largest is a bound, and nearly the (k+1)-th score itself
// (two of a query's nearest seldom share 8 columns); no ids, no list to keep in
// order. Otherwise cand_idx[q] receives the candidates' ids.
//
// The epilogue sets the pace (K = 64 leaves the tensor pipe 31 to 42% busy), and
// of it the warp that is slowest, since all others wait for it within a tile. Per
// tile a warp reads its 64 columns at once and takes minima of 8 columns (three
// values an instruction); only an 8-column group in which some row's minimum
// passes that row's threshold is looked at again, all rows of the warp together, a
// candidate costing two predicated stores. Rows are cut back when one is full
// (cand_cut, bound_cut). Taking the rows one by one, with a search of the row's
// slots for every candidate, the two scans of 1M x 50 points took 31.1 and 56.4
// ms, a search only for a full row 8.5 and 16.4; 5.8 and 11.7 ms now.
template <int KA, bool F8, bool BOUND = false>
__global__ void __launch_bounds__(KNN_THREADS, 1)
    k_knn_tc(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, uint32_t n,
             uint32_t nq, uint32_t* __restrict__ cand_idx, float* __restrict__ bound, uint32_t* status, uint32_t lim,
             uint32_t hold_tiles, const KnnScale* __restrict__ scale, const uint32_t* __restrict__ rptr,
             const uint2* __restrict__ rngs, const float* __restrict__ qcap, const uint32_t* __restrict__ gorder) {
    using L = KnnSmem<KA>;
    extern __shared__ __align__(1024) unsigned char raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
    unsigned char* sA = smem + L::A_OFF;
    unsigned char* sB = smem + L::B_OFF;
    float* cs = (float*)(smem + L::C_OFF);
    uint32_t* ci = (uint32_t*)(smem + L::I_OFF);
    uint64_t* bars = (uint64_t*)(smem + L::BAR_OFF);
    uint64_t* full = bars;                 // [L::STAGES] B tile landed
    uint64_t* empty = bars + L::STAGES;       // [L::STAGES] B tile consumed by the MMAs
    // an accumulator per (buffer, query tile), handed over on its own: the warps
    // of one query tile work while the other's products are under way
    uint64_t* accfull = bars + 2 * L::STAGES;  // [2][QT] accumulator ready
    uint64_t* accempty = accfull + 2 * QT;     // [2][QT] accumulator drained
    uint64_t* afull = accempty + 2 * QT;       // query tiles landed
    uint64_t* aempty = afull + 1;              // query tiles no longer read
    uint32_t* misc = (uint32_t*)(smem + L::MISC_OFF);
    volatile uint32_t* abort_flag = misc + 1;

    const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const uint32_t ntiles = (n + TILE - 1) / TILE;          // point tiles (B)
    const uint32_t ngroups = (nq + QT * TILE - 1) / (QT * TILE);  // query tile groups (A)
    // the i-th group of this CTA, ngroups when there is none
    auto group_at = [&](uint32_t i) -> uint32_t {
        const uint64_t pos = (uint64_t)i * gridDim.x + ((i & 1) && gorder ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
        return pos >= ngroups ? ngroups : (gorder ? gorder[pos] : (uint32_t)pos);
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < L::STAGES; ++s) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, 1);
        }
        for (int b = 0; b < 2 * QT; ++b) {
            mbar_init(accfull + b, 1);
            mbar_init(accempty + b, NUM_EPI_WARPS / QT);
        }
        mbar_init(afull, 1);
        mbar_init(aempty, 1);
        misc[1] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(misc)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = misc[0];

    if (warp == 0) {
        // ---------------- TMA producer
        if (lane == 0) {
            uint64_t it = 0;                    // B tiles issued, all groups
            uint32_t stage = 0, s_parity = 0;  // the stage in turn
            uint32_t gi = 0;
            bool a_in_flight = false;
            for (uint32_t g; (g = group_at(gi)) < ngroups && !*abort_flag; ++gi) {
                if (gi > 0 && !mbar_wait(aempty, (gi - 1) & 1, lim)) {
                    *abort_flag = 1;
                    break;
                }
                mbar_expect_tx(afull, QT * L::TILE_BYTES);
                a_in_flight = true;
                for (int q = 0; q < QT; ++q)
                    tma_load_2d(sA + q * L::TILE_BYTES, &tmA, afull, 0, (int)(g * QT * TILE + q * TILE));
                if (hold_tiles) {  // test hook: no point tile is ever issued
                    ++gi;
                    break;
                }
                TileWalk walk(rptr, rngs, g, ntiles);
                const uint32_t cnt = walk.count();
                for (uint32_t t = 0; t < cnt; ++t, ++it) {
                    const uint32_t tile = walk.next();
                    // a stage's first use passes at once: its barrier is in phase 0
                    if (!mbar_wait(empty + stage, s_parity ^ 1u, lim)) {
                        *abort_flag = 1;
                        break;
                    }
                    if (*abort_flag) break;
                    mbar_expect_tx(full + stage, L::TILE_BYTES);
                    tma_load_2d(sB + stage * L::TILE_BYTES, &tmB, full + stage, 0, (int)(tile * TILE));
                    if (++stage == (uint32_t)L::STAGES) {
                        stage = 0;
                        s_parity ^= 1u;
                    }
                }
            }
            // drain: the copies issued last (one per stage, and the query tiles)
            // must land before the CTA exits (waits with the default limit)
            if (*abort_flag || hold_tiles) {
                for (uint64_t x = it > L::STAGES ? it - L::STAGES : 0; x < it; ++x)
                    mbar_wait(full + (x % L::STAGES), (uint32_t)((x / L::STAGES) & 1));
                if (a_in_flight && gi > 0) mbar_wait(afull, (gi - 1) & 1);
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer. One warp issues every product, so its
        // instructions are on each tile's path: the whole warp walks the tiles
        // (addresses and descriptors are then uniform), one lane issues, and
        // stages and parities are counted, not divided. With a descriptor built
        // for every product and 64-bit remainders the issue alone took 1040
        // cycles of a tile's 2200 (300 to 500 now), the products 512.
        const uint32_t idesc = F8 ? idesc_e4m3_128x128() : idesc_16bit_128x128(f16_exp(scale) != INT32_MIN);
        const uint64_t adesc = smem_desc<KA>(smem_u32(sA)), bdesc = smem_desc<KA>(smem_u32(sB));
        constexpr uint32_t TILE_STEP = L::TILE_BYTES >> 4;  // of a descriptor's start address
        const bool issuer = elect_one();
        uint64_t* last = nullptr;  // the newest accumulator commit and its parity
        uint32_t last_parity = 0;
        uint32_t s = 0, s_parity = 0, b = 0, b_parity = 0;  // the B stage and accumulator buffer in turn
        uint32_t gi = 0;
        bool ok = true;
        for (uint32_t g; ok && (g = group_at(gi)) < ngroups && !__any_sync(0xFFFFFFFFu, *abort_flag != 0); ++gi) {
            ok = __all_sync(0xFFFFFFFFu, mbar_wait(afull, gi & 1, lim));
            if (!ok) break;
            fence_after();
            const uint32_t cnt = __shfl_sync(0xFFFFFFFFu, TileWalk(rptr, rngs, g, ntiles).count(), 0);
            for (uint32_t t = 0; t < cnt; ++t) {
                ok = __all_sync(0xFFFFFFFFu, mbar_wait(full + s, s_parity, lim));
                const uint64_t bd = bdesc + s * TILE_STEP;
#pragma unroll
                for (int q = 0; q < QT; ++q) {
                    const uint32_t acc = b * QT + q;
                    // a buffer's first use passes at once: its barrier is in phase 0
                    if (ok) ok = __all_sync(0xFFFFFFFFu, mbar_wait(accempty + acc, b_parity ^ 1u, lim));
                    if (!ok) break;
                    fence_after();
                    const uint64_t ad = adesc + q * TILE_STEP;
                    if (issuer) {
#pragma unroll
                        for (int kk = 0; kk < KA / 16; ++kk) {  // 32 bytes of K per MMA
                            if constexpr (F8)
                                mma_e4m3(tmem + acc * TILE, ad + kk * 2, bd + kk * 2, idesc, kk > 0 ? 1u : 0u);
                            else
                                mma_16bit(tmem + acc * TILE, ad + kk * 2, bd + kk * 2, idesc, kk > 0 ? 1u : 0u);
                        }
                        mma_commit(accfull + acc);
                    }
                    last = accfull + acc;
                    last_parity = b_parity;
                }
                if (!ok) break;
                if (issuer) mma_commit(empty + s);
                if (++s == (uint32_t)L::STAGES) {
                    s = 0;
                    s_parity ^= 1u;
                }
                b ^= 1u;
                b_parity ^= b ^ 1u;  // both buffers used
            }
            if (ok && issuer) mma_commit(aempty);
        }
        if (!ok) *abort_flag = 1;
        // drain: MMAs complete in issue order, so once the last tile's
        // accumulator commit has arrived none is left writing TMEM or
        // arriving on this CTA's barriers (waits with the default limit)
        if (__any_sync(0xFFFFFFFFu, *abort_flag != 0) && last) mbar_wait(last, last_parity);
        __syncwarp();
    } else {
        // ---------------- epilogue: 16 warps; warp % 4 selects the TMEM lane quarter
        // (hardware rule), (warp - 2) / 4 the (query tile, column half) it reads
        const int ew = warp - 2;
        const int combo = ew >> 2;
        const int q = combo / HALVES;           // query tile
        const int h = combo % HALVES;           // column half
        const int lq = warp & 3;                // lane quarter
        const int row = lq * 32 + lane;         // row within the query tile
        const uint32_t owner = combo * TILE + row;  // candidate-buffer column
        constexpr uint32_t S = SLOT_STRIDE;
        uint32_t b = 0, b_parity = 0;  // the accumulator buffer in turn
        uint32_t gi = 0;
        for (uint32_t g; (g = group_at(gi)) < ngroups && !__any_sync(0xFFFFFFFFu, *abort_flag != 0); ++gi) {
            const uint64_t qrow = (uint64_t)g * QT * TILE + q * TILE + row;
            const float capv = (!BOUND && qcap && qrow < nq) ? qcap[qrow] : INFINITY;
            float thr = qrow < nq ? capv : -INFINITY;  // rows past the last query take nothing
            uint32_t cnt = 0;      // candidates held
            uint32_t off = owner;  // where the next one goes
            TileWalk walk(rptr, rngs, g, ntiles);
            const uint32_t tcnt = walk.count();
            for (uint32_t t = 0; t < tcnt; ++t) {
                const uint32_t tile = walk.next();
                const uint32_t acc = b * QT + q;
                if (!__all_sync(0xFFFFFFFFu, mbar_wait(accfull + acc, b_parity, lim))) {
                    *abort_flag = 1;
                    break;
                }
                fence_after();
                const uint32_t taddr = tmem + ((uint32_t)(lq * 32) << 16) + acc * TILE + h * (TILE / HALVES);
                float r[64];
                tmem_ld64(taddr, r);
                auto release = [&] {  // the accumulator is no longer read
                    fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(accempty + acc);
                };
                if constexpr (BOUND) release();
                b ^= 1u;
                b_parity ^= b ^ 1u;
                const uint32_t base_idx = tile * TILE + h * (TILE / HALVES);
                if (base_idx + 64 > n) {  // the last tile's rows past the points hold zeros, not scores
#pragma unroll
                    for (int j = 0; j < 64; ++j)
                        if (base_idx + j >= n) r[j] = INFINITY;
                }
                float m[8];
#pragma unroll
                for (int j8 = 0; j8 < 8; ++j8) {
                    const float* x = r + j8 * 8;
                    m[j8] = fminf(fmin3(x[0], x[1], x[2]), fmin3(fmin3(x[3], x[4], x[5]), x[6], x[7]));
                }
                const float mall = fminf(fmin3(m[0], m[1], m[2]), fmin3(fmin3(m[3], m[4], m[5]), m[6], m[7]));
                if (!__any_sync(0xFFFFFFFFu, mall < thr)) {
                    if constexpr (!BOUND) release();
                    continue;
                }
                if constexpr (BOUND) {
                    if (__any_sync(0xFFFFFFFFu, cnt > BOUND_SLOTS - 8)) {  // a tile adds up to 8
                        thr = fminf(thr, bound_cut(cs, owner, cnt));
                        cnt = cnt < BOUND_KEEP ? cnt : BOUND_KEEP;
                        off = cnt * S + owner;
                    }
#pragma unroll
                    for (int j8 = 0; j8 < 8; ++j8) {
                        if (m[j8] < thr) {
                            cs[off] = m[j8];
                            ++cnt;
                            off += S;
                        }
                    }
                } else {
                    // the 8-column groups with a candidate, read again one at a time:
                    // the same few instructions for all of them (unrolled over the 64
                    // columns they were fetched anew for each hit), and the columns'
                    // registers are free for them
                    unsigned groups = 0;
#pragma unroll
                    for (int j8 = 0; j8 < 8; ++j8)
                        groups |= (__any_sync(0xFFFFFFFFu, m[j8] < thr) ? 1u : 0u) << j8;
#pragma unroll 1
                    while (groups) {
                        __syncwarp();  // the lanes part below, at their stores and in cand_cut
                        const uint32_t j8 = (uint32_t)__ffs(groups) - 1;
                        groups &= groups - 1;
                        float x[8];
                        tmem_ld8(taddr + j8 * 8, x);
                        const uint32_t id = base_idx + j8 * 8;
                        if (id + 8 > n) {
#pragma unroll
                            for (int j = 0; j < 8; ++j)
                                if (id + j >= n) x[j] = INFINITY;
                        }
#pragma unroll
                        for (int j4 = 0; j4 < 8; j4 += 4) {
                            uint32_t more = cnt;
#pragma unroll
                            for (int j = j4; j < j4 + 4; ++j) more += x[j] < thr ? 1u : 0u;
                            if (__any_sync(0xFFFFFFFFu, more > (uint32_t)CAND_SLOTS)) {
                                thr = fminf(thr, cand_cut(cs, ci, owner, cnt, capv));
                                cnt = cnt < RCAND ? cnt : RCAND;
                                off = cnt * S + owner;
                            }
#pragma unroll
                            for (int j = j4; j < j4 + 4; ++j)
                                if (x[j] < thr) {
                                    cs[off] = x[j];
                                    ci[off] = id + j;
                                    ++cnt;
                                    off += S;
                                }
                        }
                    }
                    release();
                }
            }
            if (__any_sync(0xFFFFFFFFu, *abort_flag != 0)) break;
            if constexpr (BOUND) {
                bound_cut(cs, owner, cnt);
                if (qrow < nq)
                    for (int s2 = 0; s2 < BOUND_KEEP; ++s2)
                        bound[(qrow * HALVES + h) * BOUND_KEEP + s2] = cs[s2 * S + owner];
            } else {
                cand_cut(cs, ci, owner, cnt, capv);
                if (qrow < nq)
                    for (uint32_t s2 = 0; s2 < (uint32_t)RCAND; ++s2)
                        cand_idx[qrow * RTOTAL + h * RCAND + s2] = s2 < cnt ? ci[s2 * S + owner] : 0xFFFFFFFFu;
            }
        }
    }
    fence_before();
    __syncthreads();
    fence_after();
    if (threadIdx.x == 0 && *abort_flag) atomicOr(status, DEV_TIMEOUT);
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS)
                     : "memory");
    }
}

// ------------------------------------------------------------ FP32 candidate search
// The FP32 arm: squared distances computed on the CUDA cores as
// sum_t (q_t - c_t)^2, the re-rank's own operations in the same order
// (dimensions past d are zero on both sides and add exactly nothing), so the
// candidates are the exact FP32 nearest points, with no norm expansion and no
// reduced-precision operand. A thread holds F32_Q queries' coordinates in
// registers; points stream through shared memory in tiles of F32_TILE (every
// thread reads the same point: broadcast loads).
//
// Bound by instruction issue with two warps a scheduler: 2 DP operations a pair (DP:
// d rounded up to 4, a register array's size), and the candidate slots leave room
// for four blocks of two warps an SM. At 30,011 x 50 the issue slots are 62% busy,
// the FMA pipe 45%, the shared-memory pipe 29%; between issues a warp waits for
// its own last operation or a broadcast load. One query a thread, which halves the
// operations a 16-byte load feeds, took 8.7 ms there, two (and two or four points
// at a time) take 6.3. The work
// items (F32_QUERIES queries x a half of the points, the half's RCAND best in its
// half of the candidate slots) are cut into equal runs of point tiles, one run a
// resident block, so that a few items fill the chip too: a block per item took
// 275 us at 1,000 x 30 points, 780 at 5,003 x 30 and 57.3 ms at 100,000 x 50, the
// runs take 47, 500 and 53.8; at 30,011 x 50 both take 6.3 ms. More queries a thread
// or more warps would need more slots than shared memory holds. An item that
// several blocks share goes through their lists in scratch (k_f32_merge).
//
// A candidate is two predicated stores into the query's F32_SLOTS
// slots; when a row of the warp is nearly full, all rows are cut back to their
// RCAND best together. The floor is 2.5 ms of FP32 operations; one query a thread,
// a search of the row for every insertion and DP = 64 for all d > 32 took 9.1 ms.
constexpr int F32_THREADS = 64;
constexpr int F32_Q = 2;  // queries a thread
constexpr int F32_QUERIES = F32_THREADS * F32_Q;
constexpr int F32_TILE = 32;
constexpr int F32_SLOTS = 44;
constexpr int F32_GROUP = 4;  // points taken together: eight independent sums a thread

// Cuts a row of `cnt` candidates to its RCAND best by (distance, id): the last one
// takes the worst one's slot until RCAND are left. Returns the worst distance kept,
// or thr with fewer.
__device__ __noinline__ float f32_cut(float* cs, uint32_t* ci, uint32_t cnt, float thr) {
    while (cnt >= (uint32_t)RCAND) {
        float worst = -INFINITY;
        uint32_t at = 0, last = 0;  // the first and the last slot that hold the worst
#pragma unroll 8
        for (uint32_t s = 0; s < cnt; ++s) {
            const float x = cs[s * F32_QUERIES];
            if (x >= worst) last = s;
            if (x > worst) {
                worst = x;
                at = s;
            }
        }
        thr = worst;
        if (cnt == (uint32_t)RCAND) break;
        if (at != last)  // equal ones: the highest id goes
            for (uint32_t s = at + 1; s <= last; ++s)
                if (cs[s * F32_QUERIES] == worst && ci[s * F32_QUERIES] > ci[at * F32_QUERIES]) at = s;
        --cnt;
        cs[at * F32_QUERIES] = cs[cnt * F32_QUERIES];
        ci[at * F32_QUERIES] = ci[cnt * F32_QUERIES];
    }
    return thr;
}

// The runs: unit u is tile u % per of item u / per, block b takes units
// [first(b), first(b + 1)).
struct F32Plan {
    uint64_t units, per;
    uint32_t blocks;
    __host__ __device__ uint64_t first(uint64_t b) const { return b * units / blocks; }
    __host__ __device__ uint64_t block_of(uint64_t u) const {
        uint64_t b = u * blocks / units;
        while (first(b + 1) <= u) ++b;
        while (first(b) > u) --b;
        return b;
    }
};

template <int DP>
__global__ void __launch_bounds__(F32_THREADS) k_knn_fp32(const float* __restrict__ X, uint64_t n, uint32_t d,
                                                          uint64_t q0, uint64_t nq, F32Plan plan,
                                                          uint32_t* __restrict__ cand_idx,
                                                          unsigned long long* __restrict__ shared_lists) {
    extern __shared__ __align__(16) unsigned char smem[];
    float* tile = (float*)smem;                                // [F32_TILE][DP]
    float* cs = tile + F32_TILE * DP + threadIdx.x;            // [F32_SLOTS][F32_QUERIES], this thread's columns
    uint32_t* ci = (uint32_t*)(cs + F32_SLOTS * F32_QUERIES);  // at 0 and F32_THREADS; the ids beside them
    const uint32_t t = threadIdx.x;
    const uint64_t u0 = plan.first(blockIdx.x), u1 = plan.first(blockIdx.x + 1);
    for (uint64_t unit = u0; unit < u1;) {
        const uint64_t item = unit / plan.per, half = item % HALVES;
        const uint64_t stop = (item + 1) * plan.per < u1 ? (item + 1) * plan.per : u1;  // this block's part of it
        const uint64_t lq0 = item / HALVES * F32_QUERIES + t;
        float q[F32_Q][DP], thr[F32_Q];
        uint32_t cnt[F32_Q];
#pragma unroll
        for (int u = 0; u < F32_Q; ++u) {
            const uint64_t lq = lq0 + u * F32_THREADS;
#pragma unroll
            for (int j = 0; j < DP; ++j) q[u][j] = (lq < nq && (uint32_t)j < d) ? X[(q0 + lq) * d + j] : 0.0f;
            thr[u] = lq < nq ? INFINITY : -INFINITY;
            cnt[u] = 0;
        }
        // the points of the item's tiles [unit, stop)
        const uint64_t h0 = half * plan.per;  // the half's first tile
        const uint64_t p0 = (h0 + unit % plan.per) * F32_TILE;
        const uint64_t p1 = min(n, (h0 + (stop - 1) % plan.per + 1) * F32_TILE);
        for (uint64_t base = p0; base < p1; base += F32_TILE) {
            __syncthreads();  // the previous tile is no longer read
            for (uint32_t e = t; e < (uint32_t)(F32_TILE * DP); e += F32_THREADS) {
                const uint32_t p = e / DP, j = e % DP;
                tile[e] = (base + p < p1 && j < d) ? X[(base + p) * d + j] : 0.0f;
            }
            __syncthreads();
            const uint32_t points = (p1 - base < (uint64_t)F32_TILE) ? (uint32_t)(p1 - base) : (uint32_t)F32_TILE;
            for (uint32_t g = 0; g < points; g += F32_GROUP) {
#pragma unroll
                for (int u = 0; u < F32_Q; ++u) {
                    if (__any_sync(0xFFFFFFFFu, cnt[u] > F32_SLOTS - F32_GROUP)) {
                        thr[u] = f32_cut(cs + u * F32_THREADS, ci + u * F32_THREADS, cnt[u], thr[u]);
                        cnt[u] = cnt[u] < (uint32_t)RCAND ? cnt[u] : (uint32_t)RCAND;
                    }
                }
                // rows past the last point are zeros in the tile: computed, not taken
                float acc[F32_GROUP][F32_Q];
#pragma unroll
                for (int v = 0; v < F32_GROUP; ++v)
#pragma unroll
                    for (int u = 0; u < F32_Q; ++u) acc[v][u] = 0.0f;
                const float4* c4 = (const float4*)(tile + g * DP);
#pragma unroll
                for (int j4 = 0; j4 < DP / 4; ++j4) {
#pragma unroll
                    for (int v = 0; v < F32_GROUP; ++v) {
                        const float4 c = c4[v * (DP / 4) + j4];
#pragma unroll
                        for (int u = 0; u < F32_Q; ++u) {
                            float df = __fsub_rn(q[u][4 * j4], c.x);
                            acc[v][u] = __fmaf_rn(df, df, acc[v][u]);
                            df = __fsub_rn(q[u][4 * j4 + 1], c.y);
                            acc[v][u] = __fmaf_rn(df, df, acc[v][u]);
                            df = __fsub_rn(q[u][4 * j4 + 2], c.z);
                            acc[v][u] = __fmaf_rn(df, df, acc[v][u]);
                            df = __fsub_rn(q[u][4 * j4 + 3], c.w);
                            acc[v][u] = __fmaf_rn(df, df, acc[v][u]);
                        }
                    }
                }
#pragma unroll
                for (int v = 0; v < F32_GROUP; ++v) {
#pragma unroll
                    for (int u = 0; u < F32_Q; ++u) {
                        if (acc[v][u] < thr[u] && g + v < points) {
                            cs[cnt[u] * F32_QUERIES + u * F32_THREADS] = acc[v][u];
                            ci[cnt[u] * F32_QUERIES + u * F32_THREADS] = (uint32_t)(base + g + v);
                            ++cnt[u];
                        }
                    }
                }
            }
        }
        const bool whole = unit == item * plan.per && stop == (item + 1) * plan.per;
        unsigned long long* part = shared_lists + (2 * (uint64_t)blockIdx.x + (unit == u0 ? 0 : 1)) * F32_QUERIES * RCAND;
#pragma unroll
        for (int u = 0; u < F32_Q; ++u) {
            const uint64_t lq = lq0 + u * F32_THREADS;
            f32_cut(cs + u * F32_THREADS, ci + u * F32_THREADS, cnt[u], thr[u]);
            if (lq >= nq) continue;
            const uint32_t kept = cnt[u] < (uint32_t)RCAND ? cnt[u] : (uint32_t)RCAND;
            if (whole) {
                uint32_t* out = cand_idx + lq * RTOTAL + half * RCAND;
                for (uint32_t s2 = 0; s2 < (uint32_t)RCAND; ++s2)
                    out[s2] = s2 < kept ? ci[s2 * F32_QUERIES + u * F32_THREADS] : 0xFFFFFFFFu;
            } else {
                unsigned long long* out = part + (uint64_t)(t + u * F32_THREADS) * RCAND;
                for (uint32_t s2 = 0; s2 < (uint32_t)RCAND; ++s2) {
                    const uint32_t at = s2 * F32_QUERIES + u * F32_THREADS;
                    out[s2] = s2 < kept ? (unsigned long long)__float_as_uint(cs[at]) << 32 | ci[at] : ~0ull;
                }
            }
        }
        unit = stop;
    }
}

// The RCAND best of every item that several blocks shared, a warp per query: the
// list so far ascending, the next one descending, the smaller of each pair are
// the best of both. A key is the distance's bits over the id.
__device__ __forceinline__ unsigned long long warp_sort_keys(unsigned long long v, bool descending) {
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
    for (uint32_t k = 2; k <= 32; k <<= 1)
#pragma unroll
        for (uint32_t j = k >> 1; j; j >>= 1) {
            const unsigned long long o = __shfl_xor_sync(0xFFFFFFFFu, v, j);
            const bool up = ((lane & k) == 0) != descending;
            v = up == ((lane & j) == 0) ? (o < v ? o : v) : (o < v ? v : o);
        }
    return v;
}

__global__ void k_f32_merge(uint64_t nq, uint64_t items, F32Plan plan,
                            const unsigned long long* __restrict__ shared_lists, uint32_t* __restrict__ cand_idx) {
    static_assert(RCAND == 32, "a lane per candidate");
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t i = warp; i < items * F32_QUERIES; i += nwarps) {  // warp-uniform
        const uint64_t item = i / F32_QUERIES, ql = i % F32_QUERIES, lq = item / HALVES * F32_QUERIES + ql;
        if (lq >= nq) continue;
        const uint64_t b0 = plan.block_of(item * plan.per), b1 = plan.block_of((item + 1) * plan.per - 1);
        if (b0 == b1) continue;  // written by its block
        unsigned long long best = ~0ull;
        for (uint64_t b = b0; b <= b1; ++b) {
            const uint64_t slot = 2 * b + (plan.first(b) / plan.per == item ? 0 : 1);
            const unsigned long long v =
                warp_sort_keys(shared_lists[(slot * F32_QUERIES + ql) * RCAND + lane], b > b0);
            best = b == b0 ? v : warp_sort_keys(v < best ? v : best, false);
        }
        cand_idx[lq * RTOTAL + item % HALVES * RCAND + lane] = best == ~0ull ? 0xFFFFFFFFu : (uint32_t)best;
    }
}

template <int DP>
void candidates_fp32_dp(Ctx& c, const float* dX, uint64_t n, uint32_t d, uint64_t q0, uint64_t nq, uint32_t* cand_idx) {
    const size_t sm = (size_t)F32_TILE * DP * 4 + (size_t)F32_SLOTS * F32_QUERIES * 8;
    SC_CUDA(cudaFuncSetAttribute(k_knn_fp32<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    int resident = 0;
    SC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, k_knn_fp32<DP>, F32_THREADS, sm));
    const uint64_t items = (nq + F32_QUERIES - 1) / F32_QUERIES * HALVES;
    F32Plan plan;
    plan.per = ((n + F32_TILE - 1) / F32_TILE + HALVES - 1) / HALVES;  // tiles of a half
    plan.units = items * plan.per;
    plan.blocks = (uint32_t)std::min<uint64_t>(plan.units, (uint64_t)c.sm_count * std::max(resident, 1));
    if (!plan.units) return;
    DBuf<unsigned long long> lists(c, (uint64_t)plan.blocks * 2 * F32_QUERIES * RCAND);
    k_knn_fp32<DP><<<plan.blocks, F32_THREADS, sm, c.stream>>>(dX, n, d, q0, nq, plan, cand_idx, lists.get());
    k_f32_merge<<<grid_for(items * F32_QUERIES * 32, 256), 256, 0, c.stream>>>(nq, items, plan, lists.get(), cand_idx);
    SC_LAUNCH_CHECK();
    c.launches += 2;
}

// DP = d rounded up to a multiple of 4.
template <int DP = 4>
void candidates_fp32(Ctx& c, const float* dX, uint64_t n, uint32_t d, uint64_t q0, uint64_t nq, uint32_t* cand_idx) {
    if constexpr (DP < 64) {
        if (d > (uint32_t)DP) return candidates_fp32<DP + 4>(c, dX, n, d, q0, nq, cand_idx);
    }
    candidates_fp32_dp<DP>(c, dX, n, d, q0, nq, cand_idx);
}

// ------------------------------------------------------------ exact re-rank
__device__ __forceinline__ uint64_t rerank_key(const float* __restrict__ X, uint64_t n, uint32_t d, uint64_t q,
                                               uint32_t j) {
    if (j >= n) return ~0ull;
    const float* a = X + q * d;
    const float* b = X + (uint64_t)j * d;
    float acc = 0.0f;
    for (uint32_t t = 0; t < d; ++t) {
        const float diff = __fsub_rn(a[t], b[t]);
        acc = __fmaf_rn(diff, diff, acc);
    }
    // (distance, self first, index); acc >= 0 so its bits order like the value
    return ((uint64_t)__float_as_uint(acc) << 32) | (j == (uint32_t)q ? 0u : j + 1u);
}

__device__ __forceinline__ uint64_t warp_sort32(uint64_t key) {
    const unsigned lane = threadIdx.x & 31u;
    for (int size = 2; size <= 32; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            const uint64_t other = __shfl_xor_sync(0xFFFFFFFFu, key, stride);
            const bool up = ((lane & size) == 0);
            const bool lower = (lane & stride) == 0;
            const uint64_t mn = key < other ? key : other, mx = key < other ? other : key;
            key = (lower == up) ? mn : mx;
        }
    }
    return key;
}

// A query's list from its 64 candidates a, b (two per lane): their keys (key(id)),
// the 32 smallest kept by a merge-split of two sorted halves, ascending over the
// lanes. A row of more equal points than the candidates hold may lack the query
// itself: it comes first all the same, unless a coordinate is not finite (its
// distance to itself is then none).
template <class Key>
__device__ __forceinline__ uint64_t rerank_list(uint32_t a, uint32_t b, uint32_t self, Key key) {
    const unsigned FULL = 0xFFFFFFFFu, lane = threadIdx.x & 31u;
    const uint64_t ka = warp_sort32(key(a)), kb = warp_sort32(key(b));
    const uint64_t kbr = __shfl_sync(FULL, kb, 31 - lane);
    uint64_t k = ka < kbr ? ka : kbr;  // the 32 smallest, as a bitonic sequence
    for (int stride = 16; stride > 0; stride >>= 1) {
        const uint64_t other = __shfl_xor_sync(FULL, k, stride);
        k = (lane & stride) == 0 ? (k < other ? k : other) : (k < other ? other : k);
    }
    if (!__any_sync(FULL, a == self || b == self) && key(self) == 0) {  // warp-uniform
        const uint64_t before = __shfl_up_sync(FULL, k, 1);
        k = lane ? before : 0;
    }
    return k;
}

// One warp per query: exact FP32 distances of its RTOTAL = 64 candidates, the
// first k+1 written.
// Queries are points q0 .. q0 + nq - 1; rows of cand_idx / out_* are local.
__global__ void k_knn_rerank(const float* __restrict__ X, uint64_t n, uint32_t d, uint32_t k, uint64_t q0,
                             uint64_t nq, const uint32_t* __restrict__ cand_idx, uint32_t* __restrict__ out_idx,
                             float* __restrict__ out_d2) {
    const unsigned lane = threadIdx.x & 31u;
    const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t lq = warp; lq < nq; lq += nwarps) {
        const uint64_t q = q0 + lq;
        const uint32_t* cand = cand_idx + lq * RTOTAL;
        const uint64_t key = rerank_list(cand[lane], cand[32 + lane], (uint32_t)q,
                                         [&](uint32_t j) { return rerank_key(X, n, d, q, j); });
        if (lane <= k) {
            const uint32_t tag = (uint32_t)key;
            const uint32_t idx = (key == ~0ull) ? 0xFFFFFFFFu : (tag == 0 ? (uint32_t)q : tag - 1u);
            out_idx[lq * (k + 1) + lane] = idx;
            out_d2[lq * (k + 1) + lane] = key == ~0ull ? INFINITY : __uint_as_float((uint32_t)(key >> 32));
        }
    }
}

// ------------------------------------------------------------ sigma and connectivities
// sigma_i: median of the positive distances among the k+1 (neighborhood/mod.rs:480-499;
// the kd-tree path's sqrt(median(d^2)), :105-124, is the same element), 1 if none;
// or the k-th neighbour's distance.
__global__ void k_knn_sigma(const float* __restrict__ d2, uint64_t n, uint32_t k, int kth, float* sigma) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const float* r = d2 + i * (k + 1);
        // with fewer than k + 1 points the trailing slots are empty (infinite):
        // only the neighbours the search returned count, as in the reference
        uint32_t m = 0;
        while (m <= k && isfinite(r[m])) ++m;
        if (kth) {
            sigma[i] = m ? sqrtf(r[m - 1]) : 1.0f;
            continue;
        }
        uint32_t pos = 0;
        for (uint32_t t = 0; t < m; ++t) pos += r[t] > 0.0f;
        if (pos == 0) {
            sigma[i] = 1.0f;
            continue;
        }
        // rows are sorted ascending, positive entries are the last `pos` of the m
        uint32_t first = m - pos;
        sigma[i] = sqrtf(r[first + pos / 2]);
    }
}

// Connectivity weight of :139-163 in f32, operation for operation.
__device__ __forceinline__ float gauss_w(float dist_sq, float si, float sj, bool* ok) {
    float si2 = __fmul_rn(si, si), sj2 = __fmul_rn(sj, sj);
    float den = __fadd_rn(si2, sj2);
    *ok = den > 0.0f;
    if (!*ok) return 0.0f;
    float num = __fmul_rn(__fmul_rn(2.0f, si), sj);
    float norm = sqrtf(__fdiv_rn(num, den));
    float ex = expf(__fdiv_rn(-dist_sq, den));
    return __fmul_rn(norm, ex);
}

// Emit (row << idbits | col) keys and weights. lower_id: only from the row
// i <= j, both directions (the reference's rule). union: every listed pair,
// both directions; duplicates are removed after the sort (a pair listed from
// both sides carries the same bits twice, so the order of emission is free).
// A thread per listed pair, coalesced reads of the lists; the slots of a block's
// pairs come from one atomic (ballots inside a warp, the warps' counts in
// shared memory). One atomic per pair on the one counter, a thread per row,
// took 9.9 ms at 1M x 15 lists, this 0.39 ms.
constexpr int PAIR_THREADS = 256;
__global__ void __launch_bounds__(PAIR_THREADS)
    k_knn_pairs(const uint32_t* __restrict__ idx, const float* __restrict__ d2, uint64_t n, uint32_t k,
                const float* __restrict__ sigma, int sym_union, int squared, int idbits, unsigned long long* keys,
                float* w, unsigned long long* count) {
    __shared__ uint32_t s_cnt[PAIR_THREADS / 32];
    __shared__ unsigned long long s_base;
    const unsigned lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    const uint64_t total = n * (k + 1);
    for (uint64_t base = blockIdx.x * (uint64_t)PAIR_THREADS; base < total;
         base += (uint64_t)gridDim.x * PAIR_THREADS) {  // block-uniform
        const uint64_t e = base + threadIdx.x;
        bool one = false, two = false;  // the pair is emitted; its mirror too
        uint64_t i = 0;
        uint32_t j = 0;
        float wt = 0.0f;
        if (e < total) {
            i = e / (k + 1);
            j = idx[e];
            // slot 0 of a row is the point itself: not a pair
            bool ok = e != i * (k + 1) && j < n && (sym_union ? j != i : i <= j);
            if (ok) {
                // HNSW path: squares the returned distance; kd-tree path: already squared
                const float r = d2[e];
                const float dist_sq = squared ? r : __fmul_rn(sqrtf(r), sqrtf(r));
                wt = gauss_w(dist_sq, sigma[i], sigma[j], &ok);
                one = ok && wt > 1e-14f;
                two = one && i != j;
            }
        }
        const unsigned b1 = __ballot_sync(0xFFFFFFFFu, one), b2 = __ballot_sync(0xFFFFFFFFu, two);
        if (lane == 0) s_cnt[wid] = (uint32_t)(__popc(b1) + __popc(b2));
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t sum = 0;
            for (int t = 0; t < PAIR_THREADS / 32; ++t) {
                const uint32_t c = s_cnt[t];
                s_cnt[t] = sum;
                sum += c;
            }
            s_base = sum ? atomicAdd(count, (unsigned long long)sum) : 0ull;
        }
        __syncthreads();
        if (one) {
            const uint64_t pos = s_base + s_cnt[wid] + __popc(b1 & below) + __popc(b2 & below);
            keys[pos] = ((unsigned long long)i << idbits) | j;
            w[pos] = wt;
            if (two) {
                keys[pos + 1] = ((unsigned long long)j << idbits) | i;
                w[pos + 1] = wt;
            }
        }
        __syncthreads();  // s_cnt and s_base are reused
    }
}

__global__ void k_dedupe_flags(const unsigned long long* __restrict__ keys, uint64_t N, uint8_t* keep) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < N;
         i += (uint64_t)gridDim.x * blockDim.x)
        keep[i] = (i == 0 || keys[i] != keys[i - 1]);
}

__global__ void k_split_rowcol(const unsigned long long* __restrict__ keys, uint64_t N, int idbits, uint32_t* rows,
                               uint32_t* cols) {
    const unsigned long long low = (1ull << idbits) - 1ull;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < N;
         i += (uint64_t)gridDim.x * blockDim.x) {
        rows[i] = (uint32_t)(keys[i] >> idbits);
        cols[i] = (uint32_t)(keys[i] & low);
    }
}

__global__ void k_ptr_from_rows(const uint32_t* __restrict__ rows, uint64_t N, uint64_t R, uint64_t* start) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i <= N;
         i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t r = i < N ? rows[i] : R;
        uint64_t prev = i == 0 ? 0 : (uint64_t)rows[i - 1] + 1;
        for (uint64_t q = prev; q <= r && q <= R; ++q) start[q] = i;
    }
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        SC_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q));
        if (q != cudaDriverEntryPointSuccess || !p) fail(SC_E_CUDA, "cuTensorMapEncodeTiled is unavailable");
        fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
    }
    return fn;
}

// 2-D map of n rows of `row_bytes` bytes, tiles of 128 rows, swizzled by the row size.
CUtensorMap make_map(const void* base, uint64_t n, uint32_t row_bytes, bool bytes_type) {
    CUtensorMap m;
    const uint32_t esize = bytes_type ? 1 : 2;
    cuuint64_t dims[2] = {(cuuint64_t)(row_bytes / esize), (cuuint64_t)n};
    cuuint64_t strides[1] = {(cuuint64_t)row_bytes};
    cuuint32_t box[2] = {(cuuint32_t)(row_bytes / esize), (cuuint32_t)TILE};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = encode_fn()(&m, bytes_type ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                             (void*)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                             row_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) fail(SC_E_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return m;
}

// Scores are |y|^2 - 2 x.y from 16-bit operands x^, y^ with FP32 accumulation.
// A point within Y of the origin scores within a Y + b Y^2 of the exact value:
// |x.y - x^.y^| <= |x - x^| |y| + |x^| |y - y^|, with |y - y^| <= rho |y| (k_knn_prep
// measured rho and each |x - x^|), gives a; the norm's two terms and up to 64
// FP32 accumulations of terms that sum to at most 2 |x| |y| + |y|^2 stay below
// b = 2^-13. Measured residuals in place of the unit roundoff: on a mixture of
// 200k x 50 points the margin of the median query is 0.54 (f16) or 3.8 (BF16),
// from the unit roundoff of BF16 it was 6.8, at a 15th neighbour's squared
// distance of 83.
struct ScoreMargin {
    double a, b;
};
__device__ __forceinline__ ScoreMargin score_margin(double nx, double rx, const KnnScale* sc) {
    const double rho = (double)__uint_as_float(sc->rho);
    return ScoreMargin{2.0 * (rx + (nx + rx) * rho) * (1.0 + 0x1.0p-20), 0x1.0p-13};
}

// k + 1 points' squared FP32 distances against any real distance: 2^-16 covers
// the rounding of either side.
constexpr double KTH_SLACK = 1.0 + 0x1.0p-14;

__device__ __forceinline__ float up_or_inf(double v) {
    return v < INFINITY ? __double2float_ru(v) : INFINITY;  // NaN: no bound
}

// An upper bound on each query's (k+1)-th squared distance from the minima of a
// bounding scan: the (k+1)-th smallest t of the query's two ascending lists is
// the score of a point with k others at or below it. Every one of them obeys
// d^2 <= t + |x|^2 + a Y + b Y^2 with Y = |x| + d; the larger root of that
// quadratic bounds d. Query r is point q0 + r.
__global__ void k_bound_kth(const float* __restrict__ minima, uint64_t nq, uint64_t q0, uint32_t k1,
                            const float* __restrict__ nx, const float* __restrict__ rx,
                            const KnnScale* __restrict__ sc, float* __restrict__ kb) {
    const int e = f16_exp(sc);
    const double unit = e != INT32_MIN ? ldexp(1.0, -2 * e) : 1.0;  // scores in the points' units
    for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < nq; r += (uint64_t)gridDim.x * blockDim.x) {
        const float* l0 = minima + r * (HALVES * BOUND_KEEP);
        const float* l1 = l0 + BOUND_KEEP;
        uint32_t i = 0, j = 0;
        float t = INFINITY;
        for (uint32_t s = 0; s < k1; ++s) {
            const float a = i < (uint32_t)BOUND_KEEP ? l0[i] : INFINITY, b = j < (uint32_t)BOUND_KEEP ? l1[j] : INFINITY;
            if (a <= b) ++i;
            else ++j;
            t = fminf(a, b);
        }
        if (!(t < INFINITY)) {
            kb[r] = INFINITY;
            continue;
        }
        const double x = nx[q0 + r];
        const ScoreMargin m = score_margin(x, rx[q0 + r], sc);
        const double p = m.a + 2.0 * m.b * x, q = (double)t * unit + x * x + m.a * x + m.b * x * x;
        const double disc = p * p + 4.0 * (1.0 - m.b) * q;  // negative only by rounding, at distance 0
        const double dist = (p + sqrt(disc > 0.0 ? disc : 0.0)) / (2.0 * (1.0 - m.b));
        kb[r] = up_or_inf(dist * dist * KTH_SLACK);
    }
}

// The same bound where the first scan kept whole lists: their (k+1)-th FP32 distance.
__global__ void k_list_kth(const float* __restrict__ d2, const uint32_t* __restrict__ perm, uint64_t n, uint32_t k1,
                           float* __restrict__ kb) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        kb[i] = up_or_inf((double)d2[(uint64_t)perm[i] * k1 + k1 - 1] * KTH_SLACK);
}

// The score bound the last scan starts from (query r is the point ord[r], or q0
// + r without ord, and its bound kb[r] then): a point that can reach the
// query's list lies within d^2 <= kb, so it scores at most kb - |x|^2 plus the
// margin at Y = |x| + d. Rounded up, and one step more: a candidate's score must
// be below the cap also where every term is zero (k + 1 points at the origin).
__global__ void k_score_cap(const float* __restrict__ kb, uint64_t nq, uint64_t q0, const uint32_t* __restrict__ ord,
                            const float* __restrict__ nx, const float* __restrict__ rx,
                            const KnnScale* __restrict__ sc, float* __restrict__ cap) {
    const int e = f16_exp(sc);
    const double unit = e != INT32_MIN ? ldexp(1.0, 2 * e) : 1.0;
    for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < nq; r += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = ord ? ord[r] : q0 + r;
        const double d2 = kb[ord ? i : r], x = nx[i], low = x * (1.0 - 0x1.0p-15);
        const ScoreMargin m = score_margin(x, rx[i], sc);
        const double Y = x + sqrt(d2);
        cap[r] = nextafterf(up_or_inf((d2 - low * low + m.a * Y + m.b * Y * Y) * unit), INFINITY);
    }
}

// What a scan starts from (device arrays, all nullable).
struct TileLists {
    const uint32_t* rptr = nullptr;    // the pruned search's tile ranges of each query group: ngroups + 1
    const uint2* rngs = nullptr;       // (first tile, tile count)
    const float* cap = nullptr;        // per query (launch order): the score bound of k_knn_tc's qcap
    const uint32_t* gorder = nullptr;  // the groups by descending tile count
};

// Whether the 2 x BOUND_KEEP minima of a bounding scan leave room beside the
// k + 1 points they bound; otherwise a first scan keeps whole candidate lists.
bool few_bound(uint32_t k1) { return 2 * BOUND_KEEP >= (int)k1 + 8; }

// A scan of the queries' tiles: candidate ids to cand_idx, or (BOUND) score
// minima to bound.
template <int KA, bool F8, bool BOUND>
void launch_tc(Ctx& c, const CUtensorMap& ta, const CUtensorMap& tb, uint64_t n, uint64_t nq, uint32_t* cand_idx,
               float* bound, const KnnScale* scale, const TileLists& tl) {
    using L = KnnSmem<KA>;
    SC_CUDA(cudaFuncSetAttribute(k_knn_tc<KA, F8, BOUND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::BYTES));
    const uint32_t ngroups = (uint32_t)((nq + QT * TILE - 1) / (QT * TILE));
    const unsigned grid = std::min<unsigned>(ngroups, (unsigned)c.sm_count);
    k_knn_tc<KA, F8, BOUND><<<grid, KNN_THREADS, L::BYTES, c.stream>>>(
        ta, tb, (uint32_t)n, (uint32_t)nq, cand_idx, bound, c.d_status, c.wait_limit, c.knn_hold_tiles, scale, tl.rptr,
        tl.rngs, tl.cap, tl.gorder);
    SC_LAUNCH_CHECK();
    c.launches++;
}

// The contraction's operands of the points X. The query operand's tensor map
// starts at row q0 (64 or 128 bytes per row, so every row start is a legal TMA
// base) and has nq rows.
struct TcOperands {
    DBuf<uint8_t> A, B;
    DBuf<float> nx, rx;  // 16-bit: each row's norm and rounding error (k_knn_prep)
    CUtensorMap ta{}, tb{};
    int kind = 0;  // 0: 16-bit KA = 32, 1: 16-bit KA = 64, 2: e4m3
    const KnnScale* scale = nullptr;
    uint32_t row_bytes() const { return kind == 1 ? 128u : 64u; }
};

// scale: the point set's ranges (k_knn_scales has run).
void prep_operands(Ctx& c, const float* dX, uint64_t n, uint32_t d, uint64_t q0, uint64_t nq, int precision,
                   KnnScale* scale, TcOperands& op) {
    op.kind = precision == SC_KNN_FP8 ? 2 : d <= 30 ? 0 : 1;
    op.scale = scale;
    const uint64_t rb = op.row_bytes();
    op.A.alloc(c, n * rb);
    op.B.alloc(c, n * rb);
    if (op.kind == 2) {
        k_knn_prep_f8<<<grid_for(n, 256), 256, 0, c.stream>>>(dX, n, d, scale, op.A.get(), op.B.get());
    } else {
        op.nx.alloc(c, n);
        op.rx.alloc(c, n);
        uint16_t *A = (uint16_t*)op.A.get(), *B = (uint16_t*)op.B.get();
        const unsigned grid = grid_for(n * 32, 256, 148u * 8u);
        if (op.kind == 0) k_knn_prep<32><<<grid, 256, 0, c.stream>>>(dX, n, d, scale, A, B, op.nx.get(), op.rx.get());
        else k_knn_prep<64><<<grid, 256, 0, c.stream>>>(dX, n, d, scale, A, B, op.nx.get(), op.rx.get());
    }
    SC_LAUNCH_CHECK();
    c.launches++;
    op.ta = make_map(op.A.get() + q0 * rb, nq, (uint32_t)rb, op.kind == 2);
    op.tb = make_map(op.B.get(), n, (uint32_t)rb, op.kind == 2);
}

void launch_keep(Ctx& c, const TcOperands& op, uint64_t n, uint64_t nq, uint32_t* cidx, const TileLists& tl) {
    if (op.kind == 2) launch_tc<32, true, false>(c, op.ta, op.tb, n, nq, cidx, nullptr, op.scale, tl);
    else if (op.kind == 0) launch_tc<32, false, false>(c, op.ta, op.tb, n, nq, cidx, nullptr, op.scale, tl);
    else launch_tc<64, false, false>(c, op.ta, op.tb, n, nq, cidx, nullptr, op.scale, tl);
}

// Bounds every query's (k+1)-th squared distance (kb, query order) by a scan of
// 16-bit scores. minima: 2 x BOUND_KEEP words per query.
void launch_bound(Ctx& c, const TcOperands& op, uint64_t n, uint64_t q0, uint64_t nq, uint32_t k1, float* minima,
                  const TileLists& tl, float* kb) {
    if (op.kind == 0) launch_tc<32, false, true>(c, op.ta, op.tb, n, nq, nullptr, minima, op.scale, tl);
    else launch_tc<64, false, true>(c, op.ta, op.tb, n, nq, nullptr, minima, op.scale, tl);
    k_bound_kth<<<grid_for(nq, 256), 256, 0, c.stream>>>(minima, nq, q0, k1, op.nx.get(), op.rx.get(), op.scale, kb);
    SC_LAUNCH_CHECK();
    c.launches++;
}

// Candidates of the queries q0 .. q0 + nq - 1 against all n points. 16-bit
// operands take two scans, as the pruned search does: the first bounds each
// query's (k+1)-th distance, the second starts from that bound, so its rows
// hold some twenty candidates instead of taking 32 (1 + ln(n / 64)) one after
// another. One scan from +inf took 1.33 ms at 5,003 x 30 points, the two take
// 0.15 ms. One scan for lists too long for the bounding scan's minima (k > 23)
// and for e4m3, whose scores are too coarse for a useful bound.
void candidates(Ctx& c, const float* dX, uint64_t n, uint32_t d, uint32_t k, uint64_t q0, uint64_t nq, int precision,
                uint32_t* cand_idx) {
    DBuf<KnnScale> scale(c, 1);
    zero(c, scale.get(), 1);
    k_knn_scales<<<grid_for(n, 256), 256, 0, c.stream>>>(dX, n, d, scale.get());
    SC_LAUNCH_CHECK();
    c.launches++;
    TcOperands op;
    prep_operands(c, dX, n, d, q0, nq, precision, scale.get(), op);
    TileLists tl;
    DBuf<float> kb, cap;
    if (op.kind != 2 && few_bound(k + 1)) {
        kb.alloc(c, nq);
        cap.alloc(c, nq);
        launch_bound(c, op, n, q0, nq, k + 1, (float*)cand_idx, tl, kb.get());
        k_score_cap<<<grid_for(nq, 256), 256, 0, c.stream>>>(kb.get(), nq, q0, nullptr, op.nx.get(), op.rx.get(),
                                                             op.scale, cap.get());
        SC_LAUNCH_CHECK();
        c.launches++;
        tl.cap = cap.get();
    }
    launch_keep(c, op, n, nq, cand_idx, tl);
}

// ------------------------------------------------------------ exact pruning
// Points are grouped by a deterministic k-means (fixed-point sums, ties to the
// lower centroid) and sorted by group, so every 128-row tile is spatially
// coherent. A query group first scans the tiles of its own clusters; the k + 1
// smallest score minima bound each query's (k+1)-th distance from above
// (k_bound_kth). A cluster b can hold a closer point only if a lower bound on
// |q - x| over x in b is at most that distance: the ball bound |q - c_b| - r_b
// and the slab bound of the direction u from the query's cluster centre to
// c_b (every x in b projects into [lo, hi] on u, so |q - x| >= the distance
// from <q, u> to [lo, hi]). The second pass scans the own tiles and those of
// every cluster some query of the group cannot exclude, narrowed to the fine
// cells (~256 points) a ball bound cannot exclude; skipped points are provably
// farther than the query's (k+1)-th neighbour, so the result is the full
// search's. The first pass keeps score minima alone (it only yields the bound)
// and walks each group's nearest cells first; the second starts every query's
// candidate rows from a proven score bound derived from the first pass's
// bound (k_score_cap). Both passes take their tile lists from the device.
constexpr int KM_ITERS = 8;
constexpr uint32_t KM_SAMPLE = 65536;  // points the Lloyd steps run on

// Nearest centroid of every point (squared FP32 distance, ties to the lower id).
__global__ void k_km_assign(const float* __restrict__ X, uint64_t n, uint32_t d, const float* __restrict__ cent,
                            uint32_t K, uint32_t* assign) {
    // centroid rows padded to a multiple of 4 floats, read as float4
    extern __shared__ __align__(16) float s_cent[];
    const uint32_t dp = (d + 3) & ~3u;
    for (uint32_t i = threadIdx.x; i < K * dp; i += blockDim.x) {
        const uint32_t c = i / dp, j = i % dp;
        s_cent[i] = j < d ? cent[(uint64_t)c * d + j] : 0.0f;
    }
    __syncthreads();
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        // the point in registers (d <= 62): the centroid loop then reads only
        // shared memory, every lane the same words (a broadcast)
        float x[64];
#pragma unroll
        for (int j = 0; j < 64; ++j) x[j] = (uint32_t)j < d ? X[i * d + j] : 0.0f;
        float best = INFINITY;
        uint32_t bc = 0;
        for (uint32_t c = 0; c < K; ++c) {
            const float4* m4 = reinterpret_cast<const float4*>(s_cent + (uint64_t)c * dp);
            float acc = 0.0f;
#pragma unroll
            for (int q = 0; q < 16; ++q)
                if ((uint32_t)(4 * q) < d) {
                    const float4 mv = m4[q];
                    const float mm[4] = {mv.x, mv.y, mv.z, mv.w};
#pragma unroll
                    for (int t = 0; t < 4; ++t)
                        if ((uint32_t)(4 * q + t) < d) {
                            const float df = __fsub_rn(x[4 * q + t], mm[t]);
                            acc = __fmaf_rn(df, df, acc);
                        }
                }
            if (acc < best) {
                best = acc;
                bc = c;
            }
        }
        assign[i] = bc;
    }
}

// Per-cluster coordinate sums in fixed point (x * 2^s rounded; integer adds are
// associative, so the centroids do not depend on the order) and counts. A warp
// per point, a lane per coordinate, four points' loads in flight: with a point a
// lane the lanes of one cluster (most of a warp's, with few clusters) added to the
// same word one after another, 92 us a step for 65,536 x 50 points in 24 clusters;
// 27 now.
__global__ void __launch_bounds__(256) k_km_accum(const float* __restrict__ X, uint64_t n, uint32_t d,
                                                  const uint32_t* __restrict__ assign, uint32_t K, double scale,
                                                  unsigned long long* sum, unsigned* cnt) {
    extern __shared__ unsigned long long s_sum[];
    unsigned* s_cnt = (unsigned*)(s_sum + K * d);
    for (uint32_t i = threadIdx.x; i < K * d; i += blockDim.x) s_sum[i] = 0;
    for (uint32_t i = threadIdx.x; i < K; i += blockDim.x) s_cnt[i] = 0;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t i0 = warp; i0 < n; i0 += 4 * nwarps) {  // warp-uniform
        uint32_t c[4];
        float x[4][2];  // d <= 62
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const uint64_t i = i0 + t * nwarps;
            c[t] = i < n ? assign[i] : 0u;
#pragma unroll
            for (int h = 0; h < 2; ++h) x[t][h] = i < n && lane + 32 * h < d ? X[i * d + lane + 32 * h] : 0.0f;
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            if (i0 + t * nwarps >= n) break;
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (lane + 32 * h < d)
                    atomicAdd(s_sum + c[t] * d + lane + 32 * h,
                              (unsigned long long)__double2ll_rn((double)x[t][h] * scale));
            if (lane == 0) atomicAdd(s_cnt + c[t], 1u);
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < K * d; i += blockDim.x)
        if (s_sum[i]) atomicAdd(sum + i, s_sum[i]);
    for (uint32_t i = threadIdx.x; i < K; i += blockDim.x)
        if (s_cnt[i]) atomicAdd(cnt + i, s_cnt[i]);
}

// Farthest-point seeding, step t >= 1: centre t - 1 is the sample point that key
// t - 1 names (step 1: the first point); d2min[i] = min(d2min[i], |x_i - c|^2);
// key t receives the point farthest from every centre chosen so far (ties to the
// lower index), so separated groups of points each get a centre before any group
// gets a second. A key is the distance's bits (non-negative floats order like
// them) over the complement of the index, so one atomicMax per block finds it:
// a second launch of one block for the search took 16 of a step's 23 us, 2.8 ms
// for 121 centres; a step takes 7.3 us now. One more step (update == 0) only
// writes the last centre.
__global__ void __launch_bounds__(256) k_seed_step(const float* __restrict__ Xs, uint64_t n, uint32_t d, uint32_t t,
                                                   int update, float* d2min, unsigned long long* keys,
                                                   float* __restrict__ cent) {
    __shared__ float s_c[64];
    __shared__ unsigned long long s_key[8];
    const uint32_t pick = t == 1 ? 0u : ~(uint32_t)keys[t - 1];
    for (uint32_t j = threadIdx.x; j < d; j += blockDim.x) {
        const float v = Xs[(uint64_t)pick * d + j];
        s_c[j] = v;
        if (blockIdx.x == 0) cent[(uint64_t)(t - 1) * d + j] = v;
    }
    if (!update) return;
    __syncthreads();
    unsigned long long key = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        float acc = 0.0f;
        for (uint32_t j = 0; j < d; ++j) {
            const float df = __fsub_rn(Xs[i * d + j], s_c[j]);
            acc = __fmaf_rn(df, df, acc);
        }
        const float m = fminf(d2min[i], acc);
        d2min[i] = m;
        const unsigned long long k = ((unsigned long long)__float_as_uint(m) << 32) | (uint32_t)~(uint32_t)i;
        key = k > key ? k : key;
    }
    for (int o = 16; o; o >>= 1) {
        const unsigned long long k = __shfl_xor_sync(0xFFFFFFFFu, key, o);
        key = k > key ? k : key;
    }
    if ((threadIdx.x & 31) == 0) s_key[threadIdx.x >> 5] = key;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (uint32_t w = 1; w < (blockDim.x >> 5); ++w) key = s_key[w] > key ? s_key[w] : key;
        atomicMax(keys + t, key);
    }
}

// New centroids; an empty cluster keeps its centroid.
__global__ void k_km_update(const unsigned long long* __restrict__ sum, const unsigned* __restrict__ cnt, uint32_t K,
                            uint32_t d, double inv_scale, float* cent) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < K * d; i += gridDim.x * blockDim.x) {
        const uint32_t c = i / d;
        if (cnt[c]) cent[i] = (float)((double)(long long)sum[i] * inv_scale / (double)cnt[c]);
    }
}

__global__ void k_gather_rows(const float* __restrict__ X, const uint32_t* __restrict__ rows, uint64_t m, uint32_t d,
                              float* out) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m * d; i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = X[(uint64_t)rows[i / d] * d + i % d];
}

__global__ void k_iota_u32(uint32_t* x, uint64_t n) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        x[i] = (uint32_t)i;
}

// Order-preserving map of floats to unsigned integers (for atomic min / max).
__device__ __forceinline__ unsigned ord32(float x) {
    const unsigned b = __float_as_uint(x);
    return (b >> 31) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float unord32(unsigned k) {
    return __uint_as_float((k >> 31) ? (k & 0x7FFFFFFFu) : ~k);
}

// Fine cell of every point inside its coarse cluster (points sorted by coarse
// cluster): the nearest of the cluster's fine centres, its points at local
// positions 0, FINE, 2 FINE, ... (ties to the lower cell). Sorting by fine cell
// then makes each group of 256 consecutive queries one spatially tight cell,
// so its queries need similar clusters.
constexpr uint32_t FINE = 256;

// |x - m|^2 of a point in registers (zeros past d) and a row of row_pad(d) floats
// that starts on 16 bytes (zeros past d: those terms add +0), summed in
// ascending order. 8 values are on their way at once: read one or four at a
// time, the loads (the same address for every thread of a warp) set the pace of
// the kernels below (fine cells of 1M x 50: 2.3 ms with one, 2.0 with four, 1.4
// now).
__host__ __device__ __forceinline__ uint32_t row_pad(uint32_t d) { return (d + 7) & ~7u; }
__device__ __forceinline__ float sq_dist_padded(const float (&x)[64], const float* __restrict__ m, uint32_t d) {
    const float4* m4 = reinterpret_cast<const float4*>(m);
    float acc = 0.0f;
#pragma unroll
    for (int j = 0; j < 64; j += 8)
        if ((uint32_t)j < d) {
            float4 v[2];
#pragma unroll
            for (int t = 0; t < 2; ++t) v[t] = m4[j / 4 + t];
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                float df = __fsub_rn(x[j + 4 * t], v[t].x);
                acc = __fmaf_rn(df, df, acc);
                df = __fsub_rn(x[j + 4 * t + 1], v[t].y);
                acc = __fmaf_rn(df, df, acc);
                df = __fsub_rn(x[j + 4 * t + 2], v[t].z);
                acc = __fmaf_rn(df, df, acc);
                df = __fsub_rn(x[j + 4 * t + 3], v[t].w);
                acc = __fmaf_rn(df, df, acc);
            }
        }
    return acc;
}

// rows[i] of src (rows of d floats) as row i of dst (rows of dp, zeros past d).
__global__ void k_gather_rows_padded(const float* __restrict__ src, const uint32_t* __restrict__ rows, uint64_t n,
                                     uint32_t d, uint32_t dp, float* dst) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n * dp; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t j = (uint32_t)(i % dp);
        dst[i] = j < d ? src[(uint64_t)rows[i / dp] * d + j] : 0.0f;
    }
}

__global__ void k_fine_assign(const float* __restrict__ Xs, uint64_t n, uint32_t d, const uint32_t* __restrict__ cl,
                              const float* __restrict__ fcent, uint32_t dp, const uint32_t* __restrict__ fbase,
                              uint32_t* fine) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t b = cl[i];
        const uint32_t f0 = fbase[b], f1 = fbase[b + 1];
        float x[64];  // the point in registers (d <= 62), zeros past d
#pragma unroll
        for (int j = 0; j < 64; ++j) x[j] = (uint32_t)j < d ? Xs[i * d + j] : 0.0f;
        float best = INFINITY;
        uint32_t bf = f0;
        for (uint32_t f = f0; f < f1; ++f) {
            const float acc = sq_dist_padded(x, fcent + (uint64_t)f * dp, d);
            if (acc < best) {
                best = acc;
                bf = f;
            }
        }
        fine[i] = bf;
    }
}

// start[q] = the first of the sorted points whose cluster is q or more, q = 0 .. K.
__global__ void k_cluster_starts(const uint32_t* __restrict__ cl, uint64_t n, uint32_t K, uint64_t* start) {
    for (uint32_t q = threadIdx.x; q <= K; q += blockDim.x) {
        uint64_t lo = 0, hi = n;
        while (lo < hi) {
            const uint64_t mid = (lo + hi) >> 1;
            if (cl[mid] < q) lo = mid + 1;
            else hi = mid;
        }
        start[q] = lo;
    }
}

// Unit vectors between the centres, a thread per (a, b): Ua[a][b] = Ub[b][a] =
// (c_b - c_a) / |c_b - c_a| in rows of dp floats (zeros past d, and for a zero
// direction, which bounds nothing).
__global__ void k_directions(const float* __restrict__ cent, uint32_t K, uint32_t d, uint32_t dp, float* Ua,
                             float* Ub) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < K * K; i += gridDim.x * blockDim.x) {
        const uint32_t a = i / K, b = i % K;
        double nrm = 0.0;
        for (uint32_t j = 0; j < d; ++j) {
            const double t = (double)cent[(uint64_t)b * d + j] - (double)cent[(uint64_t)a * d + j];
            nrm += t * t;
        }
        nrm = sqrt(nrm);
        for (uint32_t j = 0; j < dp; ++j) {
            float u = 0.0f;
            if (j < d && nrm != 0.0)
                u = (float)(((double)cent[(uint64_t)b * d + j] - (double)cent[(uint64_t)a * d + j]) / nrm);
            Ua[((uint64_t)a * K + b) * dp + j] = u;
            Ub[((uint64_t)b * K + a) * dp + j] = u;
        }
    }
}

// A chunk of consecutive sorted points of one cluster (blocks of the extent
// and bound kernels).
struct Chunk {
    uint32_t cluster;
    uint64_t begin, end;
};

// Per chunk (one block): the radius of its cluster around the centre, and the
// extent [lo, hi] of its points along every direction u_{a,b} from a centre a
// to its own centre b. Ub[b][a][j] (FP32) is staged in shared memory; warps
// reduce by shuffles, the block in shared memory, and one thread per direction
// updates the global extents (order-preserving integer min / max).
__global__ void k_cluster_extent(const float* __restrict__ Xs, uint32_t d, const Chunk* __restrict__ chunks,
                                 const float* __restrict__ cent, const float* __restrict__ Ub, uint32_t K,
                                 unsigned* rad, unsigned* lo, unsigned* hi) {
    extern __shared__ __align__(16) float sm[];
    const uint32_t dp = (d + 3) & ~3u;
    float* su = sm;                                    // K * dp
    unsigned* slo = (unsigned*)(su + (size_t)K * dp);  // K
    unsigned* shi = slo + K;                          // K
    __shared__ unsigned srad;
    const Chunk ch = chunks[blockIdx.x];
    const uint32_t b = ch.cluster;
    for (uint32_t i = threadIdx.x; i < K * dp; i += blockDim.x) su[i] = Ub[(uint64_t)b * K * dp + i];
    for (uint32_t i = threadIdx.x; i < K; i += blockDim.x) {
        slo[i] = 0xFFFFFFFFu;
        shi[i] = 0u;
    }
    if (threadIdx.x == 0) srad = 0u;
    __syncthreads();
    const unsigned FULL = 0xFFFFFFFFu;
    for (uint64_t base = ch.begin; base < ch.end; base += blockDim.x) {
        const uint64_t i = base + threadIdx.x;
        const uint64_t ii = i < ch.end ? i : ch.end - 1;  // idle lanes repeat a point: min / max unchanged
        float x[64];
#pragma unroll
        for (int j = 0; j < 64; ++j) x[j] = (uint32_t)j < d ? Xs[ii * d + j] : 0.0f;
        float r2 = 0.0f;
#pragma unroll
        for (int j = 0; j < 64; ++j)
            if ((uint32_t)j < d) {
                const float df = x[j] - cent[b * d + j];
                r2 = __fmaf_rn(df, df, r2);
            }
        unsigned kr = ord32(sqrtf(r2));
        for (int o = 16; o; o >>= 1) kr = max(kr, __shfl_xor_sync(FULL, kr, o));
        if ((threadIdx.x & 31) == 0) atomicMax(&srad, kr);
        for (uint32_t a = 0; a < K; ++a) {
            const float4* u4 = reinterpret_cast<const float4*>(su + (size_t)a * dp);
            float p = 0.0f;  // terms past d are +0: the same sum
#pragma unroll
            for (int j = 0; j < 16; ++j)
                if ((uint32_t)(4 * j) < d) {
                    const float4 u = u4[j];
                    p = __fmaf_rn(x[4 * j], u.x, p);
                    p = __fmaf_rn(x[4 * j + 1], u.y, p);
                    p = __fmaf_rn(x[4 * j + 2], u.z, p);
                    p = __fmaf_rn(x[4 * j + 3], u.w, p);
                }
            unsigned kl = ord32(p), kh = kl;
            for (int o = 16; o; o >>= 1) {
                kl = min(kl, __shfl_xor_sync(FULL, kl, o));
                kh = max(kh, __shfl_xor_sync(FULL, kh, o));
            }
            if ((threadIdx.x & 31) == 0) {
                atomicMin(slo + a, kl);
                atomicMax(shi + a, kh);
            }
        }
    }
    __syncthreads();
    for (uint32_t a = threadIdx.x; a < K; a += blockDim.x) {
        atomicMin(lo + (uint64_t)a * K + b, slo[a]);
        atomicMax(hi + (uint64_t)a * K + b, shi[a]);
    }
    if (threadIdx.x == 0) atomicMax(rad + b, srad);
}

// For every sorted query (chunks of its own cluster a, one block each): the
// clusters whose lower bound does not exclude them given its current (k+1)-th
// distance, as the bits of its own mask (words 64-bit words per query). FP32 with margins: `eps` bounds the
// rounding of a projection or a distance (a few ulps of the largest |x| times
// d), so every bound used is below the exact one.
__global__ void k_cluster_needs(const float* __restrict__ Xs, uint32_t d, const Chunk* __restrict__ chunks,
                                const float* __restrict__ kb, const float* __restrict__ cent,
                                const unsigned* __restrict__ rad,
                                const float* __restrict__ Ua, const unsigned* __restrict__ lo,
                                const unsigned* __restrict__ hi, uint32_t K, float eps, uint32_t words,
                                unsigned long long* mask) {
    extern __shared__ __align__(16) float sm[];
    // rows of dp floats, read as float4: one load feeds eight operations (one
    // float at a time the loads set the pace: 3.9 ms at 1M x 50, 1.65 now)
    const uint32_t dp = (d + 3) & ~3u;
    float* su = sm;                        // K * dp: directions from a to every b
    float* sc = su + (size_t)K * dp;       // K * dp: centres
    float* sr = sc + (size_t)K * dp;       // K: radii
    float* sl = sr + K;                    // K: lo[a][b]
    float* sh = sl + K;                    // K: hi[a][b]
    const Chunk ch = chunks[blockIdx.x];
    const uint32_t a = ch.cluster;
    for (uint32_t i = threadIdx.x; i < K * dp; i += blockDim.x) {
        su[i] = Ua[(uint64_t)a * K * dp + i];
        sc[i] = i % dp < d ? cent[(uint64_t)(i / dp) * d + i % dp] : 0.0f;
    }
    for (uint32_t b = threadIdx.x; b < K; b += blockDim.x) {
        sr[b] = unord32(rad[b]);
        sl[b] = unord32(lo[(uint64_t)a * K + b]);
        sh[b] = unord32(hi[(uint64_t)a * K + b]);
    }
    __syncthreads();
    for (uint64_t base = ch.begin; base < ch.end; base += blockDim.x) {
        const uint64_t i = base + threadIdx.x;
        const bool ok = i < ch.end;
        const uint64_t ii = ok ? i : ch.end - 1;
        float x[64];
#pragma unroll
        for (int j = 0; j < 64; ++j) x[j] = (uint32_t)j < d ? Xs[ii * d + j] : 0.0f;
        const float kd2 = kb[ii];
        // no (k+1)-th neighbour among the own clusters: every cluster is needed
        const float kth = isfinite(kd2) ? sqrtf(kd2) * (1.0f + 1e-5f) + eps : INFINITY;
        unsigned long long m[4] = {0ull, 0ull, 0ull, 0ull};
        for (uint32_t b = 0; b < K; ++b) {
            bool need = false;
            if (b != a) {
                const float4* m4 = reinterpret_cast<const float4*>(sc + (size_t)b * dp);
                const float4* u4 = reinterpret_cast<const float4*>(su + (size_t)b * dp);
                float dc = 0.0f, p = 0.0f;  // terms past d are +0: the same sums
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    if ((uint32_t)(4 * j) < d) {
                        const float4 m = m4[j], u = u4[j];
                        float df = x[4 * j] - m.x;
                        dc = __fmaf_rn(df, df, dc);
                        p = __fmaf_rn(x[4 * j], u.x, p);
                        df = x[4 * j + 1] - m.y;
                        dc = __fmaf_rn(df, df, dc);
                        p = __fmaf_rn(x[4 * j + 1], u.y, p);
                        df = x[4 * j + 2] - m.z;
                        dc = __fmaf_rn(df, df, dc);
                        p = __fmaf_rn(x[4 * j + 2], u.z, p);
                        df = x[4 * j + 3] - m.w;
                        dc = __fmaf_rn(df, df, dc);
                        p = __fmaf_rn(x[4 * j + 3], u.w, p);
                    }
                const float ball = sqrtf(dc) * (1.0f - 1e-5f) - sr[b] - eps;
                const float slab = fmaxf(sl[b] - p, p - sh[b]) - 2.0f * eps;
                need = fmaxf(ball, slab) <= kth;
            }
            if (need) m[b / 64] |= 1ull << (b % 64);
        }
        if (ok)
            for (uint32_t w = 0; w < words; ++w) mask[ii * words + w] = m[w];
    }
}

// Pass-2 order of the queries: by own cluster, then by a hash of the set of
// clusters the query needs, so each group of 256 holds queries needing the
// same clusters and the union a group scans stays close to what one needs.
__global__ void k_need_keys(const unsigned long long* __restrict__ mask, const uint32_t* __restrict__ cl, uint64_t n,
                            uint32_t words, unsigned long long* keys, uint32_t* pos) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t h = 0x2545F4914F6CDD1Dull;
        for (uint32_t w = 0; w < words; ++w) h = splitmix(h ^ mask[i * words + w]);
        keys[i] = ((unsigned long long)cl[i] << 32) | (h >> 32);
        pos[i] = (uint32_t)i;
    }
}

// Rows of an operand (row_bytes, a multiple of 16) gathered in the order `ord`.
__global__ void k_gather_operand_rows(const uint4* __restrict__ src, const uint32_t* __restrict__ ord, uint64_t n,
                                      uint32_t row_vec, uint4* dst) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n * row_vec;
         i += (uint64_t)gridDim.x * blockDim.x)
        dst[i] = src[(uint64_t)ord[i / row_vec] * row_vec + i % row_vec];
}

// Per pass-2 group (one warp): the OR of its queries' masks, and the clusters
// of its first and last query (the group's own clusters lie between them).
__global__ void k_group_needs(const unsigned long long* __restrict__ mask, const uint32_t* __restrict__ ord,
                              const uint32_t* __restrict__ cl, uint64_t n, uint32_t words, uint64_t ngroups,
                              unsigned long long* gmask, uint32_t* gown) {
    const unsigned lane = threadIdx.x & 31u;
    const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t g = warp; g < ngroups; g += nwarps) {
        const uint64_t b = g * (QT * TILE), e = min(n, b + QT * TILE);
        for (uint32_t w = 0; w < words; ++w) {
            unsigned long long acc = 0ull;
            for (uint64_t i = b + lane; i < e; i += 32) acc |= mask[(uint64_t)ord[i] * words + w];
            for (int o = 16; o; o >>= 1) acc |= __shfl_xor_sync(0xFFFFFFFFu, acc, o);
            if (lane == 0) gmask[g * words + w] = acc;
        }
        if (lane == 0) {
            gown[2 * g] = cl[ord[b]];
            gown[2 * g + 1] = cl[ord[e - 1]];
        }
    }
}

// Points per fine cell (cells numbered in sorted order: a cell's points are
// contiguous) and the radius of every cell around its centre (the sample
// point that defined it).
__global__ void k_cell_count(const uint32_t* __restrict__ cell, uint64_t n, unsigned* cnt) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        atomicAdd(cnt + cell[i], 1u);
}

__global__ void k_cell_radius(const float* __restrict__ Xs, uint64_t n, uint32_t d, const uint32_t* __restrict__ cell,
                              const float* __restrict__ fcent, uint32_t dp, unsigned* crad) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t f = cell[i];
        float r2 = 0.0f;
        for (uint32_t j = 0; j < d; ++j) {
            const float df = Xs[i * d + j] - fcent[(uint64_t)f * dp + j];
            r2 = __fmaf_rn(df, df, r2);
        }
        atomicMax(crad + f, ord32(sqrtf(r2)));
    }
}

// Per pass-2 group (one block, a thread per query): the fine cells of the
// group's candidate clusters (its own clusters and every cluster one of its
// queries needs) that the ball bound |q - c_f| - r_f cannot exclude for at
// least one query, as bits of the group's cell bitmap. The group's queries
// are neighbours in the sorted order (one or a few fine cells), so a ball
// around them (centre: their mean, radius: the farthest of them) first
// excludes, for all queries at once, every cell with
// |g - c_f| - r_g - r_f > max kth; only the remaining cells are tested per
// query. Both tests carry the same rounding margins, the group test twice.
// Bound by the instructions of the tests: 8.3 ms at 1M x 50 with every warp
// testing every kept cell, a block per cluster in the first test and one float
// a load; 4.4 with a warp per cluster there, warps that start at different
// cells and skip the settled ones, and float4 rows; 4.1 with two of them a step.
// Stopping at a partial sum that excludes the cell for the whole warp made it
// slower (5.8): the cells the group ball keeps are mostly near.
__global__ void k_group_cells(const float* __restrict__ Xs, uint64_t n, uint32_t d, const uint32_t* __restrict__ ord,
                              const float* __restrict__ kb, const unsigned long long* __restrict__ gmask,
                              const uint32_t* __restrict__ gown,
                              uint32_t words, uint32_t K, const uint32_t* __restrict__ fbase,
                              const float* __restrict__ fcent, const unsigned* __restrict__ crad, float eps,
                              uint32_t cwords, const unsigned long long* __restrict__ qmask,
                              const uint32_t* __restrict__ qcl, unsigned* gcell) {
    const uint64_t g = blockIdx.x;
    const uint64_t r = g * (QT * TILE) + threadIdx.x;
    const bool ok = r < n;
    const uint64_t sq = ok ? ord[r] : ord[n - 1];
    const uint32_t dp = row_pad(d);
    float x[64];
#pragma unroll
    for (int j = 0; j < 64; ++j) x[j] = (uint32_t)j < d ? Xs[sq * d + j] : 0.0f;
    const float kd2 = kb[sq];
    const float kth = isfinite(kd2) ? sqrtf(kd2) * (1.0f + 1e-5f) + eps : INFINITY;
    extern __shared__ unsigned s_bits[];  // cwords: the result, then cwords: cells the group ball keeps
    unsigned* s_maybe = s_bits + cwords;
    __shared__ float s_c[64];
    __shared__ unsigned s_r, s_k;  // group radius and max kth (ordered bits)
    for (uint32_t w = threadIdx.x; w < cwords; w += blockDim.x) s_bits[w] = s_maybe[w] = 0u;
    for (uint32_t j = threadIdx.x; j < 64; j += blockDim.x) s_c[j] = 0.0f;
    if (threadIdx.x == 0) s_r = s_k = 0u;
    __syncthreads();
    // group centre: the mean of its queries, summed in a fixed order (a warp
    // per dimension, lanes over the queries, a fixed tree)
    const uint64_t g0 = g * (QT * TILE), gcount = n - g0 < (uint64_t)(QT * TILE) ? n - g0 : (uint64_t)(QT * TILE);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (uint32_t j = wid; j < d; j += nw) {
        float acc = 0.0f;
        for (uint64_t t = lane; t < gcount; t += 32) acc += Xs[(uint64_t)ord[g0 + t] * d + j];
        for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
        if (lane == 0) s_c[j] = acc / (float)gcount;
    }
    __syncthreads();
    if (ok) {
        float dq = 0.0f;
#pragma unroll
        for (int j = 0; j < 64; ++j)
            if ((uint32_t)j < d) {
                const float df = x[j] - s_c[j];
                dq = __fmaf_rn(df, df, dq);
            }
        atomicMax(&s_r, ord32(sqrtf(dq)));
        atomicMax(&s_k, ord32(kth));
    }
    __syncthreads();
    const float rg = unord32(s_r) * (1.0f + 1e-5f), kmax = unord32(s_k);
    const uint32_t a0 = gown[2 * g], a1 = gown[2 * g + 1];
    // the group-ball test: a warp per candidate cluster, a lane per cell (a
    // cluster holds some tens of cells)
    for (uint32_t b = wid; b < K; b += nw) {
        const bool cand = (b >= a0 && b <= a1) || ((gmask[g * words + b / 64] >> (b % 64)) & 1ull);
        if (!cand) continue;  // uniform over the warp
        for (uint32_t f = fbase[b] + lane; f < fbase[b + 1]; f += 32) {
            const float4* m4 = reinterpret_cast<const float4*>(fcent + (uint64_t)f * dp);
            float dc = 0.0f;
            for (uint32_t j = 0; j < dp; j += 4) {
                const float4 v = m4[j / 4];
                float df = s_c[j] - v.x;
                dc = __fmaf_rn(df, df, dc);
                df = s_c[j + 1] - v.y;
                dc = __fmaf_rn(df, df, dc);
                df = s_c[j + 2] - v.z;
                dc = __fmaf_rn(df, df, dc);
                df = s_c[j + 3] - v.w;
                dc = __fmaf_rn(df, df, dc);
            }
            if (!(sqrtf(dc) * (1.0f - 1e-5f) - rg - unord32(crad[f]) - 2.0f * eps > kmax))
                atomicOr(s_maybe + f / 32, 1u << (f % 32));
        }
    }
    __syncthreads();
    // the per-query test on the cells the group ball kept, for the queries
    // whose own cluster or needs hold the cell's cluster (the group scans the
    // union of its queries' needs; each query tests only its own). One query
    // that needs a cell settles it for the group, so the warps start at
    // different words and pass over the cells that another has already set.
    const uint32_t myown = qcl[sq];
    const unsigned long long* mym = qmask + sq * words;
    const volatile unsigned* v_bits = s_bits;
    const uint32_t rot = wid * cwords / nw;
    for (uint32_t base = 0; base < cwords; base += 32) {
        const uint32_t at = (rot + base + lane) % cwords;
        const unsigned kept = base + lane < cwords ? s_maybe[at] : 0u;
        unsigned left = __ballot_sync(0xFFFFFFFFu, kept != 0u);
        while (left) {
            const int l = __ffs(left) - 1;
            left &= left - 1;
            unsigned bits = __shfl_sync(0xFFFFFFFFu, kept, l);
            const uint32_t wd = (rot + base + l) % cwords;
            uint32_t b = 0;  // the cluster of the word's first cell (cells ascend, so does b)
            for (uint32_t hi = K, f = wd * 32 + (uint32_t)(__ffs(bits) - 1); hi - b > 1;) {
                const uint32_t mid = (b + hi) >> 1;
                if (fbase[mid] <= f) b = mid;
                else hi = mid;
            }
            while (bits) {
                const uint32_t bit = (uint32_t)(__ffs(bits) - 1), f = wd * 32 + bit;
                bits &= bits - 1;
                while (fbase[b + 1] <= f) ++b;
                const bool mine = ok && !((v_bits[wd] >> bit) & 1u) &&
                                  (b == myown || ((mym[b / 64] >> (b % 64)) & 1ull));
                if (!__any_sync(0xFFFFFFFFu, mine)) continue;
                const float dc = sq_dist_padded(x, fcent + (uint64_t)f * dp, d);
                const bool need = mine && sqrtf(dc) * (1.0f - 1e-5f) - unord32(crad[f]) - eps <= kth;
                // one shared OR per warp that needs the cell
                if (__ballot_sync(0xFFFFFFFFu, need) && lane == 0) atomicOr(s_bits + wd, 1u << bit);
            }
        }
    }
    __syncthreads();
    for (uint32_t w = threadIdx.x; w < cwords; w += blockDim.x) gcell[g * cwords + w] = s_bits[w];
}

// Pass 1's tile order, a block per query group: the group's own-cluster tiles
// [tb[g], te[g]) sorted by the distance from the group's centre (the mean of
// its queries) to the centroid of the cell holding each tile's first point,
// nearest first, ties by tile id; each tile one range of length 1 at
// out[rptr[g] ..]. Nearest points first tighten the rows' thresholds within
// the first tiles. More tiles than ORDER_CAP keep ascending order from the
// group's own tile.
constexpr int ORDER_CAP = 2048;
__global__ void k_order_tiles(const float* __restrict__ Xs, uint64_t n, uint32_t d, const uint32_t* __restrict__ tb,
                              const uint32_t* __restrict__ te, const uint32_t* __restrict__ tile_cell,
                              const float* __restrict__ fcent, const uint32_t* __restrict__ rptr, uint2* out) {
    __shared__ float s_c[64];
    __shared__ float s_key[ORDER_CAP];
    __shared__ uint32_t s_tile[ORDER_CAP];
    const uint64_t g = blockIdx.x;
    const uint64_t g0 = g * (QT * TILE), gcount = n - g0 < (uint64_t)(QT * TILE) ? n - g0 : (uint64_t)(QT * TILE);
    const uint32_t t0 = tb[g], t1 = te[g], cnt = t1 - t0;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (cnt > (uint32_t)ORDER_CAP) {  // ascending from the group's own tile, wrapping round
        const uint32_t own = (uint32_t)(g0 / TILE);
        const uint32_t first = own >= t0 && own < t1 ? own : t0;
        for (uint32_t k = threadIdx.x; k < cnt; k += blockDim.x) {
            uint32_t t = first + k;
            if (t >= t1) t -= cnt;
            out[rptr[g] + k] = make_uint2(t, 1u);
        }
        return;
    }
    for (uint32_t j = wid; j < d; j += nw) {
        float acc = 0.0f;
        for (uint64_t t = lane; t < gcount; t += 32) acc += Xs[(g0 + t) * d + j];
        for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
        if (lane == 0) s_c[j] = acc / (float)gcount;
    }
    __syncthreads();
    uint32_t P = 1;
    while (P < cnt) P <<= 1;
    for (uint32_t k = threadIdx.x; k < P; k += blockDim.x) {
        float key = INFINITY;
        uint32_t t = 0xFFFFFFFFu;
        if (k < cnt) {
            t = t0 + k;
            const float* m = fcent + (uint64_t)tile_cell[t] * row_pad(d);
            key = 0.0f;
            for (uint32_t j = 0; j < d; ++j) {
                const float df = s_c[j] - m[j];
                key = __fmaf_rn(df, df, key);
            }
        }
        s_key[k] = key;
        s_tile[k] = t;
    }
    __syncthreads();
    // bitonic sort of (key, tile) ascending
    for (uint32_t size = 2; size <= P; size <<= 1)
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
            for (uint32_t k = threadIdx.x; k < P; k += blockDim.x) {
                const uint32_t o = k ^ stride;
                if (o > k) {
                    const bool up = (k & size) == 0;
                    const float ka = s_key[k], kb = s_key[o];
                    const uint32_t ta = s_tile[k], tb2 = s_tile[o];
                    const bool gt = ka > kb || (ka == kb && ta > tb2);
                    if (gt == up) {
                        s_key[k] = kb;
                        s_key[o] = ka;
                        s_tile[k] = tb2;
                        s_tile[o] = ta;
                    }
                }
            }
            __syncthreads();
        }
    for (uint32_t k = threadIdx.x; k < cnt; k += blockDim.x) out[rptr[g] + k] = make_uint2(s_tile[k], 1u);
}

__global__ void k_u64_to_u32(const uint64_t* __restrict__ in, uint64_t n, uint32_t* out) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = (uint32_t)in[i];
}

// The pass-2 tile ranges of every group (a thread per group) from its cell
// bitmap: each run of consecutive set cells is a run of adjacent points
// [cstart[first], cstart[last + 1]); those become tile ranges, merged where
// they touch or overlap.
// Without rptr it counts the ranges into cnt; with it, it writes them from
// rptr[g], adds the group's tile count to *tiles and leaves its sort key.
__global__ void k_group_ranges(const unsigned* __restrict__ gcell, uint32_t cwords, uint32_t F,
                               const uint64_t* __restrict__ cstart, uint64_t ngroups,
                               const uint32_t* __restrict__ rptr, uint64_t* cnt, uint2* rngs,
                               unsigned long long* tiles, uint32_t* gkey) {
    for (uint64_t g = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; g < ngroups;
         g += (uint64_t)gridDim.x * blockDim.x) {
        const unsigned* bits = gcell + g * cwords;
        uint64_t cur_b = 0, cur_e = 0, sum = 0;
        bool open = false;
        uint32_t k = 0, out = rptr ? rptr[g] : 0;
        auto emit = [&](uint64_t b, uint64_t e) {
            if (rptr) rngs[out + k] = make_uint2((uint32_t)b, (uint32_t)(e - b));
            sum += e - b;
            ++k;
        };
        uint32_t f = 0;
        while (f < F) {
            const unsigned m = bits[f / 32] >> (f % 32);
            if (m == 0) {  // no set bit left in this word
                f = (f / 32 + 1) * 32;
                continue;
            }
            f += (uint32_t)(__ffs(m) - 1);
            const uint32_t run0 = f;
            while (f < F) {
                const uint32_t avail = 32 - f % 32;
                const unsigned zeros = ~bits[f / 32] >> (f % 32);  // first clear bit at or after f
                if (zeros == 0) {
                    f += avail;
                    continue;
                }
                f += (uint32_t)(__ffs(zeros) - 1);
                break;
            }
            const uint32_t run1 = f < F ? f : F;
            const uint64_t pb = cstart[run0], pe = cstart[run1];
            if (pe <= pb) continue;
            const uint64_t tb = pb / TILE, te = (pe + TILE - 1) / TILE;
            if (open && tb <= cur_e) {
                cur_e = cur_e > te ? cur_e : te;
            } else {
                if (open) emit(cur_b, cur_e);
                cur_b = tb;
                cur_e = te;
                open = true;
            }
        }
        if (open) emit(cur_b, cur_e);
        if (rptr) {
            atomicAdd(tiles, (unsigned long long)sum);
            gkey[g] = ~(uint32_t)sum;  // ascending keys: descending tile counts
        } else {
            cnt[g] = k;
        }
    }
}

// The exact re-rank on the cluster-sorted copy Xs (the same FP32 values as X,
// so the same distances): row r is the sorted query ord[r] (ord nullable:
// r itself), candidates are sorted positions, ties are broken on original ids
// exactly as k_knn_rerank, and the lists land in the original query's row.
__global__ void k_knn_rerank_sorted(const float* __restrict__ Xs, uint64_t n, uint32_t d, uint32_t k,
                                    const uint32_t* __restrict__ ord, const uint32_t* __restrict__ perm,
                                    const uint32_t* __restrict__ cand_idx, uint32_t* __restrict__ out_idx,
                                    float* __restrict__ out_d2) {
    const unsigned lane = threadIdx.x & 31u;
    const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t r = warp; r < n; r += nwarps) {
        const uint64_t sq = ord ? ord[r] : r;
        const uint32_t q = perm[sq];
        auto key = [&](uint32_t js) -> uint64_t {
            if (js >= n) return ~0ull;
            const float* a = Xs + sq * d;
            const float* b = Xs + (uint64_t)js * d;
            float acc = 0.0f;
            for (uint32_t t = 0; t < d; ++t) {
                const float diff = __fsub_rn(a[t], b[t]);
                acc = __fmaf_rn(diff, diff, acc);
            }
            const uint32_t j = perm[js];
            return ((uint64_t)__float_as_uint(acc) << 32) | (j == q ? 0u : j + 1u);
        };
        const uint32_t* cand = cand_idx + r * RTOTAL;
        const uint64_t kk = rerank_list(cand[lane], cand[32 + lane], (uint32_t)sq, key);
        if (lane <= k) {
            const uint32_t tag = (uint32_t)kk;
            const uint32_t idx = (kk == ~0ull) ? 0xFFFFFFFFu : (tag == 0 ? q : tag - 1u);
            out_idx[(uint64_t)q * (k + 1) + lane] = idx;
            out_d2[(uint64_t)q * (k + 1) + lane] = kk == ~0ull ? INFINITY : __uint_as_float((uint32_t)(kk >> 32));
        }
    }
}

void knn_check(uint64_t n, uint64_t d, uint64_t k, const sc_knn_opts& opts) {
    if (d == 0 || d > 62) fail(SC_E_UNSUPPORTED, "kNN supports 1..62 dimensions, got %llu", (unsigned long long)d);
    if (k + 1 > 32) fail(SC_E_UNSUPPORTED, "kNN supports k <= 31");
    if (n >= 0xFFFFFFFFull) fail(SC_E_TOO_MANY_NODES, "too many points");
    if (opts.precision != SC_KNN_FP32 && opts.precision != SC_KNN_BF16 && opts.precision != SC_KNN_FP8)
        fail(SC_E_INVALID_ARGUMENT, "unknown kNN precision %d", opts.precision);
    if (opts.precision == SC_KNN_FP8 && d > 61)
        fail(SC_E_UNSUPPORTED, "the FP8 contraction supports 1..61 dimensions, got %llu", (unsigned long long)d);
}

constexpr uint64_t PRUNE_MIN_POINTS = 65536;

uint32_t prune_clusters(const Ctx& c, uint64_t n) {
    if (c.knn_clusters == 1 || n < PRUNE_MIN_POINTS) return 0;
    if (c.knn_clusters) return std::min<uint32_t>(c.knn_clusters, 256);
    // more clusters bound tighter (measured on 4M points x 30: 16% of the tiles
    // scanned with 256 clusters, 45% with 32); about 8192 points per cluster
    return (uint32_t)std::min<uint64_t>(256, std::max<uint64_t>(16, n / 8192));
}

// The exact k+1 nearest points of every point by the pruned search (see
// "exact pruning" above); the same lists as the full scan.
// Device time between events recorded on the context's stream.
struct StageTimer {
    Ctx& c;
    std::vector<cudaEvent_t> ev;
    explicit StageTimer(Ctx& ctx) : c(ctx) {}
    ~StageTimer() {
        for (cudaEvent_t e : ev) cudaEventDestroy(e);
    }
    void mark() {
        cudaEvent_t e;
        SC_CUDA(cudaEventCreate(&e));
        ev.push_back(e);
        SC_CUDA(cudaEventRecord(e, c.stream));
    }
    double ms(size_t a, size_t b) {
        SC_CUDA(cudaEventSynchronize(ev[b]));
        float t = 0.0f;
        SC_CUDA(cudaEventElapsedTime(&t, ev[a], ev[b]));
        return t;
    }
};

void knn_search_pruned(Ctx& c, const float* dX, uint64_t n, uint32_t d, uint32_t k, int precision, uint32_t K,
                       uint32_t* idx, float* d2) {
    const uint32_t k1 = k + 1;
    static const bool trace = std::getenv("SC_TRACE") != nullptr;
    StageTimer tm(c);
    tm.mark();
    // 1. deterministic k-means: K centroids from evenly spaced points, KM_ITERS Lloyd steps
    DBuf<KnnScale> scale_words(c, 1);
    zero(c, scale_words.get(), 1);
    k_knn_scales<<<grid_for(n, 256), 256, 0, c.stream>>>(dX, n, d, scale_words.get());
    SC_LAUNCH_CHECK();
    c.launches++;
    DBuf<float> cent(c, (uint64_t)K * d);
    const KnnScale hmx = to_host(c, scale_words.get());
    float maxabs, maxnorm;
    std::memcpy(&maxabs, &hmx.maxabs, 4);
    std::memcpy(&maxnorm, &hmx.maxnorm, 4);
    // sums of n coordinates of magnitude <= maxabs stay below 2^62 in fixed point
    const double span = std::max(1e-30, (double)maxabs * (double)n);
    const int e = std::min(40, (int)std::floor(62.0 - std::log2(span)) - 1);
    const double scale = std::ldexp(1.0, e), inv_scale = std::ldexp(1.0, -e);
    // Lloyd steps on an evenly spaced sample of the points (a few hundred per
    // centroid is plenty for bounds that hold whatever the clusters), then one
    // assignment of every point
    const uint64_t ns = std::min<uint64_t>(n, (uint64_t)KM_SAMPLE);
    std::vector<uint32_t> srows(ns);
    for (uint64_t i = 0; i < ns; ++i) srows[i] = (uint32_t)(i * n / ns);
    DBuf<uint32_t> d_srows(c, ns);
    DBuf<float> Xsub(c, ns * d);
    h2d(c, d_srows.get(), srows.data(), ns);
    k_gather_rows<<<grid_for(ns * d, 256), 256, 0, c.stream>>>(dX, d_srows.get(), ns, d, Xsub.get());
    SC_LAUNCH_CHECK();
    c.launches++;
    {
        // farthest-point seeds: the first sample point, then the farthest from all chosen so far
        DBuf<float> d2min(c, ns);
        DBuf<unsigned long long> keys(c, K + 1);
        SC_CUDA(cudaMemsetAsync(d2min.get(), 0x7F, ns * sizeof(float), c.stream));  // a huge finite value
        zero(c, keys.get(), K + 1);
        for (uint32_t t = 1; t <= K; ++t)
            k_seed_step<<<t < K ? grid_for(ns, 256) : 1, 256, 0, c.stream>>>(Xsub.get(), ns, d, t, t < K, d2min.get(),
                                                                             keys.get(), cent.get());
        SC_LAUNCH_CHECK();
        c.launches += K;
    }
    DBuf<uint32_t> assign(c, n);
    DBuf<unsigned long long> sums(c, (uint64_t)K * d);
    DBuf<unsigned> cnt(c, K);
    const size_t sm_assign = (size_t)K * ((d + 3) & ~3u) * 4, sm_accum = (size_t)K * d * 8 + (size_t)K * 4;
    SC_CUDA(cudaFuncSetAttribute(k_km_assign, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_assign));
    SC_CUDA(cudaFuncSetAttribute(k_km_accum, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_accum));
    for (int it = 0; it < KM_ITERS; ++it) {
        k_km_assign<<<grid_for(ns, 256, (unsigned)c.sm_count * 4), 256, sm_assign, c.stream>>>(
            Xsub.get(), ns, d, cent.get(), K, assign.get());
        zero(c, sums.get(), (uint64_t)K * d);
        zero(c, cnt.get(), K);
        k_km_accum<<<grid_for(ns * 32, 256, (unsigned)c.sm_count), 256, sm_accum, c.stream>>>(
            Xsub.get(), ns, d, assign.get(), K, scale, sums.get(), cnt.get());
        k_km_update<<<grid_for((uint64_t)K * d, 256), 256, 0, c.stream>>>(sums.get(), cnt.get(), K, d, inv_scale,
                                                                         cent.get());
        SC_LAUNCH_CHECK();
        c.launches += 3;
    }
    k_km_assign<<<grid_for(n, 256, (unsigned)c.sm_count * 4), 256, sm_assign, c.stream>>>(dX, n, d, cent.get(), K,
                                                                                          assign.get());
    SC_LAUNCH_CHECK();
    c.launches++;
    Xsub.release();
    tm.mark();  // 1: k-means
    // 2. points sorted by cluster (stable: ascending point id inside a cluster)
    DBuf<uint32_t> iota(c, n), cl_s(c, n), perm0(c, n);
    k_iota_u32<<<grid_for(n, 256), 256, 0, c.stream>>>(iota.get(), n);
    SC_LAUNCH_CHECK();
    c.launches++;
    sort_pairs(c, assign.get(), cl_s.get(), iota.get(), perm0.get(), n, bits_for(K - 1));
    assign.release();
    iota.release();
    DBuf<float> Xs(c, n * d);
    k_gather_rows<<<grid_for(n * d, 256), 256, 0, c.stream>>>(dX, perm0.get(), n, d, Xs.get());
    SC_LAUNCH_CHECK();
    c.launches++;
    DBuf<uint64_t> d_start(c, K + 1);
    k_cluster_starts<<<1, 512, 0, c.stream>>>(cl_s.get(), n, K, d_start.get());
    SC_LAUNCH_CHECK();
    c.launches++;
    std::vector<uint64_t> start(K + 1);
    {
        Mailbox mb(c);
        const uint64_t* hs = mb.get(d_start.get(), K + 1);
        mb.wait();
        std::copy(hs, hs + K + 1, start.begin());
    }
    // 3. fine cells inside every cluster, then the final order: (cluster, cell)
    std::vector<uint32_t> fbase(K + 1, 0);
    for (uint32_t q = 0; q < K; ++q) fbase[q + 1] = fbase[q] + (uint32_t)((start[q + 1] - start[q] + FINE - 1) / FINE);
    DBuf<uint32_t> d_fbase(c, K + 1), fine(c, n), fine_s(c, n), perm(c, n);
    h2d(c, d_fbase.get(), fbase.data(), K + 1);
    // each cell's centre: the sample point that defines it (read before Xs is re-sorted)
    const uint32_t F = fbase[K];
    std::vector<uint32_t> cell_rows(F);
    for (uint32_t q = 0; q < K; ++q)
        for (uint32_t j = 0; j < fbase[q + 1] - fbase[q]; ++j) cell_rows[fbase[q] + j] = (uint32_t)(start[q] + (uint64_t)j * FINE);
    DBuf<uint32_t> d_cell_rows(c, std::max<uint32_t>(F, 1));
    const uint32_t dp = (d + 3) & ~3u;  // rows of the direction tables, read as float4
    const uint32_t fp = row_pad(d);     // rows of the cells' centres
    DBuf<float> fcent(c, (uint64_t)std::max<uint32_t>(F, 1) * fp);
    h2d(c, d_cell_rows.get(), cell_rows.data(), F);
    k_gather_rows_padded<<<grid_for((uint64_t)F * fp, 256), 256, 0, c.stream>>>(Xs.get(), d_cell_rows.get(), F, d, fp,
                                                                             fcent.get());
    k_fine_assign<<<grid_for(n, 256), 256, 0, c.stream>>>(Xs.get(), n, d, cl_s.get(), fcent.get(), fp, d_fbase.get(),
                                                           fine.get());
    SC_LAUNCH_CHECK();
    c.launches += 2;
    sort_pairs(c, fine.get(), fine_s.get(), perm0.get(), perm.get(), n, bits_for(std::max<uint32_t>(F, 2) - 1));
    fine.release();
    perm0.release();
    k_gather_rows<<<grid_for(n * d, 256), 256, 0, c.stream>>>(dX, perm.get(), n, d, Xs.get());
    SC_LAUNCH_CHECK();
    c.launches++;
    // each cell's points (contiguous in the final order) and radius around its centre
    DBuf<unsigned> ccnt(c, std::max<uint32_t>(F, 1)), crad(c, std::max<uint32_t>(F, 1));
    zero(c, ccnt.get(), F);
    zero(c, crad.get(), F);
    k_cell_count<<<grid_for(n, 256), 256, 0, c.stream>>>(fine_s.get(), n, ccnt.get());
    k_cell_radius<<<grid_for(n, 256), 256, 0, c.stream>>>(Xs.get(), n, d, fine_s.get(), fcent.get(), fp, crad.get());
    SC_LAUNCH_CHECK();
    c.launches += 2;
    std::vector<unsigned> h_ccnt(F);
    d2h(c, h_ccnt.data(), ccnt.get(), F);
    sync(c);
    fine_s.release();
    std::vector<uint64_t> cstart(F + 1, 0);
    for (uint32_t f = 0; f < F; ++f) cstart[f + 1] = cstart[f] + h_ccnt[f];
    tm.mark();  // 2: sorted by cluster and cell
    // 4. cluster extents: radius, and [lo, hi] along every direction between centres
    DBuf<float> d_Ua(c, (uint64_t)K * K * dp), d_Ub(c, (uint64_t)K * K * dp);
    k_directions<<<grid_for((uint64_t)K * K, 128), 128, 0, c.stream>>>(cent.get(), K, d, dp, d_Ua.get(), d_Ub.get());
    SC_LAUNCH_CHECK();
    c.launches++;
    const uint64_t ngroups = (n + QT * TILE - 1) / (QT * TILE);
    const uint64_t ntiles = (n + TILE - 1) / TILE;
    // chunks: inside one cluster for the extents; inside one cluster and one query group for the bounds
    std::vector<Chunk> ch_ext, ch_need;
    for (uint32_t q = 0; q < K; ++q) {
        for (uint64_t p0 = start[q]; p0 < start[q + 1]; p0 += 2048)
            ch_ext.push_back(Chunk{q, p0, std::min<uint64_t>(start[q + 1], p0 + 2048)});
        for (uint64_t p0 = start[q]; p0 < start[q + 1];) {
            const uint64_t grp_end = (p0 / (QT * TILE) + 1) * (QT * TILE);
            const uint64_t p1 = std::min<uint64_t>(start[q + 1], grp_end);
            ch_need.push_back(Chunk{q, p0, p1});
            p0 = p1;
        }
    }
    DBuf<Chunk> d_ch_ext(c, ch_ext.size()), d_ch_need(c, ch_need.size());
    h2d(c, d_ch_ext.get(), ch_ext.data(), ch_ext.size());
    h2d(c, d_ch_need.get(), ch_need.data(), ch_need.size());
    DBuf<unsigned> rad(c, K), lo(c, (uint64_t)K * K), hi(c, (uint64_t)K * K);
    zero(c, rad.get(), K);
    zero(c, hi.get(), (uint64_t)K * K);
    SC_CUDA(cudaMemsetAsync(lo.get(), 0xFF, (uint64_t)K * K * 4, c.stream));
    const size_t sm_ext = (size_t)K * dp * 4 + (size_t)K * 8;
    SC_CUDA(cudaFuncSetAttribute(k_cluster_extent, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_ext));
    k_cluster_extent<<<(unsigned)ch_ext.size(), 256, sm_ext, c.stream>>>(Xs.get(), d, d_ch_ext.get(), cent.get(),
                                                                         d_Ub.get(), K, rad.get(), lo.get(), hi.get());
    SC_LAUNCH_CHECK();
    c.launches++;
    // 5. operands of the sorted points
    TcOperands op;
    prep_operands(c, Xs.get(), n, d, 0, n, precision, scale_words.get(), op);
    tm.mark();  // 3: extents and operands
    // the points of the clusters that query group g lies in
    auto own = [&](uint64_t g, std::vector<std::pair<uint64_t, uint64_t>>& pts) {
        auto cluster_of = [&](uint64_t i) {
            return (uint64_t)(std::upper_bound(start.begin(), start.end(), i) - start.begin()) - 1;
        };
        const uint64_t a0 = cluster_of(g * QT * TILE), a1 = cluster_of(std::min<uint64_t>(n, (g + 1) * QT * TILE) - 1);
        pts.emplace_back(start[a0], start[a1 + 1]);
    };
    DBuf<uint32_t> cidx(c, n * RTOTAL);
    // the candidates' exact re-rank, queries in the order `ord` (nullable: the sorted order)
    auto rerank = [&](const uint32_t* ord, uint32_t* out_idx, float* out_d2) {
        k_knn_rerank_sorted<<<grid_for(n * 32, 256), 256, 0, c.stream>>>(Xs.get(), n, d, k, ord, perm.get(),
                                                                        cidx.get(), out_idx, out_d2);
        SC_LAUNCH_CHECK();
        c.launches++;
    };
    // query groups by descending tile count (stable), from their negated counts
    DBuf<uint32_t> gkey(c, ngroups), gkey_s(c, ngroups), giota(c, ngroups), gorder(c, ngroups);
    k_iota_u32<<<grid_for(ngroups, 256), 256, 0, c.stream>>>(giota.get(), ngroups);
    SC_LAUNCH_CHECK();
    c.launches++;
    auto order_groups = [&]() {
        sort_pairs(c, gkey.get(), gkey_s.get(), giota.get(), gorder.get(), ngroups, 32);
    };
    // 6. pass 1: every query group against its own clusters, nearest cells first
    // (k_order_tiles: the rows' thresholds tighten within the first tiles, so
    // fewer later scores are kept; pass 1 only yields the bounds of pass 2: kb,
    // each sorted query's (k+1)-th squared distance from above)
    std::vector<uint32_t> rptr(ngroups + 1, 0);
    uint64_t tiles1 = 0;
    DBuf<float> kb(c, n);
    {
        std::vector<uint32_t> h_tb(ngroups), h_te(ngroups), h_key(ngroups);
        std::vector<std::pair<uint64_t, uint64_t>> pts;
        for (uint64_t g = 0; g < ngroups; ++g) {
            pts.clear();
            own(g, pts);
            h_tb[g] = (uint32_t)(pts[0].first / TILE);
            h_te[g] = (uint32_t)((pts[0].second + TILE - 1) / TILE);
            tiles1 += h_te[g] - h_tb[g];
            h_key[g] = ~(h_te[g] - h_tb[g]);
            if (tiles1 > 0xFFFFFFFFull)
                fail(SC_E_UNSUPPORTED, "pruned kNN lists exceed 2^32 tiles: use more clusters or the full scan");
            rptr[g + 1] = (uint32_t)tiles1;
        }
        std::vector<uint32_t> tile_cell(ntiles);
        for (uint64_t t = 0, f = 0; t < ntiles; ++t) {
            while (f + 1 < F && cstart[f + 1] <= t * TILE) ++f;
            tile_cell[t] = (uint32_t)f;
        }
        DBuf<uint32_t> d_tb(c, ngroups), d_te(c, ngroups), d_tc(c, ntiles), d_rp(c, ngroups + 1);
        DBuf<uint2> d_rg(c, std::max<uint64_t>(tiles1, 1));
        h2d(c, d_tb.get(), h_tb.data(), ngroups);
        h2d(c, d_te.get(), h_te.data(), ngroups);
        h2d(c, d_tc.get(), tile_cell.data(), ntiles);
        h2d(c, d_rp.get(), rptr.data(), ngroups + 1);
        k_order_tiles<<<(unsigned)ngroups, 256, 0, c.stream>>>(Xs.get(), n, d, d_tb.get(), d_te.get(), d_tc.get(),
                                                               fcent.get(), d_rp.get(), d_rg.get());
        SC_LAUNCH_CHECK();
        c.launches++;
        h2d(c, gkey.get(), h_key.data(), ngroups);
        order_groups();
        const TileLists tl{d_rp.get(), d_rg.get(), nullptr, gorder.get()};
        if (op.kind != 2 && few_bound(k1)) {
            launch_bound(c, op, n, 0, n, k1, (float*)cidx.get(), tl, kb.get());
        } else {
            DBuf<uint32_t> idx1(c, n * k1);
            DBuf<float> d21(c, n * k1);
            launch_keep(c, op, n, n, cidx.get(), tl);
            rerank(nullptr, idx1.get(), d21.get());
            k_list_kth<<<grid_for(n, 256), 256, 0, c.stream>>>(d21.get(), perm.get(), n, k1, kb.get());
            SC_LAUNCH_CHECK();
            c.launches++;
        }
        sync(c);  // the host arrays above must outlive the copies
    }
    tm.mark();  // 4: pass 1
    // 7. the clusters every group still needs
    const uint32_t words = (K + 63) / 64;
    DBuf<unsigned long long> mask(c, n * words);
    // rounding of an FP32 projection, distance or radius: a few ulps of the
    // largest coordinate norm times d
    const float R = std::sqrt(std::max(maxnorm, 0.0f)) + 1.0f;
    const float eps = 8.0f * (float)d * std::ldexp(1.0f, -24) * 2.0f * R;
    tm.mark();  // 5: bounds begin (after pass 1)
    const size_t sm_need = (size_t)K * dp * 8 + (size_t)K * 12;
    SC_CUDA(cudaFuncSetAttribute(k_cluster_needs, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_need));
    k_cluster_needs<<<(unsigned)ch_need.size(), QT * TILE, sm_need, c.stream>>>(
        Xs.get(), d, d_ch_need.get(), kb.get(), cent.get(), rad.get(), d_Ua.get(), lo.get(), hi.get(), K, eps, words,
        mask.get());
    SC_LAUNCH_CHECK();
    c.launches++;
    // pass-2 order: by own cluster, then by need set; groups of 256 in that order
    DBuf<unsigned long long> nkeys(c, n), nkeys_s(c, n);
    DBuf<uint32_t> npos(c, n), ord(c, n);
    k_need_keys<<<grid_for(n, 256), 256, 0, c.stream>>>(mask.get(), cl_s.get(), n, words, nkeys.get(), npos.get());
    SC_LAUNCH_CHECK();
    c.launches++;
    tm.mark();  // 6: cluster needs done
    sort_pairs(c, nkeys.get(), nkeys_s.get(), npos.get(), ord.get(), n, 32 + bits_for(K - 1));
    nkeys.release();
    nkeys_s.release();
    npos.release();
    DBuf<unsigned long long> gmask(c, ngroups * words);
    DBuf<uint32_t> gown(c, ngroups * 2);
    k_group_needs<<<grid_for(ngroups * 32, 256), 256, 0, c.stream>>>(mask.get(), ord.get(), cl_s.get(), n, words,
                                                                   ngroups, gmask.get(), gown.get());
    SC_LAUNCH_CHECK();
    c.launches++;
    // the cells each group scans: those of its candidate clusters a query cannot exclude
    tm.mark();  // 7: order and group needs done
    const uint32_t cwords = (F + 31) / 32;
    DBuf<unsigned> gcell(c, ngroups * cwords);
    zero(c, gcell.get(), ngroups * cwords);
    SC_CUDA(cudaFuncSetAttribute(k_group_cells, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(cwords * 8)));
    k_group_cells<<<(unsigned)ngroups, QT * TILE, cwords * 8, c.stream>>>(Xs.get(), n, d, ord.get(), kb.get(),
                                                                gmask.get(), gown.get(), words, K, d_fbase.get(),
                                                                fcent.get(), crad.get(), eps, cwords, mask.get(),
                                                                cl_s.get(), gcell.get());
    SC_LAUNCH_CHECK();
    c.launches++;
    tm.mark();  // 8: group cells done
    // the query operand in pass-2 order
    TcOperands op2;
    {
        const uint32_t row_bytes = op.row_bytes();
        op2.kind = op.kind;
        op2.scale = op.scale;
        op2.A.alloc(c, n * row_bytes);
        k_gather_operand_rows<<<grid_for(n * row_bytes / 16, 256), 256, 0, c.stream>>>(
            (const uint4*)op.A.get(), ord.get(), n, row_bytes / 16, (uint4*)op2.A.get());
        SC_LAUNCH_CHECK();
        c.launches++;
        op2.ta = make_map(op2.A.get(), n, row_bytes, op.kind == 2);
        op2.tb = op.tb;
    }
    // score bounds of the 16-bit search from the pass-1 bounds (FP8 scores
    // carry too coarse an error for a useful bound: none)
    DBuf<float> qcap;
    if (op.kind != 2) {
        qcap.alloc(c, n);
        k_score_cap<<<grid_for(n, 256), 256, 0, c.stream>>>(kb.get(), n, 0, ord.get(), op.nx.get(), op.rx.get(),
                                                            op.scale, qcap.get());
        SC_LAUNCH_CHECK();
        c.launches++;
    }
    sync(c);
    tm.mark();  // 9: bounds
    mask.release();
    // 8. pass 2: every cell a query of the group cannot exclude (cells in point
    // order), the tile lists built on the device from the cell bitmaps
    DBuf<uint64_t> d_cstart(c, F + 1);
    h2d(c, d_cstart.get(), cstart.data(), F + 1);
    DBuf<uint64_t> gcnt(c, ngroups + 1), r64(c, ngroups + 1);
    DBuf<uint32_t> d_rptr2(c, ngroups + 1);
    zero(c, gcnt.get(), ngroups + 1);
    DBuf<unsigned long long> d_tiles2(c, 1);
    zero(c, d_tiles2.get(), 1);
    k_group_ranges<<<grid_for(ngroups, 128), 128, 0, c.stream>>>(gcell.get(), cwords, F, d_cstart.get(), ngroups,
                                                                 nullptr, gcnt.get(), nullptr, nullptr, nullptr);
    exclusive_sum(c, gcnt.get(), r64.get(), ngroups + 1);
    const uint64_t nranges = to_host(c, r64.get() + ngroups);
    if (nranges > 0xFFFFFFFFull)
        fail(SC_E_UNSUPPORTED, "pruned kNN lists exceed 2^32 ranges: use more clusters or the full scan");
    k_u64_to_u32<<<grid_for(ngroups + 1, 256), 256, 0, c.stream>>>(r64.get(), ngroups + 1, d_rptr2.get());
    DBuf<uint2> d_rngs2(c, std::max<uint64_t>(nranges, 1));
    k_group_ranges<<<grid_for(ngroups, 128), 128, 0, c.stream>>>(gcell.get(), cwords, F, d_cstart.get(), ngroups,
                                                                 d_rptr2.get(), nullptr, d_rngs2.get(),
                                                                 d_tiles2.get(), gkey.get());
    SC_LAUNCH_CHECK();
    c.launches += 3;
    const uint64_t tiles2 = to_host(c, d_tiles2.get());
    tm.mark();  // 10: lists built
    order_groups();
    launch_keep(c, op2, n, n, cidx.get(), TileLists{d_rptr2.get(), d_rngs2.get(), qcap.get(), gorder.get()});
    rerank(ord.get(), idx, d2);
    tm.mark();  // 11: pass 2
    c.knn_stats.ms_cluster = tm.ms(0, 3);
    c.knn_stats.ms_pass1 = tm.ms(3, 4);
    c.knn_stats.ms_bounds = tm.ms(4, 10);
    c.knn_stats.ms_pass2 = tm.ms(10, 11);
    c.knn_stats.clusters = K;
    c.knn_stats.tiles_scanned = tiles1 + tiles2;
    c.knn_stats.tiles_pass1 = tiles1;
    c.knn_stats.tiles_full = ngroups * ntiles;
    if (trace)
        std::fprintf(stderr,
                     "[sc] knn pruned n=%llu K=%u cells=%u: k-means %.1f ms, sort %.1f ms, extents %.1f ms, pass1 "
                     "%.1f ms (%.2f%% of tiles), needs %.1f ms, order %.1f ms, cells %.1f ms, copy %.1f ms, lists "
                     "%.1f ms, pass2 %.1f ms (%.2f%%)\n",
                     (unsigned long long)n, K, F, tm.ms(0, 1), tm.ms(1, 2), tm.ms(2, 3), tm.ms(3, 4),
                     100.0 * tiles1 / (double)(ngroups * ntiles), tm.ms(5, 6), tm.ms(6, 7), tm.ms(7, 8),
                     tm.ms(8, 9), tm.ms(9, 10), tm.ms(10, 11), 100.0 * tiles2 / (double)(ngroups * ntiles));
}

// Exact (brute-force) k+1 nearest points of the queries q0 .. q0 + nq - 1
// among all n points of the device array dX: 64 candidates per query (the 32
// best of each half of the candidate columns) from the 16-bit or FP8 tensor-core
// scores, or the 32 best exact FP32 distances of either half of the points from
// the CUDA cores, ranked exactly in FP32. idx/d2 are nq x (k+1), self first, then
// ascending squared distance, ties by lower index (of equal candidates that a row
// has no room for, those of lower index stay).
void knn_search_device(Ctx& c, const float* dX, uint64_t n, uint64_t d, uint64_t k, uint64_t q0, uint64_t nq,
                       int precision, uint32_t* idx, float* d2) {
    c.knn_stats = sc_knn_stats{};
    if (!nq) return;
    if (precision != SC_KNN_FP32 && q0 == 0 && nq == n) {
        const uint32_t K = prune_clusters(c, n);
        if (K) {
            knn_search_pruned(c, dX, n, (uint32_t)d, (uint32_t)k, precision, K, idx, d2);
            check_device_status(c);
            return;
        }
    }
    {
        const uint64_t groups = (nq + QT * TILE - 1) / (QT * TILE), tiles = (n + TILE - 1) / TILE;
        c.knn_stats.tiles_scanned = c.knn_stats.tiles_full = groups * tiles;
    }
    DBuf<uint32_t> cidx(c, nq * RTOTAL);
    if (precision != SC_KNN_FP32) candidates(c, dX, n, (uint32_t)d, (uint32_t)k, q0, nq, precision, cidx.get());
    else candidates_fp32(c, dX, n, (uint32_t)d, q0, nq, cidx.get());
    k_knn_rerank<<<grid_for(nq * 32, 256), 256, 0, c.stream>>>(dX, n, (uint32_t)d, (uint32_t)k, q0, nq,
                                                                cidx.get(), idx, d2);
    SC_LAUNCH_CHECK();
    c.launches++;
    check_device_status(c);
}

// Gaussian connectivities (neighborhood/mod.rs:105-163, :480-544) from the
// device k+1 lists of all n points (squared distances): sigma per point,
// weights, symmetrisation, duplicate removal, CSR. earlier: a download that
// still runs on the context's staging lanes.
void knn_connectivities_device(Ctx& c, const uint32_t* idx, const float* d2, uint64_t n, uint64_t k,
                               const sc_knn_opts& opts, uint64_t* conn_ptrs, uint32_t* conn_nbrs, float* conn_w,
                               uint64_t conn_cap, uint64_t* conn_nnz, DevGraph** graph_out,
                               Download* earlier = nullptr) {
    DBuf<float> sigma(c, n);
    DBuf<unsigned long long> keys(c, 2 * n * k + 1), keys_s(c, 2 * n * k + 1);
    DBuf<float> w(c, 2 * n * k + 1), w_s(c, 2 * n * k + 1);
    DBuf<unsigned long long> cnt(c, 1);
    zero(c, cnt.get(), 1);
    // ids of idbits bits each: the sort's radix passes cover the bits in use only
    const int idbits = bits_for(n);
    if (n) {
        k_knn_sigma<<<grid_for(n, 256), 256, 0, c.stream>>>(d2, n, (uint32_t)k, opts.sigma == SC_SIGMA_KTH,
                                                            sigma.get());
        k_knn_pairs<<<grid_for(n * (k + 1), PAIR_THREADS), PAIR_THREADS, 0, c.stream>>>(
            idx, d2, n, (uint32_t)k, sigma.get(), opts.sym == SC_SYM_UNION, opts.squared_kiddo, idbits, keys.get(),
            w.get(), cnt.get());
        SC_LAUNCH_CHECK();
        c.launches += 2;
    }
    uint64_t N = to_host(c, cnt.get());
    sort_pairs(c, keys.get(), keys_s.get(), w.get(), w_s.get(), N, 2 * idbits);
    DBuf<uint8_t> keep(c, N);
    DBuf<unsigned long long> ukeys(c, N);
    DBuf<float> uw(c, N);
    uint64_t M = N;
    if (N) {
        k_dedupe_flags<<<grid_for(N, 256), 256, 0, c.stream>>>(keys_s.get(), N, keep.get());
        c.launches++;
        DBuf<uint64_t> m(c, 1);
        select_flagged(c, keys_s.get(), keep.get(), ukeys.get(), m.get(), N);
        select_flagged(c, w_s.get(), keep.get(), uw.get(), m.get(), N);
        M = to_host(c, m.get());
    }
    DBuf<uint32_t> rows(c, M), cols(c, M);
    DBuf<uint64_t> ptr(c, n + 1);
    if (M) {
        k_split_rowcol<<<grid_for(M, 256), 256, 0, c.stream>>>(ukeys.get(), M, idbits, rows.get(), cols.get());
        c.launches++;
    }
    k_ptr_from_rows<<<grid_for(M + 1, 256), 256, 0, c.stream>>>(rows.get(), M, n, ptr.get());
    SC_LAUNCH_CHECK();
    c.launches++;
    if (conn_nnz) *conn_nnz = M;
    Download csr(c);  // while the graph is built
    if (earlier) earlier->finish();  // the lanes serve one download at a time
    if (conn_ptrs) {
        if (M > conn_cap) fail(SC_E_INVALID_ARGUMENT, "conn_capacity %llu < %llu entries",
                               (unsigned long long)conn_cap, (unsigned long long)M);
        csr.add(conn_ptrs, ptr.get(), ptr.bytes());
        csr.add(conn_nbrs, cols.get(), M * sizeof(uint32_t));
        csr.add(conn_w, uw.get(), M * sizeof(float));
        csr.start();
    }
    std::unique_ptr<DevGraph> graph;
    if (graph_out) graph.reset(graph_from_csr(c, ptr.get(), n + 1, cols.get(), M, uw.get(), M, nullptr, 0, true));
    csr.finish();
    if (graph_out) *graph_out = graph.release();
}

__global__ void k_sqrt(const float* __restrict__ a, uint64_t n, float* b) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        b[i] = sqrtf(a[i]);
}

// The distances a caller sees: the squared ones, or their roots in `roots`.
const float* distances_out(Ctx& c, const float* d2, uint64_t count, int squared, bool wanted, DBuf<float>& roots) {
    if (squared || !wanted || !count) return d2;
    roots.alloc(c, count);
    k_sqrt<<<grid_for(count, 256), 256, 0, c.stream>>>(d2, count, roots.get());
    SC_LAUNCH_CHECK();
    c.launches++;
    return roots.get();
}

}  // namespace

// knn_arrayd_* (neighborhood/mod.rs:51-202, :359-578) with exact search.
void knn_gaussian(Ctx& c, const float* X, uint64_t n, uint64_t d, uint64_t k, const sc_knn_opts& opts,
                  uint32_t* knn_index, float* knn_dist, uint64_t* conn_ptrs, uint32_t* conn_nbrs, float* conn_w,
                  uint64_t conn_cap, uint64_t* conn_nnz, DevGraph** graph_out) {
    knn_check(n, d, k, opts);
    DBuf<float> dX(c, n * d);
    upload(c, dX.get(), X, n * d * sizeof(float));
    DBuf<uint32_t> idx(c, n * (k + 1));
    DBuf<float> d2(c, n * (k + 1));
    knn_search_device(c, dX.get(), n, d, k, 0, n, opts.precision, idx.get(), d2.get());
    DBuf<float> roots;
    const float* dist = distances_out(c, d2.get(), n * (k + 1), opts.squared_kiddo, knn_dist != nullptr, roots);
    Download lists(c);  // while the connectivities are built
    lists.add(knn_index, idx.get(), idx.bytes());
    lists.add(knn_dist, dist, d2.bytes());
    lists.start();
    if (conn_ptrs || graph_out)
        knn_connectivities_device(c, idx.get(), d2.get(), n, k, opts, conn_ptrs, conn_nbrs, conn_w, conn_cap, conn_nnz,
                                  graph_out, &lists);
    lists.finish();
}

// Times the search of all rows of X under candidate cluster counts (1: the
// full scan) and keeps the fastest on the context. Every candidate returns the
// same lists, so this changes speed only. Returns the number of candidates.
uint32_t knn_autotune(Ctx& c, const float* X, uint64_t n, uint64_t d, uint64_t k, const sc_knn_opts& opts,
                      uint32_t* chosen, double* ms_chosen, double* ms_full) {
    knn_check(n, d, k, opts);
    DBuf<float> dX(c, n * d);
    upload(c, dX.get(), X, n * d * sizeof(float));
    DBuf<uint32_t> idx(c, n * (k + 1));
    DBuf<float> d2(c, n * (k + 1));
    std::vector<uint32_t> cand{1};
    for (uint32_t K : {32u, 64u, 128u, 256u})
        if (n >= PRUNE_MIN_POINTS && (uint64_t)K * 4096 <= n) cand.push_back(K);
    const uint32_t saved = c.knn_clusters;
    double best = INFINITY, full = 0.0;
    uint32_t pick = 1;
    cudaEvent_t e0, e1;
    SC_CUDA(cudaEventCreate(&e0));
    SC_CUDA(cudaEventCreate(&e1));
    try {
        // warm-up: modules, pools, first-call costs
        c.knn_clusters = cand.back();
        knn_search_device(c, dX.get(), n, d, k, 0, n, opts.precision, idx.get(), d2.get());
        for (uint32_t K : cand) {
            c.knn_clusters = K;
            SC_CUDA(cudaEventRecord(e0, c.stream));
            knn_search_device(c, dX.get(), n, d, k, 0, n, opts.precision, idx.get(), d2.get());
            SC_CUDA(cudaEventRecord(e1, c.stream));
            SC_CUDA(cudaEventSynchronize(e1));
            float ms = 0.0f;
            SC_CUDA(cudaEventElapsedTime(&ms, e0, e1));
            if (K == 1) full = ms;
            if (ms < best) {
                best = ms;
                pick = K;
            }
        }
    } catch (...) {
        c.knn_clusters = saved;
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        throw;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    c.knn_clusters = pick;
    if (chosen) *chosen = pick;
    if (ms_chosen) *ms_chosen = best;
    if (ms_full) *ms_full = full;
    return (uint32_t)cand.size();
}

// The k+1 lists of the query rows [q0, q1) only (one shard of a multi-GPU
// build); squared FP32 distances.
void knn_search(Ctx& c, const float* X, uint64_t n, uint64_t d, uint64_t k, uint64_t q0, uint64_t q1,
                const sc_knn_opts& opts, uint32_t* knn_index, float* knn_d2) {
    knn_check(n, d, k, opts);
    if (q0 > q1 || q1 > n) fail(SC_E_INVALID_ARGUMENT, "query rows [%llu, %llu) are not inside [0, %llu)",
                                (unsigned long long)q0, (unsigned long long)q1, (unsigned long long)n);
    const uint64_t nq = q1 - q0;
    DBuf<float> dX(c, n * d);
    upload(c, dX.get(), X, n * d * sizeof(float));
    DBuf<uint32_t> idx(c, nq * (k + 1));
    DBuf<float> d2(c, nq * (k + 1));
    knn_search_device(c, dX.get(), n, d, k, q0, nq, opts.precision, idx.get(), d2.get());
    Download lists(c);
    lists.add(knn_index, idx.get(), idx.bytes());
    lists.add(knn_d2, d2.get(), d2.bytes());
    lists.start();
    lists.finish();
}

// Connectivities from gathered host lists (all n rows, squared distances).
void knn_connectivities(Ctx& c, const uint32_t* knn_index, const float* knn_d2, uint64_t n, uint64_t k,
                        const sc_knn_opts& opts, uint64_t* conn_ptrs, uint32_t* conn_nbrs, float* conn_w,
                        uint64_t conn_cap, uint64_t* conn_nnz, DevGraph** graph_out) {
    if (k + 1 > 32) fail(SC_E_UNSUPPORTED, "kNN supports k <= 31");
    if (n >= 0xFFFFFFFFull) fail(SC_E_TOO_MANY_NODES, "too many points");
    DBuf<uint32_t> idx(c, n * (k + 1));
    DBuf<float> d2(c, n * (k + 1));
    h2d(c, idx.get(), knn_index, n * (k + 1));
    h2d(c, d2.get(), knn_d2, n * (k + 1));
    knn_connectivities_device(c, idx.get(), d2.get(), n, k, opts, conn_ptrs, conn_nbrs, conn_w, conn_cap, conn_nnz,
                              graph_out);
}

}  // namespace sc
