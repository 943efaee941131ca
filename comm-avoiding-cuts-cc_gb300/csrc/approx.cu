// approx_cut: the GB300 form of ApproximateCut::run (src/ApproximateCut.cpp:10-79).
//
// For levels i = 1 .. ceil(ln W) the reference keeps each edge of each of `copies` disjoint
// copies iff Binomial(w, 2^-i) > 0 (std::binomial_distribution, :39-48), relabels copy j to
// v + j n, runs the iterated-sparse-sampling CC on the union and stops at the first level with
// more than `copies` components; the answer is 2^level.
//
// Here each level hooks the kept edges of every copy into one union-find over n * copies vertices
// (the CC of the disjoint union is the union-find of all kept edges), then the roots are counted. On
// larger graphs a sample of the edges comes first: it leaves one giant component per copy, and of the
// other edges only those with an end outside the giant of some copy are tested and hooked at all
// (run_level). The keep test is integer-only and counter-addressed:
// P(Binomial(w, q) > 0) = 1 - (1 - q)^w, so the pair is kept iff the u64 draw x >= F(i, w) with
// F = (1 - 2^-i)^w in 0.64 fixed point by square-and-multiply over truncating 64x64->128-bit
// products; x is draw e_local of stream (seed + r, i, j, 1), r the virtual rank whose slice
// holds the edge (ApproximateCut::loadFromInput, ApproximateCut.hpp:64-68) and e_local its
// index in that slice. oracle/approx.c replays the same rule on the host.
//
// The level count is the reference's ceil(ln w) of each rank's own slice weight (`w` at :19-30
// is the calling rank's local sum), the smallest over ranks: the ranks step through the levels'
// collectives together, so the reference's run is defined only while every rank is still in its
// loop, and the smallest count gives its answer wherever it has one.
//
// Seed replay (approx_run with ref_stream): the keep test instead consumes the reference's own
// draws. Rank r's engine is sitmo::prng_engine(seed + r) (ApproximateCut.hpp:35, .cpp:33), read in
// the reference's order: per level, for each copy, for each slice edge one
// std::binomial_distribution<int>(w, 2^-i) draw, then one raw output for the level's CC seed
// (:50-58). With w = 1 that draw (libstdc++'s waiting-time method) takes exactly one
// generate_canonical<double, 53> value U from the two outputs x0, x1 as (x0 + x1 2^32) / 2^64,
// and returns 1 iff -ln(1 - U) <= -ln(1 - 2^-i). So the draw for copy j and slice edge e of
// level i reads outputs k and k + 1, k = (i - 1) (2 C len_r + 1) + 2 (j len_r + e), and every
// edge of every copy is tested independently on the device. The test is an integer comparison
// of U 2^64 with a threshold per level (see stream_keep) that decides exactly as the logarithms
// do; no floating point runs on the device.
// Graphs with other weights draw a variable number of outputs per edge (a sequential chain per
// rank), so the replay takes unit weights only.
#include "cac_internal.h"
#include "grid_loop.cuh"
#include "pdl.cuh"
#include "sitmo.cuh"

#include <algorithm>
#include <cmath>
#include <vector>

namespace cac {
namespace {

constexpr int kThreads = 256;
// Graphs with fewer edges (and more than kSmallN vertices) hook every edge in one pass: there a level is a few
// launches either way.
constexpr uint64_t kSampledEdges = 1u << 15;
constexpr uint32_t kSampleParts = 128;        // a sampling round takes 128ths of the edges
constexpr int kHops = 32;                     // longest walk of a compression between rounds
constexpr double kRoundDegree[] = {0.8, 0.8, 0.8, 0.8, 1.6};  // kept edges per vertex in each round
constexpr uint32_t kGiantSample = 1024;       // vertices looked at to find a copy's giant component
constexpr int kStreamThreads = 1024;          // CTA of the pass over the other edges (the bitmap fills shared memory)
constexpr uint32_t kSmemWords = 48 * 1024;    // bitmap words in shared memory (1.57 M vertices)
__device__ __forceinline__ uint64_t keep_threshold(uint32_t level, uint32_t w) {
    const uint64_t base = 0ull - (1ull << (64 - level));
    uint64_t res = base, b = base;
    uint32_t e = w - 1;
    while (e) {
        if (e & 1) res = mulhi64(res, b);
        b = mulhi64(b, b);
        e >>= 1;
    }
    return res;
}

// The forest of all copies: parent of vertex x in copy j at x * copies + j, so that what one edge needs
// of all copies lies side by side (4 copies: one 16-byte access per end). Parents are vertices of the
// same copy, never larger than the child; roots are their own parents.
struct Forest {
    uint32_t *par;
    uint32_t copies;
    __device__ __forceinline__ uint32_t &at(uint32_t x, uint32_t j) const { return par[x * copies + j]; }
};

__device__ __forceinline__ uint32_t afind(const Forest &F, uint32_t j, uint32_t v) {  // with path halving
    uint32_t cur = F.at(v, j);
    if (cur != v) {
        uint32_t prev = v, next;
        while (cur > (next = F.at(cur, j))) {
            F.at(prev, j) = next;
            prev = cur;
            cur = next;
        }
    }
    return cur;
}

__device__ __forceinline__ void aunite(const Forest &F, uint32_t j, uint32_t a, uint32_t b) {
    uint32_t ra = afind(F, j, a), rb = afind(F, j, b);
    while (ra != rb) {
        if (ra < rb) {
            const uint32_t old = atomicCAS(&F.at(rb, j), rb, ra);
            if (old == rb) return;
            rb = old;
        } else {
            const uint32_t old = atomicCAS(&F.at(ra, j), ra, rb);
            if (old == ra) return;
            ra = old;
        }
    }
}

__device__ __forceinline__ uint32_t root_of(const Forest &F, uint32_t j, uint32_t cur) {  // without writes
    uint32_t next;
    while ((next = F.at(cur, j)) != cur) cur = next;
    return cur;
}

// Singletons, one thread per vertex of 4 copies, else per vertex and copy, and the root count at 0.
__global__ void approx_init(const Forest F, uint32_t n, unsigned int *count) {
    pdl_wait();
    if (blockIdx.x == 0 && threadIdx.x == 0) *count = 0;
    if (F.copies == 4)
        grid_stride(n, [&](uint32_t x) { reinterpret_cast<uint4 *>(F.par)[x] = make_uint4(x, x, x, x); });
    else
        grid_stride(n * F.copies, [&](uint32_t i) { F.par[i] = i / F.copies; });
}

// The draws are taken by quads: a quad is 4 consecutive edges of one rank's slice, local
// indices 4 lq .. 4 lq + 3, whose 4 draws are the 4 words of one sitmo block (counter lq). Rank
// r < P - 1 owns Qf = ceil(portion / 4) quads, the last rank the rest of the edges (all of them when
// portion is 0).
struct Level {
    const uint32_t *U, *V, *Wt;
    uint32_t m, n, level, seed, ranks, portion, Qf, Q;
    uint64_t keep_max;     // seed replay: stream_threshold(level)
    uint32_t from, to;     // the quads of a sampling round: groups g of 64 with from <= g % kSampleParts < to
    Forest F;
    uint32_t *giants;      // copies: the root of each copy's giant component
    uint32_t *member;      // n: bit j: in the giant of copy j
    uint32_t *bits;        // n bits: in the giant of every copy
    uint2 *list;           // (edge, copies it has to be tested in), the first `cap` survivors
    uint32_t cap;
    uint32_t *count;       // survivors
};

struct Quad {
    uint32_t r, lq, base, len;  // its rank, its index there, the rank's first edge and edge count
};
__device__ __forceinline__ Quad quad_of(const Level &L, uint32_t gq) {
    Quad q;
    q.r = L.ranks - 1;
    if (L.portion) q.r = min(gq / L.Qf, L.ranks - 1);
    q.lq = gq - q.r * L.Qf;
    q.base = q.r * L.portion;
    q.len = q.r + 1 < L.ranks ? L.portion : L.m - q.base;
    return q;
}

// Binomial(1, p) > 0 on the reference's draws: U = generate_canonical<double, 53> of outputs x0, x1
// (x0 + x1 2^32 rounded to a double, scaled by 2^-64, clamped below 1); kept iff
// -ln(1 - U) <= -ln(1 - p) (libstdc++'s waiting-time test with t = 1). ln is increasing, and for
// p = 2^-i <= 1/2 every double next to b = 1 - p lies at least two units in the last place of
// ln(b) away from it in logarithm, so any logarithm accurate to within one unit decides as
// fl(1 - U) >= b does. That test is made here in integers: with R = U 2^64 (x0 + x1 2^32 rounded
// to 53 significant bits, to nearest, ties to even), fl(1 - U) >= b iff 1 - R 2^-64 is at least
// the midpoint between b and the double below it (a tie rounds to b, whose significand is even
// for i <= 52), i.e. iff R <= T(i) with T(1) = 2^63 + 2^9 and T(i) = 2^(64-i) + 2^10 for
// 2 <= i <= 52 (levels stop at ceil(ln W) <= 45). R = 2^64 is U = 1, clamped below 1: never kept.
__host__ __device__ __forceinline__ uint64_t stream_threshold(uint32_t level) {
    return level == 1 ? (1ull << 63) + (1ull << 9) : (1ull << (64 - level)) + (1ull << 10);
}

__device__ __forceinline__ bool stream_keep(uint64_t S, uint64_t T) {  // S = x0 + x1 2^32
    const int sh = 11 - __clzll(S);  // bits below the 53-bit significand
    if (sh <= 0) return S <= T;
    const uint64_t q = S >> sh, rem = S & ((1ull << sh) - 1), half = 1ull << (sh - 1);
    const uint64_t qr = q + ((rem > half || (rem == half && (q & 1))) ? 1 : 0);
    if (qr >> (64 - sh)) return false;
    return (qr << sh) <= T;
}

// Seed replay, unit weights: the quad's 4 draws read the 8 consecutive outputs k0 .. k0 + 7 of the
// rank's engine (output k = half k & 1 of word k >> 1, low half first: lib/prng_engine.hpp:195-212;
// words 4b .. 4b + 3 form sitmo block b). Draw d's two outputs give S = x0 + x1 2^32, which is
// word (k0 >> 1) + d itself when k0 is even and the high half of that word joined to the low half
// of the next when k0 is odd; the words lie in the blocks k0 >> 3 and the one after it.
__device__ __forceinline__ uint64_t stream_output(const Level &L, uint32_t j, uint32_t len, uint32_t local) {
    return (uint64_t)(L.level - 1) * (2 * (uint64_t)L.F.copies * len + 1) + 2 * ((uint64_t)j * len + local);
}

// The kept edges of quad q in copy j, bit d for its edge d (edges past the slice's end: 0).
// Thresholds: `table` holds those of weights below kTable (a square-and-multiply of up to 16 wide
// products each, as many instructions as the cipher for a quad of small weights).
constexpr uint32_t kTable = 256;
__device__ __forceinline__ void fill_thresholds(uint64_t *table, uint32_t level) {  // (a barrier follows)
    for (uint32_t w = threadIdx.x; w < kTable; w += blockDim.x) table[w] = w ? keep_threshold(level, w) : 0;
}

template <bool kRef>
__device__ __forceinline__ uint32_t quad_keeps(const Level &L, const Quad &q, uint32_t j, const uint64_t *table) {
    const uint32_t here = min(4u, q.len - 4 * q.lq);
    uint32_t mask = 0;
    if constexpr (kRef) {
        const uint64_t k0 = stream_output(L, j, q.len, 4 * q.lq);
        const uint64_t b0 = k0 >> 3;
        const unsigned a = (unsigned)(k0 >> 1) & 3u;  // first word inside block b0
        const bool odd = k0 & 1;
        const uint32_t key = L.seed + q.r;
        const u64x4 A = sitmo_block(key, 0, 0, 0, b0, 0, 0, 0);
        u64x4 B = A;
        if (a != 0 || odd) B = sitmo_block(key, 0, 0, 0, b0 + 1, 0, 0, 0);
        const uint64_t w[8] = {A.x[0], A.x[1], A.x[2], A.x[3], B.x[0], B.x[1], B.x[2], B.x[3]};
        uint64_t S[4];
#define CAC_QUAD_DRAWS(A0)                                                                     \
    _Pragma("unroll") for (int d = 0; d < 4; d++) S[d] =                                       \
        odd ? ((w[(A0) + d] >> 32) | (w[(A0) + d + 1] << 32)) : w[(A0) + d];
        switch (a) {
            case 0: CAC_QUAD_DRAWS(0) break;
            case 1: CAC_QUAD_DRAWS(1) break;
            case 2: CAC_QUAD_DRAWS(2) break;
            default: CAC_QUAD_DRAWS(3) break;
        }
#undef CAC_QUAD_DRAWS
#pragma unroll
        for (int d = 0; d < 4; d++) mask |= (uint32_t)stream_keep(S[d], L.keep_max) << d;
    } else {
        const u64x4 o = sitmo_block(L.seed + q.r, L.level, j, 1, q.lq, 0, 0, 0);
#pragma unroll
        for (uint32_t d = 0; d < 4; d++) {
            const uint32_t w = d < here ? L.Wt[q.base + 4 * q.lq + d] : 0;
            const uint64_t least = w < kTable ? table[w] : keep_threshold(L.level, w);
            mask |= (uint32_t)(w != 0 && o.x[d] >= least) << d;
        }
    }
    return mask & ((1u << here) - 1);
}

// Whether edge e is kept in copy j, on its own.
template <bool kRef>
__device__ __forceinline__ bool edge_kept(const Level &L, uint32_t e, uint32_t j) {
    const uint32_t r = L.portion ? min(e / L.portion, L.ranks - 1) : L.ranks - 1;
    const uint32_t base = r * L.portion, local = e - base;
    if constexpr (kRef) {
        const uint64_t k0 = stream_output(L, j, r + 1 < L.ranks ? L.portion : L.m - base, local);
        const uint64_t w0 = draw64(L.seed + r, 0, 0, 0, 0, k0 >> 1);
        if (!(k0 & 1)) return stream_keep(w0, L.keep_max);
        return stream_keep((w0 >> 32) | (draw64(L.seed + r, 0, 0, 0, 0, (k0 >> 1) + 1) << 32), L.keep_max);
    } else {
        const uint32_t w = L.Wt[e];
        return w != 0 && draw64(L.seed + r, L.level, j, 1, 0, local) >= keep_threshold(L.level, w);
    }
}

// Hooks the kept edges of some quads, a thread per quad and copy, the copies of a quad in neighbouring
// lanes (what an end needs of 4 copies is one 16-byte access).
//   kRound  a sampling round: the forest is nearly flat, and every kept edge between two parents makes the smaller
//           one the parent of the larger, the smallest of all winning (an atomic without a return value:
//           no walk, no retry; a link that loses is found again by the pass over all edges). Late
//           rounds have few large trees, whose roots would take thousands of such writes each: a table
//           of the CTA's writes (lossy; root -> smallest parent given) stops those that change nothing.
//   kAll    every quad, by union walks
enum QuadPass { kRound, kAll };
constexpr uint32_t kGiven = 1024;
template <bool kRef, QuadPass kPass>
__device__ __forceinline__ void hook_quads(const Level &L, unsigned long long *given, const uint64_t *table) {
    const uint32_t C = L.F.copies, lane = threadIdx.x & 31, side = min(C, 32u), per = 32 / side;  // quads per warp
    if (lane >= side * per) return;
    // the pass's quads, numbered: all, or those of the round
    const uint32_t w = L.to - L.from, groups = (L.Q + 63) / 64, last = groups % kSampleParts;
    const uint64_t count = kPass == kAll ? L.Q
                                         : (uint64_t)64 * (groups / kSampleParts * w + (last > L.from ? min(last, L.to) - L.from : 0));
    const uint32_t warps = (gridDim.x * kThreads) >> 5;
    for (uint64_t i = (uint64_t)((blockIdx.x * kThreads + threadIdx.x) >> 5) * per + lane / side; i < count;
         i += (uint64_t)warps * per) {
        uint32_t gq = (uint32_t)i;
        if (kPass == kRound) {
            const uint32_t g = (uint32_t)(i >> 6);
            gq = (g / w * kSampleParts + L.from + g % w) * 64 + ((uint32_t)i & 63u);
            if (gq >= L.Q) continue;
        }
        const Quad q = quad_of(L, gq);
        const uint32_t e0 = q.base + 4 * q.lq;
        for (uint32_t j = lane % side; j < C; j += side) {
            const uint32_t mask = quad_keeps<kRef>(L, q, j, table);
            uint32_t a[4], b[4];
#pragma unroll
            for (uint32_t d = 0; d < 4; d++) {
                a[d] = b[d] = 0;
                if ((mask >> d) & 1u) {
                    a[d] = __ldg(L.U + e0 + d);
                    b[d] = __ldg(L.V + e0 + d);
                }
            }
#pragma unroll
            for (uint32_t d = 0; d < 4; d++)
                if ((mask >> d) & 1u) {
                    a[d] = L.F.at(a[d], j);
                    b[d] = L.F.at(b[d], j);
                }
#pragma unroll
            for (uint32_t d = 0; d < 4; d++) {
                if (a[d] == b[d]) continue;
                if (kPass == kAll) {
                    aunite(L.F, j, a[d], b[d]);
                } else {
                    const uint32_t hi = max(a[d], b[d]) * C + j, lo = min(a[d], b[d]);
                    volatile unsigned long long *t = &given[hi * 2654435761u >> 22];
                    const unsigned long long had = *t;
                    if ((uint32_t)(had >> 32) == hi && (uint32_t)had <= lo) continue;
                    atomicMin(&L.F.par[hi], lo);
                    *t = (unsigned long long)hi << 32 | lo;
                }
            }
        }
    }
}

template <bool kRef, QuadPass kPass>
__global__ void __launch_bounds__(kThreads) approx_quads(const Level L) {
    __shared__ unsigned long long given[kPass == kRound ? kGiven : 1];
    __shared__ uint64_t table[kRef ? 1 : kTable];
    if (kPass == kRound)
        for (uint32_t i = threadIdx.x; i < kGiven; i += kThreads) given[i] = ~0ull;
    if (!kRef) fill_thresholds(table, L.level);
    __syncthreads();
    pdl_wait();
    hook_quads<kRef, kPass>(L, given, table);
}

// All edges after the sampling rounds, a warp per 256-edge tile as in the filter of the
// connected-components path: an edge with both ends in the giant of every copy is dropped unseen
// (whatever its draws say, it joins nothing); of the others, the copies in which an end is outside the
// giant are noted in the survivor list (the first L.cap; past that only counted). kShared: the bitmap fits
// shared memory.
template <bool kRef, bool kShared>
__global__ void __launch_bounds__(kStreamThreads) approx_stream(const Level L) {
    pdl_wait();
    extern __shared__ uint32_t sbits[];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    if (kShared) {
        for (uint32_t i = threadIdx.x; i < (L.n + 31) / 32; i += blockDim.x) sbits[i] = L.bits[i];
        __syncthreads();
    }
    const uint32_t *bits = kShared ? sbits : L.bits;
    auto inside = [&](uint32_t x) { return (bits[x >> 5] >> (x & 31)) & 1u; };
    const uint32_t tiles = (uint32_t)(((uint64_t)L.m + 255) / 256);
    const uint32_t all = L.F.copies >= 32 ? 0xFFFFFFFFu : (1u << L.F.copies) - 1;
    for (uint32_t i = blockIdx.x * nwarps + warp; i < tiles; i += gridDim.x * nwarps) {
        const uint32_t e0 = i * 256;
        uint32_t a[8], b[8], e[8], keep = 0;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint32_t x = e0 + 128 * h + 4 * lane;
            uint4 ua = make_uint4(0, 0, 0, 0), va = ua;
            if (x + 3 < L.m) {
                ua = __ldcs(reinterpret_cast<const uint4 *>(L.U + x));
                va = __ldcs(reinterpret_cast<const uint4 *>(L.V + x));
            } else {
                if (x < L.m) ua.x = L.U[x], va.x = L.V[x];
                if (x + 1 < L.m) ua.y = L.U[x + 1], va.y = L.V[x + 1];
                if (x + 2 < L.m) ua.z = L.U[x + 2], va.z = L.V[x + 2];
            }
            a[4 * h] = ua.x, a[4 * h + 1] = ua.y, a[4 * h + 2] = ua.z, a[4 * h + 3] = ua.w;
            b[4 * h] = va.x, b[4 * h + 1] = va.y, b[4 * h + 2] = va.z, b[4 * h + 3] = va.w;
#pragma unroll
            for (int d = 0; d < 4; d++) e[4 * h + d] = x + d;
        }
#pragma unroll
        for (int d = 0; d < 8; d++) {  // (an edge past the end is 0-0: a loop)
            keep |= (uint32_t)(a[d] != b[d] && !(inside(a[d]) && inside(b[d]))) << d;
        }
        if (!__any_sync(0xffffffffu, keep)) continue;
        uint32_t need[8];
#pragma unroll
        for (int d = 0; d < 8; d++) need[d] = (keep >> d) & 1u ? all & ~(L.member[a[d]] & L.member[b[d]]) : 0;
        const uint32_t mine = __popc(keep);
        uint32_t incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += y;
        }
        uint32_t at = 0;
        if (lane == 31) at = atomicAdd(L.count, incl);
        at = __shfl_sync(0xffffffffu, at, 31) + incl - mine;
#pragma unroll
        for (int d = 0; d < 8; d++) {
            if (!((keep >> d) & 1u)) continue;
            if (at < L.cap) L.list[at] = make_uint2(e[d], need[d]);
            at++;
        }
    }
}

// What the stream pass left: one thread per (survivor, copy), or, where the survivors are more than their
// list holds, every quad by union walks (a quad's 4 draws cost as much as one survivor's).
template <bool kRef>
__global__ void __launch_bounds__(kThreads) approx_rest(const Level L) {
    pdl_wait();
    const uint32_t count = *L.count;
    if (count > L.cap) {
        __shared__ uint64_t table[kRef ? 1 : kTable];
        if (!kRef) fill_thresholds(table, L.level);
        __syncthreads();
        hook_quads<kRef, kAll>(L, nullptr, table);
        return;
    }
    const uint64_t items = (uint64_t)count * L.F.copies;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < items; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t at = (uint32_t)(i / L.F.copies), j = (uint32_t)(i - (uint64_t)at * L.F.copies);
        const uint2 x = L.list[at];
        if (((x.y >> j) & 1u) && edge_kept<kRef>(L, x.x, j)) aunite(L.F, j, L.U[x.x], L.V[x.x]);
    }
}

// Weight sum of every rank's slice. Slices as GraphInputIterator::loadSlice
// (src/input/GraphInputIterator.hpp:77-93): rank r < P - 1 owns [r portion, (r + 1) portion), the
// last rank the rest. Ranks along blockIdx.y (strided).
__global__ void approx_slice_sums(const uint32_t *__restrict__ w, uint64_t m, uint32_t ranks, uint64_t portion,
                                  unsigned long long *sums) {
    for (uint32_t r = blockIdx.y; r < ranks; r += gridDim.y) {
        const uint64_t from = (uint64_t)r * portion, to = r + 1 < ranks ? from + portion : m;
        unsigned long long acc = 0;
        for (uint64_t e = from + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < to;
             e += (uint64_t)gridDim.x * blockDim.x)
            acc += w[e];
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if ((threadIdx.x & 31) == 0 && acc) atomicAdd(&sums[r], acc);
    }
}

// An ancestor of v in copy j, the root unless it is more than kHops away.
__device__ __forceinline__ uint32_t near_of(const Forest &F, uint32_t j, uint32_t cur) {
    uint32_t next;
    for (int k = 0; k < kHops && (next = F.at(cur, j)) != cur; k++) cur = next;
    return cur;
}

// Compression between the rounds, a thread per vertex and 4 copies: their parents in one load, the 4
// grandparents requested together, then the longer chains. With other numbers of copies a thread per vertex
// and copy, neighbouring lanes on neighbouring words (37 copies of 300,000 vertices: 38 us; 184 us by
// vertices). Walks end after kHops parents: heavy paths
// numbered along their length make chains of that length, and the rounds do not need a flat forest (what
// a link at a vertex that is no root any more separates is joined again by the pass over all edges).
__global__ void approx_compress(const Forest F, uint32_t n) {
    pdl_wait();
    if (F.copies == 4) {
        uint4 *p4 = reinterpret_cast<uint4 *>(F.par);
        grid_stride(n, [&](uint32_t x) {
            const uint4 p = p4[x];
            const uint32_t g0 = F.par[4 * p.x], g1 = F.par[4 * p.y + 1], g2 = F.par[4 * p.z + 2], g3 = F.par[4 * p.w + 3];
            const uint32_t r0 = g0 == p.x ? g0 : near_of(F, 0, g0), r1 = g1 == p.y ? g1 : near_of(F, 1, g1);
            const uint32_t r2 = g2 == p.z ? g2 : near_of(F, 2, g2), r3 = g3 == p.w ? g3 : near_of(F, 3, g3);
            if (r0 != p.x || r1 != p.y || r2 != p.z || r3 != p.w) p4[x] = make_uint4(r0, r1, r2, r3);
        });
    } else {
        grid_stride(n * F.copies, [&](uint32_t i) {
            const uint32_t x = i / F.copies, r = near_of(F, i - x * F.copies, x);
            if (r != x) F.par[i] = r;
        });
    }
}

// The giant component of each copy (one CTA per copy): the most frequent root among kGiantSample
// vertices spread over the copy (the mode of each warp's 32, counted over all; ties to the smaller
// root). The choice decides which edges are dropped unseen, never the partition.
__global__ void __launch_bounds__(kGiantSample) approx_giants(const Level L) {
    pdl_wait();
    __shared__ uint32_t cand[kGiantSample / 32], cnt[kGiantSample / 32];
    __shared__ unsigned long long best;
    const uint32_t i = threadIdx.x, lane = i & 31, w = i >> 5;
    const uint32_t r = root_of(L.F, blockIdx.x, (uint32_t)(((uint64_t)i * 2654435761u) % L.n));
    const uint32_t same = __match_any_sync(0xffffffffu, r);
    const uint32_t c = __popc(same);
    const uint32_t top = __reduce_max_sync(0xffffffffu, c);
    const uint32_t lo = __reduce_min_sync(0xffffffffu, c == top ? r : 0xFFFFFFFFu);
    if (lane == 0) {
        cand[w] = lo;
        cnt[w] = 0;
    }
    if (i == 0) best = 0;
    __syncthreads();
    for (uint32_t k = 0; k < kGiantSample / 32; k++)
        if (r == cand[k]) atomicAdd(&cnt[k], 1u);
    __syncthreads();
    if (i < kGiantSample / 32) atomicMax(&best, ((unsigned long long)cnt[i] << 32) | (0xFFFFFFFFu - cand[i]));
    __syncthreads();
    if (i == 0) L.giants[blockIdx.x] = 0xFFFFFFFFu - (uint32_t)best;
    if (blockIdx.x == 0 && i == 0) *L.count = 0;
}

// Each vertex's giant memberships, and the bitmap of the vertices that are in the giant of every copy
// (a warp per 32 vertices). The forest need not be flat: walks without writes.
__global__ void approx_members(const Level L) {
    pdl_wait();
    const uint32_t lane = threadIdx.x & 31, C = L.F.copies;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5, words = (L.n + 31) / 32;
    const uint32_t all = C >= 32 ? 0xFFFFFFFFu : (1u << C) - 1;
    for (uint32_t wd = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; wd < words; wd += warps) {
        const uint32_t x = wd * 32 + lane;
        uint32_t in = 0;
        if (x < L.n) {
            if (C == 4) {
                const uint4 p = reinterpret_cast<const uint4 *>(L.F.par)[x];
                const uint32_t g0 = L.F.par[4 * p.x], g1 = L.F.par[4 * p.y + 1];
                const uint32_t g2 = L.F.par[4 * p.z + 2], g3 = L.F.par[4 * p.w + 3];
                const uint4 g = *reinterpret_cast<const uint4 *>(L.giants);
                in = (uint32_t)((g0 == p.x ? g0 : root_of(L.F, 0, g0)) == g.x) |
                     (uint32_t)((g1 == p.y ? g1 : root_of(L.F, 1, g1)) == g.y) << 1 |
                     (uint32_t)((g2 == p.z ? g2 : root_of(L.F, 2, g2)) == g.z) << 2 |
                     (uint32_t)((g3 == p.w ? g3 : root_of(L.F, 3, g3)) == g.w) << 3;
            } else {
                for (uint32_t j = 0; j < C; j++) in |= (uint32_t)(root_of(L.F, j, x) == L.giants[j]) << j;
            }
            L.member[x] = in;
        }
        const uint32_t word = __ballot_sync(0xffffffffu, in == all);
        if (lane == 0) L.bits[wd] = word;
    }
}

__global__ void approx_count_roots(const Forest F, uint32_t n, unsigned int *count) {
    pdl_wait();
    uint32_t c = 0;
    grid_stride(n, [&](uint32_t x) {
        if (F.copies == 4) {
            const uint4 p = reinterpret_cast<const uint4 *>(F.par)[x];
            c += (uint32_t)(p.x == x) + (uint32_t)(p.y == x) + (uint32_t)(p.z == x) + (uint32_t)(p.w == x);
        } else {
            for (uint32_t j = 0; j < F.copies; j++) c += F.at(x, j) == x;
        }
    });
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, c);
}

// Small graphs: one CTA per (copy, level), the copy's forest in shared memory, several levels in one
// launch. A thread takes a quad at a time; links are unions with path halving (shared CAS of the larger
// root onto the smaller). A copy that has become one tree is decided, whatever its other edges: on the dense
// graphs of small n that takes a few n ln n of them. The root count goes to the host's page.
//   Bound by the cipher of the levels that are decided last (all quads) and by the launch and its wait, of
// which there was one of each, and three kernels or more, per level. Level by level over the whole
// device (and, to 2^15 edges, a thread per edge and a block per draw) / here: R-MAT scale 9, m = 2,048 40 / 29 us;
// G(16,000, m = 128,000), 8 levels 623 / 163 us; G(1000, m = 125,000), 10 levels 2.0 ms / 121 us; R-MAT scale 14,
// m = 114,688, disconnected and so decided by its first level 161 / 141 us (75 by rounds, which run no other level).
//   The rule (approx_is_small): the forest fits in 64 KB of shared memory, and one CTA's pass over the edges is
// no longer than two levels of rounds over the whole device (70 us each): with 2^20 edges it would be 0.9 ms.
constexpr uint32_t kSmallThreads = 1024, kSmallN = 16384, kSmallM = 1u << 17;

__device__ __forceinline__ uint32_t small_find(volatile uint32_t *par, uint32_t v) {
    uint32_t p = par[v];
    while (p != v) {
        const uint32_t g = par[p];
        if (g == p) return p;
        par[v] = g;  // (a vertex that is no root never becomes one: any ancestor may be written)
        v = g;
        p = par[v];
    }
    return v;
}

template <bool kRef>
__global__ void __launch_bounds__(kSmallThreads) approx_small(const Level base, uint32_t *__restrict__ roots) {
    extern __shared__ uint32_t par[];
    __shared__ uint32_t s_links;
    __shared__ uint64_t table[kRef ? 1 : kTable];
    Level L = base;
    L.level += blockIdx.y;
    L.keep_max = stream_threshold(L.level);
    const uint32_t j = blockIdx.x, lane = threadIdx.x & 31;
    for (uint32_t v = threadIdx.x; v < L.n; v += kSmallThreads) par[v] = v;
    if (threadIdx.x == 0) s_links = 0;
    if (!kRef) fill_thresholds(table, L.level);
    __syncthreads();
    for (uint32_t q0 = threadIdx.x - lane; q0 < L.Q; q0 += kSmallThreads) {
        // other warps add to the count meanwhile: one lane's look at it decides for the warp, whose lanes
        // meet again in the sum below
        const uint32_t seen = lane == 0 ? *(volatile uint32_t *)&s_links : 0;
        if (__shfl_sync(0xffffffffu, seen, 0) + 1 >= L.n) break;
        uint32_t links = 0;
        if (q0 + lane < L.Q) {
            const Quad q = quad_of(L, q0 + lane);
            const uint32_t mask = quad_keeps<kRef>(L, q, j, table), e0 = q.base + 4 * q.lq;
            uint32_t a[4], b[4];
#pragma unroll
            for (uint32_t d = 0; d < 4; d++) {
                a[d] = b[d] = 0;
                if ((mask >> d) & 1u) {
                    a[d] = __ldg(L.U + e0 + d);
                    b[d] = __ldg(L.V + e0 + d);
                }
            }
#pragma unroll 1
            for (uint32_t d = 0; d < 4; d++) {
                uint32_t x = d == 0 ? a[0] : d == 1 ? a[1] : d == 2 ? a[2] : a[3];
                uint32_t y = d == 0 ? b[0] : d == 1 ? b[1] : d == 2 ? b[2] : b[3];
                while (x != y) {
                    x = small_find(par, x);
                    y = small_find(par, y);
                    if (x == y) break;
                    const uint32_t hi = max(x, y), lo = min(x, y);
                    if (atomicCAS(&par[hi], hi, lo) == hi) {
                        links++;
                        break;
                    }
                }
            }
        }
        links = __reduce_add_sync(0xffffffffu, links);
        if (lane == 0 && links) atomicAdd(&s_links, links);
    }
    __syncthreads();
    if (threadIdx.x == 0) roots[blockIdx.y * gridDim.x + j] = L.n - s_links;
}

// Device memory of one call, given back (in the stream's order) when the call ends.
struct Temporary {
    cac_ctx *ctx;
    void *p = nullptr;
    size_t bytes = 0;
    explicit Temporary(cac_ctx *c) : ctx(c) {}
    Temporary(const Temporary &) = delete;
    Temporary &operator=(const Temporary &) = delete;
    ~Temporary() { stream_free(ctx, p, bytes); }
    int get(size_t n) {
        bytes = n;
        return stream_alloc(ctx, &p, n);
    }
};

bool approx_is_small(uint32_t n, uint64_t m) { return n <= kSmallN && m <= kSmallM; }

// The hooks of one level (the forest already holds singletons).
// Union walks from singletons make long parent chains that every walk then pays for (15 M edges, 4
// copies: 480 us for the first eighth of the edges, 85 us for each of the last). So the forest is built
// in rounds on small parts of the edges, flattened after each: with kRoundDegree kept edges per vertex
// in each, 98.7% of a random graph's vertices are in the giant component after the fifth (counted on
// G(10^6, M); two rounds of twice the edges leave it in small trees). Then some 1.3% of the vertices of
// a copy are outside, about 2.6% of its edges are tested one by one, and the rest cost two bitmap
// lookups for all copies together.
// Bound by: the draws (one or two cipher blocks per quad and copy) and L2 gathers of the rounds at 10^7
// edges, kernel boundaries at 10^6. Measured per query against eight slices of union walks: G(10^6,
// 15.2 M edges), unit weights, 4 copies, 1.97 -> 0.75 ms; G(10^5, 1.4 M edges), weights to 42, six
// levels, 1.79 -> 0.61 ms.
// The rounds need the forest alone, so they come first also where there is no survivor list and every quad
// is tested after them: G(10^6, 15.2 M edges) in a budget without room for it 1.28 ms by slices, 1.74 by one pass from
// singletons, 0.65 so; 37 copies of G(300,000, 3.9 M edges), two levels, 5.6, 15.4 and 4.8 ms.
template <bool kRef>
int run_level(cac_ctx *ctx, Level L, double kept_degree, bool rounds) {
    cudaStream_t s = ctx->stream;
    auto grid = [&](uint64_t work, int per_sm) {
        return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((work + kThreads - 1) / kThreads, (uint64_t)ctx->num_sms * per_sm));
    };
    const unsigned gc = grid(L.F.copies == 4 ? L.n : (uint64_t)L.n * L.F.copies, 8), gq = grid((uint64_t)L.Q * L.F.copies, 8);
    double sum = 0;
    for (double d : kRoundDegree) sum += d;
    if (rounds) {
        double upto = 0;
        L.to = 0;
        for (double d : kRoundDegree) {
            upto += d;
            L.from = L.to;
            L.to = std::min(kSampleParts, (uint32_t)std::ceil(kSampleParts * std::min(1.0, upto / kept_degree)));
            if (L.to == L.from) continue;
            CAC_CUDA_TRY(launch_pdl(approx_quads<kRef, kRound>, gq, kThreads, 0, s, L));
            CAC_CUDA_TRY(launch_pdl(approx_compress, gc, kThreads, 0, s, L.F, L.n));
        }
    }
    if (!L.list || kept_degree < sum) {  // too few edges for a giant component in every copy
        CAC_CUDA_TRY(launch_pdl(approx_quads<kRef, kAll>, gq, kThreads, 0, s, L));
    } else {
        CAC_CUDA_TRY(launch_pdl(approx_giants, L.F.copies, kGiantSample, 0, s, L));
        CAC_CUDA_TRY(launch_pdl(approx_members, gc, kThreads, 0, s, L));
        const uint32_t words = (L.n + 31) / 32;
        const bool shared = words <= kSmemWords;
        auto kern = shared ? approx_stream<kRef, true> : approx_stream<kRef, false>;
        CAC_TRY(smem_optin(ctx, kern));
        const uint64_t tiles = ((uint64_t)L.m + 255) / 256;
        const unsigned gt = (unsigned)std::min<uint64_t>(tiles / (kStreamThreads / 32) + 1, (uint64_t)ctx->num_sms);
        CAC_CUDA_TRY(launch_pdl(kern, gt, kStreamThreads, shared ? words * 4 : 0, s, L));
        CAC_CUDA_TRY(launch_pdl(approx_rest<kRef>, (unsigned)ctx->num_sms * 8, kThreads, 0, s, L));
    }
    CAC_CUDA_TRY(cudaGetLastError());
    return CAC_OK;
}

}  // namespace

// ApproximateCut.cpp:30: (unsigned) ceil(log(w)), w a rank's slice weight (none for w = 0)
static uint32_t level_count(uint64_t w) { return w ? (uint32_t)std::ceil(std::log((double)w)) : 0; }

int approx_run(cac_ctx *ctx, const cac_graph *g, double p, uint32_t seed, uint32_t ranks, bool ref_stream,
               cac_approx_result *res) {
    cudaStream_t s = ctx->stream;
    *res = cac_approx_result{};
    const uint32_t copies = approx_copies(p);
    res->copies = copies;
    const uint64_t nv = (uint64_t)g->n * copies;
    if (nv >= 0xFFFFFFFFull) {
        set_error("approx_cut: n * copies must stay below 2^32");
        return CAC_ERR_UNSUPPORTED;
    }
    const uint64_t portion = g->m / ranks;
    if (ref_stream && !g->unit_weights) {
        set_error("approx_cut seed replay: every edge weight must be 1 (a weighted edge draws a variable number "
                  "of outputs)");
        return CAC_ERR_UNSUPPORTED;
    }
    // Levels: the smallest ceil(ln w_r) over the ranks' slices. More ranks than edges leave every
    // slice but the last empty: no level runs. Unit weights: w_r is the slice length; one rank:
    // the graph's total weight; otherwise the slice sums are taken on the device.
    const bool stats = ranks > 1 && portion > 0 && !g->unit_weights;
    // quads of 4 edges per rank slice
    const uint64_t Qf = (portion + 3) / 4;
    const uint64_t Q = portion == 0 ? (g->m + 3) / 4 : (ranks - 1) * Qf + (g->m - (uint64_t)(ranks - 1) * portion + 3) / 4;
    const bool large = g->m >= kSampledEdges && Q < 0xFFFFFFFFull;
    const size_t base_bytes = align_up(nv * 4 + 4) + 256 + (stats ? align_up((uint64_t)ranks * 8) : 0);
    const uint64_t cap = g->m / 8 + 1024;
    const size_t more = align_up((uint64_t)g->n * 4) + align_up(((uint64_t)g->n + 31) / 32 * 4) +
                        align_up(cap * 8) + 256;
    // the survivor list needs a byte an edge more than the forest: without it (it does not fit the
    // budget, or there are more copies than a mask has bits) every edge is tested after the rounds. Under a budget it is
    // the query's own (5 us a call) and not the arena's, which keeps what it has: room that other calls need
    bool sampled = large && copies <= 32;
    Temporary extra(ctx);
    CAC_TRY(arena_reserve(ctx, base_bytes + (sampled && !ctx->budget ? more : 0)));
    arena_reset(ctx);
    if (sampled && ctx->budget) sampled = ctx->held + more <= ctx->budget && extra.get(more) == CAC_OK;
    uint32_t *par = (uint32_t *)arena_take(ctx, nv * 4 + 4);
    unsigned int *d_count = (unsigned int *)arena_take(ctx, 16);
    CAC_CUDA_TRY(cudaEventRecord(ctx->ev[0], s));
    uint32_t iterations = level_count(g->total_weight);
    if (ranks > 1 && portion == 0) {
        iterations = 0;
    } else if (ranks > 1 && g->unit_weights) {
        iterations = level_count(portion);  // the last slice holds at least `portion` edges
    } else if (stats) {
        unsigned long long *d_sums = (unsigned long long *)arena_take(ctx, (uint64_t)ranks * 8);
        CAC_CUDA_TRY(cudaMemsetAsync(d_sums, 0, (uint64_t)ranks * 8, s));
        const uint64_t longest = g->m - (uint64_t)(ranks - 1) * portion;
        const uint32_t gy = std::min<uint32_t>(ranks, 65535u);
        const uint32_t gx = (uint32_t)std::max<uint64_t>(
            1, std::min<uint64_t>((longest + 4 * kThreads - 1) / (4 * kThreads),
                                  std::max<uint64_t>(1, (uint64_t)ctx->num_sms * 8 / gy)));
        approx_slice_sums<<<dim3(gx, gy), kThreads, 0, s>>>(g->w, g->m, ranks, portion, d_sums);
        CAC_CUDA_TRY(cudaGetLastError());
        std::vector<unsigned long long> h(ranks);  // ranks <= m here
        CAC_CUDA_TRY(cudaMemcpyAsync(h.data(), d_sums, (uint64_t)ranks * 8, cudaMemcpyDeviceToHost, s));
        CAC_CUDA_TRY(cudaStreamSynchronize(s));
        iterations = UINT32_MAX;
        for (uint32_t r = 0; r < ranks; r++) iterations = std::min(iterations, level_count(h[r]));
    }
    const int gi = (int)std::max<uint64_t>(1, std::min<uint64_t>(((copies == 4 ? g->n : nv) + kThreads - 1) / kThreads, ctx->num_sms * 8));
    uint32_t first = 0;
    if (ref_stream) iterations = std::min<uint32_t>(iterations, 52);  // ceil(ln W) <= 45 for W < 2^64
    Level L{};
    L.U = g->u;
    L.V = g->v;
    L.Wt = g->w;
    L.m = (uint32_t)g->m;
    L.n = g->n;
    L.F = Forest{par, copies};
    L.seed = seed;
    L.ranks = ranks;
    L.portion = (uint32_t)portion;
    L.Qf = (uint32_t)Qf;
    L.Q = (uint32_t)Q;
    if (sampled) {
        char *at = static_cast<char *>(extra.p ? extra.p : arena_take(ctx, more));
        auto take = [&](size_t bytes) {
            char *p = at;
            at += align_up(bytes);
            return p;
        };
        L.member = (uint32_t *)take((uint64_t)g->n * 4);
        L.bits = (uint32_t *)take(((uint64_t)g->n + 31) / 32 * 4);
        L.list = (uint2 *)take(cap * 8);
        L.cap = (uint32_t)cap;
        L.giants = (uint32_t *)take(256);
        L.count = L.giants + 32;
    }
    iterations = std::min<uint32_t>(iterations, 63);
    const bool small = approx_is_small(g->n, g->m) && copies <= 8192;  // (the host's page holds a launch's counts)
    if (small) {
        auto kern = ref_stream ? approx_small<true> : approx_small<false>;
        CAC_TRY(smem_optin(ctx, kern));
        // as many levels as fill the device with one CTA per SM
        const uint32_t wide = std::max<uint32_t>(1, std::min<uint32_t>((uint32_t)ctx->num_sms, 8192) / copies);
        for (uint32_t level = 1; level <= iterations && !first; level += wide) {
            const uint32_t here = std::min(wide, iterations + 1 - level);
            L.level = level;
            kern<<<dim3(copies, here), kSmallThreads, (size_t)g->n * 4, s>>>(L, ctx->pinned_u32);
            CAC_CUDA_TRY(cudaGetLastError());
            CAC_CUDA_TRY(cudaStreamSynchronize(s));
            for (uint32_t i = 0; i < here && !first; i++) {
                uint64_t total = 0;
                for (uint32_t j = 0; j < copies; j++) total += ctx->pinned_u32[i * copies + j];
                if (total > copies) first = level + i;
            }
        }
    }
    const double mean_weight = g->m ? (double)g->total_weight / (double)g->m : 0;
    for (uint32_t level = 1; level <= iterations && !small; level++) {
        approx_init<<<gi, kThreads, 0, s>>>(L.F, g->n, d_count);
        L.level = level;
        L.keep_max = stream_threshold(level);  // p = 2^-level (ApproximateCut.cpp:37)
        if (g->m) {
            const double kept = 1 - std::pow(1 - std::ldexp(1.0, -(int)level), mean_weight);  // share of the edges
            const double degree = 2.0 * g->m * kept / std::max<uint32_t>(1, g->n);
            CAC_TRY(ref_stream ? run_level<true>(ctx, L, degree, large) : run_level<false>(ctx, L, degree, large));
        }
        CAC_CUDA_TRY(launch_pdl(approx_count_roots, (unsigned)gi, kThreads, 0, s, L.F, g->n, d_count));
        CAC_CUDA_TRY(cudaGetLastError());
        CAC_CUDA_TRY(cudaMemcpyAsync(ctx->pinned_u32, d_count, 4, cudaMemcpyDeviceToHost, s));
        CAC_CUDA_TRY(cudaStreamSynchronize(s));
        if (ctx->pinned_u32[0] > copies) {
            first = level;
            break;
        }
    }
    CAC_CUDA_TRY(cudaEventRecord(ctx->ev[1], s));
    CAC_CUDA_TRY(cudaStreamSynchronize(s));
    CAC_CUDA_TRY(cudaEventElapsedTime(&res->device_ms, ctx->ev[0], ctx->ev[1]));
    res->level = first;
    res->cut = 1ull << first;
    res->trials = copies * first;
    return CAC_OK;
}

}  // namespace cac
