// Connected components: the GB300 form of the reference's iterated-sparse-sampling CC
// (src/UnweightedIteratedSparseSampling.cpp:40-72, src/IteratedSparseSampling.hpp:160-295).
//
// Reference round structure            ->  here
//   root scatters per-rank draw counts    host restates edgesToSamplePerProcessor (cc_plan)
//   rank r draws engine()%slice samples   cc_sample_draws / cc_sample_round: sitmo stream
//     with sitmo(seed + r)                  (seed + r, 0, 0, 0), output k = word k % 8 of block
//                                           k / 8, the reference's k-th engine output; it picks
//                                           a 32-edge chunk of the slice (coalesced) instead of
//                                           one edge
//   root: shuffle + prefix union-find     rounds of root links in HBM (the smallest root an edge
//     to one component (Boost sets)         leads to becomes the parent), flattened in between
//   bcast map, rewrite slice, drop loops  cc_edge_pass: one streaming pass over every edge;
//     and repeat while edges remain         edges whose endpoints already share a root are the
//                                           dropped loops, the rest hook (the final round): lock-
//                                           free union-find (atomicCAS hooking of the larger root
//                                           under the smaller, so roots are component minima)
//   relabel by first appearance           roots = minima, so label = exclusive scan of the
//                                           root flags (label_components)
//
// Memory layout in HBM: edge endpoints as two uint32 arrays u[m], v[m] (structure of arrays,
// 16-byte vector loads, 4 edges per load pair); parent[n] uint32 (L2-resident for n up to
// tens of millions: 129 MB of L2); per-tile root counts; labels[n].
#include "cac_internal.h"
#include "grid_loop.cuh"
#include "pdl.cuh"
#include "sitmo.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>
#include <type_traits>

namespace cac {
namespace {

constexpr int kThreads = 256;
constexpr int kTileItems = 4;                        // vertices per thread in the labelling tiles
constexpr int kTile = kThreads * kTileItems;         // vertices per labelling tile
constexpr size_t kPinnedBytes = 60 * 1024;           // ctx pinned staging available for rank descriptors
constexpr int kEdgeThreads = 1024;                   // closing-pass CTA (one per SM: the bitmap fills smem)
constexpr uint32_t kSmemBitmapWords = 48 * 1024;     // 192 KB of bitmap in shared memory (1.57M vertices)
constexpr uint32_t kGiantSample = 1024;              // vertices sampled to find the giant component
constexpr uint32_t kSampleChunk = 32;                // consecutive edges behind one sampling draw
// Edges per vertex (as degrees: half as many) in each round of forest building. Union walks from
// singletons make long parent chains that every walk then pays for, so the forest is built in rounds on
// disjoint parts of the edges, flattened after each; in a round every edge between two roots makes the
// smaller one the parent of the larger, the smallest of all winning. With these sizes 98.7% of a
// random graph's vertices are in the giant component after the fifth (counted on G(10^6, M); two rounds
// of twice the edges leave it in small trees).
constexpr double kRoundDegree[] = {0.8, 0.8, 0.8, 0.8, 1.6};
constexpr uint32_t kRoundParts = 128;                // without draws: rounds are 128ths of the 256-edge tiles
// Without draws, smaller or sparser graphs hook every edge in one pass (up to one edge per vertex at each
// end a random graph has small trees only, and disjoint edges have no more): G(10^6, M) with average degree 0.1 takes 41 us
// in one pass and 48 in rounds, with 1.05 93 and 84, with 3 863 and 127, G(17000, M) with degree 2 87 and 66; a perfect
// matching of 300,000 vertices 33 and 46, of 10^6 relabelled 49 and 69.
constexpr uint64_t kRoundEdges = 1u << 13;
// Between these average degrees, and while the forest lies in the L2 (64 MB), the rounds are those of sparse_rounds, of
// kFullRounds - 1 below kFewRoundEdges edges. Device us by them and by edge_rounds: G(10^6, M) of degree 1 86 and 81, 1.25
// 106 and 118, 2.25 145 and 626, 2.5 147 and 118, 3 167 and 121; a 1000 x 1000 grid (4) 132 and 110. Degree 2 on 16 M
// vertices 1165 and 1416, on 20 M 1554 and 1870, on 26 M 2379 and 2249; degree 2.3 1287 and 1625, 1720 and 1477, 2632 and 2259.
constexpr double kSparseLow = 1.2, kSparseDegree = 2.4;
constexpr uint32_t kSparseVertices = 1u << 24;
constexpr uint64_t kFewRoundEdges = 1u << 18;
constexpr uint32_t kProbes = 128;
constexpr int kHops = 32;                            // longest walk of a compression between rounds
constexpr int kRoundThreads = 1024;                  // CTA of a round: the more threads, the more links the table sees
constexpr uint32_t kMaxRegions = 1024;               // filter CTAs (regions of the survivor buffer)
// survivor-hook CTAs per SM: about one survivor per thread on BA n=1,024,000 (0.6 M survivors);
// 8 against 4: 20 vs 22.5 us there, 47 vs 63.5 us on R-MAT scale 22; 16 no better
constexpr unsigned kSurvivorBlocksPerSm = 8;
constexpr uint32_t kStreamPieces = 8;                // sample pieces (and gaps) of a host edge list
constexpr uint32_t kErrWord = 9;                     // a query's error word (after its count and giant root)
constexpr uint32_t kErrBadId = 1;                    // an edge endpoint was >= n (the edge was skipped)
constexpr uint32_t kFullRounds = 4;                  // most rounds of sparse_rounds after its first
constexpr uint32_t kOpenWord = 10;                   // the open edges that each of them found
constexpr uint32_t kQueryWords = kOpenWord + kFullRounds;  // words in use of the total's 64

struct RankDesc {
    uint64_t slice_off;
    uint64_t slice_len;
    uint64_t draws;      // chunk draws of this rank
    uint64_t block_off;  // first sitmo block (8 chunk draws) of this rank in the flattened launch
    uint64_t draw_off;   // first chunk draw of this rank in the flattened draw list
    uint32_t key0;       // seed + rank
    uint32_t pad;
};

// Root of v with path halving. Invariant: parent[x] <= x, roots satisfy parent[r] == r.
__device__ __forceinline__ uint32_t find_root(uint32_t *par, uint32_t v) {
    uint32_t cur = par[v];
    if (cur != v) {
        uint32_t prev = v, next;
        while (cur > (next = par[cur])) {
            par[prev] = next;
            prev = cur;
            cur = next;
        }
    }
    return cur;
}

// Root of v without writes. Used where no hooking happens any more: a path-halving write by
// one thread could otherwise overwrite another thread's just-stored `parent[i] = root` with a
// non-root ancestor and leave i uncompressed.
__device__ __forceinline__ uint32_t find_root_ro(const uint32_t *par, uint32_t v) {
    uint32_t cur = v, next;
    while ((next = par[cur]) != cur) cur = next;
    return cur;
}

// Merge the sets of a and b: hook the larger representative under the smaller with CAS;
// a failed CAS returns the node's new parent and the walk continues from there.
__device__ __forceinline__ void unite(uint32_t *par, uint32_t a, uint32_t b) {
    uint32_t ra = find_root(par, a), rb = find_root(par, b);
    while (ra != rb) {
        if (ra < rb) {
            uint32_t old = atomicCAS(&par[rb], rb, ra);
            if (old == rb) return;
            rb = old;
        } else {
            uint32_t old = atomicCAS(&par[ra], ra, rb);
            if (old == ra) return;
            ra = old;
        }
    }
}

__device__ __forceinline__ void edge_hook(uint32_t *par, uint32_t a, uint32_t b) {
    const uint32_t pa = par[a], pb = par[b];
    if (pa == pb) return;  // already one component: the reference drops this edge as a loop
    unite(par, pa, pb);
}

// Edge lists handed in by the caller (host arrays of cac_cc_edges, device arrays of
// cac_cc_noalloc) are not validated beforehand: an endpoint >= n skips the edge and sets the
// query's error word instead of indexing past the parent array.
template <bool kCheck>
__device__ __forceinline__ void edge_hook_checked(uint32_t *par, uint32_t a, uint32_t b, uint32_t n, uint32_t *err) {
    if (kCheck && (a >= n || b >= n)) {
        atomicOr(err, kErrBadId);
        return;
    }
    edge_hook(par, a, b);
}

__global__ void cc_init(uint32_t *par, uint32_t n) {
    pdl_wait();
    grid_stride(n, [&](uint32_t i) { par[i] = i; });
}

// The draws of the sampling round, one thread per sitmo block (8 draws of one rank). The reference
// draws single edges (engine() % slice, a random 8-byte gather each); here draw k of rank r
// (32-bit output k of stream (seed + r, 0, 0, 0), word k % 8 of block k / 8) selects chunk
// (output % chunks) of kSampleChunk consecutive edges of the rank's slice. The chunk is stored as
// (first edge | edge count << 32) at the draw's flattened index.
__global__ void cc_sample_draws(const RankDesc *__restrict__ ranks, int nranks, uint64_t nblocks,
                                uint64_t *__restrict__ chunks) {
    pdl_wait();
    for (uint64_t gb = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; gb < nblocks;
         gb += (uint64_t)gridDim.x * blockDim.x) {
        int lo = 0, hi = nranks - 1;  // last rank whose first block <= gb
        while (lo < hi) {
            int mid = (lo + hi + 1) >> 1;
            if (ranks[mid].block_off <= gb) lo = mid; else hi = mid - 1;
        }
        const RankDesc rd = ranks[lo];
        const uint64_t blk = gb - rd.block_off;  // sitmo block index within the rank's stream
        const u64x4 o = sitmo_block(rd.key0, 0, 0, 0, blk, 0, 0, 0);
        const uint64_t nchunks = (rd.slice_len + kSampleChunk - 1) / kSampleChunk;
        const uint64_t end = rd.slice_off + rd.slice_len;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const uint64_t k = blk * 8 + j;
            if (k >= rd.draws) break;  // rd.draws counts chunk draws
            const uint64_t word = o.x[j >> 1];
            const uint32_t x = (j & 1) ? (uint32_t)(word >> 32) : (uint32_t)word;
            const uint64_t first = rd.slice_off + (x % nchunks) * kSampleChunk;
            const uint64_t count = min((uint64_t)kSampleChunk, end - first);
            chunks[rd.draw_off + k] = first | (count << 32);
        }
    }
}

// The links of one CTA's part of a round, gathered in shared memory: root -> smallest root it is linked
// to. Late rounds have few large trees, whose roots would take thousands of atomics from every CTA at
// once; here each takes one. A root whose entry belongs to another is linked in memory directly; the roots
// of kProbes vertices, among which the large trees are, get their entries first.
template <uint32_t kLinks>  // a power of two
struct Links {
    uint32_t key[kLinks], val[kLinks];
    static __device__ __forceinline__ uint32_t entry(uint32_t r) { return (uint32_t)(((uint64_t)(r * 2654435761u) * kLinks) >> 32); }
    __device__ __forceinline__ void clear() {
        for (uint32_t i = threadIdx.x; i < kLinks; i += blockDim.x) key[i] = val[i] = 0xFFFFFFFFu;
        __syncthreads();
    }
    __device__ __forceinline__ void claim_large(const uint32_t *par, uint32_t n) {
        if (threadIdx.x < kProbes) {
            const uint32_t r = par[(uint32_t)(((uint64_t)(threadIdx.x * 0x9E3779B9u) * n) >> 32)];
            atomicCAS(&key[entry(r)], 0xFFFFFFFFu, r);
        }
        __syncthreads();
    }
    // a and b: parents of an edge's ends in a flat forest
    __device__ __forceinline__ void add(uint32_t *par, uint32_t a, uint32_t b) {
        if (a == b) return;
        const uint32_t hi = max(a, b), lo = min(a, b), x = entry(hi);
        uint32_t k = *(volatile uint32_t *)&key[x];
        if (k == 0xFFFFFFFFu) k = atomicCAS(&key[x], 0xFFFFFFFFu, hi);
        if (k != hi && k != 0xFFFFFFFFu) atomicMin(&par[hi], lo);
        else if (*(volatile uint32_t *)&val[x] > lo) atomicMin(&val[x], lo);
    }
    __device__ __forceinline__ void flush(uint32_t *par) {
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < kLinks; i += blockDim.x)
            if (val[i] != 0xFFFFFFFFu) atomicMin(&par[key[i]], val[i]);
    }
};

// The first round: every vertex is still its own root, and any smaller end will do as its parent (a
// store; hubs take thousands of links here, and atomics on them took 110 us on R-MAT scale 22).
__device__ __forceinline__ void first_link(uint32_t *par, uint32_t a, uint32_t b) {
    if (a != b) par[max(a, b)] = min(a, b);
}

// One round on the chunks of the draw range [d0, d1): a warp takes two chunks at a time (coalesced loads
// of their edges, all in flight together).
template <bool kFirst, bool kCheck>
__global__ void __launch_bounds__(kRoundThreads, 2) cc_sample_round(uint32_t *par, const uint32_t *__restrict__ u,
                                                            const uint32_t *__restrict__ v,
                                                            const uint64_t *__restrict__ chunks, uint64_t d0, uint64_t d1,
                                                            uint32_t n, uint32_t *err) {
    __shared__ typename std::conditional<kFirst, char, Links<4 * kRoundThreads>>::type links;
    if constexpr (!kFirst) links.clear();
    pdl_wait();
    if constexpr (!kFirst) links.claim_large(par, n);
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t d = d0 + (((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5); d < d1; d += 2 * warps) {
        uint64_t c[2];
        uint32_t a[2], b[2];
#pragma unroll
        for (int k = 0; k < 2; k++) c[k] = d + k * warps < d1 ? chunks[d + k * warps] : 0;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            a[k] = b[k] = 0;
            if (lane < (uint32_t)(c[k] >> 32)) {
                const uint64_t e = (c[k] & 0xFFFFFFFFull) + lane;
                a[k] = __ldg(u + e);
                b[k] = __ldg(v + e);
                if (kCheck && (a[k] >= n || b[k] >= n)) {
                    atomicOr(err, kErrBadId);
                    a[k] = b[k] = 0;
                }
            }
        }
        if (!kFirst) {
#pragma unroll
            for (int k = 0; k < 2; k++) {
                a[k] = par[a[k]];
                b[k] = par[b[k]];
            }
        }
#pragma unroll
        for (int k = 0; k < 2; k++) {
            if constexpr (kFirst) first_link(par, a[k], b[k]);
            else links.add(par, a[k], b[k]);
        }
    }
    if constexpr (!kFirst) links.flush(par);
}

// Rounds on the edges that an earlier round left open (their ends under different parents): what comes after one
// that found few of them is left out.
struct OpenCount {
    const uint32_t *before = nullptr;  // the open edges that the round before found, or null: not to be left out
    uint32_t few = 0;
    __device__ __forceinline__ bool skip() const { return before && *before <= few; }
};

// One round on the 256-edge tiles t with from <= t % kRoundParts < to, a warp per tile, its lane l on
// edges l, 32 + l, ... (all loads of the eight in flight together).
template <bool kFirst, bool kCheck, int kNT>
__global__ void __launch_bounds__(kNT, 2048 / kNT) cc_edge_round(uint32_t *par, const uint32_t *__restrict__ u,
                                                          const uint32_t *__restrict__ v, uint64_t m, uint32_t from,
                                                          uint32_t to, uint32_t n, uint32_t *err) {
    __shared__ typename std::conditional<kFirst, char, Links<4 * kNT>>::type links;
    if constexpr (!kFirst) links.clear();
    pdl_wait();
    if constexpr (!kFirst && kNT == kRoundThreads) links.claim_large(par, n);
    const uint32_t lane = threadIdx.x & 31, w = to - from;
    const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5, tiles = (m + 255) / 256;
    for (uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;; i += warps) {
        const uint64_t t = i / w * kRoundParts + from + i % w;
        if (t >= tiles) break;
        uint32_t a[8], b[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const uint64_t e = t * 256 + 32 * k + lane;
            a[k] = b[k] = 0;
            if (e < m) {
                a[k] = __ldg(u + e);
                b[k] = __ldg(v + e);
            }
            if (kCheck && (a[k] >= n || b[k] >= n)) {
                atomicOr(err, kErrBadId);
                a[k] = b[k] = 0;
            }
        }
        if (!kFirst) {
#pragma unroll
            for (int k = 0; k < 8; k++) {
                a[k] = par[a[k]];
                b[k] = par[b[k]];
            }
        }
#pragma unroll
        for (int k = 0; k < 8; k++) {
            if constexpr (kFirst) first_link(par, a[k], b[k]);
            else links.add(par, a[k], b[k]);
        }
    }
    if constexpr (!kFirst) links.flush(par);
}

// One round on all edges, a CTA per contiguous range of tiles, which writes the open ones (as the pairs of
// their ends' parents) to its region of `list`, as cc_filter does with its survivors.
template <bool kCheck, int kNT>
__global__ void __launch_bounds__(kNT, 2048 / kNT) cc_open_edges(uint32_t *par, const uint32_t *__restrict__ u,
                                                          const uint32_t *__restrict__ v, uint64_t m, uint32_t n,
                                                          uint2 *__restrict__ list, uint32_t *__restrict__ counts,
                                                          uint32_t *open, uint32_t *err) {
    __shared__ Links<4 * kNT> links;
    __shared__ uint32_t s_n;
    links.clear();
    if (threadIdx.x == 0) s_n = 0;
    pdl_wait();
    if (kNT == kRoundThreads) links.claim_large(par, n);
    else __syncthreads();
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t tiles = (m + 255) / 256, per = (tiles + gridDim.x - 1) / gridDim.x;
    const uint64_t t0 = min(tiles, (uint64_t)blockIdx.x * per), t1 = min(tiles, t0 + per);
    uint2 *out = list + t0 * 256;
    for (uint64_t t = t0 + (threadIdx.x >> 5); t < t1; t += kNT / 32) {
        uint32_t a[8], b[8], mine = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const uint64_t e = t * 256 + 32 * k + lane;
            a[k] = b[k] = 0;
            if (e < m) {
                a[k] = __ldg(u + e);
                b[k] = __ldg(v + e);
            }
            if (kCheck && (a[k] >= n || b[k] >= n)) {
                atomicOr(err, kErrBadId);
                a[k] = b[k] = 0;
            }
        }
#pragma unroll
        for (int k = 0; k < 8; k++) {
            a[k] = par[a[k]];
            b[k] = par[b[k]];
        }
#pragma unroll
        for (int k = 0; k < 8; k++) {
            mine += a[k] != b[k];
            links.add(par, a[k], b[k]);
        }
        if (!__any_sync(0xffffffffu, mine)) continue;
        uint32_t incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += y;
        }
        uint32_t at = 0;
        if (lane == 31) at = atomicAdd(&s_n, incl);
        at = __shfl_sync(0xffffffffu, at, 31) + incl - mine;
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (a[k] != b[k]) out[at++] = make_uint2(a[k], b[k]);
    }
    links.flush(par);
    if (threadIdx.x == 0) {
        counts[blockIdx.x] = s_n;
        if (s_n) atomicAdd(open, s_n);
    }
}

// An ancestor of v, the root unless it is more than kHops away.
__device__ __forceinline__ uint32_t find_near(const uint32_t *par, uint32_t v) {
    uint32_t cur = v, next;
    for (int k = 0; k < kHops && (next = par[cur]) != cur; k++) cur = next;
    return cur;
}

// Compression between the rounds, 4 consecutive vertices per thread: one 16-byte load of their parents,
// then the grandparents of all four requested together (most chains end there), then the longer chains;
// one 16-byte store. The last n % 4 vertices are done one by one. Walks end after kHops parents: a path
// whose vertices are numbered along it makes chains of its own length, and walking these to the end
// took 9 ms for 300,000 vertices; cut short, every compression divides the depth by kHops. The rounds
// do not need a flat forest: a link made at a vertex that is no root any more replaces that vertex's
// parent by another vertex of its component, and what that separates is joined again by the passes over
// all edges.
__global__ void cc_compress4(uint32_t *par, uint32_t n, const OpenCount left) {
    pdl_wait();
    if (left.skip()) return;
    uint4 *p4 = reinterpret_cast<uint4 *>(par);
    const uint32_t n4 = n / 4;
    if (blockIdx.x == 0 && threadIdx.x < (n & 3u)) {
        const uint32_t x = 4 * n4 + threadIdx.x;
        par[x] = find_near(par, x);
    }
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += gridDim.x * blockDim.x) {
        const uint4 p = p4[i];
        const uint32_t v0 = 4 * i;
        uint32_t r0 = p.x, r1 = p.y, r2 = p.z, r3 = p.w;
        const uint32_t g0 = r0 != v0 ? par[r0] : r0, g1 = r1 != v0 + 1 ? par[r1] : r1;
        const uint32_t g2 = r2 != v0 + 2 ? par[r2] : r2, g3 = r3 != v0 + 3 ? par[r3] : r3;
        r0 = g0 == r0 ? r0 : find_near(par, g0);
        r1 = g1 == r1 ? r1 : find_near(par, g1);
        r2 = g2 == r2 ? r2 : find_near(par, g2);
        r3 = g3 == r3 ? r3 : find_near(par, g3);
        if (r0 != p.x || r1 != p.y || r2 != p.z || r3 != p.w) p4[i] = make_uint4(r0, r1, r2, r3);
    }
}

// Compression of [0, n) (the parent array is 256-byte aligned).
void compress_all(cac_ctx *ctx, uint32_t *par, uint32_t n, cudaStream_t s, OpenCount left = {});

// A byte per 32 vertices, a bit per four of them (read as words): for graphs whose bitmap does not fit in
// shared memory. They take no scratch of their own (the arena keeps what it once had, and under a budget other
// calls need the room), but lie in memory that is idle between the sample and the labels: `spare`, of `bytes`.
size_t quad_bytes(uint32_t nwords) { return nwords > kSmemBitmapWords ? (size_t)(nwords + 3) / 4 * 4 : 0; }
uint8_t *quads_in(void *spare, size_t bytes, uint32_t nwords) {
    const size_t need = quad_bytes(nwords);
    return need && need <= bytes ? static_cast<uint8_t *>(spare) : nullptr;
}

// The end of the sampling round in one launch: full compression, the giant component and its
// membership bitmap. Every CTA (kGiantSample threads) first finds the giant itself, from the
// roots of the same kGiantSample vertices (fixed spread of positions): every warp finds the mode
// of its 32 samples (__match_any_sync groups equal roots; ties to the smaller root), each of those
// 32 candidates is counted over all samples with shared atomics, and the candidate with the
// largest count wins (ties: the smaller root). The walks only read and no hook runs during this
// kernel, so every CTA sees the same roots and picks the same giant. The choice only decides which
// edges the filter can drop, never the labels. Then its warps take 32-vertex words: each lane walks its vertex to the root,
// writes the root back when it differs (only roots are written, as in cc_compress4), and the
// warp's ballot of (root == giant) is the word. CTA 0 records the giant for the next kernels.
__global__ void __launch_bounds__(kGiantSample) cc_compress_giant_bitmap(uint32_t *par, uint32_t n, uint32_t *giant,
                                                                         uint32_t *bits, uint8_t *quads) {
    pdl_wait();
    __shared__ uint32_t cand[kGiantSample / 32], cnt[kGiantSample / 32];
    __shared__ unsigned long long best;
    const uint32_t i = threadIdx.x, lane = i & 31, w = i >> 5;
    const uint32_t r = find_root_ro(par, (uint32_t)(((uint64_t)i * 2654435761u) % n));
    const uint32_t same = __match_any_sync(0xffffffffu, r);
    const uint32_t c = __popc(same);
    const uint32_t top = __reduce_max_sync(0xffffffffu, c);
    const uint32_t lo = __reduce_max_sync(0xffffffffu, c == top ? 0xFFFFFFFFu - r : 0u);
    if (lane == 0) {
        cand[w] = 0xFFFFFFFFu - lo;
        cnt[w] = 0;
    }
    if (i == 0) best = 0;
    __syncthreads();
#pragma unroll 8
    for (uint32_t k = 0; k < kGiantSample / 32; k++)
        if (r == cand[k]) atomicAdd(&cnt[k], 1u);
    __syncthreads();
    if (i < kGiantSample / 32)
        atomicMax(&best, ((unsigned long long)cnt[i] << 32) | (0xFFFFFFFFu - cand[i]));
    __syncthreads();
    const uint32_t g = 0xFFFFFFFFu - (uint32_t)(best & 0xFFFFFFFFu);
    if (blockIdx.x == 0 && i == 0) *giant = g;
    const uint64_t nw = ((uint64_t)n + 31) / 32;
    const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t wd = ((uint64_t)blockIdx.x * blockDim.x + i) >> 5; wd < nw; wd += warps) {
        const uint64_t x = wd * 32 + lane;
        bool in = false;
        if (x < n) {
            const uint32_t p = par[x];
            const uint32_t root = p == (uint32_t)x ? p : find_root_ro(par, p);
            if (root != p) par[x] = root;
            in = root == g;
        }
        const uint32_t word = __ballot_sync(0xffffffffu, in);
        if (lane == 0) bits[wd] = word;
        if (quads && lane == 0) {  // a bit per four vertices: all of them are in the giant
            uint32_t b = word & (word >> 1);
            b &= b >> 2;
            b &= 0x11111111u;
            b = (b | b >> 3) & 0x03030303u;
            b = (b | b >> 6) & 0x000F000Fu;
            quads[wd] = (uint8_t)(b | b >> 12);
        }
    }
}

// Closing pass without a sampling round: every edge hooks, 4 edges per thread step through
// 16-byte streaming loads. kFlat: after rounds, when most edges have found equal parents: the 8 parents are requested
// together. From singletons the walks make the forest as they go, and what one has read before the others' links
// is old by then (cac_cc_noalloc, which has this pass alone: paths of 10^6 vertices numbered along them 0.22 ms an edge at a
// time and 0.42 with parents ahead, backwards 5.5 and 16.3; 62,500 disjoint cliques of 16 0.31 and 0.27).
template <bool kVec, bool kCheck, bool kFlat>
__global__ void __launch_bounds__(kThreads) cc_edge_pass(uint32_t *par, const uint32_t *__restrict__ u,
                                                         const uint32_t *__restrict__ v, uint64_t m, uint32_t n,
                                                         uint32_t *err) {
    pdl_wait();
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint64_t done = 0;
    if (kVec) {
        const uint64_t m4 = m >> 2;
        const uint4 *u4 = reinterpret_cast<const uint4 *>(u);
        const uint4 *v4 = reinterpret_cast<const uint4 *>(v);
        for (uint64_t i = tid; i < m4; i += stride) {
            const uint4 qa = __ldcs(u4 + i), qb = __ldcs(v4 + i);
            uint32_t a[4] = {qa.x, qa.y, qa.z, qa.w}, b[4] = {qb.x, qb.y, qb.z, qb.w};
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (kCheck && (a[k] >= n || b[k] >= n)) {
                    atomicOr(err, kErrBadId);
                    a[k] = b[k] = 0;
                }
            if (kFlat) {
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    a[k] = par[a[k]];
                    b[k] = par[b[k]];
                }
#pragma unroll
                for (int k = 0; k < 4; k++)  // (equal parents: one component already, the reference drops the edge as a loop)
                    if (a[k] != b[k]) unite(par, a[k], b[k]);
            } else {
#pragma unroll
                for (int k = 0; k < 4; k++) edge_hook(par, a[k], b[k]);
            }
        }
        done = m4 << 2;
    }
    for (uint64_t e = done + tid; e < m; e += stride)
        edge_hook_checked<kCheck>(par, __ldcs(u + e), __ldcs(v + e), n, err);
}

// Filter pass after the sampling round (the reference's slice rewrite that drops loops,
// IteratedSparseSampling.hpp:160-172): a pure streaming read of every edge; edges with both
// endpoints in the giant component are dropped, the others are appended to this CTA's region of
// `surv` (region = the CTA's contiguous range of 256-edge tiles, so no global counter is
// contended). A warp owns a tile: lane l reads edges 4l..4l+3 and 128+4l..128+4l+3 of it with
// two fully coalesced 512-byte loads per endpoint array, keeps 8 edges in flight, and appends its
// survivors after one warp scan and one shared-memory atomic.
//   The membership bitmap is staged in shared memory. Above kSmemBitmapWords it does not fit: a lane
// whose word is elsewhere makes a 32-byte access of the L2 each time, and these bound the pass (R-MAT scale 22,
// 30% of the endpoints: 262 us). Staged instead is the bitmap of whole quads of vertices in the
// giant (up to 6.3 M vertices; the ids beyond it, and those of other quads, are looked up in the full one): 98% of
// R-MAT's endpoints are in such quads although 40% of its vertices are isolated, since a vertex and its
// neighbours in the numbering have like degrees. Where few are (a giant of half the vertices, spread
// evenly), the first part of the full bitmap is the better one: a CTA counts what its first two tiles per
// warp find in the quads and takes the other if that is less than the share of ids it would hold.
// R-MAT scale 22, 67 M edges: 204 us (the full bitmap's first part alone 262 us).
template <bool kAllSmem, bool kCheck>
__global__ void __launch_bounds__(kEdgeThreads) cc_filter(const uint32_t *__restrict__ u,
                                                          const uint32_t *__restrict__ v, uint64_t tiles,
                                                          const uint32_t *__restrict__ gbits, uint32_t nwords,
                                                          const uint32_t *__restrict__ quads, uint2 *__restrict__ surv, uint32_t *__restrict__ counts,
                                                          uint32_t n, uint32_t *err) {
    pdl_wait();
    extern __shared__ uint32_t sbits[];
    __shared__ uint32_t s_n, s_found;
    const uint32_t swords = min(nwords, (uint32_t)kSmemBitmapWords);
    // words staged: of the quads' bitmap first, where the full one does not fit
    uint32_t qwords = kAllSmem || !quads ? 0u : min((nwords + 3) / 4, (uint32_t)kSmemBitmapWords);
    if (!qwords)
        for (uint32_t i = threadIdx.x; i < swords; i += blockDim.x) sbits[i] = gbits[i];
    else
        for (uint32_t i = threadIdx.x; i < qwords; i += blockDim.x) sbits[i] = quads[i];
    if (threadIdx.x == 0) s_n = s_found = 0;
    __syncthreads();
    const uint64_t per = (tiles + gridDim.x - 1) / gridDim.x;
    const uint64_t t0 = min(tiles, (uint64_t)blockIdx.x * per), t1 = min(tiles, t0 + per);
    uint2 *out = surv + t0 * 256;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    // the word that holds x's bit, or all ones if its quad is in the giant (loads are predicated, not
    // branched to: those of the 16 endpoints of a lane's tile are in flight together)
    auto look = [&](uint32_t x) -> uint32_t {
        const uint32_t w = x >> 5;
        if (kAllSmem) return sbits[w];
        const uint32_t at = qwords ? x >> 7 : w, staged = qwords ? qwords : swords;
        uint32_t word = sbits[at < staged ? at : 0];
        const bool known = at < staged && (!qwords || (word >> (x >> 2 & 31)) & 1u);
        if (qwords) word = 0xFFFFFFFFu;
        if (!known) word = __ldg(gbits + w);
        return word;
    };
    const uint4 *u4 = reinterpret_cast<const uint4 *>(u);
    const uint4 *v4 = reinterpret_cast<const uint4 *>(v);
    auto process = [&](const uint4 &ua, const uint4 &ub, const uint4 &va, const uint4 &vb) {
        const uint32_t a[8] = {ua.x, ua.y, ua.z, ua.w, ub.x, ub.y, ub.z, ub.w};
        const uint32_t b[8] = {va.x, va.y, va.z, va.w, vb.x, vb.y, vb.z, vb.w};
        uint32_t keep = 0, bad = 0;
        uint32_t wa[8], wb[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const bool ok = !kCheck || (a[k] < n && b[k] < n);  // an invalid edge is neither tested nor kept
            bad |= !ok;
            wa[k] = look(ok ? a[k] : 0u);
            wb[k] = look(ok ? b[k] : 0u);
            if (kCheck && !ok) wa[k] = wb[k] = 0xFFFFFFFFu;
        }
#pragma unroll
        for (int k = 0; k < 8; k++) keep |= (~((wa[k] >> (a[k] & 31)) & (wb[k] >> (b[k] & 31))) & 1u) << k;
        if (kCheck && bad) atomicOr(err, kErrBadId);
        const uint32_t cnt = __popc(keep);
        uint32_t incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
        if (total == 0) return;
        uint32_t base = 0;
        if (lane == 31) base = atomicAdd(&s_n, total);
        base = __shfl_sync(0xffffffffu, base, 31) + incl - cnt;
#pragma unroll
        for (int k = 0; k < 8; k++)
            if ((keep >> k) & 1u) out[base++] = make_uint2(a[k], b[k]);
    };
    // two tiles per warp step: all eight 512-byte loads are issued before either tile is used
    auto step = [&](uint64_t t) {
        const bool two = t + 1 < t1;
        const uint4 z = make_uint4(0, 0, 0, 0);
        const uint4 ua = __ldcs(u4 + t * 64 + lane), ub = __ldcs(u4 + t * 64 + 32 + lane);
        const uint4 va = __ldcs(v4 + t * 64 + lane), vb = __ldcs(v4 + t * 64 + 32 + lane);
        const uint4 uc = two ? __ldcs(u4 + (t + 1) * 64 + lane) : z, ud = two ? __ldcs(u4 + (t + 1) * 64 + 32 + lane) : z;
        const uint4 vc = two ? __ldcs(v4 + (t + 1) * 64 + lane) : z, vd = two ? __ldcs(v4 + (t + 1) * 64 + 32 + lane) : z;
        process(ua, ub, va, vb);
        if (two) process(uc, ud, vc, vd);
    };
    uint64_t t = t0 + 2 * (uint64_t)warp;
    if constexpr (!kAllSmem) {
        // what the quads would find in the CTA's first tiles (one endpoint in eight)
        uint32_t found = 0;
        if (t < t1) {
            const uint32_t x[2] = {__ldg(u + t * 256 + 4 * lane), __ldg(v + t * 256 + 4 * lane)};
#pragma unroll
            for (int k = 0; k < 2; k++) found += x[k] >> 7 < qwords && (sbits[x[k] >> 7] >> (x[k] >> 2 & 31)) & 1u;
        }
        found = __reduce_add_sync(0xffffffffu, found);
        if (lane == 0 && found) atomicAdd(&s_found, found);
        const uint64_t warps_in = t1 > t0 ? min((uint64_t)nwarps, (t1 - t0 + 1) / 2) : 0;
        __syncthreads();
        if (qwords && (uint64_t)s_found * nwords < 64 * warps_in * swords) {
            __syncthreads();
            for (uint32_t i = threadIdx.x; i < swords; i += blockDim.x) sbits[i] = gbits[i];
            qwords = 0;
            __syncthreads();
        }
    }
    for (; t < t1; t += 2 * (uint64_t)nwarps) step(t);
    __syncthreads();
    if (threadIdx.x == 0) counts[blockIdx.x] = s_n;
}

// Exclusive prefix of the region counts: four per thread, then a block scan of the sums.
__device__ __forceinline__ void region_prefix(const uint32_t *__restrict__ counts, uint32_t nregions, uint32_t *pre) {
    __shared__ uint32_t wsum[kThreads / 32];
    static_assert(kMaxRegions == 4 * kThreads, "four region counts per thread");
    uint32_t c[4], local = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const uint32_t r = 4 * threadIdx.x + k;
        c[k] = r < nregions ? counts[r] : 0;
        local += c[k];
    }
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = local;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    uint32_t before = 0;
    for (uint32_t w = 0; w < warp; w++) before += wsum[w];
    uint32_t acc = before + incl - local;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const uint32_t r = 4 * threadIdx.x + k;
        if (r <= nregions) pre[r] = acc;
        acc += c[k];
    }
    if (threadIdx.x == kThreads - 1 && nregions == kMaxRegions) pre[kMaxRegions] = acc;
    __syncthreads();
}

__device__ __forceinline__ uint2 region_edge(const uint2 *__restrict__ list, const uint32_t *pre, uint32_t nregions,
                                             uint64_t region_stride, uint32_t i) {
    uint32_t lo = 0, hi = nregions - 1;  // last region whose first edge <= i
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (pre[mid] <= i) lo = mid; else hi = mid - 1;
    }
    return list[(uint64_t)lo * region_stride + (i - pre[lo])];
}

// One more round on the edges that cc_open_edges left.
__global__ void __launch_bounds__(kThreads, 8) cc_list_round(uint32_t *par, const uint2 *__restrict__ list,
                                                          const uint32_t *__restrict__ counts, uint32_t nregions,
                                                          uint64_t region_stride, const OpenCount left, uint32_t *open) {
    __shared__ Links<4 * kThreads> links;
    __shared__ uint32_t pre[kMaxRegions + 1];
    __shared__ uint32_t s_open;
    links.clear();
    if (threadIdx.x == 0) s_open = 0;
    pdl_wait();
    if (left.skip()) return;
    region_prefix(counts, nregions, pre);
    uint32_t mine = 0;
    grid_stride(pre[nregions], [&](uint32_t i) {
        const uint2 e = region_edge(list, pre, nregions, region_stride, i);
        const uint32_t a = par[e.x], b = par[e.y];
        mine += a != b;
        links.add(par, a, b);
    });
    if (mine) atomicAdd(&s_open, mine);
    links.flush(par);
    if (threadIdx.x == 0 && s_open) atomicAdd(open, s_open);
}

// Union of the surviving edges (the reference's next round on the remaining slice). Regions of
// the filter CTAs are addressed through the prefix of their counts.
__global__ void __launch_bounds__(kThreads) cc_hook_survivors(uint32_t *par, const uint2 *__restrict__ surv,
                                                              const uint32_t *__restrict__ counts, uint32_t nregions,
                                                              uint64_t region_stride) {
    pdl_wait();
    __shared__ uint32_t pre[kMaxRegions + 1];
    region_prefix(counts, nregions, pre);
    grid_stride(pre[nregions], [&](uint32_t i) {
        const uint2 e = region_edge(surv, pre, nregions, region_stride, i);
        edge_hook(par, e.x, e.y);
    });
}

__device__ __forceinline__ uint32_t block_sum(uint32_t x, uint32_t *sh) {
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) sh[w] = x;
    __syncthreads();
    uint32_t t = 0;
    if (threadIdx.x < 32) {
        t = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0;
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    }
    return t;  // valid in thread 0
}

// Per-tile root counts. kCompress: with a full compression (roots only are written).
template <bool kCompress>
__global__ void __launch_bounds__(kThreads) cc_count_roots(uint32_t *par, uint32_t n, uint32_t *tile_counts) {
    pdl_wait();
    __shared__ uint32_t sh[32];
    const uint64_t base = (uint64_t)blockIdx.x * kTile;
    uint32_t c = 0;
#pragma unroll
    for (int k = 0; k < kTileItems; k++) {
        const uint64_t i = base + (uint64_t)k * kThreads + threadIdx.x;
        if (kCompress) {
            const uint32_t r = i < n ? find_root_ro(par, (uint32_t)i) : 0;
            if (i < n) par[i] = r;
            c += i < n && r == (uint32_t)i;
        } else {
            c += i < n && par[i] == (uint32_t)i;
        }
    }
    const uint32_t t = block_sum(c, sh);
    if (threadIdx.x == 0) tile_counts[blockIdx.x] = t;
}

// Exclusive scan of the tile counts by one block, chunk by chunk; writes the total.
__global__ void __launch_bounds__(1024) cc_scan_tiles(const uint32_t *counts, uint32_t *offsets, uint32_t ntiles,
                                                      uint32_t *total) {
    pdl_wait();
    __shared__ uint32_t sh[32];
    __shared__ uint32_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (uint32_t base = 0; base < ntiles; base += blockDim.x) {
        const uint32_t i = base + threadIdx.x;
        const uint32_t x = i < ntiles ? counts[i] : 0;
        // inclusive warp scan
        uint32_t s = x;
        const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
            if (l >= o) s += y;
        }
        if (l == 31) sh[w] = s;
        __syncthreads();
        if (w == 0) {
            uint32_t t = l < (int)(blockDim.x >> 5) ? sh[l] : 0;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
                if (l >= o) t += y;
            }
            sh[l] = t;
        }
        __syncthreads();
        const uint32_t warp_off = w ? sh[w - 1] : 0;
        if (i < ntiles) offsets[i] = carry + warp_off + s - x;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry += warp_off + s;
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}

// Rank of every root: tile offset + exclusive scan of root flags inside the tile. kOwn: the CTA sums the
// counts of the tiles before its own (counts), and the last one writes the total; else the offsets
// come from cc_scan_tiles. Labels of a null array are not written.
template <bool kOwn>
__global__ void __launch_bounds__(kThreads) cc_rank_roots(const uint32_t *par, uint32_t n, const uint32_t *offsets,
                                                          const uint32_t *counts, uint32_t *total, uint32_t *labels) {
    pdl_wait();
    __shared__ uint32_t sh[32];
    __shared__ uint32_t s_before;
    if (kOwn) {
        uint32_t x = 0;
        for (uint32_t t = threadIdx.x; t < blockIdx.x; t += kThreads) x += counts[t];
        x = block_sum(x, sh);
        if (threadIdx.x == 0) {
            s_before = x;
            if (blockIdx.x == gridDim.x - 1) *total = x + counts[blockIdx.x];
        }
        __syncthreads();
    }
    if (!labels) return;
    const uint64_t base = (uint64_t)blockIdx.x * kTile + (uint64_t)threadIdx.x * kTileItems;
    uint32_t flags = 0, c = 0;
#pragma unroll
    for (int k = 0; k < kTileItems; k++) {
        const uint64_t i = base + k;
        const uint32_t f = (i < n) && par[i] == (uint32_t)i;
        flags |= f << k;
        c += f;
    }
    // exclusive scan of c over the block (thread order == vertex order inside the tile)
    uint32_t s = c;
    const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
        if (l >= o) s += y;
    }
    if (l == 31) sh[w] = s;
    __syncthreads();
    if (w == 0) {
        uint32_t t = l < (kThreads >> 5) ? sh[l] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
            if (l >= o) t += y;
        }
        sh[l] = t;
    }
    __syncthreads();
    uint32_t r = (kOwn ? s_before : offsets[blockIdx.x]) + (w ? sh[w - 1] : 0) + s - c;
#pragma unroll
    for (int k = 0; k < kTileItems; k++) {
        if ((flags >> k) & 1u) labels[base + k] = r++;
    }
}

// Every other vertex takes its root's label (4 vertices per thread, their parents and grandparents
// requested together; a vertex further down writes its root back, which shortens the walks of others).
__global__ void __launch_bounds__(kThreads) cc_label_all(uint32_t *par, uint32_t n, uint32_t *labels) {
    pdl_wait();
    const uint32_t stride = gridDim.x * blockDim.x;
    grid_stride(n, [&](uint32_t i0) {
        uint32_t p[4], r[4];
#pragma unroll
        for (uint32_t k = 0; k < 4; k++) p[k] = i0 + (uint64_t)k * stride < n ? par[i0 + k * stride] : 0;
#pragma unroll
        for (uint32_t k = 0; k < 4; k++) r[k] = par[p[k]];
#pragma unroll
        for (uint32_t k = 0; k < 4; k++)
            if (r[k] != p[k]) r[k] = find_root_ro(par, r[k]);
#pragma unroll
        for (uint32_t k = 0; k < 4; k++) {
            const uint32_t i = i0 + k * stride;
            if (i0 + (uint64_t)k * stride >= n || r[k] == i) continue;
            if (r[k] != p[k]) par[i] = r[k];
            labels[i] = labels[r[k]];
        }
    }, 4);
}

// Count and labels of a finished forest. Up to kOwnTiles tiles each ranking CTA sums the counts before
// its own (saves a launch; the sums together read ntiles^2 / 2 counts).
constexpr uint32_t kOwnTiles = 4096;
// flat: the forest's trees are a few links deep; those of union walks from singletons are compressed with the count,
// tile after tile, before every vertex walks to its root at once.
int label_components(int sms, uint32_t *par, uint32_t n, uint32_t ntiles, uint32_t *counts, uint32_t *offsets,
                     uint32_t *total, uint32_t *labels, bool flat, cudaStream_t s) {
    const uint32_t *cpar = par, *ccounts = counts, *coffsets = offsets;
    CAC_CUDA_TRY(launch_pdl(flat ? cc_count_roots<false> : cc_count_roots<true>, ntiles, kThreads, 0, s, par, n, counts));
    if (ntiles <= kOwnTiles) {
        CAC_CUDA_TRY(launch_pdl(cc_rank_roots<true>, ntiles, kThreads, 0, s, cpar, n, coffsets, ccounts, total, labels));
    } else {
        CAC_CUDA_TRY(launch_pdl(cc_scan_tiles, 1, 1024, 0, s, ccounts, offsets, ntiles, total));
        if (labels)
            CAC_CUDA_TRY(launch_pdl(cc_rank_roots<false>, ntiles, kThreads, 0, s, cpar, n, coffsets, ccounts, total, labels));
    }
    if (labels) {
        const uint64_t blocks = ((uint64_t)n + 4 * kThreads - 1) / (4 * kThreads);
        CAC_CUDA_TRY(launch_pdl(cc_label_all, (unsigned)std::min<uint64_t>(blocks, (uint64_t)sms * 8), kThreads, 0, s, par, n,
                                labels));
    }
    return CAC_OK;
}

// A whole query in one CTA, the forest in shared memory (small graphs: the launches of the form above
// cost more than their work). Three passes over the edges -- the smallest neighbour as parent, the same
// between roots, union walks for what is left -- with a compression after each, which walks to the root after the
// last only (see cc_compress4; the last pass joins all edges whatever the first two left), then every thread
// ranks the roots of its own run of vertices. The count, the error word and, for host labels, the labels
// go straight into pinned host memory, so that the one wait after the launch is the whole read-back.
// Bound by the latency of its passes (shared-memory unions, edges from L2). Measured per query, labels
// into a host array, against the 16 launches: R-MAT scale 10 with 8192 edges 94 -> 26 us, G(16000, M) with
// 64,000 edges 133 -> 78. Device time at 16,320 vertices: a path numbered along its length 171 -> 55 (61 with walks to the
// root after every pass), relabelled 106 -> 39, a ring lattice of degree 8 224 -> 62, a star 33 -> 28.
constexpr int kSmallThreads = 1024;
template <bool kCheck>
__global__ void __launch_bounds__(kSmallThreads) cc_small(const uint32_t *__restrict__ u, const uint32_t *__restrict__ v,
                                                          uint32_t m, uint32_t n, uint32_t *labels, uint32_t *out) {
    extern __shared__ uint32_t dyn[];
    uint32_t *par = dyn, *lab = dyn + n;
    __shared__ uint32_t wsum[kSmallThreads / 32], bad;
    const uint32_t t = threadIdx.x;
    for (uint32_t i = t; i < n; i += kSmallThreads) par[i] = i;
    if (t == 0) bad = 0;
    __syncthreads();
    for (int pass = 0; pass < 3; pass++) {
        for (uint32_t e0 = t; e0 < m; e0 += 4 * kSmallThreads) {
            uint32_t a[4], b[4];
#pragma unroll
            for (uint32_t k = 0; k < 4; k++) {
                const uint32_t e = e0 + k * kSmallThreads;
                a[k] = b[k] = 0;
                if (e < m) {
                    a[k] = __ldg(u + e);
                    b[k] = __ldg(v + e);
                }
                if (kCheck && (a[k] >= n || b[k] >= n)) {
                    bad = kErrBadId;
                    a[k] = b[k] = 0;
                }
            }
#pragma unroll
            for (uint32_t k = 0; k < 4; k++) {
                if (a[k] == b[k]) continue;
                if (pass == 0) {
                    atomicMin(&par[max(a[k], b[k])], min(a[k], b[k]));
                } else if (pass == 1) {
                    const uint32_t x = par[a[k]], y = par[b[k]];
                    if (x != y) atomicMin(&par[max(x, y)], min(x, y));
                } else {
                    edge_hook(par, a[k], b[k]);
                }
            }
        }
        __syncthreads();
        for (uint32_t i = t; i < n; i += kSmallThreads) par[i] = pass < 2 ? find_near(par, i) : find_root_ro(par, i);
        __syncthreads();
    }
    // ranks: thread t owns the vertices [t per, (t + 1) per)
    const uint32_t per = (n + kSmallThreads - 1) / kSmallThreads, i0 = min(n, t * per), i1 = min(n, i0 + per);
    uint32_t c = 0;
    for (uint32_t i = i0; i < i1; i++) c += par[i] == i;
    uint32_t incl = c;
    const uint32_t lane = t & 31, w = t >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
    }
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    uint32_t r = incl - c;
    for (uint32_t k = 0; k < w; k++) r += wsum[k];
    if (t == kSmallThreads - 1) {
        out[0] = r + c;
        out[kErrWord] = kCheck ? bad : 0;
    }
    if (!labels) return;
    for (uint32_t i = i0; i < i1; i++)
        if (par[i] == i) lab[i] = r++;
    __syncthreads();
    for (uint32_t i = t; i < n; i += kSmallThreads) labels[i] = lab[par[i]];
}

// CTAs of cc_compress_giant_bitmap: two per SM (kGiantSample threads each), fewer for small n.
unsigned giant_grid(cac_ctx *ctx, uint32_t n) {
    const uint64_t words = ((uint64_t)n + 31) / 32;
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((words + 31) / 32, (uint64_t)ctx->num_sms * 2));
}

int grid_for(cac_ctx *ctx, uint64_t work, int per_sm) {
    const uint64_t need = (work + kThreads - 1) / kThreads;
    const uint64_t cap = (uint64_t)ctx->num_sms * per_sm;
    return (int)std::max<uint64_t>(1, std::min(need, cap));
}

void compress_all(cac_ctx *ctx, uint32_t *par, uint32_t n, cudaStream_t s, OpenCount left) {
    launch_pdl(cc_compress4, grid_for(ctx, n / 4, 8), kThreads, 0, s, par, n, left);
}

}  // namespace

CCPlan cc_plan(uint32_t n, uint64_t m, uint32_t ranks) {
    // UnweightedIteratedSparseSampling::loadSlice (.cpp:5-21) and edgesToSamplePerProcessor
    // (.cpp:80-128), same float expressions and uint32 wrap-around.
    CCPlan p;
    p.slice_off.resize(ranks);
    p.slice_len.resize(ranks);
    p.draws.assign(ranks, 0);
    const uint64_t portion = m / ranks;
    std::vector<int> avail(ranks), per(ranks, 0);
    uint32_t total = 0;
    for (uint32_t r = 0; r < ranks; r++) {
        p.slice_off[r] = portion * r;
        p.slice_len[r] = (r == ranks - 1) ? m - portion * r : portion;
        avail[r] = (int)p.slice_len[r];
        total += (uint32_t)avail[r];
    }
    const uint32_t want = (uint32_t)(std::pow((float)n, 1.0f + 0.09f / 2) * (1.0f + 0.2f));
    uint32_t to_sample = std::min(want, total);
    const uint32_t threshold = (uint32_t)(3.0f / (0.2f * 0.2f) * std::log((float)ranks / 0.9f));
    uint32_t remaining = to_sample;
    for (uint32_t i = 0; i < ranks; i++) {
        if ((uint32_t)avail[i] <= threshold) {
            per[i] = avail[i];
            remaining -= (uint32_t)avail[i];
            to_sample -= (uint32_t)avail[i];
        }
    }
    for (uint32_t i = 0; i < ranks; i++) {
        if (per[i] != 0) continue;
        const int share = (int)((float)to_sample * (float)avail[i] / (float)total);
        per[i] = std::min(share, avail[i]);
        remaining -= (uint32_t)per[i];
    }
    for (uint32_t sp = 0; remaining > 0 && sp < ranks; sp++) {
        if (avail[sp] > per[sp]) {
            const uint32_t delta = std::min((uint32_t)(avail[sp] - per[sp]), remaining);
            per[sp] += (int)delta;
            remaining -= delta;
        }
    }
    for (uint32_t r = 0; r < ranks; r++) {
        // a rank asked for its whole slice returns the slice itself (.cpp:28-29): those edges
        // are covered by the closing pass, so nothing is drawn for it.
        p.draws[r] = ((uint64_t)per[r] == p.slice_len[r]) ? 0 : (uint64_t)per[r];
    }
    return p;
}

size_t cc_scratch_bytes(uint32_t n, uint32_t ranks, uint64_t m) {
    const size_t ntiles = ((size_t)n + kTile - 1) / kTile;
    const size_t nwords = ((size_t)n + 31) / 32;
    return align_up((size_t)n * 4) + 2 * align_up(ntiles * 4 + 4) + align_up(256) +
           align_up(sizeof(RankDesc) * (size_t)ranks) + align_up(nwords * 4 + 4) + align_up(kMaxRegions * 4) +
           align_up((m + 4 * (uint64_t)kMaxRegions) * 8);
}

namespace {

// Everything one query enqueues, resolved on the host.
struct CCLaunch {
    uint32_t n = 0;
    uint64_t m = 0;
    const uint32_t *u = nullptr, *v = nullptr;
    uint32_t *labels = nullptr;
    uint32_t ranks = 1;
    uint32_t *par = nullptr, *counts = nullptr, *offsets = nullptr, *total = nullptr, *giant = nullptr;
    uint32_t *bits = nullptr, *region_counts = nullptr;
    uint2 *surv = nullptr;
    RankDesc *d_ranks = nullptr;
    const RankDesc *h_ranks = nullptr;
    uint32_t ntiles = 0, nwords = 0;
    uint8_t *quads = nullptr;                    // see quad_bytes
    uint64_t blocks = 0, draws = 0, drawn = 0;  // sitmo blocks, chunk draws, sampled edges
    uint64_t *chunks = nullptr;                  // per draw: first edge | count << 32
    uint32_t *err = nullptr;                     // total + kErrWord
    bool vec = false;
    bool check = false;                          // endpoints not validated: every kernel checks them
};

int record(cac_ctx *ctx, int i, bool capturing) {
    if (capturing) CAC_CUDA_TRY(cudaEventRecordWithFlags(ctx->ev[i], ctx->stream, cudaEventRecordExternal));
    else CAC_CUDA_TRY(cudaEventRecord(ctx->ev[i], ctx->stream));
    return CAC_OK;
}

auto pick_edge_round(bool first, bool check, bool wide) {
    if (first) return check ? (wide ? cc_edge_round<true, true, kRoundThreads> : cc_edge_round<true, true, kThreads>)
                            : (wide ? cc_edge_round<true, false, kRoundThreads> : cc_edge_round<true, false, kThreads>);
    return check ? (wide ? cc_edge_round<false, true, kRoundThreads> : cc_edge_round<false, true, kThreads>)
                 : (wide ? cc_edge_round<false, false, kRoundThreads> : cc_edge_round<false, false, kThreads>);
}

unsigned round_grid(cac_ctx *ctx, uint64_t warps, int threads = kRoundThreads) {
    const uint64_t per = threads / 32;
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((warps + per - 1) / per, (uint64_t)ctx->num_sms * 2048 / threads));
}

// Forest building without draws (every rank returns its whole slice) on few edges per vertex: a round on all
// edges, another that lists those still open, and some more on the list, each left out when the one before found
// few open. What is left after the partial rounds below near the threshold of a giant component are open edges
// between few large trees, and union walks of these are slow: each reads and swaps the same roots, and a line of the L2
// serves about one access per ns (500,000 open edges of G(3 10^6, degree 2): 790 us). In a round they cost a CTA's
// table entry each. Few: as many as are walked in the time of a round.
//   Bound by the kernel boundaries (a round and its compression take 6 us) and, from 10^6 edges on, by the gathers of
// parents from the L2 (3 M edges 50 us; on the list 10 to 20). Device us by one pass of union walks / by the partial rounds / so:
// G(300,000, M) of degree 1.5 192 / 110 / 81, 1.75 116 / 218 / 81, 2 242 / 216 / 83; G(10^6, M) of degree 1.25 135 / 118 / 106,
// 2 441 / 352 / 132; G(3 10^6, M) of degree 1.5 376 / 442 / 205, 2 400 / 808 / 267; paths of 10^6 numbered along
// them 232 / 181 / 155, relabelled 168 / 144 / 136; random trees 118 / 123 / 122. What a pass joins at once pays for the
// launches: stars of 300,000 vertices 34 / 46 / 48.
int sparse_rounds(cac_ctx *ctx, const CCLaunch &L, cudaStream_t s) {
    const uint64_t tiles = (L.m + 255) / 256;
    const bool wide = tiles >= (uint64_t)ctx->num_sms * (kRoundThreads / 32);
    const int threads = wide ? kRoundThreads : kThreads;
    const uint32_t regions = std::min<uint32_t>(round_grid(ctx, tiles, threads), kMaxRegions);
    const uint64_t region = (tiles + regions - 1) / regions * 256;
    CAC_CUDA_TRY(launch_pdl(pick_edge_round(true, L.check, wide), round_grid(ctx, tiles, threads), threads, 0, s, L.par, L.u,
                            L.v, L.m, 0u, kRoundParts, L.n, L.err));
    compress_all(ctx, L.par, L.n, s);
    uint32_t *open = L.total + kOpenWord;
    auto kern = wide ? (L.check ? cc_open_edges<true, kRoundThreads> : cc_open_edges<false, kRoundThreads>)
                     : (L.check ? cc_open_edges<true, kThreads> : cc_open_edges<false, kThreads>);
    CAC_CUDA_TRY(launch_pdl(kern, regions, threads, 0, s, L.par, L.u, L.v, L.m, L.n, L.surv, L.region_counts, open, L.err));
    compress_all(ctx, L.par, L.n, s);
    const unsigned grid = (unsigned)std::min<uint64_t>((L.m + 4 * kThreads - 1) / (4 * kThreads), (uint64_t)ctx->num_sms * 8);
    for (uint32_t k = 1; k < (L.m < kFewRoundEdges ? kFullRounds - 1 : kFullRounds); k++) {
        const OpenCount left{open++, (uint32_t)(L.m / 128 + 4096)};
        CAC_CUDA_TRY(launch_pdl(cc_list_round, grid, kThreads, 0, s, L.par, static_cast<const uint2 *>(L.surv),
                                static_cast<const uint32_t *>(L.region_counts), regions, region, left, open));
        compress_all(ctx, L.par, L.n, s, left);
    }
    return CAC_OK;
}

// The same on more edges: the rounds of kRoundDegree on
// parts of the edges; where these take all edges before a giant component forms, one more round over all
// of them, after which some hundred of 375,000 edges are left to the union walks (counted on G(300000, M),
// average degree 2.5; 104,000 without it). Bound by the kernel boundaries (a round and its compression
// take 6 us each). Measured against one pass of union walks: G(300000, M) of average degree 2.5 166 ->
// 90 us a query, G(10^6, M) of degree 3 863 -> 127.
int edge_rounds(cac_ctx *ctx, const CCLaunch &L, cudaStream_t s, bool *flat) {
    const double degree = 2.0 * (double)L.m / L.n;
    *flat = L.m >= kRoundEdges && degree > 1;
    if (!*flat) return CAC_OK;
    if (degree >= kSparseLow && degree < kSparseDegree && L.n <= kSparseVertices) return sparse_rounds(ctx, L, s);
    auto round = [&](uint32_t from, uint32_t to) -> int {
        const uint64_t warps = (L.m / 256 / kRoundParts + 1) * (to - from);
        const bool wide = warps >= (uint64_t)ctx->num_sms * (kRoundThreads / 32), first = from == 0 && to < kRoundParts;
        const int threads = wide ? kRoundThreads : kThreads;
        auto kern = pick_edge_round(first, L.check, wide);
        CAC_CUDA_TRY(launch_pdl(kern, round_grid(ctx, warps, threads), threads, 0, s, L.par, L.u, L.v, L.m, from, to, L.n, L.err));
        compress_all(ctx, L.par, L.n, s);
        return CAC_OK;
    };
    double upto = 0;
    uint32_t to = 0;
    for (double d : kRoundDegree) {
        upto += d;
        const uint32_t from = to;
        to = std::min(kRoundParts, (uint32_t)std::ceil(kRoundParts * std::min(1.0, upto / degree)));
        if (to > from) CAC_TRY(round(from, to));
    }
    if (to == kRoundParts) CAC_TRY(round(0, kRoundParts));
    return CAC_OK;
}

template <bool kFlat>
auto pick_edge_pass(bool vec, bool check) {
    return vec ? (check ? cc_edge_pass<true, true, kFlat> : cc_edge_pass<true, false, kFlat>)
               : (check ? cc_edge_pass<false, true, kFlat> : cc_edge_pass<false, false, kFlat>);
}

// Enqueues the whole query on the ctx stream (directly, or into a graph being captured).
int cc_enqueue(cac_ctx *ctx, const CCLaunch &L, bool capturing) {
    cudaStream_t s = ctx->stream;
    const uint32_t n = L.n;
    const uint64_t m = L.m;
    bool flat = true;  // what the closing pass leaves: trees a few links deep, or those of union walks alone
    CAC_TRY(record(ctx, 0, capturing));
    CAC_CUDA_TRY(cudaMemsetAsync(L.err, 0, (kQueryWords - kErrWord) * 4, s));
    CAC_CUDA_TRY(launch_pdl(cc_init, grid_for(ctx, n, 8), kThreads, 0, s, L.par, n));
    if (L.draws > 0 && m > 0) {
        CAC_CUDA_TRY(cudaMemcpyAsync(L.d_ranks, L.h_ranks, sizeof(RankDesc) * L.ranks, cudaMemcpyHostToDevice, s));
        // (Drawing inside the hooking CTAs instead of in one kernel up front measured slower: the rank
        // search and the block cipher then sit on every round's critical path.)
        CAC_CUDA_TRY(launch_pdl(cc_sample_draws, grid_for(ctx, L.blocks, 8), kThreads, 0, s,
                                static_cast<const RankDesc *>(L.d_ranks), (int)L.ranks, L.blocks, L.chunks));
        // the rounds: kRoundDegree, the last one with all draws that are left
        constexpr uint32_t rounds = sizeof(kRoundDegree) / sizeof(kRoundDegree[0]);
        uint64_t d1 = 0;
        double edges = 0;
        for (uint32_t k = 0; k < rounds && d1 < L.draws; k++) {
            const uint64_t d0 = d1;
            edges += kRoundDegree[k] * n / 2;
            d1 = k + 1 == rounds ? L.draws : std::min<uint64_t>(L.draws, (uint64_t)(edges / kSampleChunk) + 1);
            auto round = k == 0 ? (L.check ? cc_sample_round<true, true> : cc_sample_round<true, false>)
                                : (L.check ? cc_sample_round<false, true> : cc_sample_round<false, false>);
            CAC_CUDA_TRY(launch_pdl(round, round_grid(ctx, (d1 - d0 + 1) / 2), kRoundThreads, 0, s, L.par, L.u, L.v,
                                    static_cast<const uint64_t *>(L.chunks), d0, d1, n, L.err));
            if (d1 < L.draws) compress_all(ctx, L.par, n, s);
        }
        CAC_CUDA_TRY(launch_pdl(cc_compress_giant_bitmap, giant_grid(ctx, n), kGiantSample, 0, s, L.par, n, L.giant,
                                L.bits, L.quads));
    }
    CAC_TRY(record(ctx, 1, capturing));
    if (m > 0) {
        if (L.draws > 0) {
            // a sampling round ran, so a giant component exists: filter, then hook the survivors
            const size_t sm = (size_t)std::min(L.nwords, kSmemBitmapWords) * 4;
            const uint64_t tiles = L.vec ? m >> 8 : 0;  // 256-edge tiles; the rest goes to the scalar pass
            const uint32_t regions = (uint32_t)std::max<uint64_t>(
                1, std::min<uint64_t>({(uint64_t)ctx->num_sms, (uint64_t)kMaxRegions, tiles}));
            const uint64_t per = (tiles + regions - 1) / regions;
            if (tiles) {
                auto filt = L.nwords <= kSmemBitmapWords ? (L.check ? cc_filter<true, true> : cc_filter<true, false>)
                                                         : (L.check ? cc_filter<false, true> : cc_filter<false, false>);
                CAC_CUDA_TRY(launch_pdl(filt, regions, kEdgeThreads, sm, s, L.u, L.v, tiles,
                                        static_cast<const uint32_t *>(L.bits), L.nwords,
                                        reinterpret_cast<const uint32_t *>(L.quads), L.surv, L.region_counts, n,
                                        L.err));
            }
            CAC_TRY(record(ctx, 4, capturing));
            if (tiles)
                CAC_CUDA_TRY(launch_pdl(cc_hook_survivors, (unsigned)ctx->num_sms * kSurvivorBlocksPerSm, kThreads, 0, s,
                                        L.par, static_cast<const uint2 *>(L.surv),
                                        static_cast<const uint32_t *>(L.region_counts), regions, per * 256));
            const uint64_t done = tiles * 256;
            if (done < m)
                (L.check ? cc_edge_pass<false, true, true> : cc_edge_pass<false, false, true>)<<<grid_for(ctx, m - done, 8), kThreads,
                                                                                       0, s>>>(
                    L.par, L.u + done, L.v + done, m - done, n, L.err);
        } else {
            CAC_TRY(edge_rounds(ctx, L, s, &flat));
            const int grid = grid_for(ctx, (m + 3) / 4, 8);
            auto pass = flat ? pick_edge_pass<true>(L.vec, L.check) : pick_edge_pass<false>(L.vec, L.check);
            pass<<<grid, kThreads, 0, s>>>(L.par, L.u, L.v, m, n, L.err);
            CAC_TRY(record(ctx, 4, capturing));
        }
    } else {
        CAC_TRY(record(ctx, 4, capturing));
    }
    CAC_TRY(record(ctx, 2, capturing));
    // (A single-pass count and rank by decoupled look-back measured slower: BA n=1,024,000 20.4 vs
    // 18.5 us, R-MAT scale 22 48.6 vs 34.0 us for the labelling.)
    CAC_TRY(label_components(ctx->num_sms, L.par, n, L.ntiles, L.counts, L.offsets, L.total, L.labels, flat, s));
    CAC_CUDA_TRY(cudaGetLastError());
    CAC_CUDA_TRY(cudaMemcpyAsync(ctx->pinned_u32, L.total, (kErrWord + 1) * 4, cudaMemcpyDeviceToHost, s));
    CAC_TRY(record(ctx, 3, capturing));
    return CAC_OK;
}

// The query's error word, copied back with its count.
int check_ids_word(cac_ctx *ctx, uint32_t n) {
    if (ctx->pinned_u32[kErrWord] & kErrBadId) {
        set_error("connected components: an edge endpoint is >= n = " + std::to_string(n) +
                  " (such edges were skipped; the labels are not valid)");
        return CAC_ERR_INVALID;
    }
    return CAC_OK;
}

bool same_key(const CCGraphKey &a, const CCGraphKey &b) {
    return a.u == b.u && a.v == b.v && a.labels == b.labels && a.n == b.n && a.m == b.m && a.seed == b.seed &&
           a.ranks == b.ranks && a.arena_base == b.arena_base && a.arena_cap == b.arena_cap && a.check == b.check;
}

}  // namespace

void cc_graph_reset(cac_ctx *ctx) {
    if (ctx->cc_exec) cudaGraphExecDestroy(ctx->cc_exec);
    ctx->cc_exec = nullptr;
    ctx->cc_key = CCGraphKey{};
    if (ctx->cc_stream_exec) cudaGraphExecDestroy(ctx->cc_stream_exec);
    ctx->cc_stream_exec = nullptr;
    ctx->cc_stream_key = CCStreamKey{};
}

// One CTA (cc_small): the two arrays of n words fit its shared memory, host labels the ctx's pinned page,
// and one SM still reads the edges faster than a dozen launches run. Device us by one CTA / by the launches, random
// graphs: 300 vertices, 65,537 edges 37 / 67, 131,072 64 / 62, 262,144 119 / 72; 2000 vertices 43 / 71, 74 / 66, 154 / 71; 6000
// 43 / 74, 74 / 74, 138 / 74; 16,000 68 / 88, 84 / 86, 146 / 87: the two meet at twice the line whatever the vertices.
constexpr uint32_t kSmallVertices = (64 * 1024 - 256) / 4;
constexpr uint64_t kSmallEdges = 1u << 16;
bool cc_is_small(uint32_t n, uint64_t m) { return n && n <= kSmallVertices && m <= kSmallEdges; }

int cc_run_small(cac_ctx *ctx, uint32_t n, uint64_t m, const uint32_t *d_u, const uint32_t *d_v, uint32_t *labels,
                 int labels_where, cac_cc_result *res, bool check_ids) {
    cudaStream_t s = ctx->stream;
    uint32_t *stage = ctx->pinned_u32 + 64;
    uint32_t *out = !labels ? nullptr : labels_where == CAC_DEVICE ? labels : stage;
    auto kern = check_ids ? cc_small<true> : cc_small<false>;
    CAC_TRY(smem_optin(ctx, kern));
    CAC_CUDA_TRY(cudaEventRecord(ctx->ev[0], s));
    kern<<<1, kSmallThreads, 2 * n * sizeof(uint32_t), s>>>(d_u, d_v, (uint32_t)m, n, out, ctx->pinned_u32);
    CAC_CUDA_TRY(cudaGetLastError());
    CAC_CUDA_TRY(cudaEventRecord(ctx->ev[3], s));
    CAC_CUDA_TRY(cudaStreamSynchronize(s));
    CAC_TRY(check_ids_word(ctx, n));
    if (out == stage) std::memcpy(labels, stage, (size_t)n * 4);
    if (res) {
        *res = cac_cc_result{};
        res->num_components = ctx->pinned_u32[0];
        res->rounds = m > 0 ? 1u : 0u;
        CAC_CUDA_TRY(cudaEventElapsedTime(&res->device_ms, ctx->ev[0], ctx->ev[3]));
        res->edge_pass_ms = res->device_ms;
    }
    return CAC_OK;
}

int cc_run(cac_ctx *ctx, uint32_t n, uint64_t m, const uint32_t *d_u, const uint32_t *d_v, uint32_t seed,
           uint32_t ranks, uint32_t *d_labels, cac_cc_result *res, bool check_ids) {
    if (ranks == 0) ranks = 1;
    cudaStream_t s = ctx->stream;
    if (n == 0) {
        if (res) *res = cac_cc_result{};
        return CAC_OK;
    }
    if (cc_is_small(n, m)) return cc_run_small(ctx, n, m, d_u, d_v, d_labels, CAC_DEVICE, res, check_ids);
    const CCPlan plan = cc_plan(n, m, ranks);
    uint64_t chunk_slots = 1;
    for (uint32_t r = 0; r < ranks; r++) chunk_slots += (plan.draws[r] + kSampleChunk - 1) / kSampleChunk;
    CCLaunch L;
    L.n = n;
    L.m = m;
    L.u = d_u;
    L.v = d_v;
    L.labels = d_labels;
    L.ranks = ranks;
    L.ntiles = (uint32_t)(((uint64_t)n + kTile - 1) / kTile);
    L.nwords = (uint32_t)(((uint64_t)n + 31) / 32);
    L.vec = ((reinterpret_cast<uintptr_t>(d_u) | reinterpret_cast<uintptr_t>(d_v)) & 15) == 0;
    L.check = check_ids;

    CAC_TRY(arena_reserve(ctx, cc_scratch_bytes(n, ranks, m) + align_up(chunk_slots * 8)));
    arena_reset(ctx);
    L.par = (uint32_t *)arena_take(ctx, (size_t)n * 4);
    L.counts = (uint32_t *)arena_take(ctx, (size_t)L.ntiles * 4 + 4);
    L.offsets = (uint32_t *)arena_take(ctx, (size_t)L.ntiles * 4 + 4);
    L.total = (uint32_t *)arena_take(ctx, 256);
    L.giant = L.total + 8;
    L.err = L.total + kErrWord;
    L.d_ranks = (RankDesc *)arena_take(ctx, sizeof(RankDesc) * ranks);
    L.bits = (uint32_t *)arena_take(ctx, (size_t)L.nwords * 4 + 4);
    L.region_counts = (uint32_t *)arena_take(ctx, kMaxRegions * 4);
    L.surv = (uint2 *)arena_take(ctx, (m + 4 * (uint64_t)kMaxRegions) * 8);
    L.chunks = (uint64_t *)arena_take(ctx, chunk_slots * 8);
    L.quads = quads_in(L.chunks, chunk_slots * 8, L.nwords);  // (the last round has read the draws by then)

    // rank descriptors go through the ctx's pinned staging page when they fit (async copy)
    std::vector<RankDesc> hv;
    RankDesc *hr = nullptr;
    const bool pinned = sizeof(RankDesc) * ranks <= kPinnedBytes;
    if (pinned) {
        hr = reinterpret_cast<RankDesc *>(ctx->pinned_u32 + 64);
    } else {
        hv.resize(ranks);
        hr = hv.data();
    }
    for (uint32_t r = 0; r < ranks; r++) {
        const uint64_t chunk_draws = (plan.draws[r] + kSampleChunk - 1) / kSampleChunk;
        hr[r].slice_off = plan.slice_off[r];
        hr[r].slice_len = plan.slice_len[r];
        hr[r].draws = chunk_draws;
        hr[r].block_off = L.blocks;
        hr[r].draw_off = L.draws;
        hr[r].key0 = seed + r;
        hr[r].pad = 0;
        L.blocks += (chunk_draws + 7) / 8;
        L.draws += chunk_draws;
        L.drawn += chunk_draws * kSampleChunk;
    }
    L.h_ranks = hr;
    if (L.draws > 0 && m > 0) {
        CAC_TRY(smem_optin(ctx, cc_filter<true, true>));
        CAC_TRY(smem_optin(ctx, cc_filter<false, true>));
        CAC_TRY(smem_optin(ctx, cc_filter<true, false>));
        CAC_TRY(smem_optin(ctx, cc_filter<false, false>));
    }

    // Repeated identical queries replay a captured CUDA graph: one launch instead of a dozen
    // kernel launches and copies. The first sighting of a key runs directly; the second captures.
    CCGraphKey key{d_u, d_v, d_labels, n, m, seed, ranks, ctx->arena.base, ctx->arena.cap, check_ids};
    if (!pinned) {
        cc_graph_reset(ctx);
        CAC_TRY(cc_enqueue(ctx, L, false));
    } else if (same_key(key, ctx->cc_key) && ctx->cc_exec) {
        CAC_CUDA_TRY(cudaGraphLaunch(ctx->cc_exec, s));
    } else if (same_key(key, ctx->cc_key)) {
        cudaGraph_t graph = nullptr;
        CAC_CUDA_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        const int st = cc_enqueue(ctx, L, true);
        const cudaError_t ce = cudaStreamEndCapture(s, &graph);
        if (st != CAC_OK) {
            if (graph) cudaGraphDestroy(graph);
            return st;
        }
        CAC_CUDA_TRY(ce);
        const cudaError_t ie = cudaGraphInstantiate(&ctx->cc_exec, graph, 0);
        cudaGraphDestroy(graph);
        if (ie != cudaSuccess) {
            ctx->cc_exec = nullptr;
            cudaGetLastError();
            CAC_TRY(cc_enqueue(ctx, L, false));
        } else {
            CAC_CUDA_TRY(cudaGraphLaunch(ctx->cc_exec, s));
        }
    } else {
        cc_graph_reset(ctx);
        ctx->cc_key = key;
        CAC_TRY(cc_enqueue(ctx, L, false));
    }
    CAC_CUDA_TRY(cudaStreamSynchronize(s));
    CAC_TRY(check_ids_word(ctx, n));
    if (res) {
        res->num_components = ctx->pinned_u32[0];
        res->rounds = (L.draws > 0 ? 1u : 0u) + (m > 0 ? 1u : 0u);  // sampling round + closing pass
        res->sampled_edges = L.drawn;
        CAC_CUDA_TRY(cudaEventElapsedTime(&res->device_ms, ctx->ev[0], ctx->ev[3]));
        CAC_CUDA_TRY(cudaEventElapsedTime(&res->edge_pass_ms, ctx->ev[1], ctx->ev[4]));
        CAC_CUDA_TRY(cudaEventElapsedTime(&res->sample_ms, ctx->ev[0], ctx->ev[1]));
        CAC_CUDA_TRY(cudaEventElapsedTime(&res->hook_ms, ctx->ev[4], ctx->ev[2]));
        CAC_CUDA_TRY(cudaEventElapsedTime(&res->label_ms, ctx->ev[2], ctx->ev[3]));
    }
    return CAC_OK;
}

// Device address of a pinned (page-locked, mapped) host array, or null for pageable memory.
static const uint32_t *pinned_device_view(const uint32_t *h) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, h) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return a.type == cudaMemoryTypeHost ? static_cast<const uint32_t *>(a.devicePointer) : nullptr;
}

// Connected components of an edge list that is still in host memory (cac_cc_edges). The
// host-to-device link (about 209 GB/s on a GB300 host, measured for copy-engine copies and for
// kernels reading pinned host memory alike) is the bound: BA n=1,024,000 needs 0.63 ms to cross it
// and 0.23 ms to solve once resident. So the edges cross in an order that lets the ctx stream do
// its work behind the copy:
//   1. kStreamPieces evenly spaced pieces, together as large as the reference's sample budget
//      (edgesToSamplePerProcessor: n^1.045 * 1.2 edges), land first: pulled by one kernel from
//      pinned host arrays while the copy engine starts on the gaps, else as one strided copy per
//      array. They are hooked piece by piece, one edge per thread, with a full compression after
//      each: this is the sampling round (the pieces are spread over the whole list, so an edge list
//      sorted by vertex still yields a sample of the whole graph).
//   2. The giant component of the sample is fixed as a bitmap.
//   3. The gaps between the pieces cross on the copy stream, each streamed through the filter as
//      it lands: edges with both ends in the giant component are dropped, the others hooked.
// What is left after the last byte arrives is one gap's filter and the labelling. Labels -- rank
// of each component's smallest vertex -- are the same as cc_run's for any edge order and sample.
// h_labels (optional) receives the labels before the call returns. A repeated call with the same
// buffers replays the whole sequence as one captured CUDA graph.
namespace {

// Everything one streamed query enqueues, resolved on the host.
struct StreamLaunch {
    uint32_t n = 0;
    uint64_t m = 0;
    const uint32_t *h_u = nullptr, *h_v = nullptr;  // host edge arrays (copy-engine source)
    const uint32_t *z_u = nullptr, *z_v = nullptr;  // their device views when pinned and aligned, else null
    uint32_t *d_u = nullptr, *d_v = nullptr, *d_labels = nullptr, *h_labels = nullptr;
    uint32_t *par = nullptr, *counts = nullptr, *offsets = nullptr, *total = nullptr, *giant = nullptr;
    uint32_t *bits = nullptr, *region_counts = nullptr;
    uint2 *surv = nullptr;
    uint32_t ntiles = 0, nwords = 0;
    uint8_t *quads = nullptr;                    // see quad_bytes
    bool vec = false, filtered = false;
    std::vector<std::pair<uint64_t, uint64_t>> parts;  // (first edge, count): pieces, then gaps
};

// Copies the sample pieces of a pinned host edge list into the device arrays: kernel loads of
// pinned host memory cross the link at the copy engine's rate, and one launch moves all pieces
// (the copy engine would take one copy per piece and array). Piece i is the 16-byte words
// [i * seg4, i * seg4 + piece4) of each array.
__global__ void cc_pull_pieces(const uint4 *__restrict__ hu, const uint4 *__restrict__ hv, uint4 *__restrict__ du,
                               uint4 *__restrict__ dv, uint64_t seg4, uint64_t piece4, uint32_t pieces) {
    pdl_wait();
    const uint64_t total = piece4 * pieces;
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < total; k += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = k / piece4, x = i * seg4 + (k - i * piece4);
        const uint4 a = hu[x], b = hv[x];
        du[x] = a;
        dv[x] = b;
    }
}

int stream_enqueue(cac_ctx *ctx, const StreamLaunch &L, bool capturing) {
    cudaStream_t s = ctx->stream;
    const uint32_t n = L.n;
    CAC_TRY(record(ctx, 0, capturing));
    cc_init<<<grid_for(ctx, n, 8), kThreads, 0, s>>>(L.par, n);
    CAC_CUDA_TRY(cudaMemsetAsync(L.total + kErrWord, 0, 4, s));
    // the copies start after everything already queued on the ctx stream (the staging buffers
    // may still be read by the previous query)
    cudaEvent_t *ev = ctx->chunk_ev;
    CAC_CUDA_TRY(cudaEventRecord(ev[0], s));
    CAC_CUDA_TRY(cudaStreamWaitEvent(ctx->copy_stream, ev[0], 0));
    // The pieces land first: pulled by a kernel on the ctx stream from pinned host arrays (the
    // copy engine meanwhile starts on the gaps), else as one strided copy per array ahead of the
    // gaps on the copy stream.
    const uint64_t seg = L.filtered ? L.parts[1].first : 0, piece = L.filtered ? L.parts[0].second : 0;
    if (L.filtered && L.z_u) {
        cc_pull_pieces<<<grid_for(ctx, piece / 4 * kStreamPieces, 8), kThreads, 0, s>>>(
            reinterpret_cast<const uint4 *>(L.z_u), reinterpret_cast<const uint4 *>(L.z_v),
            reinterpret_cast<uint4 *>(L.d_u), reinterpret_cast<uint4 *>(L.d_v), seg / 4, piece / 4, kStreamPieces);
    } else if (L.filtered) {
        CAC_CUDA_TRY(cudaMemcpy2DAsync(L.d_u, seg * 4, L.h_u, seg * 4, piece * 4, kStreamPieces,
                                       cudaMemcpyHostToDevice, ctx->copy_stream));
        CAC_CUDA_TRY(cudaMemcpy2DAsync(L.d_v, seg * 4, L.h_v, seg * 4, piece * 4, kStreamPieces,
                                       cudaMemcpyHostToDevice, ctx->copy_stream));
        CAC_CUDA_TRY(cudaEventRecord(ev[1], ctx->copy_stream));
    }
    for (size_t c = L.filtered ? kStreamPieces : 0; c < L.parts.size(); c++) {
        const uint64_t e0 = L.parts[c].first, len = L.parts[c].second;
        CAC_CUDA_TRY(cudaMemcpyAsync(L.d_u + e0, L.h_u + e0, len * 4, cudaMemcpyHostToDevice, ctx->copy_stream));
        CAC_CUDA_TRY(cudaMemcpyAsync(L.d_v + e0, L.h_v + e0, len * 4, cudaMemcpyHostToDevice, ctx->copy_stream));
        CAC_CUDA_TRY(cudaEventRecord(ev[1 + c], ctx->copy_stream));
    }
    for (size_t c = 0; c < L.parts.size(); c++) {
        const uint64_t e0 = L.parts[c].first, len = L.parts[c].second;
        // a part copied by the copy engine is waited for (the strided piece copy: before piece 0)
        if (!L.filtered || c >= kStreamPieces || (c == 0 && !L.z_u)) CAC_CUDA_TRY(cudaStreamWaitEvent(s, ev[1 + c], 0));
        if (!L.filtered || c < kStreamPieces) {
            // a piece of the sample (or, unfiltered, a chunk): every edge hooks, one edge per
            // thread (union walks are latency chains, so more of them run at once), then the
            // trees are flattened so the next part's walks stay one or two hops long
            cc_edge_pass<false, true, false><<<grid_for(ctx, len, 8), kThreads, 0, s>>>(L.par, L.d_u + e0, L.d_v + e0, len, n,
                                                                           L.total + kErrWord);
            if (L.filtered && c + 1 == kStreamPieces) {
                cc_compress_giant_bitmap<<<giant_grid(ctx, n), kGiantSample, 0, s>>>(L.par, n, L.giant, L.bits, L.quads);
                CAC_TRY(record(ctx, 1, capturing));
            } else if (c + 1 < L.parts.size()) {
                compress_all(ctx, L.par, n, s);
            }
        } else {
            const uint64_t tiles = len >> 8;  // 256-edge tiles; the rest goes to the scalar pass
            const uint32_t regions = (uint32_t)std::max<uint64_t>(
                1, std::min<uint64_t>({(uint64_t)ctx->num_sms, (uint64_t)kMaxRegions, tiles}));
            const uint64_t tper = (tiles + regions - 1) / regions;
            if (tiles) {
                const size_t sm = (size_t)std::min(L.nwords, kSmemBitmapWords) * 4;
                auto filt = L.nwords <= kSmemBitmapWords ? cc_filter<true, true> : cc_filter<false, true>;
                filt<<<regions, kEdgeThreads, sm, s>>>(L.d_u + e0, L.d_v + e0, tiles, L.bits, L.nwords,
                                                       reinterpret_cast<const uint32_t *>(L.quads), L.surv,
                                                       L.region_counts, n, L.total + kErrWord);
                cc_hook_survivors<<<(unsigned)ctx->num_sms * kSurvivorBlocksPerSm, kThreads, 0, s>>>(L.par, L.surv, L.region_counts,
                                                                                   regions, tper * 256);
            }
            const uint64_t done = tiles * 256;
            if (done < len)
                cc_edge_pass<false, true, false><<<grid_for(ctx, len - done, 8), kThreads, 0, s>>>(
                    L.par, L.d_u + e0 + done, L.d_v + e0 + done, len - done, n, L.total + kErrWord);
        }
    }
    if (!L.filtered) CAC_TRY(record(ctx, 1, capturing));
    CAC_TRY(record(ctx, 2, capturing));
    CAC_TRY(label_components(ctx->num_sms, L.par, n, L.ntiles, L.counts, L.offsets, L.total, L.d_labels, L.filtered, s));
    CAC_CUDA_TRY(cudaGetLastError());
    CAC_CUDA_TRY(cudaMemcpyAsync(ctx->pinned_u32, L.total, (kErrWord + 1) * 4, cudaMemcpyDeviceToHost, s));
    CAC_TRY(record(ctx, 3, capturing));
    if (L.d_labels && L.h_labels)
        CAC_CUDA_TRY(cudaMemcpyAsync(L.h_labels, L.d_labels, (size_t)n * 4, cudaMemcpyDeviceToHost, s));
    return CAC_OK;
}

bool same_stream_key(const CCStreamKey &a, const CCStreamKey &b) {
    return a.h_u == b.h_u && a.h_v == b.h_v && a.h_labels == b.h_labels && a.d_u == b.d_u && a.d_v == b.d_v &&
           a.d_labels == b.d_labels && a.n == b.n && a.m == b.m && a.zero_copy == b.zero_copy &&
           a.arena_base == b.arena_base && a.arena_cap == b.arena_cap;
}

}  // namespace

int cc_run_streamed(cac_ctx *ctx, uint32_t n, uint64_t m, const uint32_t *h_u, const uint32_t *h_v, uint32_t *d_u,
                    uint32_t *d_v, uint32_t *d_labels, uint32_t *h_labels, cac_cc_result *res) {
    cudaStream_t s = ctx->stream;
    if (res) *res = cac_cc_result{};
    if (n == 0) return CAC_OK;
    if (!ctx->copy_stream) {
        CAC_CUDA_TRY(cudaStreamCreateWithFlags(&ctx->copy_stream, cudaStreamNonBlocking));
        for (auto &e : ctx->chunk_ev) CAC_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
    StreamLaunch L;
    L.n = n;
    L.m = m;
    L.h_u = h_u;
    L.h_v = h_v;
    L.d_u = d_u;
    L.d_v = d_v;
    L.d_labels = d_labels;
    L.h_labels = h_labels;
    L.ntiles = (uint32_t)(((uint64_t)n + kTile - 1) / kTile);
    L.nwords = (uint32_t)(((uint64_t)n + 31) / 32);
    L.vec = ((reinterpret_cast<uintptr_t>(d_u) | reinterpret_cast<uintptr_t>(d_v)) & 15) == 0;
    // Segment i of the list is [i * seg, (i + 1) * seg), the last one running to m; its piece is
    // the first `piece` edges, its gap the rest. seg and piece are multiples of 256 edges, so
    // every piece and gap starts 1 KB aligned and all but the last gap are whole filter tiles.
    const uint64_t budget = std::min<uint64_t>(m, (uint64_t)(std::pow((float)n, 1.0f + 0.09f / 2) * (1.0f + 0.2f)));
    const uint64_t seg = (m / kStreamPieces) & ~255ull;
    const uint64_t piece = seg ? std::min<uint64_t>(seg, ((budget + kStreamPieces - 1) / kStreamPieces + 255) & ~255ull)
                               : 0;
    L.filtered = L.vec && seg > 0;
    const uint64_t max_gap = L.filtered ? m - (kStreamPieces - 1) * seg - piece : 0;
    CAC_TRY(arena_reserve(ctx, align_up((size_t)n * 4) + 2 * align_up((size_t)L.ntiles * 4 + 4) + align_up(256) +
                                   (L.filtered ? align_up((size_t)L.nwords * 4 + 4) + align_up(kMaxRegions * 4) +
                                                     align_up((max_gap + 4 * (uint64_t)kMaxRegions) * 8)
                                               : 0)));
    arena_reset(ctx);
    L.par = (uint32_t *)arena_take(ctx, (size_t)n * 4);
    L.counts = (uint32_t *)arena_take(ctx, (size_t)L.ntiles * 4 + 4);
    L.offsets = (uint32_t *)arena_take(ctx, (size_t)L.ntiles * 4 + 4);
    L.total = (uint32_t *)arena_take(ctx, 256);
    L.giant = L.total + 8;
    if (L.filtered) {
        L.bits = (uint32_t *)arena_take(ctx, (size_t)L.nwords * 4 + 4);
        L.region_counts = (uint32_t *)arena_take(ctx, kMaxRegions * 4);
        L.surv = (uint2 *)arena_take(ctx, (max_gap + 4 * (uint64_t)kMaxRegions) * 8);
        if (d_labels) L.quads = quads_in(d_labels, (size_t)n * 4, L.nwords);  // (labels are written last)
        CAC_TRY(smem_optin(ctx, cc_filter<true, true>));
        CAC_TRY(smem_optin(ctx, cc_filter<false, true>));
        CAC_TRY(smem_optin(ctx, cc_filter<true, false>));
        CAC_TRY(smem_optin(ctx, cc_filter<false, false>));
        // pinned, 16-byte aligned host arrays: the pieces are pulled by a kernel
        L.z_u = pinned_device_view(h_u);
        L.z_v = pinned_device_view(h_v);
        if (!L.z_u || !L.z_v || ((reinterpret_cast<uintptr_t>(L.z_u) | reinterpret_cast<uintptr_t>(L.z_v)) & 15))
            L.z_u = L.z_v = nullptr;
        for (uint32_t i = 0; i < kStreamPieces; i++) L.parts.push_back({i * seg, piece});
        for (uint32_t i = 0; i < kStreamPieces; i++) {
            const uint64_t g0 = i * seg + piece, g1 = (i + 1 == kStreamPieces) ? m : (i + 1) * seg;
            if (g1 > g0) L.parts.push_back({g0, g1 - g0});
        }
    } else if (m) {
        // no filter: the whole list in kStreamPieces chunks with 16-byte aligned starts
        const uint64_t per = ((m + kStreamPieces - 1) / kStreamPieces + 1023) & ~1023ull;
        for (uint64_t e0 = 0; e0 < m; e0 += per) L.parts.push_back({e0, std::min(per, m - e0)});
    }

    // A repeated identical call replays a captured CUDA graph, as cc_run does: the first sighting
    // of a key runs directly, the second captures.
    CCStreamKey key{h_u, h_v, h_labels, d_u, d_v, d_labels, n, m, L.z_u != nullptr, ctx->arena.base, ctx->arena.cap};
    if (same_stream_key(key, ctx->cc_stream_key) && ctx->cc_stream_exec) {
        CAC_CUDA_TRY(cudaGraphLaunch(ctx->cc_stream_exec, s));
    } else if (same_stream_key(key, ctx->cc_stream_key)) {
        cudaGraph_t graph = nullptr;
        CAC_CUDA_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        const int st = stream_enqueue(ctx, L, true);
        const cudaError_t ce = cudaStreamEndCapture(s, &graph);
        if (st != CAC_OK) {
            if (graph) cudaGraphDestroy(graph);
            return st;
        }
        CAC_CUDA_TRY(ce);
        const cudaError_t ie = cudaGraphInstantiate(&ctx->cc_stream_exec, graph, 0);
        cudaGraphDestroy(graph);
        if (ie != cudaSuccess) {
            ctx->cc_stream_exec = nullptr;
            cudaGetLastError();
            CAC_TRY(stream_enqueue(ctx, L, false));
        } else {
            CAC_CUDA_TRY(cudaGraphLaunch(ctx->cc_stream_exec, s));
        }
    } else {
        if (ctx->cc_stream_exec) cudaGraphExecDestroy(ctx->cc_stream_exec);
        ctx->cc_stream_exec = nullptr;
        ctx->cc_stream_key = key;
        CAC_TRY(stream_enqueue(ctx, L, false));
    }
    CAC_CUDA_TRY(cudaStreamSynchronize(s));
    CAC_TRY(check_ids_word(ctx, n));
    if (res) {
        res->num_components = ctx->pinned_u32[0];
        res->rounds = (L.filtered ? 1u : 0u) + (m > 0 ? 1u : 0u);  // sample pieces + streamed gaps
        res->sampled_edges = L.filtered ? kStreamPieces * piece : 0;
        CAC_CUDA_TRY(cudaEventElapsedTime(&res->device_ms, ctx->ev[0], ctx->ev[3]));
        CAC_CUDA_TRY(cudaEventElapsedTime(&res->sample_ms, ctx->ev[0], ctx->ev[1]));
        CAC_CUDA_TRY(cudaEventElapsedTime(&res->edge_pass_ms, ctx->ev[1], ctx->ev[2]));
        CAC_CUDA_TRY(cudaEventElapsedTime(&res->label_ms, ctx->ev[2], ctx->ev[3]));
    }
    return CAC_OK;
}

}  // namespace cac

// ---------------------------------------------------------------------------------------------
// Allocation-free connected components (cac_cc_noalloc).
//
// Some callers cannot allocate device memory: a plugin running inside a host framework whose
// device memory is owned by that framework's allocator, or a latency-bound serving path that
// must not take cudaMalloc's implicit synchronisation. For them this entry point runs the
// single-pass form of the CC query (hook every edge, compress, count, label) with all of its
// scratch in one file-scope device array of fixed size, so it performs no device allocation of
// its own. The array belongs to this module: every GPU that loads the library holds it (16 MiB
// for the parent array plus 33 KiB of tile counters and offsets) until the process exits.
namespace cac {
namespace {

constexpr uint32_t kNoAllocMaxVertices = 1u << 22;  // 4,194,304 vertices
constexpr uint32_t kNoAllocMaxTiles = (kNoAllocMaxVertices + kTile - 1) / kTile;
constexpr int kNoAllocMaxDevices = 64;

struct NoAllocScratch {
    uint32_t parent[kNoAllocMaxVertices];
    uint32_t counts[kNoAllocMaxTiles + 1];
    uint32_t offsets[kNoAllocMaxTiles + 1];
    uint32_t total[64];
};

__device__ __align__(256) NoAllocScratch g_noalloc_scratch;

// The component count, or 0xFFFFFFFF when an edge endpoint was >= n (the edge was skipped).
__global__ void cc_noalloc_count(const uint32_t *total, uint32_t *out) {
    pdl_wait();
    *out = total[kErrWord] ? 0xFFFFFFFFu : total[0];
}

// Per-device set-up, with that device current: the device address of the scratch array (its
// host-side name is only a stand-in) and the SM count used to size the grids. A device counts as
// set up only once both succeeded, so a call that failed here (for instance one made while its
// stream was being captured, when the module may still have to be loaded) is retried in full by
// the next call instead of failing for the rest of the process.
struct NoAllocDevice {
    std::mutex mu;
    bool ready = false;
    NoAllocScratch *scratch = nullptr;
    int sms = 0;
};
NoAllocDevice g_noalloc_devices[kNoAllocMaxDevices];

cudaError_t noalloc_setup(NoAllocDevice &D, int dev) {
    std::lock_guard<std::mutex> lock(D.mu);
    if (D.ready) return cudaSuccess;
    void *p = nullptr;
    int sms = 0;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) {
        cudaGetLastError();  // not sticky: the next call tries again
        return e;
    }
    D.scratch = reinterpret_cast<NoAllocScratch *>(p);
    D.sms = sms;
    D.ready = true;
    return cudaSuccess;
}

}  // namespace
}  // namespace cac

extern "C" int cac_cc_noalloc(uint32_t n, uint64_t m, const uint32_t *u_dev, const uint32_t *v_dev,
                              uint32_t *labels_dev, uint32_t *num_components_dev, void *stream) {
    using namespace cac;
    if (n > kNoAllocMaxVertices) {
        set_error("cac_cc_noalloc: n = " + std::to_string(n) + " exceeds the allocation-free limit of " +
                  std::to_string(kNoAllocMaxVertices) + " vertices; use cac_cc for larger graphs");
        return CAC_ERR_INVALID;
    }
    if (m > 0xFFFFFFFFull || (m && (!u_dev || !v_dev))) {
        set_error("cac_cc_noalloc: invalid edge arrays (m must be < 2^32 and u/v non-null when m > 0)");
        return CAC_ERR_INVALID;
    }
    int dev = 0;
    CAC_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kNoAllocMaxDevices) {
        set_error("cac_cc_noalloc: device ordinal " + std::to_string(dev) + " out of range");
        return CAC_ERR_INVALID;
    }
    NoAllocDevice &D = g_noalloc_devices[dev];
    const cudaError_t se = noalloc_setup(D, dev);
    if (se != cudaSuccess) {
        set_error(std::string("cac_cc_noalloc: scratch set-up failed (the call may be retried): ") +
                  cudaGetErrorString(se));
        return CAC_ERR_CUDA;
    }
    cudaStream_t s = (cudaStream_t)stream;
    NoAllocScratch *S = D.scratch;
    auto grid = [&](uint64_t work) {
        return (int)std::max<uint64_t>(1, std::min<uint64_t>((work + kThreads - 1) / kThreads, (uint64_t)D.sms * 8));
    };
    if (n == 0) {
        // no vertices: 0 components, or 0xFFFFFFFF when there are edges (every endpoint is >= n)
        if (num_components_dev) CAC_CUDA_TRY(cudaMemsetAsync(num_components_dev, m ? 0xFF : 0, 4, s));
        return CAC_OK;
    }
    // Nothing in the scratch needs to start at zero: parent[] is initialised by cc_init, the tile
    // counters and the total are fully written before they are read.
    const uint32_t ntiles = (uint32_t)(((uint64_t)n + kTile - 1) / kTile);
    cc_init<<<grid(n), kThreads, 0, s>>>(S->parent, n);
    CAC_CUDA_TRY(cudaMemsetAsync(S->total + kErrWord, 0, 4, s));
    if (m > 0) {
        const bool vec = ((reinterpret_cast<uintptr_t>(u_dev) | reinterpret_cast<uintptr_t>(v_dev)) & 15) == 0;
        if (vec) cc_edge_pass<true, true, false><<<grid((m + 3) / 4), kThreads, 0, s>>>(S->parent, u_dev, v_dev, m, n,
                                                                                 S->total + kErrWord);
        else cc_edge_pass<false, true, false><<<grid(m), kThreads, 0, s>>>(S->parent, u_dev, v_dev, m, n, S->total + kErrWord);
    }
    CAC_TRY(label_components(D.sms, S->parent, n, ntiles, S->counts, S->offsets, S->total, labels_dev, false, s));
    if (num_components_dev) cc_noalloc_count<<<1, 1, 0, s>>>(S->total, num_components_dev);
    CAC_CUDA_TRY(cudaGetLastError());
    return CAC_OK;
}
