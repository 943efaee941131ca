// Minimum cut: the GB300 form of the reference's square_root low-concurrency trial loop
// (src/SquareRootCut.cpp:86-148) with every trial of every virtual rank in flight at once.
//
// One trial (virtual rank r, index i) = the reference's SequentialSquareRootCut::compute
// (src/SequentialSquareRootCut.cpp:4-67) followed by one Karger-Stein trial
// (src/karger-stein/co_mincut.h:176-223):
//   Stage 1  iss_shrink_kernel, one CTA per trial: rounds of (vertex count) weighted draws over
//            the edges that are not loops, contracted in draw order by a shared-memory union-find
//            until t = min(n, ceil(2 sqrt(m) + 1)) vertices remain; vertices renamed to the rank
//            of their smallest member.
//   Stage 2  dense_build_kernel: the t x t adjacency matrix of the contracted graph in HBM
//            (u64 entries, global atomics per edge).
//   Stage 3  Karger-Stein, level-synchronous over all trials of a wave:
//              prep_rows_kernel  row sums + 32-column block prefixes of the matrices that came
//                                without them
//              contract_kernel   one CTA per child: draws (row by a scan of the row sums, block
//                                by its prefixes, column by a scan of the block), contraction in draw
//                                order until max(ceil(n/sqrt 2)+1, 128) vertices, labels by rank
//                                of the smallest member, member lists by counting sort
//              quotient_tri_kernel / quotient_tile_kernel / quotient_shared_row_kernel
//                                the child's matrix: a few output rows at a time as one tile in shared
//                                memory, member rows summed on the way in, joined columns added to their
//                                groups' first ones, those stored; at large N a CTA per output row
//              sw_leaf_kernel    one warp per leaf (n <= 128), four vertices per lane:
//                                Stoer-Wagner maximum-adjacency
//                                phases with Nagamochi-Ono-Ibaraki contractions on the matrix held
//                                in shared memory (its lower triangle); atomicMin into the
//                                trial's cut
// The random stream of every draw is addressed by (seed + r, i, tag, 0) and (round, draw index),
// tag 1 for Stage 1 and 1 + h for the Karger-Stein child with heap index h, so a CPU replay of
// the same trial reproduces it bit for bit (oracle/mincut.c).
#include "cac_internal.h"
#include "sitmo.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <type_traits>
#include <utility>

namespace cac {
namespace {

constexpr uint32_t kSharedRows = 8;         // output rows per CTA of the shared-row quotient

constexpr uint32_t kMaxSmemVertices = kMaxDenseVertices;  // union-find of a contraction held in shared memory
constexpr int kBatch = 1024;                  // draws gathered before the ordered contraction
constexpr int kNT = 512;                      // threads of the per-trial / per-task CTAs
constexpr uint32_t kLeafN = 128;              // nodes up to this size are solved exactly
constexpr uint32_t kRootFlag = 0x80000000u;   // a contraction's vertex word: label, first of its group
constexpr uint32_t kDropped = 0xFFFFFFFFu;    // task whose source matrix has no edges left
constexpr uint64_t kU64Max = 0xFFFFFFFFFFFFFFFFull;

// Stage 1 of one trial: its graph, its contraction target and its stream key, its scratch.
struct ShrinkDesc {
    const uint32_t *U, *V, *W;
    uint64_t m;
    uint64_t *pre;     // ceil(m / 4): inclusive prefix of the non-loop weights at the end of each four edges
    uint32_t *lab;     // n: output labels (rank of the smallest member)
    uint32_t *k_out;   // output: number of vertices left
    uint32_t n, target;
    uint32_t k0, idx;  // stream key words 0, 1: seed + virtual rank, trial index within the rank
};

// Stage 2 of one trial: scatter its (relabelled) edges into its k x k matrix.
struct DenseDesc {
    const uint32_t *U, *V, *W;
    const uint32_t *lab;  // nullable: identity
    void *mat;            // k x k, u32 entries when `small`, else u64
    uint64_t m;
    uint32_t k, small;
    // planned ahead: k is the trial's target, checked against Stage 1's own count before any write
    const uint32_t *k_act = nullptr;
    uint32_t *err = nullptr;
};

struct SrcDesc {
    const void *mat;      // N x N row-major, u32 entries when `small`, else u64
    uint64_t *rowsum;     // N row sums
    uint64_t *blk;        // N x nb: per row, inclusive prefix of 32-column block sums
    uint64_t *cut;        // the trial's cut (root matrices deliver the minimum weighted degree bound)
    uint32_t N, nb;
    uint32_t is_root, small;  // small: the graph's total weight is below 2^32
};

struct TaskDesc {
    uint64_t tag;         // stream key word 2 (1 + heap index)
    uint64_t *cut;        // the trial's cut
    uint16_t *lab;        // N labels (output; all vertices and counts are at most 16384)
    uint16_t *memb_off;   // k + 1 offsets (output)
    uint16_t *members;    // N vertices grouped by label, each group's smallest first (output)
    uint16_t *cols;       // the quotient's column lists (output, see kColHead)
    uint32_t *rows;       // k: label | member offset << 16, by falling group size (output)
    uint32_t src;         // index into the SrcDesc array
    uint32_t target;
    uint32_t round;
    uint32_t k0, idx;     // stream key words 0, 1
    uint32_t brief;       // a child planned to be solved or built from its triangle: only the labels and first
                          // vertices are wanted
};

struct LeafDesc {
    const void *mat;          // u32 entries when `small`, else u64
    uint64_t *cut;
    const uint64_t *rowsum;   // the N row sums written with the matrix (a quotient's), or null
    uint32_t N;
    uint32_t small;  // entries fit in 32 bits
};

// Node matrices are stored with u32 entries when the graph's total weight is below 2^32 (every
// entry, row sum and cut of every node fits), else u64.
// Kernels that read or write node matrices are instantiated for one entry width Tm each and
// skip the nodes of the other width; the host launches the u64 instance only when some node of
// the step needs it.
// Row stride of an N x N node matrix: N rounded up to a multiple of 4 entries, so that every row
// starts on a 16-byte boundary (16-byte loads). Entries past column N - 1 are never used.
__host__ __device__ __forceinline__ uint64_t ld_of(uint32_t N) { return ((uint64_t)N + 3) & ~(uint64_t)3; }

// Column lists that a contraction leaves for the quotient, u16 entries:
//   [0, kEll)  joined[j]: how many small groups have more than j members beside their first
//   [kColMulti], [kColBig], [kColEll]  small groups with joined members, big groups, list entries
//   from kColHead: the k groups' first (smallest) vertices in label order; then, list by list
//   j = 0 .. kEll - 1, the joined[j] small groups' member j + 1 (groups by falling size, so that the
//   groups still going are a prefix); then the small groups' first vertices in the same order. Each
//   part is padded to an even count. Big groups have more than kEll members beside their first.
constexpr uint32_t kEll = 32, kColMulti = 32, kColBig = 33, kColEll = 34, kColHead = 64;
// u32 words of a contraction's output arrays: rows, then lab, members, memb_off and cols (u16)
__host__ __device__ __forceinline__ uint32_t even16(uint32_t x) { return (x + 1) / 2; }
inline uint32_t task_words(uint32_t N) {
    return N + 2 * even16(N) + even16(N + 1) + even16(kColHead + N + N / 2 + 4);
}

template <typename Tm>
__device__ __forceinline__ bool width_is(uint32_t small) {
    return (small != 0) == (sizeof(Tm) == 4);
}

// ---------------------------------------------------------------- block helpers

template <int NT>
__device__ __forceinline__ uint64_t block_excl_scan_u64(uint64_t x, uint64_t &total) {
    __shared__ uint64_t warp_tot[NT / 32];
    const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint64_t s = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t y = __shfl_up_sync(0xffffffffu, s, o);
        if (l >= o) s += y;
    }
    if (l == 31) warp_tot[w] = s;
    __syncthreads();
    if (w == 0) {
        uint64_t t = l < NT / 32 ? warp_tot[l] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t y = __shfl_up_sync(0xffffffffu, t, o);
            if (l >= o) t += y;
        }
        if (l < NT / 32) warp_tot[l] = t;
    }
    __syncthreads();
    const uint64_t off = w ? warp_tot[w - 1] : 0;
    total = warp_tot[NT / 32 - 1];
    __syncthreads();
    return off + s - x;
}

template <int NT>
__device__ __forceinline__ uint32_t block_excl_scan_u32(uint32_t x, uint32_t &total) {
    uint64_t t64;
    const uint64_t r = block_excl_scan_u64<NT>(x, t64);
    total = (uint32_t)t64;
    return (uint32_t)r;
}

__device__ __forceinline__ uint32_t sfind_ro(const uint32_t *par, uint32_t x) {
    uint32_t nx;
    while ((nx = par[x]) != x) x = nx;
    return x;
}

// Contract the draw pairs sb[0, nb) into the shared-memory union-find `par` (roots are component
// minima) in draw order until *s_count reaches target -- the sequential rule of the trial.
// With need = count - target links still allowed, the next `need` draws are linked by all threads
// at once (CAS of the larger root onto the smaller, finds without compression): each draw links
// at most once, so the count cannot fall below target, and since draws after the one that reaches
// target link nothing, the partition equals the sequential one. A successful CAS always joins
// two different components, so the number of links is the exact count drop. Repeated until the
// target or the end of the batch; the last few links (need <= kWarpTail) are made by one warp the
// same way, without block barriers. Endpoints of linked draws are pointed at their roots after each step.
constexpr uint32_t kWarpTail = 32;

template <int NT>
__device__ void contract_batch(uint32_t *par, const uint2 *sb, uint32_t nb, uint32_t target, uint32_t *s_count,
                               uint32_t *s_nlog) {
    volatile uint32_t *vp = par;
    uint32_t j0 = 0;
    for (;;) {
        __syncthreads();
        const uint32_t c = *s_count;
        if (c <= target || j0 >= nb) break;
        const uint32_t need = c - target;
        if (need <= kWarpTail) {
            __syncthreads();  // every warp has read *s_count before the tail writes it
            if (threadIdx.x < 32) {
                // 32 draws at a time: those that are loops already stay so; the first `left` others are
                // linked (at most once each, so the count cannot fall below target), the rest looked at again
                const uint32_t lane = threadIdx.x;
                uint32_t cc = c;
                for (uint32_t j = j0; j < nb && cc > target;) {
                    uint32_t x = 0, y = 0;
                    if (j + lane < nb) {
                        x = sb[j + lane].x;
                        y = sb[j + lane].y;
                        while (vp[x] != x) x = vp[x];
                        while (vp[y] != y) y = vp[y];
                    }
                    const uint32_t open = __ballot_sync(0xffffffffu, x != y), left = cc - target;
                    const bool mine = x != y && (uint32_t)__popc(open & ((1u << lane) - 1)) < left;
                    const uint32_t taken = __ballot_sync(0xffffffffu, mine);
                    bool linked = false;
                    while (mine && x != y) {
                        const uint32_t hi = x > y ? x : y, lo = x > y ? y : x;
                        linked = atomicCAS(&par[hi], hi, lo) == hi;
                        if (linked) break;
                        x = hi;  // hi was linked meanwhile: find both roots again
                        y = lo;
                        while (vp[x] != x) x = vp[x];
                        while (vp[y] != y) y = vp[y];
                    }
                    cc -= __popc(__ballot_sync(0xffffffffu, linked));
                    j += taken != open ? 32 - __clz(taken) : 32;
                    __syncwarp();
                }
                if (lane == 0) *s_count = cc;
            }
            __syncthreads();
            break;
        }
        const uint32_t j1 = min(nb, j0 + need);
        if (threadIdx.x == 0) *s_nlog = 0;
        __syncthreads();
        for (uint32_t j = j0 + threadIdx.x; j < j1; j += NT) {
            uint32_t x = sb[j].x, y = sb[j].y;
            for (;;) {
                while (vp[x] != x) x = vp[x];
                while (vp[y] != y) y = vp[y];
                if (x == y) break;
                const uint32_t hi = x > y ? x : y, lo = x > y ? y : x;
                if (atomicCAS(&par[hi], hi, lo) == hi) {
                    atomicAdd(s_nlog, 1u);
                    break;
                }
                x = hi;  // hi was linked meanwhile: find both roots again
                y = lo;
            }
        }
        __syncthreads();
        for (uint32_t j = j0 + threadIdx.x; j < j1; j += NT) {  // point the endpoints at their roots
            const uint32_t x = sb[j].x, y = sb[j].y;
            par[x] = sfind_ro(par, x);
            par[y] = sfind_ro(par, y);
        }
        if (threadIdx.x == 0) *s_count = c - *s_nlog;
        j0 = j1;
    }
    __syncthreads();
}

// first index i in [0, len) with a[i] > y (a non-decreasing, a[len-1] > y)
__device__ __forceinline__ uint64_t upper_bound_u64(const uint64_t *a, uint64_t len, uint64_t y) {
    uint64_t lo = 0, hi = len - 1;
    while (lo < hi) {
        const uint64_t mid = (lo + hi) >> 1;
        if (a[mid] > y) hi = mid; else lo = mid + 1;
    }
    return lo;
}

// first index i in [0, end) with a[i] > y (a non-decreasing, a[end-1] > y), in global memory: seven probes in
// flight per step; `before` receives a[i-1] (0 for i = 0). In [0, end) whatever a holds: below a child that a
// run planned ahead and that stopped off its target, matrices and prefixes were never written (the run is
// redone, but these contractions still draw from them).
// kConst: nothing writes a during the kernel.
template <bool kConst>
__device__ __forceinline__ uint32_t upper_bound8(const uint64_t *a, uint32_t end, uint64_t y, uint64_t &before) {
    uint32_t lo = 0, len = end;
    before = 0;
    for (;;) {
        const uint32_t s = (len + 7) / 8;
        uint64_t x[7];
#pragma unroll
        for (uint32_t i = 0; i < 7; i++) {
            const uint64_t *p = a + min(lo + (i + 1) * s - 1, end - 1);
            x[i] = kConst ? __ldg(p) : *p;
        }
        uint32_t c = 0;
#pragma unroll
        for (uint32_t i = 0; i < 7; i++)
            if (x[i] <= y) {
                c++;
                before = x[i];
            }
        lo = min(lo + c * s, end - 1);
        if (s == 1) return lo;
        len = min(s, end - lo);
    }
}

// Rank-of-minimum relabel of a compressed min-linked union-find (roots are minima): roots get
// their rank in vertex order, every vertex its root's label. Writes `lab` (global).
template <int NT, typename LabT>
__device__ void rank_labels(const uint32_t *par, uint32_t n, LabT *lab) {
    uint32_t off = 0;
    for (uint32_t base = 0; base < n; base += NT) {
        const uint32_t v = base + threadIdx.x;
        const uint32_t f = (v < n && par[v] == v) ? 1u : 0u;
        uint32_t tot;
        const uint32_t r = block_excl_scan_u32<NT>(f, tot);
        if (f) lab[v] = (LabT)(off + r);
        off += tot;
    }
    __syncthreads();
    for (uint32_t v = threadIdx.x; v < n; v += NT) {
        const uint32_t r = par[v];
        if (r != v) lab[v] = lab[r];
    }
    __syncthreads();
}

// ---------------------------------------------------------------- stage 1

// Stage 1 of one trial per CTA. Per round: the weights of the edges that are not loops and their
// inclusive prefix in edge order, in one pass (warp w owns a contiguous range of whole coarse segments and
// scans it from 0; four consecutive edges per lane, so one warp scan per 128), kept at the end of each
// four edges, and a coarse index in shared memory of the prefix at the end of every `cs`-edge segment,
// to which the warps' offsets are added; then draws in batches, little more than the links still
// wanted (a stream block each four): a draw finds its segment in the shared
// index, its four edges by eight-way search inside the segment, less its warp's offset, and its edge from
// their weights again, by the components of the round's start (16 bits a vertex, kept beside the
// union-find); the batch is contracted in draw order.
//   Bound by latency: the passes over the edges and, per batch, the chain of a draw and of its union.
//   60 trials of ER(1000, 0.05) 26 us, the trials of a 64-graph batch 6.7 ms. With a prefix per edge (8 bytes
// written per edge and round) 32 us and 8.6 ms; with two passes over the edges (sums, then prefixes), 32 edges
// at a time, a block per draw and binary searches 39 us and 10.1 ms.
constexpr uint32_t kCoarse = 2048;      // Stage 1 coarse prefix index entries (shared memory)
constexpr uint32_t kCoarseRows = 1024;  // contraction: coarse row-prefix index entries (shared memory)

template <int NT>
__global__ void __launch_bounds__(NT) iss_shrink_kernel(const ShrinkDesc *__restrict__ descs) {
    constexpr int NW = NT / 32;
    extern __shared__ __align__(16) unsigned char dsm[];
    uint2 *sb = reinterpret_cast<uint2 *>(dsm);
    uint64_t *coarse = reinterpret_cast<uint64_t *>(dsm + kBatch * sizeof(uint2));
    uint32_t *par = reinterpret_cast<uint32_t *>(dsm + kBatch * sizeof(uint2) + kCoarse * sizeof(uint64_t));
    __shared__ uint32_t s_count, s_nlog;
    __shared__ uint64_t s_w[NW], s_off[NW];
    const ShrinkDesc D = descs[blockIdx.x];
    const uint32_t n = D.n, target = D.target;
    const uint64_t m = D.m;
    const uint32_t *__restrict__ U = D.U;
    const uint32_t *__restrict__ V = D.V;
    const uint32_t *__restrict__ Wt = D.W;
    uint64_t *pre = D.pre;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint16_t *start = reinterpret_cast<uint16_t *>(par + n);  // the components when the round began
    for (uint32_t v = threadIdx.x; v < n; v += NT) {
        par[v] = v;
        start[v] = (uint16_t)v;
    }
    if (threadIdx.x == 0) s_count = n;
    __syncthreads();
    // coarse segments of a multiple of 32 edges, at most kCoarse of them; a warp owns whole ones
    const uint64_t cs = max((uint64_t)32, ((m + kCoarse - 1) / kCoarse + 31) / 32 * 32);
    const uint32_t ncs = (uint32_t)((m + cs - 1) / cs), own = (ncs + NW - 1) / NW;
    const uint64_t wlo = min(m, (uint64_t)warp * own * cs), whi = min(m, wlo + own * cs);
    const uint32_t csg = (uint32_t)(cs / 32);
    const bool wide = (((uintptr_t)U | (uintptr_t)V | (uintptr_t)Wt) & 15) == 0;
    // edges e .. e + 3 of those below `end`, else 0-0
    auto quad_at = [&](uint64_t e, uint64_t end, uint4 &u, uint4 &v, uint4 &w) {
        u = v = w = make_uint4(0, 0, 0, 0);
        if (wide && e + 4 <= end) {
            u = __ldg(reinterpret_cast<const uint4 *>(U + e));
            v = __ldg(reinterpret_cast<const uint4 *>(V + e));
            w = __ldg(reinterpret_cast<const uint4 *>(Wt + e));
        } else {
            if (e < end) u.x = __ldg(U + e), v.x = __ldg(V + e), w.x = __ldg(Wt + e);
            if (e + 1 < end) u.y = __ldg(U + e + 1), v.y = __ldg(V + e + 1), w.y = __ldg(Wt + e + 1);
            if (e + 2 < end) u.z = __ldg(U + e + 2), v.z = __ldg(V + e + 2), w.z = __ldg(Wt + e + 2);
            if (e + 3 < end) u.w = __ldg(U + e + 3), v.w = __ldg(V + e + 3), w.w = __ldg(Wt + e + 3);
        }
    };
    for (uint64_t rnd = 0; s_count > target; rnd++) {
        uint64_t carry = 0;
        for (uint64_t e0 = wlo; e0 < whi; e0 += 128) {
            const uint64_t e = e0 + 4 * lane;
            uint4 u, v, w;
            quad_at(e, whi, u, v, w);
            const uint64_t sum = (uint64_t)(par[u.x] != par[v.x] ? w.x : 0) + (par[u.y] != par[v.y] ? w.y : 0) +
                                 (par[u.z] != par[v.z] ? w.z : 0) + (par[u.w] != par[v.w] ? w.w : 0);
            uint64_t incl = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint64_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            const uint64_t end = carry + incl;
            carry += __shfl_sync(0xffffffffu, incl, 31);
            if (e < whi) pre[e / 4] = end;
            // the end of a segment (lanes 7, 15, 23 and 31 end 32 edges) or of the list
            if ((lane & 7) == 7 && e < whi) {
                const uint32_t groups = (uint32_t)(e / 32) + 1;
                if (groups % csg == 0) coarse[groups / csg - 1] = end;
            }
            if (e < whi && e + 4 >= m) coarse[ncs - 1] = end;  // (by the warp that owns the last edge)
        }
        if (lane == 0) s_w[warp] = carry;
        __syncthreads();
        uint64_t W = 0;
        for (int i = 0; i < NW; i++) W += s_w[i];
        if (W == 0) break;  // the remaining graph has no edges between its vertices
        if (threadIdx.x < NW) {
            uint64_t before = 0;
            for (int i = 0; i < (int)threadIdx.x; i++) before += s_w[i];
            s_off[threadIdx.x] = before;
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < ncs; i += NT) coarse[i] += s_off[i / own];
        const uint32_t c_start = s_count;
        __syncthreads();
        for (uint32_t base = 0; base < c_start;) {
            const uint32_t need = s_count - target;
            const uint32_t nb = min(min((uint32_t)kBatch, c_start - base), (need + need / 8 + 32 + NT - 1) / NT * NT);
            for (uint32_t q = threadIdx.x; 4 * q < nb; q += NT) {
                const u64x4 o = sitmo_block(D.k0, D.idx, 1, 0, (base >> 2) + q, rnd, 0, 0);
#pragma unroll
                for (uint32_t i = 0; i < 4; i++) {
                    const uint64_t y = mulhi64(o.x[i], W);
                    sb[4 * q + i] = make_uint2((uint32_t)y, (uint32_t)(y >> 32));
                }
            }
            __syncthreads();
            for (uint32_t j = threadIdx.x; j < nb; j += NT) {
                const uint64_t y = (uint64_t)sb[j].y << 32 | sb[j].x;
                const uint32_t sg = (uint32_t)upper_bound_u64(coarse, ncs, y);
                const uint64_t s0 = sg * cs, off = s_off[sg / own];
                uint64_t before;
                const uint32_t quad = upper_bound8<false>(pre + s0 / 4, (uint32_t)((min(cs, m - s0) + 3) / 4), y - off, before);
                if (quad == 0) before = sg % own ? coarse[sg - 1] - off : 0;
                // the quad's edges again, with the components of the round's start
                const uint64_t e = s0 + 4 * quad;
                uint4 u, v, w;
                quad_at(e, m, u, v, w);
                const uint64_t rem = y - off - before;
                const uint64_t p1 = start[u.x] != start[v.x] ? w.x : 0, p2 = p1 + (start[u.y] != start[v.y] ? w.y : 0),
                               p3 = p2 + (start[u.z] != start[v.z] ? w.z : 0);
                const uint32_t a = rem < p1 ? u.x : rem < p2 ? u.y : rem < p3 ? u.z : u.w;
                const uint32_t b = rem < p1 ? v.x : rem < p2 ? v.y : rem < p3 ? v.z : v.w;
                sb[j] = make_uint2(a, b);
            }
            contract_batch<NT>(par, sb, nb, target, &s_count, &s_nlog);
            if (s_count <= target) break;
            base += nb;
        }
        for (uint32_t v = threadIdx.x; v < n; v += NT) {
            const uint32_t r = sfind_ro(par, v);
            par[v] = r;
            start[v] = (uint16_t)r;
        }
        __syncthreads();
    }
    rank_labels<NT>(par, n, D.lab);
    if (threadIdx.x == 0) *D.k_out = s_count;
}

// ---------------------------------------------------------------- stage 2

__global__ void dense_build_kernel(const DenseDesc *__restrict__ descs) {
    const DenseDesc D = descs[blockIdx.y];
    if (D.k_act && *D.k_act != D.k) {  // Stage 1 stopped off the target: redo the run
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(D.err, kErrPlan);
        return;
    }
    const uint64_t ldk = ld_of(D.k);
    for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < D.m; e += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t a = D.U[e], b = D.V[e];
        if (D.lab) {
            a = D.lab[a];
            b = D.lab[b];
        }
        if (a == b) continue;
        const uint32_t w = D.W[e];
        if (D.small) {
            atomicAdd(reinterpret_cast<uint32_t *>(D.mat) + (uint64_t)a * ldk + b, w);
            atomicAdd(reinterpret_cast<uint32_t *>(D.mat) + (uint64_t)b * ldk + a, w);
        } else {
            atomicAdd(reinterpret_cast<unsigned long long *>(D.mat) + (uint64_t)a * ldk + b, (unsigned long long)w);
            atomicAdd(reinterpret_cast<unsigned long long *>(D.mat) + (uint64_t)b * ldk + a, (unsigned long long)w);
        }
    }
}

// ---------------------------------------------------------------- stage 3: Karger-Stein

// last i of [0, n) with first[i] <= x (first[0] = 0), by a warp: 32 probes per step
__device__ __forceinline__ uint32_t warp_last_le(const uint64_t *__restrict__ first, uint32_t n, uint64_t x) {
    uint32_t lo = 0, len = n;  // the answer is in [lo, lo + len)
    while (len > 1) {
        const uint32_t step = (len + 31) / 32, at = lo + step * (threadIdx.x & 31);
        const uint32_t hits = __popc(__ballot_sync(0xffffffffu, at < lo + len && first[at] <= x));
        const uint32_t end = lo + len;
        lo += (hits - 1) * step;
        len = min(step, end - lo);
    }
    return lo;
}

// One warp per matrix row: 32-column block prefixes and the row sum.
//   u32 entries: 16-byte loads, four in flight (512 columns, 16 blocks); the eight lanes of a block add up
// by a transposing reduction (4 shuffles for the 4 loads), one shuffle puts the 16 sums in order and a
// 16-lane scan makes them prefixes. Row sums are below 2^32. Bound by memory and, for short rows, by the
// latency of the search for the row's source (32-way) and of its loads.
//   K4000's root (4000 rows) and 16.4 GB of children of N = 2005 of the Watts-Strogatz query: 54 us and
// 3.0 ms; with a load per 32 columns, 64-bit shuffles (10 per block) and a binary search 181 us and 6.6 ms.
template <typename Tm>
__global__ void prep_rows_kernel(const SrcDesc *__restrict__ srcs, const uint64_t *__restrict__ row_off,
                                 uint32_t nsrc, uint64_t total_rows) {
    const uint64_t gw = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t lane = threadIdx.x & 31;
    if (gw >= total_rows) return;
    const uint32_t si = warp_last_le(row_off, nsrc, gw);  // last source whose first row <= gw
    const SrcDesc S = srcs[si];
    const uint64_t i = gw - row_off[si];
    if (!width_is<Tm>(S.small)) return;
    const Tm *mat = reinterpret_cast<const Tm *>(S.mat) + i * ld_of(S.N);
    uint64_t *blk = S.blk + i * S.nb;
    uint64_t run = 0;
    if constexpr (sizeof(Tm) == 4) {
        for (uint32_t c0 = 0; c0 < S.N; c0 += 512) {
            uint32_t x[4];
            uint4 v[4];
#pragma unroll
            for (uint32_t u = 0; u < 4; u++) {
                const uint32_t c = c0 + u * 128 + lane * 4;
                v[u] = c < S.N ? __ldg(reinterpret_cast<const uint4 *>(mat + c)) : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
            for (uint32_t u = 0; u < 4; u++) {  // (entries past the last column are not defined)
                const uint32_t c = c0 + u * 128 + lane * 4;
                x[u] = v[u].x + (c + 1 < S.N ? v[u].y : 0) + (c + 2 < S.N ? v[u].z : 0) + (c + 3 < S.N ? v[u].w : 0);
            }
            // of each pair of loads a lane keeps one and hands the other over: load u = bits 2, 1 of the lane
            const bool hi = lane & 4, mid = lane & 2;
            uint32_t s0 = hi ? x[2] : x[0], s1 = hi ? x[3] : x[1];
            s0 += __shfl_xor_sync(0xffffffffu, hi ? x[0] : x[2], 4);
            s1 += __shfl_xor_sync(0xffffffffu, hi ? x[1] : x[3], 4);
            uint32_t t = mid ? s1 : s0;
            t += __shfl_xor_sync(0xffffffffu, mid ? s0 : s1, 2);
            t += __shfl_xor_sync(0xffffffffu, t, 1);
            // block b of the 16: load b / 4, lanes 8 (b % 4) ..
            const uint32_t b = lane & 15;
            uint32_t p = __shfl_sync(0xffffffffu, t, (b & 3) * 8 + (b >> 2) * 2);
#pragma unroll
            for (uint32_t o = 1; o < 16; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, p, o);
                if (b >= o) p += y;
            }
            if (lane < 16 && c0 / 32 + b < S.nb) blk[c0 / 32 + b] = run + p;
            run += __shfl_sync(0xffffffffu, p, 15);
        }
    } else {
        for (uint32_t b0 = 0; b0 < S.nb; b0 += 8) {  // eight 32-column blocks per pass, loads in flight together
            uint64_t x[8];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const uint32_t j = (b0 + u) * 32 + lane;
                x[u] = (b0 + u < S.nb && j < S.N) ? (uint64_t)__ldg(mat + j) : 0;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
                for (int u = 0; u < 8; u++) x[u] += __shfl_xor_sync(0xffffffffu, x[u], o);
            }
#pragma unroll
            for (int u = 0; u < 8; u++) {
                run += x[u];
                if (lane == u && b0 + u < S.nb) blk[b0 + u] = run;
            }
        }
    }
    if (lane == 0) {
        S.rowsum[i] = run;
        if (S.is_root) atomicMin((unsigned long long *)S.cut, (unsigned long long)run);
    }
}

// One CTA per child: contracts the child's copy of the source to its target and writes the labels, member
// lists and the quotient's lists. The row sums that came with the source are scanned here (one segment of
// `cr` rows per entry of a coarse index in shared memory; cr = 1 up to kCoarseRows vertices), so a step needs
// no kernel for their prefix. Draws are made as the contraction asks for them -- at least as many as links
// are still wanted -- not a whole round of N at once: the stream is indexed by the draw, so those not made
// change nothing. A draw: its stream block (four draws each) and position, its row by the index, its
// 32-column block by eight-way search of the row's block prefixes, its column from one 128-byte load of
// the block (u32).
//   Bound by the latency of the serial phases (block prefix and column loads, about 20 block barriers,
// the union-find), so what counts is how many CTAs an SM holds: kContractSmall threads up to
// kContractSmallN source vertices, kContractMid up to kContractMidN, else kNT.
//   With 512 threads at every size, a prefix kernel per step, whole rounds of draws (a stream block each),
// binary searches in global memory and labels read back from there, K4000's 11 levels took 1.11 ms and
// 0.09 ms of prefixes (14,336 sources of N = 182: 347 us), the three of ER(1000, 0.05) 67 us and 15 us, a
// 64-graph batch 12.7 ms and 0.57 ms; this takes 0.52 ms (129 us), 42 us and 5.3 ms.
constexpr uint32_t kContractSmall = 128, kContractSmallN = 256;
constexpr uint32_t kContractMid = 256, kContractMidN = 724;

__host__ __device__ __forceinline__ uint32_t contract_batch_cap(uint32_t N) { return N < kBatch ? (N + 3) & ~3u : kBatch; }

// the column of one 32-column block (row starts are 16-byte aligned, so the block is too): first of the
// block's `lim` entries whose running sum exceeds rem; lim if none does
__device__ __forceinline__ uint32_t block_column(const uint32_t *p, uint32_t lim, uint64_t rem) {
    uint4 x[8];
#pragma unroll
    for (int q = 0; q < 8; q++) x[q] = 4u * q < lim ? __ldg(reinterpret_cast<const uint4 *>(p) + q) : make_uint4(0, 0, 0, 0);
    uint32_t acc = 0, c = 0;
    const uint32_t r = (uint32_t)rem;  // row sums are below 2^32
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const uint32_t e[4] = {x[q].x, x[q].y, x[q].z, x[q].w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            acc += 4u * q + i < lim ? e[i] : 0u;  // (entries past the last column are not defined)
            c += acc <= r ? 1u : 0u;
        }
    }
    return min(c, lim);
}
__device__ __forceinline__ uint32_t block_column(const uint64_t *p, uint32_t lim, uint64_t rem) {
    uint64_t acc = 0;
    uint32_t c = 0;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        ulonglong2 x[8];
#pragma unroll
        for (int q = 0; q < 8; q++)
            x[q] = 16u * h + 2u * q < lim ? __ldg(reinterpret_cast<const ulonglong2 *>(p) + 8 * h + q) : make_ulonglong2(0, 0);
#pragma unroll
        for (int q = 0; q < 8; q++) {
            acc += 16u * h + 2u * q < lim ? x[q].x : 0ull;
            c += acc <= rem ? 1u : 0u;
            acc += 16u * h + 2u * q + 1 < lim ? x[q].y : 0ull;
            c += acc <= rem ? 1u : 0u;
        }
    }
    return min(c, lim);
}

template <int NT, typename Tm>
__global__ void __launch_bounds__(NT, 1024 / NT) contract_kernel(const TaskDesc *__restrict__ tasks, const SrcDesc *__restrict__ srcs,
                                                      const uint32_t *__restrict__ list, uint32_t *__restrict__ k_out,
                                                      uint32_t *err) {
    extern __shared__ __align__(16) unsigned char dsm[];
    __shared__ uint32_t s_count, s_nlog;
    const uint32_t task = list[blockIdx.x];
    const TaskDesc T = tasks[task];
    const SrcDesc S = srcs[T.src];
    if (!width_is<Tm>(S.small)) return;
    const uint32_t N = S.N, cap = contract_batch_cap(N), lane = threadIdx.x & 31;
    // row prefix at the end of every `cr`-row segment (every row when N <= kCoarseRows)
    const uint32_t cr = (N + kCoarseRows - 1) / kCoarseRows;
    const uint32_t ncr = (N + cr - 1) / cr;
    uint64_t *crow = reinterpret_cast<uint64_t *>(dsm);         // ncr entries: coarse row index
    uint2 *sb = reinterpret_cast<uint2 *>(crow + ncr);          // cap draws
    uint32_t *par = reinterpret_cast<uint32_t *>(sb + cap);     // N: union-find, then label | root flag
    uint32_t *cnt = par + N;                                    // N: labels of roots, then member offsets
    uint32_t *num = cnt + N;                                    // N: members beside the first, then scatter cursors
    const Tm *mat = reinterpret_cast<const Tm *>(S.mat);
    for (uint32_t v = threadIdx.x; v < N; v += NT) {
        par[v] = v;
        num[v] = 0;
    }
    if (threadIdx.x == 0) s_count = N;
    uint64_t W;
    {  // a thread's segments are consecutive, so one block scan orders them all
        const uint32_t per = (ncr + NT - 1) / NT, i0 = min(threadIdx.x * per, ncr), i1 = min(i0 + per, ncr);
        uint64_t sum = 0;
        for (uint32_t r = i0 * cr; r < min(i1 * cr, N); r++) sum += __ldg(S.rowsum + r);
        uint64_t run = block_excl_scan_u64<NT>(sum, W);
        for (uint32_t i = i0; i < i1; i++) {
            for (uint32_t r = i * cr; r < min((i + 1) * cr, N); r++) run += __ldg(S.rowsum + r);
            crow[i] = run;
        }
    }
    if (W == 0) {  // no edges between the vertices: the cut is 0, nothing to contract
        if (threadIdx.x == 0) {
            k_out[task] = kDropped;
            atomicMin((unsigned long long *)T.cut, 0ull);
        }
        return;
    }
    __syncthreads();
    for (uint32_t base = 0; base < N;) {
        // a little more than the links still wanted, whole passes of the CTA
        const uint32_t need = s_count - T.target;
        const uint32_t nb = min(min(cap, N - base), (need + need / 8 + 32 + NT - 1) / NT * NT);
        for (uint32_t q = threadIdx.x; 4 * q < nb; q += NT) {
            const u64x4 o = sitmo_block(T.k0, T.idx, T.tag, 0, (base >> 2) + q, T.round, 0, 0);
#pragma unroll
            for (uint32_t i = 0; i < 4; i++) {
                const uint64_t y = mulhi64(o.x[i], W);
                sb[4 * q + i] = make_uint2((uint32_t)y, (uint32_t)(y >> 32));
            }
        }
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < nb; j += NT) {
            const uint2 yy = sb[j];
            const uint64_t y = (uint64_t)yy.y << 32 | yy.x;
            // row: first whose inclusive prefix exceeds y (segment in shared memory, then inside it)
            const uint32_t sg = (uint32_t)upper_bound_u64(crow, ncr, y);
            uint32_t a = sg * cr;
            uint64_t before = sg ? crow[sg - 1] : 0;
            if (cr > 1) {
                const uint32_t r1 = min(a + cr, N) - 1;
                for (; a < r1; a++) {
                    const uint64_t x = __ldg(S.rowsum + a);
                    if (before + x > y) break;
                    before += x;
                }
            }
            const uint64_t rem = y - before;
            uint64_t left;
            const uint32_t b = upper_bound8<true>(S.blk + (uint64_t)a * S.nb, S.nb, rem, left);
            const uint32_t lim = min(32u, N - b * 32);
            uint32_t c = block_column(mat + (uint64_t)a * ld_of(N) + (uint64_t)b * 32, lim, rem - left);
            if (c >= lim) {  // cannot happen with consistent prefixes; record and clamp
                atomicOr(err, 1u);
                c = lim - 1;
            }
            sb[j] = make_uint2(a, b * 32 + c);
        }
        contract_batch<NT>(par, sb, nb, T.target, &s_count, &s_nlog);
        if (s_count <= T.target) break;
        base += nb;
    }
    const uint32_t k = s_count;
    // labels: a root's rank among the roots, every vertex its root's. groups of 32 vertices are ranked by ballots
    // and one block scan over the groups' counts (at most NT of them)
    __shared__ uint32_t s_group[NT];
    const uint32_t groups = (N + 31) / 32;
    for (uint32_t g = threadIdx.x / 32; g < groups; g += NT / 32) {
        const uint32_t v = g * 32 + lane;
        uint32_t r = v;
        if (v < N) par[v] = r = sfind_ro(par, v);
        const uint32_t roots = __ballot_sync(0xffffffffu, v < N && r == v);
        if (lane == 0) s_group[g] = __popc(roots);
    }
    __syncthreads();
    uint32_t total;
    uint32_t ex = block_excl_scan_u32<NT>(threadIdx.x < groups ? s_group[threadIdx.x] : 0, total);
    if (threadIdx.x < groups) s_group[threadIdx.x] = ex;
    __syncthreads();
    for (uint32_t g = threadIdx.x / 32; g < groups; g += NT / 32) {
        const uint32_t v = g * 32 + lane;
        const bool root = v < N && par[v] == v;
        const uint32_t roots = __ballot_sync(0xffffffffu, root);
        if (root) cnt[v] = s_group[g] + __popc(roots & ((1u << lane) - 1));
    }
    if (T.brief) {
        __syncthreads();
        for (uint32_t v = threadIdx.x; v < N; v += NT) {
            const uint32_t r = par[v], l = cnt[r];
            T.lab[v] = (uint16_t)l;
            if (r == v) T.cols[kColHead + l] = (uint16_t)v;
        }
        if (threadIdx.x == 0) k_out[task] = k;
        return;
    }
    // member lists grouped by label, and the quotient's row order and column lists (order inside a group
    // is irrelevant): num[l] first counts the group's members beside its first
    __shared__ uint32_t s_hist[kEll + 2], s_pos[kEll + 2], s_off[kEll], s_base[2];
    if (threadIdx.x < kEll + 2) s_hist[threadIdx.x] = 0;
    __syncthreads();
    for (uint32_t v = threadIdx.x; v < N; v += NT) {
        const uint32_t r = par[v], l = cnt[r];
        T.lab[v] = (uint16_t)l;
        if (r != v) atomicAdd(&num[l], 1u);
        par[v] = r == v ? l | kRootFlag : l;
    }
    __syncthreads();
    const uint32_t lgroups = (k + 31) / 32;
    for (uint32_t g = threadIdx.x / 32; g < lgroups; g += NT / 32) {
        const uint32_t l = g * 32 + lane, x = l < k ? num[l] : 0;
        if (x) atomicAdd(&s_hist[min(x, kEll + 1)], 1u);
        const uint32_t sum = __reduce_add_sync(0xffffffffu, l < k ? x + 1 : 0);
        if (lane == 0) s_group[g] = sum;
    }
    __syncthreads();
    const uint32_t nbig = s_hist[kEll + 1];
    if (threadIdx.x < kEll) {  // joined[j] = small groups with more than j: a suffix sum over the warp's lanes
        const uint32_t j = threadIdx.x;
        uint32_t joined = s_hist[j + 1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_down_sync(0xffffffffu, joined, o);
            if (j + o < 32) joined += y;
        }
        uint32_t incl = joined;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if ((int)j >= o) incl += y;
        }
        const uint32_t nell = __shfl_sync(0xffffffffu, incl, 31), nmulti = __shfl_sync(0xffffffffu, joined, 0);
        s_off[j] = incl - joined;
        s_pos[j] = joined;  // the small groups with exactly j joined members follow those with more
        T.cols[j] = (uint16_t)joined;
        if (j == 0) {
            s_pos[kEll] = 0;
            s_pos[kEll + 1] = 0;            // big groups: the head of the row order
            s_pos[0] = nbig + nmulti;       // single vertices: its tail
            T.cols[kColMulti] = (uint16_t)nmulti;
            T.cols[kColBig] = (uint16_t)nbig;
            T.cols[kColEll] = (uint16_t)nell;
            s_base[0] = kColHead + ((k + 1) & ~1u);
            s_base[1] = s_base[0] + ((nell + 1) & ~1u);
        }
    }
    ex = block_excl_scan_u32<NT>(threadIdx.x < lgroups ? s_group[threadIdx.x] : 0, total);
    if (threadIdx.x < lgroups) s_group[threadIdx.x] = ex;
    if (threadIdx.x == 0) T.memb_off[k] = (uint16_t)N;
    __syncthreads();
    uint16_t *first = T.cols + kColHead, *ell = T.cols + s_base[0], *multi = T.cols + s_base[1];
    for (uint32_t g = threadIdx.x / 32; g < lgroups; g += NT / 32) {
        const uint32_t l = g * 32 + lane, x = l < k ? num[l] : 1u;
        uint32_t incl = l < k ? x + 1 : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        const uint32_t off = s_group[g] + incl - (x + 1);
        const uint32_t single = __ballot_sync(0xffffffffu, x == 0);  // most groups: one atomic per warp
        uint32_t at = 0, pos = 0xFFFFu;
        if (lane == 0 && single) at = atomicAdd(&s_pos[0], (uint32_t)__popc(single));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(single & ((1u << lane) - 1));
        if (l < k) {
            if (x > kEll) at = atomicAdd(&s_pos[kEll + 1], 1u);
            else if (x) at = nbig + (pos = atomicAdd(&s_pos[x], 1u));
            T.rows[at] = l | off << 16;
            T.memb_off[l] = (uint16_t)off;
            cnt[l] = off;
            num[l] = pos << 16;  // becomes (position among the small groups, scatter cursor)
        }
    }
    __syncthreads();
    for (uint32_t v = threadIdx.x; v < N; v += NT) {
        const uint32_t l = par[v] & ~kRootFlag, at = cnt[l];
        if (par[v] & kRootFlag) {
            T.members[at] = (uint16_t)v;
            first[l] = (uint16_t)v;
            const uint32_t pos = num[l] >> 16;
            if (pos != 0xFFFFu) multi[pos] = (uint16_t)v;
        } else {
            const uint32_t c = atomicAdd(&num[l], 1u), rank = c & 0xFFFFu, pos = c >> 16;
            T.members[at + 1 + rank] = (uint16_t)v;
            if (pos != 0xFFFFu) ell[s_off[rank] + pos] = (uint16_t)v;
        }
    }
    if (threadIdx.x == 0) k_out[task] = k;
}

// ---------------------------------------------------------------- lower triangles in shared memory
// Entry (i, j < i) at i (i - 1) / 2 + j: the entries (x, v) of 32 consecutive v lie in 32 different banks on
// either side of x (triangular numbers take every residue of a power of two once).
__device__ __forceinline__ uint32_t tri(uint32_t i) { return i * (i - 1) / 2; }
__device__ __forceinline__ uint32_t tpos(uint32_t i, uint32_t j) { return i > j ? tri(i) + j : tri(j) + i; }

template <typename Tm>
__device__ __forceinline__ void copy_entry_async(Tm *dst, const Tm *src) {
    if constexpr (sizeof(Tm) == 4)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                     : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                     : "memory");
}

// ---------------------------------------------------------------- quotient
// Q[a][b] = sum over u in group a, v in group b of A[u][v], the diagonal zeroed, with every row's
// 32-column block prefixes and its sum (the next step's row prep). Three kernels with identical results:
// the lower triangle of a small child (quotient_tri_kernel, see tri_fits), tiles of R rows (quotient_tile_kernel)
// up to kTileMaxN source vertices (kTileMaxN64 with u64 entries), one row per CTA (quotient_shared_row_kernel) above.
//
// R output rows make a tile: R rows of N entries in shared memory, so that every column index is
// read once for R rows. The rows of a tile are interleaved in 16-byte chunks (a column's R entries
// are a constant distance apart, so one address serves R loads), for R = 4 with a spare chunk after
// each 4 so that neighbouring chunks of a row start in different banks. A CTA of 8 warps works on 8, 4, 2
// or 1 tiles at a time, 1, 2, 4 or 8 warps on each; tiles are taken from the CTA's share as warps get
// free. Per tile:
//   1. the first member row of each output row is copied in asynchronously (16 bytes per copy), the
//      other members are summed in registers meanwhile, 8 loads in flight, and added (each thread to
//      the columns that it copied);
//   2. every joined column is added to its group's first column: a thread per small group walks the
//      lists of cols (no atomics), a warp per big group sums its members;
//   3. the groups' first columns are the output row: first[b] grows with b, so the tile is read nearly
//      in order and each lane stores 4 columns of each row with 16-byte stores; 8 lanes make a
//      32-column block sum;
//   4. the block sums become prefixes.
// Weighted contraction makes groups of hundreds of members at the deeper levels, so the rows are dealt
// out by falling group size: the R rows of a tile from R different parts of the order, the tiles of a
// CTA from all over it, the largest first.
// Bound by latency within each step (loads of step 1, index -> entry chains of 2 and 3): its steps
// alone take 150 us (1) and 160 us (2 to 4) of the 340 at N = 356, where the bytes read and written
// take 135 of HBM's time. The forms that this replaces added every source column into its label's slot
// with a shared atomic. Measured on the levels of a recursion from K4000 (7 trials; us per level of
// 225 M source entries, contraction drawn by weight), old -> new: N = 182 755 -> 386, 253 540 -> 308,
// 356 473 -> 341, 709 552 -> 357, 1416 750 -> 477, 2830 553 -> 511; at 4000 one row per CTA takes 340.
constexpr uint32_t kTileThreads = 256;
constexpr uint32_t kTileRows = 256;      // most output rows per CTA
constexpr uint32_t kTileSmem = 74 * 1024;  // three CTAs per SM
// Up to these source vertices; one row per CTA above. The rows' time over the tiles' in whole queries (complete graphs,
// 2 and 16 trials; equal weights / skewed ones, which make groups of hundreds of members), u32 entries: N = 2000 1.00,
// 1.00 / 1.14, 1.07; 2900 1.00, 0.99 / 1.10, 1.02; 3200 1.01, 0.99 / 1.15, 1.04; 4000 0.99, 0.99 / 1.22, 1.04. u64 entries,
// where a row's shared atomics are 64 bits wide: 2900 1.01, 1.00 / 1.42, 1.39; 4000 0.98, 0.99 / 1.47, 1.37; 5000 1.01, 1.00 / 1.53, 1.38
// (the largest measured).
constexpr uint32_t kTileMaxN = 2900, kTileMaxN64 = 5000;

struct TilePlan {
    uint32_t rows;   // R
    uint32_t esize;  // bytes of an entry
    uint32_t smem;   // bytes of shared memory per CTA
    uint32_t tiles;  // tiles per group of warps
};

__host__ __device__ __forceinline__ uint32_t first_pad(uint32_t k) { return (k + 127) & ~127u; }
// the lists: header, first (padded), joined columns (at most two entries each)
__host__ __device__ __forceinline__ uint32_t tile_idx_bytes(uint32_t N, uint32_t k) {
    return (kColHead * 2 + first_pad(k) * 2 + (N - k + 2) * 4 + 15) & ~15u;
}
// one tile: its chunks and one of zeros, the block sums of its rows and their diagonal entries
__host__ __device__ __forceinline__ uint32_t tile_bytes(uint32_t N, uint32_t rows, uint32_t esize) {
    const uint32_t chunk = 16 * (rows == 4 ? 5 : rows);
    return (uint32_t)(ld_of(N) * esize / 16 + 1) * chunk + ((rows * ((N + 31) / 32 + 1) * esize + 15) & ~15u);
}
// tiles at a time: the most of 8, 4, 2, 1 that fit `smem`
__host__ __device__ __forceinline__ uint32_t tile_groups(uint32_t N, uint32_t k, const TilePlan &p, uint32_t smem) {
    const uint32_t idx = tile_idx_bytes(N, k), one = tile_bytes(N, p.rows, p.esize);
    const uint32_t room = smem > idx ? smem - idx : 0;
    return room >= 8 * one ? 8u : room >= 4 * one ? 4u : room >= 2 * one ? 2u : 1u;
}

// tiles per CTA
__host__ __device__ __forceinline__ uint32_t tile_per_cta(uint32_t groups, const TilePlan &p) {
    return groups * p.tiles < kTileRows / p.rows ? groups * p.tiles : kTileRows / p.rows;
}

// One child of a launch.
struct TileTask {
    const void *mat;          // N x N
    const uint16_t *cols, *members, *memb_off;
    const uint32_t *rows;
    void *q;                  // k x k
    uint64_t *rowsum;         // k row sums, then k x ceil(k / 32) block prefixes
    const uint32_t *kact;     // planned ahead: the contraction's own count, else null
    uint32_t N, k;
};
struct TileArgs {
    const TileTask *task;
    const uint64_t *first;    // their first CTAs
    uint32_t ntasks, uniform; // uniform: CTAs of every task where all have the same number, else 0
    uint32_t *err;
    TilePlan plan;
};

// asynchronous copy of 16 bytes to shared memory, past L1
__device__ __forceinline__ void copy16_async(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

__device__ __forceinline__ void vadd(uint4 &a, const uint4 &b) {
    a.x += b.x;
    a.y += b.y;
    a.z += b.z;
    a.w += b.w;
}
__device__ __forceinline__ void vadd(ulonglong2 &a, const ulonglong2 &b) {
    a.x += b.x;
    a.y += b.y;
}

__device__ __forceinline__ void tile_sync(uint32_t group, uint32_t warps) {  // the warps of one tile
    if (warps == 1) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(warps * 32) : "memory");
}

template <typename Tm, int R>
__global__ void __launch_bounds__(kTileThreads, 3) quotient_tile_kernel(const __grid_constant__ TileArgs A) {
    extern __shared__ __align__(16) unsigned char dsm[];
    using Vec = typename std::conditional<sizeof(Tm) == 4, uint4, ulonglong2>::type;
    constexpr uint32_t VEC = 16 / sizeof(Tm);        // columns per chunk
    constexpr uint32_t CS = VEC * (R == 4 ? 5 : R);  // entries from a chunk to the next of its row
    __shared__ uint32_t s_take[8], s_next;
    __shared__ uint32_t s_row[kTileRows][2];  // label | members << 16, first member position
    const uint32_t li = A.uniform ? blockIdx.x / A.uniform : warp_last_le(A.first, A.ntasks, blockIdx.x);
    const uint32_t cta = A.uniform ? blockIdx.x - li * A.uniform : (uint32_t)(blockIdx.x - A.first[li]);
    const TileTask T = A.task[li];
    const uint32_t k = T.k, N = T.N;
    if (T.kact && *T.kact != k) {  // planned ahead, and this child stopped off its target: redo the run
        if (threadIdx.x == 0) atomicOr(A.err, kErrPlan);
        return;
    }
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t ldN = ld_of(N), ldk = ld_of(k);
    const uint32_t nch = (uint32_t)(ldN / VEC), nbk = (k + 31) / 32;
    const uint32_t groups = tile_groups(N, k, A.plan, A.plan.smem), wpt = 8 / groups;  // warps per tile
    const uint32_t grp = warp / wpt, wl = warp % wpt, tl = wl * 32 + lane, tt = wpt * 32;
    const Tm *__restrict__ mat = reinterpret_cast<const Tm *>(T.mat);
    // a vertex as an entry offset in the tile (below 2^16)
    auto slot = [](uint32_t c) { return c + c / VEC * (CS - VEC); };
    uint16_t *s_cols = reinterpret_cast<uint16_t *>(dsm), *s_first = s_cols + kColHead;
    const uint32_t kpad = first_pad(k);
    const uint32_t nmulti = T.cols[kColMulti], nbig = T.cols[kColBig], nell = T.cols[kColEll];
    uint16_t *s_ell = s_first + kpad, *s_multi = s_ell + ((nell + 1) & ~1u);
    // this CTA's tiles: cta, cta + ctas, ...; tile t has the rows at t, t + ntiles, ... of the order
    const uint32_t ntiles = (k + R - 1) / R, per = tile_per_cta(groups, A.plan), ctas = (ntiles + per - 1) / per;
    for (uint32_t i = threadIdx.x; i < kColHead; i += kTileThreads) s_cols[i] = T.cols[i];
    for (uint32_t i = threadIdx.x; i < kpad; i += kTileThreads)  // (padded with the chunk of zeros)
        s_first[i] = (uint16_t)slot(i < k ? T.cols[kColHead + i] : (uint32_t)ldN);
    {
        const uint16_t *ell = T.cols + kColHead + ((k + 1) & ~1u);
        for (uint32_t i = threadIdx.x; i < ((nell + 1) & ~1u) + nmulti; i += kTileThreads) s_ell[i] = (uint16_t)slot(ell[i]);
    }
    for (uint32_t i = threadIdx.x; i < per * R; i += kTileThreads) {
        const uint32_t t = i / R * ctas + cta, at = t + i % R * ntiles;
        if (t >= ntiles) break;
        const uint32_t x = T.rows[at < k ? at : t], l = x & 0xFFFFu;  // (a repeated row stores the same again)
        s_row[i][0] = l | (uint32_t)(T.memb_off[l + 1] - T.memb_off[l]) << 16;
        s_row[i][1] = x >> 16;
    }
    if (threadIdx.x == 0) s_next = 0;
    // entry of row r at offset x: tile[x + r * VEC]
    Tm *tile = reinterpret_cast<Tm *>(dsm + tile_idx_bytes(N, k) + (size_t)grp * tile_bytes(N, R, sizeof(Tm)));
    Tm *bsum = tile + (nch + 1) * CS, *sdiag = bsum + R * nbk;
    if (tl < R * VEC) tile[nch * CS + tl] = 0;
    Tm *Q = reinterpret_cast<Tm *>(T.q);
    uint64_t *blk = T.rowsum + k;
    __syncthreads();
    for (uint32_t it = 0;; it++) {
        uint32_t mine = it;
        if (wpt == 1) {
            if (lane == 0) mine = atomicAdd(&s_next, 1u);
            mine = __shfl_sync(0xffffffffu, mine, 0);
        } else if (wpt < 8) {
            if (tl == 0) s_take[grp] = atomicAdd(&s_next, 1u);
            tile_sync(grp, wpt);
            mine = s_take[grp];
        }
        if (mine >= per || mine * ctas + cta >= ntiles) break;
        // 1. member rows
        uint32_t lab[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            lab[r] = s_row[mine * R + r][0] & 0xFFFFu;
            const uint32_t f = s_first[lab[r]], v = f / CS * VEC + f % CS;  // the slot's vertex
            const Tm *row = mat + v * ldN + tl * VEC;
            Tm *dst = tile + tl * CS + r * VEC;
            for (uint32_t c = tl; c < nch; c += tt, row += tt * VEC, dst += tt * CS) copy16_async(dst, row);
        }
        bool waited = false;
#pragma unroll 1
        for (int r = 0; r < R; r++) {
            const uint32_t size = s_row[mine * R + r][0] >> 16;
            if (size == 1) continue;
            const uint32_t q0 = s_row[mine * R + r][1] + 1, q1 = q0 + size - 1;
            for (uint32_t c = tl; c < nch; c += 2 * tt) {
                const bool two = c + tt < nch;
                Vec acc[2] = {Vec{}, Vec{}};
                for (uint32_t p = q0; p < q1; p += 4) {
                    Vec q[4][2];
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        q[u][0] = q[u][1] = Vec{};
                        if (p + u < q1) {
                            const Vec *row = reinterpret_cast<const Vec *>(mat + (uint64_t)T.members[p + u] * ldN) + c;
                            q[u][0] = __ldg(row);
                            if (two) q[u][1] = __ldg(row + tt);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        vadd(acc[0], q[u][0]);
                        vadd(acc[1], q[u][1]);
                    }
                }
                if (!waited) {
                    asm volatile("cp.async.wait_all;" ::: "memory");
                    waited = true;
                }
                Vec *d = reinterpret_cast<Vec *>(tile + c * CS + r * VEC);
                Vec x = *d;
                vadd(x, acc[0]);
                *d = x;
                if (two) {
                    d = reinterpret_cast<Vec *>(tile + (c + tt) * CS + r * VEC);
                    x = *d;
                    vadd(x, acc[1]);
                    *d = x;
                }
            }
        }
        if (!waited) asm volatile("cp.async.wait_all;" ::: "memory");
        tile_sync(grp, wpt);
        // 2. joined columns -> their groups' first columns
        for (uint32_t i = tl; i < nmulti; i += tt) {
            Tm *to = tile + s_multi[i];
            Tm acc[R];
#pragma unroll
            for (int r = 0; r < R; r++) acc[r] = to[r * VEC];
            const uint16_t *list = s_ell + i;
            const Tm *from = tile + *list;
            uint32_t joined = nmulti;
            for (uint32_t j = 1;; j++) {  // the next list entry is read ahead of this one's column
                list += joined;
                joined = j < kEll ? s_cols[j] : 0;
                const bool more = i < joined;
                const Tm *next = more ? tile + *list : nullptr;
#pragma unroll
                for (int r = 0; r < R; r++) acc[r] += from[r * VEC];
                if (!more) break;
                from = next;
            }
#pragma unroll
            for (int r = 0; r < R; r++) to[r * VEC] = acc[r];
        }
        for (uint32_t i = wl; i < nbig; i += wpt) {  // (the big groups lead the order)
            const uint32_t x = T.rows[i], l = x & 0xFFFFu, end = T.memb_off[l + 1];
            Tm acc[R] = {};
            for (uint32_t p = (x >> 16) + lane; p < end; p += 32) {
                const Tm *from = tile + slot(T.members[p]);
#pragma unroll
                for (int r = 0; r < R; r++) acc[r] += from[r * VEC];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int r = 0; r < R; r++) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], o);
            if (lane == 0)
#pragma unroll
                for (int r = 0; r < R; r++) tile[s_first[l] + r * VEC] = acc[r];
        }
        tile_sync(grp, wpt);
        // 3. first columns -> output rows and block sums (the diagonal is taken out in step 4)
        Tm *out[R];
#pragma unroll
        for (int r = 0; r < R; r++) out[r] = Q + lab[r] * ldk + lane * 4;
        for (uint32_t b0 = wl * 128; b0 < k; b0 += tt * 4) {
            const uint32_t b = b0 + lane * 4;
            Tm y[R][4];
            const uint2 f = *reinterpret_cast<const uint2 *>(s_first + b);
            const uint32_t x[4] = {f.x & 0xFFFFu, f.x >> 16, f.y & 0xFFFFu, f.y >> 16};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const Tm *from = tile + x[i];
#pragma unroll
                for (int r = 0; r < R; r++) y[r][i] = from[r * VEC];
            }
            Tm sum[R];
#pragma unroll
            for (int r = 0; r < R; r++) sum[r] = (y[r][0] + y[r][1]) + (y[r][2] + y[r][3]);
            if (b < k) {
#pragma unroll
                for (int r = 0; r < R; r++) {
                    Tm *q = out[r] + b0;
                    if constexpr (sizeof(Tm) == 4) {
                        *reinterpret_cast<uint4 *>(q) = make_uint4(y[r][0], y[r][1], y[r][2], y[r][3]);
                    } else {
                        *reinterpret_cast<ulonglong2 *>(q) = make_ulonglong2(y[r][0], y[r][1]);
                        *reinterpret_cast<ulonglong2 *>(q + 2) = make_ulonglong2(y[r][2], y[r][3]);
                    }
                }
            }
            // sums over the block's 8 lanes: the rows are halved among the lanes first, so that 4 rows take
            // 4 shuffles
            uint32_t row = 0, step = 1;
            if constexpr (R == 4) {
                const bool hi = lane & 1u;
                const Tm s0 = hi ? sum[0] : sum[2], s1 = hi ? sum[1] : sum[3];
                sum[0] = (hi ? sum[2] : sum[0]) + __shfl_xor_sync(0xffffffffu, s0, 1);
                sum[1] = (hi ? sum[3] : sum[1]) + __shfl_xor_sync(0xffffffffu, s1, 1);
                row = hi ? 2 : 0;
                step = 2;
            }
            const bool hi = lane & step;
            const Tm s0 = hi ? sum[0] : sum[1];
            sum[0] = (hi ? sum[1] : sum[0]) + __shfl_xor_sync(0xffffffffu, s0, step);
            row += hi;
#pragma unroll
            for (int o = R; o < 8; o *= 2) sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], o);
            if ((lane & 7u) < (uint32_t)R && b / 32 < nbk) bsum[row * nbk + b / 32] = sum[0];
        }
        if (tl < R) sdiag[tl] = tile[s_first[s_row[mine * R + tl][0] & 0xFFFFu] + tl * VEC];
        tile_sync(grp, wpt);
        // 4. block sums -> prefixes: `side` rows side by side in a warp, `width` lanes each
        const uint32_t width = nbk <= 8 ? 8u : nbk <= 16 ? 16u : 32u, side = 32 / width;
        for (uint32_t r0 = wl * side; r0 < (uint32_t)R; r0 += wpt * side) {
            const uint32_t r = r0 + lane / width, j1 = lane % width;
            const bool has = r < (uint32_t)R;
            const uint32_t l = has ? s_row[mine * R + r][0] & 0xFFFFu : 0;
            Tm carry = 0;
            for (uint32_t j0 = 0; j0 < nbk; j0 += width) {
                const uint32_t j = j0 + j1;
                Tm s = 0;
                if (has && j < nbk) {
                    s = bsum[r * nbk + j];
                    if (j == l / 32) {
                        s -= sdiag[r];
                        Q[l * ldk + l] = 0;
                    }
                }
                for (uint32_t o = 1; o < width; o <<= 1) {
                    const Tm y = __shfl_up_sync(0xffffffffu, s, o, width);
                    if (j1 >= o) s += y;
                }
                s += carry;
                if (has && j < nbk) blk[(uint64_t)l * nbk + j] = s;
                carry = __shfl_sync(0xffffffffu, s, width - 1, width);
            }
            if (has && j1 == 0) T.rowsum[l] = carry;
        }
    }
}

__device__ __forceinline__ void sadd(uint32_t *p, uint64_t v) { atomicAdd(p, (uint32_t)v); }
__device__ __forceinline__ void sadd(uint64_t *p, uint64_t v) {
    atomicAdd(reinterpret_cast<unsigned long long *>(p), (unsigned long long)v);
}

// Small children: one CTA per child, the child's lower triangle in shared memory. A warp per row copies the
// entries between first vertices from the source, at the columns of the first vertices (ascending, so the
// copies stay nearly coalesced); then a warp per joined vertex adds its row to its group's, from the first
// vertices' columns and from those of the joined vertices before it, with shared atomics; then a warp per
// row stores it, with its 32-column block prefixes and its sum. Half of the source is read, and a child takes
// half the instructions of its tiles, whose setup per CTA and per tile it also spares.
//   Taken while the triangle leaves room for three CTAs per SM (u32 entries: k <= 192; u64: 135): the
// children of K4000's levels of N = 255 and 182 took 320 and 350 us as tiles and take 244 and 287 us, those
// of the Watts-Strogatz query 11.7 and 14.0 ms a group, now 7.8 and 9.1. Larger ones would leave one CTA per SM
// or few warps, where the tiles keep three. Up to kTriSmallBytes six CTAs of 128 threads fit.
constexpr int kTriThreads = 256, kTriSmall = 128;
constexpr uint32_t kTriSmallBytes = 36 * 1024;
constexpr uint32_t kTriMaxK = 192, kTriMaxJoined = 96;
__host__ __device__ __forceinline__ uint32_t tri_bytes(uint32_t k, uint32_t esize) { return (k * (k - 1) / 2 + 1) * esize; }
__host__ __device__ __forceinline__ bool tri_fits(uint32_t N, uint32_t k, uint32_t small) {
    return k >= 2 && N - k <= kTriMaxJoined && tri_bytes(k, small ? 4 : 8) <= tri_bytes(kTriMaxK, 4);
}

__device__ __forceinline__ uint32_t warp_sum(uint32_t x) { return __reduce_add_sync(0xffffffffu, x); }
__device__ __forceinline__ uint64_t warp_sum(uint64_t x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

template <int NT, typename Tm>
__global__ void __launch_bounds__(NT, 768 / NT) quotient_tri_kernel(
    const TaskDesc *__restrict__ tasks, const SrcDesc *__restrict__ srcs, const uint32_t *__restrict__ list,
    const uint32_t *__restrict__ ks, const uint64_t *__restrict__ out_off, uint32_t ntasks, unsigned char *out_base,
    const uint32_t *__restrict__ k_act, uint32_t *err) {
    extern __shared__ __align__(16) unsigned char dsm[];
    constexpr uint32_t kWarps = NT / 32, Q = kTriMaxK / 32, B = kTriMaxJoined / 32;
    Tm *M = reinterpret_cast<Tm *>(dsm);
    __shared__ uint16_t s_first[kTriMaxK];
    __shared__ uint32_t s_joined[kTriMaxJoined], s_count;  // vertex | label << 16
    const uint32_t task = list[blockIdx.x], k = ks[task], lane = threadIdx.x & 31, warp = threadIdx.x / 32;
    if (k_act && k_act[task] != k) {  // planned ahead, and this child stopped off its target: redo the run
        if (threadIdx.x == 0) atomicOr(err, kErrPlan);
        return;
    }
    const TaskDesc T = tasks[task];
    const SrcDesc S = srcs[T.src];
    const uint32_t N = S.N;
    const Tm *__restrict__ mat = reinterpret_cast<const Tm *>(S.mat);
    const uint64_t ldN = ld_of(N);
    for (uint32_t l = threadIdx.x; l < kTriMaxK; l += NT) s_first[l] = l < k ? T.cols[kColHead + l] : (uint16_t)0;
    if (threadIdx.x == 0) s_count = 0;
    __syncthreads();
    for (uint32_t v0 = warp * 32; v0 < N; v0 += NT) {
        const uint32_t v = v0 + lane, l = v < N ? T.lab[v] : 0;
        const bool j = v < N && s_first[l] != v;
        const uint32_t js = __ballot_sync(0xffffffffu, j);
        uint32_t at = 0;
        if (lane == 0 && js) at = atomicAdd(&s_count, (uint32_t)__popc(js));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(js & ((1u << lane) - 1));
        if (j) s_joined[at] = v | l << 16;
    }
    uint32_t f[Q];
#pragma unroll
    for (uint32_t q = 0; q < Q; q++) f[q] = s_first[lane + 32 * q];
#pragma unroll 2
    for (uint32_t i = 1 + warp; i < k; i += kWarps) {
        const Tm *src = mat + s_first[i] * ldN;
        Tm *dst = M + tri(i) + lane;
#pragma unroll
        for (uint32_t q = 0; q < Q; q++)
            if (lane + 32 * q < i) copy_entry_async(dst + 32 * q, src + f[q]);
    }
    __syncthreads();
    const uint32_t joined = s_count;
    uint32_t other[B];  // the lane's joined vertices
#pragma unroll
    for (uint32_t q = 0; q < B; q++) other[q] = lane + 32 * q < joined ? s_joined[lane + 32 * q] : 0;
    bool waited = false;
    for (uint32_t p0 = 0; p0 < joined || !waited; p0 += 2 * kWarps) {
        Tm a[2][Q + B];
#pragma unroll
        for (uint32_t u = 0; u < 2; u++) {
            const uint32_t p = p0 + u * kWarps + warp;
            const Tm *row = mat + (p < joined ? s_joined[p] & 0xFFFFu : 0) * ldN;
#pragma unroll
            for (uint32_t q = 0; q < Q; q++) a[u][q] = p < joined && lane + 32 * q < k ? __ldg(row + f[q]) : Tm(0);
#pragma unroll
            for (uint32_t q = 0; q < B; q++)
                a[u][Q + q] = p < joined && lane + 32 * q < p ? __ldg(row + (other[q] & 0xFFFFu)) : Tm(0);
        }
        if (!waited) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            waited = true;
        }
#pragma unroll
        for (uint32_t u = 0; u < 2; u++) {
            const uint32_t p = p0 + u * kWarps + warp;
            if (p >= joined) break;
            const uint32_t to = s_joined[p] >> 16, tt = tri(to);
#pragma unroll
            for (uint32_t q = 0; q < Q + B; q++) {
                const uint32_t l = q < Q ? lane + 32 * q : other[q - Q] >> 16;
                if (a[u][q] != 0 && l != to) sadd(&M[l > to ? tri(l) + to : tt + l], a[u][q]);
            }
        }
    }
    __syncthreads();
    const uint64_t ldk = ld_of(k);
    const uint32_t nbk = (k + 31) / 32;
    Tm *out = reinterpret_cast<Tm *>(out_base + out_off[task]);
    uint64_t *sums = reinterpret_cast<uint64_t *>(out_base + out_off[ntasks + task]), *blk = sums + k;
    for (uint32_t l = warp; l < k; l += kWarps) {
        const uint32_t tl = tri(l);
        Tm x[Q], run = 0, mine = 0;  // (a row sum fits an entry)
#pragma unroll
        for (uint32_t q = 0; q < Q; q++) {
            const uint32_t c = lane + 32 * q;
            x[q] = c < k && c != l ? M[c > l ? tri(c) + l : tl + c] : Tm(0);
        }
#pragma unroll
        for (uint32_t q = 0; q < Q; q++) {
            if (lane + 32 * q < k) out[l * ldk + lane + 32 * q] = x[q];
            x[q] = warp_sum(x[q]);
        }
#pragma unroll
        for (uint32_t q = 0; q < Q; q++) {
            run += x[q];
            if (lane == q) mine = run;
        }
        if (lane < nbk) blk[(uint64_t)l * nbk + lane] = mine;
        if (lane == 0) sums[l] = run;
    }
}

// The quotient for large N: one CTA of 8 warps per group of `rows` consecutive output rows, all
// warps on the same output row at a time (labels + one row in shared memory: 5 CTAs, 40 warps per SM
// at N = 4000, where a tile leaves room for 16). The warps split the columns: 128-column chunks (one 16-byte load per lane), chunk c to warp c mod 8, four
// chunks per warp in flight. Per output row: zero the row, sum the member rows chunk by chunk and
// add every column into its label's slot (shared atomics), store the row with the diagonal zeroed
// and its 32-column block sums, then one warp turns the block sums into the block prefixes and the
// row sum (the next step's row prep). Five CTAs per SM (48 registers): measured 1-3% faster on
// K4000 than the four that 60 registers allow.
template <typename Ts, typename Tm>
__global__ void __launch_bounds__(256, 5) quotient_shared_row_kernel(const TaskDesc *__restrict__ tasks,
                                                                  const SrcDesc *__restrict__ srcs,
                                                                  const uint32_t *__restrict__ list, uint32_t nlist,
                                                                  const uint32_t *__restrict__ kdim,
                                                                  const uint64_t *__restrict__ group_task_off,
                                                                  uint32_t ntasks, uint32_t rows,
                                                                  const uint64_t *__restrict__ out_off,
                                                                  unsigned char *out_base, uint32_t lab_words,
                                                                  uint32_t kmax, const uint32_t *__restrict__ kact,
                                                                  uint32_t *err) {
    extern __shared__ __align__(16) unsigned char dsm[];
    const uint64_t gg = blockIdx.x;
    uint32_t at = 0, hi = nlist - 1;
    while (at < hi) {  // last task of the list whose first row group <= gg
        const uint32_t mid = (at + hi + 1) >> 1;
        if (group_task_off[mid] <= gg) at = mid; else hi = mid - 1;
    }
    const uint32_t lo = list[at];
    const TaskDesc T = tasks[lo];
    const SrcDesc S = srcs[T.src];
    const uint32_t k = kdim[lo];
    if (kact && kact[lo] != k) {  // planned ahead, and this child stopped off its target: redo the run
        if (threadIdx.x == 0) atomicOr(err, kErrPlan);
        return;
    }
    const uint32_t N = S.N;
    const uint32_t a0 = (uint32_t)(gg - group_task_off[at]) * rows, a1 = min(k, a0 + rows);
    if (!width_is<Tm>(S.small)) return;
    const Tm *mat = reinterpret_cast<const Tm *>(S.mat);
    constexpr int VEC = 16 / sizeof(Tm);  // columns per 16-byte load
    constexpr uint32_t NWARP = 8;
    using Vec = typename std::conditional<sizeof(Tm) == 4, uint4, ulonglong2>::type;
    const uint64_t ldN = ld_of(N);
    uint32_t *s_lab = reinterpret_cast<uint32_t *>(dsm);  // N
    Ts *qrow = reinterpret_cast<Ts *>(dsm + (size_t)lab_words * 4);  // kmax
    uint64_t *bsum = reinterpret_cast<uint64_t *>(dsm + (size_t)lab_words * 4 + (((size_t)kmax * sizeof(Ts) + 15) & ~(size_t)15));
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t i = threadIdx.x; i < N; i += blockDim.x) s_lab[i] = T.lab[i];
    Tm *Qt = reinterpret_cast<Tm *>(out_base + out_off[lo]);
    uint64_t *rowsum_out = reinterpret_cast<uint64_t *>(out_base + out_off[ntasks + lo]);
    const uint32_t small = S.small;
    const uint32_t nbk = (k + 31) / 32;
    uint64_t *blk = rowsum_out + k;
    const uint32_t nchunk = (N + 32 * VEC - 1) / (32 * VEC);
    // the row is zeroed once here, then by the output pass of every row as it reads it
    for (uint32_t b = threadIdx.x; b < k; b += blockDim.x) qrow[b] = 0;
    __syncthreads();  // labels staged, row zeroed
    for (uint32_t a = a0; a < a1; a++) {
        const uint32_t p0 = T.memb_off[a], p1 = T.memb_off[a + 1];
        for (uint32_t c0 = warp; c0 < nchunk; c0 += 4 * NWARP) {
            Tm x[4][VEC];
#pragma unroll
            for (int u = 0; u < 4; u++)
#pragma unroll
                for (int t = 0; t < VEC; t++) x[u][t] = 0;
            for (uint32_t p = p0; p < p1; p++) {
                const Vec *row = reinterpret_cast<const Vec *>(mat + (uint64_t)T.members[p] * ldN);
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const uint32_t c = (c0 + u * NWARP) * 32 * VEC + lane * VEC;
                    if (c < N) {
                        const Vec q = __ldg(row + c / VEC);
                        const Tm *e = reinterpret_cast<const Tm *>(&q);
#pragma unroll
                        for (int t = 0; t < VEC; t++) x[u][t] += e[t];
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < 4; u++)
#pragma unroll
                for (int t = 0; t < VEC; t++) {
                    const uint32_t j = (c0 + u * NWARP) * 32 * VEC + lane * VEC + t;
                    if (j < N && x[u][t]) sadd(&qrow[s_lab[j]], (uint64_t)x[u][t]);
                }
        }
        __syncthreads();  // the row is complete
        const uint64_t qb = (uint64_t)a * ld_of(k);
        for (uint32_t b0 = warp * 32; b0 < k; b0 += NWARP * 32) {
            const uint32_t b = b0 + lane;
            uint64_t v = (b < k && b != a) ? (uint64_t)qrow[b] : 0;
            if (b < k) {
                Qt[qb + b] = (Tm)v;
                qrow[b] = 0;  // for the next row (the barrier below orders it before that row's adds)
            }
            if (small) {  // every entry < 2^32: two 32-bit reductions of the 16-bit halves are exact
                const uint32_t lo16 = __reduce_add_sync(0xffffffffu, (uint32_t)(v & 0xFFFFu));
                const uint32_t hi16 = __reduce_add_sync(0xffffffffu, (uint32_t)(v >> 16));
                v = (uint64_t)lo16 + ((uint64_t)hi16 << 16);
            } else {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            }
            if (lane == 0) bsum[b0 >> 5] = v;
        }
        __syncthreads();  // block sums complete; the row may be zeroed again after the next barrier
        if (warp == 0) {
            // inclusive prefix of the block sums: lane l owns blocks [l * per, (l + 1) * per)
            const uint32_t per = (nbk + 31) / 32;
            const uint32_t j0 = lane * per, j1 = min(nbk, j0 + per);
            uint64_t own = 0;
            for (uint32_t j = j0; j < j1; j++) own += bsum[j];
            uint64_t incl = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint64_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= (uint32_t)o) incl += y;
            }
            uint64_t run = incl - own;
            for (uint32_t j = j0; j < j1; j++) {
                run += bsum[j];
                blk[(uint64_t)a * nbk + j] = run;
            }
            if (lane == 31) rowsum_out[a] = incl;
        }
    }
}

// Exact minimum cut of one leaf (n <= 128) by one warp, four vertices per lane: maximum-adjacency orderings
// as in the reference's Stoer-Wagner base case (co_mincut_base_case.hpp:52-144), with the
// Nagamochi-Ono-Ibaraki contraction rule (Nagamochi & Ibaraki 1992; Nagamochi, Ono & Ibaraki
// 1994): when vertex w's key reaches q >= lambda while vertex v is scanned, then lambda(v, w) >= q,
// so the edge (v, w) can be contracted without losing any cut below lambda, the best cut value found
// so far (initially the leaf's minimum weighted degree). Every ordering contracts all such
// certified edges plus the last two vertices (the cut of the phase updates lambda), so far fewer
// orderings are needed than the n - 1 of plain Stoer-Wagner; the returned value is the exact
// minimum cut of the leaf.
//   A vertex is one word, key << 8 | 255 - vertex, 0 once it is scanned, so the next vertex (largest
// key, smallest id) is one maximum over the warp; 32-bit words while the leaf weighs less than 2^24,
// else 64. Every certified edge and the pair (second to last, last) joins a vertex to one scanned
// before it, so when all but the first vertex of the ordering are so joined the leaf contracts to one
// vertex and the ordering's result is final (the usual case: Karger-Stein leaves of 128 vertices
// mostly finish in one ordering). Otherwise the joined vertices are merged into the roots of their
// trees, row by row.
//   The matrix is kept as its lower triangle, (i, j < i) at i (i - 1) / 2 + j: the entries (x, v) of 32
// consecutive v lie in 32 different banks on either side of x (triangular numbers take every residue
// of a power of two once), and 128 vertices take half the shared memory of the full matrix: six leaves
// per SM. It is copied in asynchronously, all rows in flight.
//   Bound by the latency of a step (maximum, four shared loads, add: about 130 cycles), not by issue or
// memory, so the step holds no branch and no barrier. A 128-thread CTA per leaf with a thread per
// vertex (a barrier and a cross-warp maximum per step, half matrix in 32 KB) took 714 us for the 14,336
// leaves of K4000's 56 trials, 73 us for the 480 of ER(1000, 0.05)'s 60 and 9.7 ms in 64 graphs' batch;
// this takes 300 us, 36 us and 3.6 ms. With the update under a branch per vertex a step took 570 cycles
// (789 us); with the unions walked by one lane a merge took 300 cycles more.
//   Keys stay below 2^56 (total graph weight checked on the host).
__device__ __forceinline__ uint64_t warp_min_u64(uint64_t x) {
    const uint32_t hi = (uint32_t)(x >> 32);
    const uint32_t top = __reduce_min_sync(0xffffffffu, hi);
    const uint32_t lo = __reduce_min_sync(0xffffffffu, hi == top ? (uint32_t)x : 0xFFFFFFFFu);
    return ((uint64_t)top << 32) | lo;
}

__device__ __forceinline__ uint64_t warp_max(uint64_t x) {
    const uint32_t hi = (uint32_t)(x >> 32);
    const uint32_t top = __reduce_max_sync(0xffffffffu, hi);
    const uint32_t lo = __reduce_max_sync(0xffffffffu, hi == top ? (uint32_t)x : 0u);
    return ((uint64_t)top << 32) | lo;
}
__device__ __forceinline__ uint32_t warp_max(uint32_t x) { return __reduce_max_sync(0xffffffffu, x); }

constexpr uint32_t kLeafThreads = 128, kLeafWarps = kLeafThreads / 32;  // they load; warp 0 solves
// The orderings; returns the leaf's minimum cut. Kt: the vertex words. root: 128 bytes of shared memory.
template <typename Tm, typename Kt>
__device__ __forceinline__ uint64_t leaf_cut(Tm *M, uint32_t N, uint64_t lambda, uint8_t *root) {
    const uint32_t lane = threadIdx.x;
    // at[q]: the vertex whose entries the lane reads in place q, 0 where it has none (the loads are not
    // predicated: what an inactive or scanned vertex reads is dropped)
    uint32_t v[4], at[4], tat[4];
    bool active[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        v[q] = lane + 32 * q;
        active[q] = v[q] < N;
        at[q] = active[q] ? v[q] : 0;
        tat[q] = tri(at[q]);
    }
    auto entry = [&](int q, uint32_t x, uint32_t tx) { return at[q] > x ? tat[q] + x : tx + at[q]; };
    uint32_t cnt = N;
    while (cnt > 1) {
        const Kt lam = (Kt)lambda << 8;
        Kt P[4];
        uint32_t mark[4];  // vertex to contract into, 255: none
#pragma unroll
        for (int q = 0; q < 4; q++) {
            P[q] = active[q] ? (Kt)(255u - v[q]) : (Kt)0;
            mark[q] = 255u;
        }
        uint32_t prev = 0;
        for (uint32_t step = 1; step < cnt; step++) {
            const Kt m01 = P[0] > P[1] ? P[0] : P[1], m23 = P[2] > P[3] ? P[2] : P[3];
            const Kt best = warp_max(m01 > m23 ? m01 : m23);
            const uint32_t sv = 255u - ((uint32_t)best & 255u), ts = tri(sv);
            prev = sv;
            Tm c[4];
#pragma unroll
            for (int q = 0; q < 4; q++) c[q] = M[entry(q, sv, ts)];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const bool open = P[q] != 0 && P[q] != best;
                const Kt next = P[q] + ((Kt)c[q] << 8);
                P[q] = open ? next : (Kt)0;
                mark[q] = open && c[q] != 0 && next >= lam ? sv : mark[q];  // lambda(sv, v) >= key: contractible
            }
        }
        const Kt m01 = P[0] > P[1] ? P[0] : P[1], m23 = P[2] > P[3] ? P[2] : P[3];
        const Kt best = warp_max(m01 > m23 ? m01 : m23);
        const uint32_t last = 255u - ((uint32_t)best & 255u);
        lambda = (uint64_t)(best >> 8) < lambda ? (uint64_t)(best >> 8) : lambda;
        // one vertex left when every vertex but the first of the ordering is joined to an earlier one
        uint32_t linked = 0;
#pragma unroll
        for (int q = 0; q < 4; q++) linked += __popc(__ballot_sync(0xffffffffu, active[q] && (mark[q] != 255u || v[q] == last)));
        if (linked + 1 >= cnt) break;
        // the roots of the marks' trees by pointer doubling (a tree is at most 127 edges deep), then
        // (prev, last) joins two of them
#pragma unroll
        for (int q = 0; q < 4; q++) root[v[q]] = (uint8_t)(mark[q] != 255u ? mark[q] : v[q]);
        __syncwarp();
        uint32_t rt[4];
#pragma unroll 1
        for (uint32_t deep = 1; deep < 128; deep *= 2) {
#pragma unroll
            for (int q = 0; q < 4; q++) rt[q] = root[root[v[q]]];
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 4; q++) root[v[q]] = (uint8_t)rt[q];
            __syncwarp();
        }
        const uint32_t into = root[prev], from = root[last];
        // each vertex that is no root is merged into its own
#pragma unroll 1
        for (int k = 0; k < 4; k++) {
            const uint32_t mine = v[0] + 32 * k;
            const uint32_t r = root[mine];
            const uint32_t to = r == from ? into : r;
            bool on = false;
#pragma unroll
            for (int q = 0; q < 4; q++) on = q == k ? active[q] : on;
            uint32_t gone = __ballot_sync(0xffffffffu, on && to != mine);
            cnt -= __popc(gone);
            while (gone) {
                const uint32_t l = __ffs(gone) - 1;
                gone &= gone - 1;
                const uint32_t y = l + 32 * k, x = __shfl_sync(0xffffffffu, to, l);
                const uint32_t tx = tri(x), ty = tri(y);
                Tm a[4], b[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    a[q] = M[entry(q, x, tx)];
                    b[q] = M[entry(q, y, ty)];
                }
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    if (active[q] && v[q] != x && v[q] != y) M[entry(q, x, tx)] = a[q] + b[q];
                    active[q] = active[q] && v[q] != y;
                }
                __syncwarp();
            }
        }
    }
    return lambda;
}

// The lower triangle, asynchronously: warp w copies rows 1 + w, 1 + w + 4, ... (a lone warp took 15 thousand
// cycles to issue the copies, about as long as an ordering takes). row(i): where row i is; col(q): the column there
// of the lane's vertex lane + 32 q.
template <typename Tm, typename Row, typename Col>
__device__ __forceinline__ void leaf_copy(Tm *M, uint32_t N, Row row, Col col) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x / 32;
    uint32_t c[4];
#pragma unroll
    for (int q = 0; q < 4; q++) c[q] = col(q);
#pragma unroll 4
    for (uint32_t i = 1 + warp; i < N; i += kLeafWarps) {
        const Tm *src = row(i);
        Tm *dst = M + tri(i) + lane;
#pragma unroll
        for (uint32_t q = 0; q < 4; q++)
            if (lane + 32 * q < i) copy_entry_async(dst + 32 * q, src + c[q]);
    }
}

// From the matrix and the degrees of the lane's vertices: lambda starts at the minimum weighted degree (a
// cut of the leaf).
template <typename Tm>
__device__ __forceinline__ void leaf_solve(Tm *M, uint32_t N, const uint64_t (&deg)[4], uint8_t *root, uint64_t *out) {
    const uint32_t lane = threadIdx.x;
    uint64_t low = kU64Max, sum = 0;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        if (lane + 32 * q < N) {
            low = deg[q] < low ? deg[q] : low;
            sum += deg[q];
        }
    }
    const uint64_t lambda = warp_min_u64(low);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    // a key never exceeds the leaf's total weight (half its degree sum, which merges only lower)
    uint64_t cut;
    if constexpr (sizeof(Tm) == 4) {
        cut = sum < (1ull << 25) ? leaf_cut<Tm, uint32_t>(M, N, lambda, root) : leaf_cut<Tm, uint64_t>(M, N, lambda, root);
    } else {
        cut = leaf_cut<Tm, uint64_t>(M, N, lambda, root);
    }
    if (lane == 0) atomicMin((unsigned long long *)out, (unsigned long long)cut);
}

template <typename Tm>
__global__ void __launch_bounds__(kLeafThreads) sw_leaf_kernel(const LeafDesc *__restrict__ leaves) {
    extern __shared__ __align__(16) unsigned char dsm[];
    Tm *M = reinterpret_cast<Tm *>(dsm);  // N (N - 1) / 2 entries and one that is read but not used
    __shared__ uint8_t root[128];
    const LeafDesc L = leaves[blockIdx.x];
    const uint32_t N = L.N, lane = threadIdx.x & 31;
    leaf_copy(M, N, [&](uint32_t i) { return reinterpret_cast<const Tm *>(L.mat) + i * ld_of(N); },
              [&](int q) { return lane + 32 * q; });
    // degrees: the row sums that came with the matrix, else summed here, a thread per vertex (by warp 0 alone it
    // took 10 us of a single leaf's 70)
    __shared__ uint64_t s_deg[kLeafThreads];
    const uint32_t v = threadIdx.x;
    s_deg[v] = L.rowsum && v < N ? __ldg(L.rowsum + v) : 0;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (!L.rowsum) {
        uint64_t sum = 0;
        for (uint32_t j = 0; j < N && v < N; j++) sum += j == v ? 0 : (uint64_t)M[tpos(v, j)];
        s_deg[v] = sum;
        __syncthreads();
    }
    if (threadIdx.x >= 32) return;
    uint64_t deg[4];
#pragma unroll
    for (int q = 0; q < 4; q++) deg[q] = s_deg[lane + 32 * q];
    leaf_solve(M, N, deg, root, L.cut);
}

// The leaf of a contraction to kLeafN vertices, straight from its source (N <= 179): its matrix, the child's
// quotient, is never written. The entries between first vertices of two groups are copied as in
// sw_leaf_kernel, at the columns of the first vertices (ascending, so the copies stay nearly coalesced);
// then the row of each joined vertex is added to its group's, four rows in flight per warp, from the first
// vertices' columns and from those of the joined vertices before it, with shared atomics. The degrees are
// the source's row sums, less twice what lies inside the groups.
//   Before, the last level's quotients were written and read back: K4000 14,336 quotients of N = 181 and
// their leaves 485 + 300 us, now 364 us; the plain Karger-Stein query on Watts-Strogatz n = 32,000 (524,288
// children of N = 130 at a time) 18.7 + 8.3 ms, now 10.4 ms, and 37 GB less memory; ER(1000, 0.05) 44 +
// 36 us, now 48 us. (One warp for the copies and the joined rows: 424 us, 13.1 ms, 64 us.)
template <typename Tm>
__global__ void __launch_bounds__(kLeafThreads) sw_child_kernel(const TaskDesc *__restrict__ tasks,
                                                                const SrcDesc *__restrict__ srcs,
                                                                const uint32_t *__restrict__ list,
                                                                const uint32_t *__restrict__ k_act, uint32_t *err) {
    extern __shared__ __align__(16) unsigned char dsm[];
    Tm *M = reinterpret_cast<Tm *>(dsm);
    __shared__ unsigned long long s_deg[kLeafN];
    __shared__ uint16_t s_first[kLeafN], s_joined[kLeafN];  // s_joined: vertex | label << 8
    __shared__ uint8_t root[kLeafN];
    const uint32_t task = list[blockIdx.x], lane = threadIdx.x & 31, warp = threadIdx.x / 32;
    const TaskDesc T = tasks[task];
    const SrcDesc S = srcs[T.src];
    const uint32_t N = S.N, k = T.target;
    if (k_act[task] != k) {  // planned ahead, and this child stopped off its target: redo the run
        if (threadIdx.x == 0) atomicOr(err, kErrPlan);
        return;
    }
    const Tm *mat = reinterpret_cast<const Tm *>(S.mat);
    const uint64_t ldN = ld_of(N);
    if (threadIdx.x < kLeafN) s_first[threadIdx.x] = threadIdx.x < k ? T.cols[kColHead + threadIdx.x] : (uint16_t)0;
    __syncthreads();
    uint32_t f[4];
#pragma unroll
    for (int q = 0; q < 4; q++) f[q] = s_first[lane + 32 * q];
    leaf_copy(M, k, [&](uint32_t i) { return mat + s_first[i] * ldN; }, [&](int q) { return f[q]; });
    if (threadIdx.x < kLeafN) s_deg[threadIdx.x] = threadIdx.x < k ? __ldg(S.rowsum + s_first[threadIdx.x]) : 0;
    __syncthreads();
    // the joined vertices, ascending (every warp counts them, warp 0 lists them)
    uint32_t joined = 0;
    for (uint32_t v0 = 0; v0 < N; v0 += 32) {
        const uint32_t v = v0 + lane, l = v < N ? T.lab[v] : 0;
        const bool j = v < N && s_first[l] != v;
        const uint32_t js = __ballot_sync(0xffffffffu, j);
        if (j && warp == 0) {
            s_joined[joined + __popc(js & ((1u << lane) - 1))] = (uint16_t)(v | l << 8);
            atomicAdd(&s_deg[l], (unsigned long long)__ldg(S.rowsum + v));
        }
        joined += __popc(js);
    }
    __syncthreads();
    uint32_t other[2];  // the lane's joined vertices: lane and lane + 32
#pragma unroll
    for (int q = 0; q < 2; q++) other[q] = lane + 32 * q < joined ? s_joined[lane + 32 * q] : 0;
    bool waited = false;
    for (uint32_t p0 = 0; p0 < joined || !waited; p0 += 4 * kLeafWarps) {
        Tm a[4][4], b[4][2];
#pragma unroll
        for (uint32_t u = 0; u < 4; u++) {
            const uint32_t p = p0 + u * kLeafWarps + warp;
            const Tm *row = mat + (p < joined ? s_joined[p] & 255u : 0) * ldN;
#pragma unroll
            for (int q = 0; q < 4; q++) a[u][q] = p < joined && lane + 32 * q < k ? __ldg(row + f[q]) : Tm(0);
#pragma unroll
            for (int q = 0; q < 2; q++) b[u][q] = p < joined && lane + 32 * q < p ? __ldg(row + (other[q] & 255u)) : Tm(0);
        }
        if (!waited) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            waited = true;
        }
#pragma unroll
        for (uint32_t u = 0; u < 4; u++) {
            const uint32_t p = p0 + u * kLeafWarps + warp;
            if (p >= joined) break;
            const uint32_t to = s_joined[p] >> 8, tt = tri(to);
#pragma unroll
            for (int q = 0; q < 6; q++) {
                const uint32_t l = q < 4 ? lane + 32 * q : other[q - 4] >> 8;
                const Tm x = q < 4 ? a[u][q] : b[u][q - 4];
                if (x == 0) continue;
                if (l == to) atomicAdd(&s_deg[to], 0ull - 2 * (unsigned long long)x);
                else sadd(&M[l > to ? tri(l) + to : tt + l], x);
            }
        }
    }
    __syncthreads();
    if (warp > 0) return;
    uint64_t deg[4];
#pragma unroll
    for (int q = 0; q < 4; q++) deg[q] = s_deg[lane + 32 * q];
    leaf_solve(M, k, deg, root, T.cut);
}

__global__ void fill_u64(uint64_t *p, uint64_t n, uint64_t value) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        p[i] = value;
}

// ---------------------------------------------------------------- host orchestration

// Device buffer owned by one call, grown on demand.
struct DevBuf {
    cac_ctx *ctx = nullptr;
    void *p = nullptr;
    size_t cap = 0;
    explicit DevBuf(cac_ctx *c) : ctx(c) {}
    ~DevBuf() { release(); }
    void release() {
        if (p) dev_free(ctx, p, cap);
        p = nullptr;
        cap = 0;
    }
    int ensure(size_t bytes) {
        if (bytes <= cap) return CAC_OK;
        CAC_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
        release();
        const size_t want = align_up(std::max<size_t>(bytes, 256), 1 << 16);
        CAC_TRY(dev_alloc(ctx, &p, want));
        cap = want;
        return CAC_OK;
    }
    template <typename T> T *as() const { return reinterpret_cast<T *>(p); }
};

// Grow-only scratch buffers kept by the ctx between calls: a fresh device allocation per query
// (cudaMalloc, and a cudaFree that waits for the whole device) cost more than the kernels of a
// small query (admission of square_root on ER(1000, 0.05): 303 us, of which about 100 us of
// kernels). Slots 0..3 belong to the Karger-Stein engine, 4..10 to admission, 11.. to the
// one-shot probes; one engine runs per ctx at a time.
enum ScratchSlot : int {
    kSlotKout, kSlotPrep, kSlotTscratch, kSlotErr, kSlotPre, kSlotLab, kSlotK, kSlotSd, kSlotDd, kSlotSparse,
    kSlotSparseCount, kSlotProbe0, kSlotProbe1, kSlotProbe2, kSlotCount
};

// Descriptor staging of one phase of an engine step: the phase's small host arrays are packed
// (16-byte aligned) into one pinned host buffer and sent with a single copy into one device
// buffer, instead of one pageable copy per array (each a driver call on the host's critical path
// between a step's read-back and its next launches). There are kSlots pinned buffers, used in turn, and
// an event after a buffer's copy guards it: it is refilled only once that copy has run, so a run that
// plans ahead can be kSlots steps ahead of the device. With one buffer the host waited for each step
// to start before it laid out the next, and the deep levels, whose thousands of tasks take the host
// longer than the device, left the device idle: K4000 5.94 ms, a 64-graph batch 72.6 ms; now 5.63 and
// 71.3 ms (with the contractions launched behind the quotients' planning, see KsEngine::step).
// The device buffer is one for all slots: copies and kernels are ordered by the stream.
struct Staging {
    static constexpr int kSlots = 3;
    struct Slot {
        unsigned char *host = nullptr;
        size_t cap = 0;
        cudaEvent_t done = nullptr;
        bool pending = false;
    };
    cac_ctx *ctx;
    DevBuf dev;
    Slot slots[kSlots];
    int at = 0;
    size_t used = 0;
    explicit Staging(cac_ctx *c) : ctx(c), dev(c) {}
    Staging(const Staging &) = delete;
    Staging &operator=(const Staging &) = delete;
    ~Staging() {
        for (Slot &sl : slots) {
            if (sl.pending) cudaEventSynchronize(sl.done);
            if (sl.host) cudaFreeHost(sl.host);
            if (sl.done) cudaEventDestroy(sl.done);
        }
    }
    template <typename T> static size_t bytes_of(const std::vector<T> &v) {
        return (sizeof(T) * std::max<size_t>(v.size(), 1) + 15) & ~(size_t)15;
    }
    int begin(size_t bytes) {
        at = (at + 1) % kSlots;
        Slot &sl = slots[at];
        if (!sl.done) CAC_CUDA_TRY(cudaEventCreateWithFlags(&sl.done, cudaEventDisableTiming));
        if (sl.pending) {
            CAC_CUDA_TRY(cudaEventSynchronize(sl.done));
            sl.pending = false;
        }
        bytes = std::max<size_t>(bytes, 16);
        if (bytes > sl.cap) {
            if (sl.host) CAC_CUDA_TRY(cudaFreeHost(sl.host));
            sl.host = nullptr;
            sl.cap = 0;
            // as large as any slot's: the same steps fall on other slots in the next run
            for (const Slot &o : slots) bytes = std::max(bytes, o.cap);
            const size_t want = align_up(bytes, 1 << 16);
            CAC_CUDA_TRY(cudaHostAlloc(reinterpret_cast<void **>(&sl.host), want, cudaHostAllocDefault));
            sl.cap = want;
        }
        CAC_TRY(dev.ensure(bytes));
        used = 0;
        return CAC_OK;
    }
    // copies v into the host buffer; returns where it will be on the device
    template <typename T> T *put(const std::vector<T> &v) {
        const size_t off = used;
        if (!v.empty()) std::memcpy(slots[at].host + off, v.data(), sizeof(T) * v.size());
        used += bytes_of(v);
        return reinterpret_cast<T *>(static_cast<unsigned char *>(dev.p) + off);
    }
    int flush() {
        if (!used) return CAC_OK;
        CAC_CUDA_TRY(cudaMemcpyAsync(dev.p, slots[at].host, used, cudaMemcpyHostToDevice, ctx->stream));
        CAC_CUDA_TRY(cudaEventRecord(slots[at].done, ctx->stream));
        slots[at].pending = true;
        return CAC_OK;
    }
};

struct CtxScratch {
    std::vector<DevBuf> slots;
    Staging leaf, pre, post;  // an engine step's leaves, then its descriptors before and after its read-back
    explicit CtxScratch(cac_ctx *ctx) : slots(kSlotCount, DevBuf(ctx)), leaf(ctx), pre(ctx), post(ctx) {}
};

CtxScratch &ctx_scratch(cac_ctx *ctx) {
    if (!ctx->ks_scratch) ctx->ks_scratch = new CtxScratch(ctx);
    return *static_cast<CtxScratch *>(ctx->ks_scratch);
}

DevBuf &scratch(cac_ctx *ctx, ScratchSlot slot) { return ctx_scratch(ctx).slots[slot]; }

template <typename T>
int upload(cac_ctx *ctx, DevBuf &buf, const std::vector<T> &v) {
    CAC_TRY(buf.ensure(sizeof(T) * std::max<size_t>(v.size(), 1)));
    if (!v.empty())
        CAC_CUDA_TRY(cudaMemcpyAsync(buf.p, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice, ctx->stream));
    return CAC_OK;
}

size_t leaf_smem(uint32_t N, bool small) { return ((size_t)N * (N - 1) / 2 + 1) * (small ? 4 : 8); }
size_t contract_smem(uint32_t N) {
    return (size_t)std::min(N, kCoarseRows) * sizeof(uint64_t) + contract_batch_cap(N) * sizeof(uint2) + (size_t)3 * N * 4;
}

}  // namespace

void ctx_scratch_free(cac_ctx *ctx) {
    delete static_cast<CtxScratch *>(ctx->ks_scratch);
    ctx->ks_scratch = nullptr;
}

// ---- Karger-Stein engine (declared in cac_internal.h) ----

KsEngine::KsEngine(cac_ctx *ctx)
    : ctx_(ctx), d_kout_(&scratch(ctx, kSlotKout)), d_prep_(&scratch(ctx, kSlotPrep)),
      d_tscratch_(&scratch(ctx, kSlotTscratch)), d_err_(&scratch(ctx, kSlotErr)) {}

KsEngine::~KsEngine() {
    cudaStreamSynchronize(ctx_->stream);
    for (const KNode &nd : nodes_) release(nd.buf);
    for (const KTask &t : carried_) release(t.src.buf);
    nodes_.clear();
    carried_.clear();
}

int KsEngine::init_err() {
    DevBuf *e = static_cast<DevBuf *>(d_err_);
    CAC_TRY(e->ensure(4));
    CAC_CUDA_TRY(cudaMemsetAsync(e->p, 0, 4, ctx_->stream));
    return CAC_OK;
}

uint32_t *KsEngine::err_word() const { return static_cast<DevBuf *>(d_err_)->as<uint32_t>(); }

int KsEngine::read_err(uint32_t *err) {
    DevBuf *e = static_cast<DevBuf *>(d_err_);
    *err = 0;
    if (!e->p) return CAC_OK;
    CAC_CUDA_TRY(cudaMemcpyAsync(err, e->p, 4, cudaMemcpyDeviceToHost, ctx_->stream));
    CAC_CUDA_TRY(cudaStreamSynchronize(ctx_->stream));
    return CAC_OK;
}

int engine_error(uint32_t err) {
    // (one cause: a run that planned ahead and missed is redone instead)
    set_error("inconsistent selection prefix in the contraction kernel (error word " + std::to_string(err) + ")");
    return CAC_ERR_CUDA;
}

int KsEngine::alloc(size_t bytes, MatBuf **out) {
    *out = nullptr;
    bytes = std::max<size_t>(bytes, 256);
    if (ctx_->budget && ctx_->held + bytes > ctx_->budget) {
        set_error("HBM budget exceeded by a Karger-Stein level buffer of " + std::to_string(bytes) + " bytes");
        return CAC_ERR_OOM;
    }
    void *p = nullptr;
    cudaError_t e = ctx_->pool ? cudaMallocFromPoolAsync(&p, bytes, ctx_->pool, ctx_->stream)
                               : cudaMallocAsync(&p, bytes, ctx_->stream);
    if (e != cudaSuccess) {
        cudaGetLastError();
        set_error(std::string("cudaMallocAsync: ") + cudaGetErrorString(e));
        return CAC_ERR_OOM;
    }
    ctx_->held += bytes;
    MatBuf *b = new MatBuf{p, bytes, 0};
    *out = b;
    return CAC_OK;
}

void KsEngine::release(MatBuf *b) {
    if (!b) return;
    if (--b->refs > 0) return;
    if (b->refs < 0) {  // released more often than referenced: keep it, report at the next step
        release_err_ = true;
        return;
    }
    if (cudaFreeAsync(b->p, ctx_->stream) != cudaSuccess) {
        cudaGetLastError();  // reported through the engine's error state, not as a sticky CUDA error
        release_err_ = true;
    }
    ctx_->held -= std::min<uint64_t>(ctx_->held, b->bytes);
    delete b;
}

void KsEngine::add(const KNode &nd) {
    nd.buf->refs++;
    nodes_.push_back(nd);
    if (nd.query >= outstanding.size()) outstanding.resize(nd.query + 1, 0);
    outstanding[nd.query]++;
}

namespace {

// A buffer that a scope has allocated and holds one reference on until it ends, however it ends.
struct Held {
    KsEngine &eng;
    MatBuf *buf = nullptr;
    explicit Held(KsEngine &e) : eng(e) {}
    Held(const Held &) = delete;
    Held &operator=(const Held &) = delete;
    ~Held() { eng.release(buf); }
    int alloc(size_t bytes) {
        CAC_TRY(eng.alloc(bytes, &buf));
        buf->refs++;
        return CAC_OK;
    }
    unsigned char *at(uint64_t off) const { return buf ? static_cast<unsigned char *>(buf->p) + off : nullptr; }
};

// Sparse roots on their way to sparse_phase, which takes over their references.
struct SparseRoots {
    KsEngine &eng;
    std::vector<SparseNode> nodes;
    explicit SparseRoots(KsEngine &e) : eng(e) {}
    SparseRoots(const SparseRoots &) = delete;
    SparseRoots &operator=(const SparseRoots &) = delete;
    ~SparseRoots() {
        for (const SparseNode &nd : nodes) eng.release(nd.buf);
    }
    std::vector<SparseNode> take() { return std::exchange(nodes, {}); }
};

}  // namespace

int KsEngine::step() {
    cudaStream_t s = ctx_->stream;
    if (release_err_) {
        set_error("Karger-Stein engine: a level buffer was released more often than referenced or could not be freed");
        return CAC_ERR_CUDA;
    }
    DevBuf &d_kout = *static_cast<DevBuf *>(d_kout_), &d_prep = *static_cast<DevBuf *>(d_prep_);
    DevBuf &d_tscratch = *static_cast<DevBuf *>(d_tscratch_);
    uint32_t *d_err = static_cast<DevBuf *>(d_err_)->as<uint32_t>();
    // the buffers of all nodes and tasks, which leave the lists here: released when the step ends, as what it
    // enqueued reads them (freeing is ordered by the stream), and at whatever point it fails
    struct Consumed {
        KsEngine &eng;
        std::vector<MatBuf *> bufs;
        ~Consumed() {
            for (MatBuf *b : bufs) eng.release(b);
        }
    } consumed{*this, {}};
    const std::vector<KNode> nodes = std::exchange(nodes_, {});
    const std::vector<KTask> carried = std::exchange(carried_, {});
    consumed.bufs.reserve(nodes.size() + carried.size());
    for (const KNode &nd : nodes) consumed.bufs.push_back(nd.buf);
    for (const KTask &t : carried) consumed.bufs.push_back(t.src.buf);

    // leaves (n <= 128) -> exact cut, one launch per entry width
    std::vector<LeafDesc> leaves;
    std::vector<KNode> inner;
    for (const KNode &nd : nodes) {
        if (nd.N <= 128) {
            if (nd.N >= 2) {
                leaves.push_back(LeafDesc{nd.mat, nd.cut, nd.pre, nd.N, nd.small});
            }
            outstanding[nd.query]--;
        } else {
            inner.push_back(nd);
        }
    }
    const size_t leaves32 = (size_t)(std::partition(leaves.begin(), leaves.end(), [](const LeafDesc &l) { return l.small != 0; }) -
                                     leaves.begin());
    auto launch_leaves = [&](const LeafDesc *d_leaves) -> int {  // (after the descriptor copy)
        uint32_t n32 = 2, n64 = 2;
        for (const LeafDesc &l : leaves) (l.small ? n32 : n64) = std::max(l.small ? n32 : n64, l.N);
        if (leaves32) {
            CAC_TRY(smem_optin(ctx_, sw_leaf_kernel<uint32_t>));
            sw_leaf_kernel<uint32_t><<<(unsigned)leaves32, kLeafThreads, leaf_smem(n32, true), s>>>(d_leaves);
        }
        if (leaves32 < leaves.size()) {
            CAC_TRY(smem_optin(ctx_, sw_leaf_kernel<uint64_t>));
            sw_leaf_kernel<uint64_t><<<(unsigned)(leaves.size() - leaves32), kLeafThreads, leaf_smem(n64, false), s>>>(d_leaves +
                                                                                                                      leaves32);
        }
        CAC_CUDA_TRY(cudaGetLastError());
        return CAC_OK;
    };
    Staging &leaf_st = ctx_scratch(ctx_).leaf, &pre_st = ctx_scratch(ctx_).pre, &post_st = ctx_scratch(ctx_).post;
    // the leaves go first: they run while the host plans the step's contractions
    if (!leaves.empty()) {
        CAC_TRY(leaf_st.begin(Staging::bytes_of(leaves)));
        const LeafDesc *dl = leaf_st.put(leaves);
        CAC_TRY(leaf_st.flush());
        CAC_TRY(launch_leaves(dl));
    }

    // sources: inner nodes (two children each) and the matrices of tasks continuing another round
    std::vector<KTask> tasks;
    std::vector<KNode> src_nodes;
    tasks.reserve(2 * inner.size() + carried.size());
    src_nodes.reserve(inner.size() + carried.size());
    for (const KNode &nd : inner) {
        src_nodes.push_back(nd);
        const uint32_t target = (uint32_t)ks_target((int)nd.N);
        for (uint64_t c = 0; c < 2; c++) tasks.push_back(KTask{nd, 2 * nd.h + c, 0, target, (uint32_t)(src_nodes.size() - 1)});
        outstanding[nd.query]++;  // two tasks replace the node
    }
    for (KTask t : carried) {
        src_nodes.push_back(t.src);
        t.src_index = (uint32_t)(src_nodes.size() - 1);
        tasks.push_back(t);
    }
    if (tasks.empty()) return CAC_OK;
    // sources whose row sums and block prefixes came with their matrix (every quotient's) skip the
    // row prep; the others (roots) are prepped here from their own list
    std::vector<SrcDesc> srcs(src_nodes.size()), psrcs;
    std::vector<uint64_t> row_off;
    uint64_t rows = 0, prep_elems = 0;
    for (size_t i = 0; i < src_nodes.size(); i++) {
        if (src_nodes[i].pre) continue;
        const uint32_t nb = (src_nodes[i].N + 31) / 32;
        prep_elems += src_nodes[i].N + (uint64_t)src_nodes[i].N * nb;
    }
    CAC_TRY(d_prep.ensure(std::max<uint64_t>(prep_elems, 1) * 8));
    uint64_t pe = 0;
    for (size_t i = 0; i < src_nodes.size(); i++) {
        const KNode &nd = src_nodes[i];
        SrcDesc &S = srcs[i];
        S.mat = nd.mat;
        S.N = nd.N;
        S.nb = (nd.N + 31) / 32;
        S.cut = nd.cut;
        S.is_root = nd.is_root;
        S.small = nd.small;
        if (nd.pre) {
            S.rowsum = nd.pre;
        } else {
            S.rowsum = d_prep.as<uint64_t>() + pe;
            pe += nd.N + (uint64_t)nd.N * S.nb;
            row_off.push_back(rows);
            rows += nd.N;
        }
        S.blk = S.rowsum + nd.N;
        if (!nd.pre) psrcs.push_back(S);
    }

    // contraction of every child
    uint64_t tscratch = 0;
    for (const KTask &t : tasks) tscratch += task_words(t.src.N);
    CAC_TRY(d_tscratch.ensure(tscratch * 4));
    std::vector<TaskDesc> td(tasks.size());
    uint64_t ts = 0;
    for (size_t i = 0; i < tasks.size(); i++) {
        const KTask &t = tasks[i];
        TaskDesc &d = td[i];
        d.tag = 1 + t.h;
        d.cut = t.src.cut;
        d.src = t.src_index;
        d.target = t.target;
        d.round = t.round;
        d.k0 = t.src.k0;
        d.idx = t.src.idx;
        d.brief = plan_ahead_ &&
                  (t.target <= kLeafN || (ctx_->quotient_forced == kQuotientAuto && tri_fits(t.src.N, t.target, t.src.small)));
        const uint32_t N = t.src.N;
        d.rows = d_tscratch.as<uint32_t>() + ts;
        d.lab = reinterpret_cast<uint16_t *>(d.rows + N);
        d.members = d.lab + 2 * even16(N);
        d.memb_off = d.members + 2 * even16(N);
        d.cols = d.memb_off + 2 * even16(N + 1);
        ts += task_words(N);
    }
    CAC_TRY(d_kout.ensure(tasks.size() * 4));
    // the contraction's launches: tasks by the size class of their source and its entry width
    std::vector<uint32_t> list;
    uint32_t list_num[6] = {}, list_max[6] = {};
    auto class_of = [](const KNode &src) {
        return (src.N <= kContractSmallN ? 4 : src.N <= kContractMidN ? 2 : 0) + (src.small ? 0 : 1);
    };
    for (const KTask &t : tasks) {
        const int c = class_of(t.src);
        list_num[c]++;
        list_max[c] = std::max(list_max[c], t.src.N);
    }
    uint32_t list_at[6] = {};
    for (int c = 1; c < 6; c++) list_at[c] = list_at[c - 1] + list_num[c - 1];
    list.resize(tasks.size());
    for (size_t i = 0; i < tasks.size(); i++) list[list_at[class_of(tasks[i].src)]++] = (uint32_t)i;
    // one descriptor copy for the sources, the row-prep list, the tasks and their launch lists
    CAC_TRY(pre_st.begin(Staging::bytes_of(srcs) + Staging::bytes_of(row_off) + Staging::bytes_of(psrcs) +
                         Staging::bytes_of(td) + Staging::bytes_of(list)));
    const SrcDesc *dv_src = pre_st.put(srcs);
    const uint64_t *dv_rowoff = pre_st.put(row_off);
    const SrcDesc *dv_psrc = pre_st.put(psrcs);
    const TaskDesc *dv_task = pre_st.put(td);
    const uint32_t *dv_list = pre_st.put(list);
    CAC_TRY(pre_st.flush());
    if (rows) {
        bool p32 = false, p64 = false;
        for (const SrcDesc &S : psrcs) (S.small ? p32 : p64) = true;
        const unsigned pg = (unsigned)((rows * 32 + 255) / 256);
        if (p32)
            prep_rows_kernel<uint32_t><<<pg, 256, 0, s>>>(dv_psrc, dv_rowoff, (uint32_t)row_off.size(), rows);
        if (p64)
            prep_rows_kernel<uint64_t><<<pg, 256, 0, s>>>(dv_psrc, dv_rowoff, (uint32_t)row_off.size(), rows);
        CAC_CUDA_TRY(cudaGetLastError());
    }
    bool t32 = false, t64 = false;  // entry widths present among the tasks' sources
    for (const KTask &t : tasks) (t.src.small ? t32 : t64) = true;
    auto launch_contractions = [&]() -> int {  // a launch per size class and entry width, the largest first
        const uint32_t *d_list = dv_list;
        auto launch = [&](auto kern, int threads, int c) -> int {
            if (!list_num[c]) return CAC_OK;
            CAC_TRY(smem_optin(ctx_, kern));
            kern<<<list_num[c], threads, contract_smem(list_max[c]), s>>>(dv_task, dv_src, d_list, d_kout.as<uint32_t>(), d_err);
            d_list += list_num[c];
            return CAC_OK;
        };
        CAC_TRY(launch(contract_kernel<kNT, uint32_t>, kNT, 0));
        CAC_TRY(launch(contract_kernel<kNT, uint64_t>, kNT, 1));
        CAC_TRY(launch(contract_kernel<kContractMid, uint32_t>, kContractMid, 2));
        CAC_TRY(launch(contract_kernel<kContractMid, uint64_t>, kContractMid, 3));
        CAC_TRY(launch(contract_kernel<kContractSmall, uint32_t>, kContractSmall, 4));
        CAC_TRY(launch(contract_kernel<kContractSmall, uint64_t>, kContractSmall, 5));
        CAC_CUDA_TRY(cudaGetLastError());
        return CAC_OK;
    };
    // the children's sizes: read back, or (planning ahead) taken to be their targets, which the
    // quotient kernels check against the contraction's own counts on the device
    std::vector<uint32_t> kk(tasks.size());
    const uint32_t *kact = nullptr;
    if (plan_ahead_) {  // the contractions are launched with the quotients, behind the previous step's
        for (size_t i = 0; i < tasks.size(); i++) kk[i] = tasks[i].target;
        kact = d_kout.as<uint32_t>();
    } else {
        CAC_TRY(launch_contractions());
        CAC_CUDA_TRY(cudaMemcpyAsync(kk.data(), d_kout.p, tasks.size() * 4, cudaMemcpyDeviceToHost, s));
        CAC_CUDA_TRY(cudaStreamSynchronize(s));
    }

    // quotient matrices of this step, in one stream-ordered buffer: each child's matrix, then
    // (after all matrices) each child's row sums and 32-column block prefixes, which the quotient
    // kernels write for the next step's draws
    std::vector<uint64_t> out_off(2 * tasks.size(), 0);
    std::vector<uint32_t> kq(tasks.size(), 0);
    uint64_t out_bytes = 0;
    std::vector<uint32_t> leaf_list[2];  // children that are leaves: solved from their sources, by entry width
    for (size_t i = 0; i < tasks.size(); i++) {
        uint32_t k = kk[i] == kDropped ? 0 : kk[i];
        if (k && k == tasks[i].target && k <= kLeafN) {
            leaf_list[tasks[i].src.small ? 0 : 1].push_back((uint32_t)i);
            k = 0;
        }
        kq[i] = k;
        out_off[i] = out_bytes;
        out_bytes += ((uint64_t)k * ld_of(k) * (tasks[i].src.small ? 4 : 8) + 15) / 16 * 16;
    }
    for (size_t i = 0; i < tasks.size(); i++) {
        out_off[tasks.size() + i] = out_bytes;
        out_bytes += ((kq[i] + (uint64_t)kq[i] * ((kq[i] + 31) / 32)) * 8 + 15) / 16 * 16;
    }
    // Three quotient kernels, identical outputs: triangles for small children, tiles up to kTileMaxN or kTileMaxN64
    // source vertices, one row per CTA above; the caller may force tiles (where they fit) or rows.
    Held out(*this);
    if (out_bytes || !leaf_list[0].empty() || !leaf_list[1].empty()) {
        if (out_bytes) CAC_TRY(out.alloc(out_bytes));
        unsigned char *obase = out.at(0);
        struct TileList {
            TilePlan plan;
            std::vector<TileTask> task;
            std::vector<uint64_t> first;
            uint64_t ctas = 0;
            uint32_t uniform = 0;
        } tl[2];
        tl[0].plan = TilePlan{4, 4, 0, 1};  // u32 entries
        tl[1].plan = TilePlan{2, 8, 0, 1};  // u64
        std::vector<uint32_t> shared, tris[3];  // (tris: u32 entries, small and larger; u64)
        std::vector<uint64_t> gto;
        uint32_t tri_k[3] = {2, 2, 2};
        uint64_t groups_shared = 0;
        uint32_t shared_n = 0, shared_k = 0;
        bool shared_small = true;
        const uint8_t forced = ctx_->quotient_forced;
        for (size_t i = 0; i < tasks.size(); i++) {
            const uint32_t N = tasks[i].src.N, k = kq[i];
            if (!k) continue;
            if (forced == kQuotientAuto && tri_fits(N, k, tasks[i].src.small)) {
                const int w = !tasks[i].src.small ? 2 : tri_bytes(k, 4) <= kTriSmallBytes ? 0 : 1;
                tris[w].push_back((uint32_t)i);
                tri_k[w] = std::max(tri_k[w], k);
                continue;
            }
            TileList &l = tl[tasks[i].src.small ? 0 : 1];
            const uint32_t need = tile_idx_bytes(N, k) +
                                  tile_groups(N, k, l.plan, kTileSmem) * tile_bytes(N, l.plan.rows, l.plan.esize);
            const bool tiles = forced == kQuotientShared                                     ? false
                               : forced == kQuotientTile || forced == kQuotientTileToo ? need <= 226 * 1024
                                                                                       : N <= (tasks[i].src.small ? kTileMaxN : kTileMaxN64);
            if (tiles) {
                l.plan.smem = std::max(l.plan.smem, need);
                l.task.push_back(TileTask{tasks[i].src.mat, td[i].cols, td[i].members, td[i].memb_off, td[i].rows,
                                          obase + out_off[i], reinterpret_cast<uint64_t *>(obase + out_off[tasks.size() + i]),
                                          kact ? kact + i : nullptr, N, k});
            } else {
                shared.push_back((uint32_t)i);
                gto.push_back(groups_shared);
                groups_shared += (k + kSharedRows - 1) / kSharedRows;
                shared_n = std::max(shared_n, N);
                shared_k = std::max(shared_k, k);
                shared_small = shared_small && tasks[i].src.small;
            }
        }
        for (TileList &l : tl) {
            // tiles per group of warps: a CTA's lists are staged once for all of them, but a last wave of
            // long CTAs costs more than the staging (448 children of N = 709: 16 tiles 357 us, 8 414; 240
            // of N = 501: 131 and 110)
            for (l.plan.tiles = 16;; l.plan.tiles /= 2) {
                l.first.clear();
                l.ctas = 0;
                uint64_t same = 0;
                bool uniform = true;
                for (const TileTask &t : l.task) {
                    const uint32_t g = tile_groups(t.N, t.k, l.plan, l.plan.smem);
                    const uint32_t per = tile_per_cta(g, l.plan), nt = (t.k + l.plan.rows - 1) / l.plan.rows;
                    const uint64_t ctas = (nt + per - 1) / per;
                    if (l.first.empty()) same = ctas;
                    uniform = uniform && ctas == same;
                    l.first.push_back(l.ctas);
                    l.ctas += ctas;
                }
                l.uniform = uniform ? (uint32_t)same : 0;
                if (l.plan.tiles == 1 || 2 * l.ctas >= (uint64_t)ctx_->num_sms * (l.plan.tiles == 16 ? 9 : 2)) break;
            }
        }
        // one descriptor copy for the output offsets, the children's sizes and the launch lists
        size_t bytes = Staging::bytes_of(out_off) + Staging::bytes_of(kq) + Staging::bytes_of(shared) +
                       Staging::bytes_of(gto) + Staging::bytes_of(leaf_list[0]) + Staging::bytes_of(leaf_list[1]) +
                       Staging::bytes_of(tris[0]) + Staging::bytes_of(tris[1]) + Staging::bytes_of(tris[2]);
        for (const TileList &l : tl) bytes += Staging::bytes_of(l.task) + Staging::bytes_of(l.first);
        CAC_TRY(post_st.begin(bytes));
        const uint64_t *dv_qoff = post_st.put(out_off);
        const uint32_t *dv_k = post_st.put(kq);
        const uint32_t *dv_shared = post_st.put(shared);
        const uint64_t *dv_gto = post_st.put(gto);
        TileArgs args[2];
        for (int i = 0; i < 2; i++)
            args[i] = TileArgs{post_st.put(tl[i].task), post_st.put(tl[i].first), (uint32_t)tl[i].task.size(), tl[i].uniform,
                               d_err, tl[i].plan};
        const uint32_t *dv_leaf32 = post_st.put(leaf_list[0]), *dv_leaf64 = post_st.put(leaf_list[1]);
        const uint32_t *dv_tri[3] = {post_st.put(tris[0]), post_st.put(tris[1]), post_st.put(tris[2])};
        CAC_TRY(post_st.flush());
        if (plan_ahead_) CAC_TRY(launch_contractions());
        if (!leaf_list[0].empty()) {
            CAC_TRY(smem_optin(ctx_, sw_child_kernel<uint32_t>));
            sw_child_kernel<uint32_t><<<(unsigned)leaf_list[0].size(), kLeafThreads, leaf_smem(kLeafN, true), s>>>(
                dv_task, dv_src, dv_leaf32, d_kout.as<uint32_t>(), d_err);
        }
        if (!leaf_list[1].empty()) {
            CAC_TRY(smem_optin(ctx_, sw_child_kernel<uint64_t>));
            sw_child_kernel<uint64_t><<<(unsigned)leaf_list[1].size(), kLeafThreads, leaf_smem(kLeafN, false), s>>>(
                dv_task, dv_src, dv_leaf64, d_kout.as<uint32_t>(), d_err);
        }
        auto launch_tri = [&](auto kern, int threads, int w) -> int {
            if (tris[w].empty()) return CAC_OK;
            CAC_TRY(smem_optin(ctx_, kern));
            kern<<<(unsigned)tris[w].size(), threads, tri_bytes(tri_k[w], w == 2 ? 8 : 4), s>>>(
                dv_task, dv_src, dv_tri[w], dv_k, dv_qoff, (uint32_t)tasks.size(), obase, kact, d_err);
            return CAC_OK;
        };
        CAC_TRY(launch_tri(quotient_tri_kernel<kTriThreads, uint32_t>, kTriThreads, 1));
        CAC_TRY(launch_tri(quotient_tri_kernel<kTriSmall, uint32_t>, kTriSmall, 0));
        CAC_TRY(launch_tri(quotient_tri_kernel<kTriThreads, uint64_t>, kTriThreads, 2));
        if (tl[0].ctas) {
            CAC_TRY(smem_optin(ctx_, quotient_tile_kernel<uint32_t, 4>));
            quotient_tile_kernel<uint32_t, 4><<<(unsigned)tl[0].ctas, kTileThreads, tl[0].plan.smem, s>>>(args[0]);
        }
        if (tl[1].ctas) {
            CAC_TRY(smem_optin(ctx_, quotient_tile_kernel<uint64_t, 2>));
            quotient_tile_kernel<uint64_t, 2><<<(unsigned)tl[1].ctas, kTileThreads, tl[1].plan.smem, s>>>(args[1]);
        }
        if (groups_shared) {
            // shared rows are u32 only when every task's sums fit (all sources small)
            const size_t words = ((size_t)shared_n + 3) & ~(size_t)3, es = shared_small ? 4 : 8;
            const size_t ssm = words * 4 + (((size_t)shared_k * es + 15) & ~(size_t)15) + ((size_t)shared_k / 32 + 1) * 8;
            std::vector<decltype(&quotient_shared_row_kernel<uint32_t, uint32_t>)> kerns;
            if (shared_small) kerns.push_back(quotient_shared_row_kernel<uint32_t, uint32_t>);
            else {
                if (t32) kerns.push_back(quotient_shared_row_kernel<uint64_t, uint32_t>);
                if (t64) kerns.push_back(quotient_shared_row_kernel<uint64_t, uint64_t>);
            }
            for (auto kern : kerns) {
                CAC_TRY(smem_optin(ctx_, kern));
                kern<<<(unsigned)groups_shared, 256, ssm, s>>>(dv_task, dv_src, dv_shared, (uint32_t)shared.size(), dv_k, dv_gto,
                                                               (uint32_t)tasks.size(), kSharedRows, dv_qoff, obase,
                                                               (uint32_t)words, shared_k, kact, d_err);
            }
        }
        CAC_CUDA_TRY(cudaGetLastError());
    }
    for (size_t i = 0; i < tasks.size(); i++) {
        const KTask &t = tasks[i];
        outstanding[t.src.query]--;
        const uint32_t k = kq[i];
        if (k == 0) continue;  // solved, or dropped: the source had no edges, its cut 0 is recorded
        KNode nd = t.src;
        nd.h = t.h;
        nd.N = k;
        nd.is_root = 0;
        nd.mat = out.at(out_off[i]);
        nd.pre = reinterpret_cast<uint64_t *>(out.at(out_off[tasks.size() + i]));
        nd.buf = out.buf;
        out.buf->refs++;
        outstanding[nd.query]++;
        if (k <= t.target) {
            nodes_.push_back(nd);
        } else {
            KTask c = t;
            c.src = nd;
            c.round += 1;
            carried_.push_back(c);
        }
    }
    return CAC_OK;
}

namespace {

// Admission of square_root queries: trial keys, per-trial cut slots, Stage 1 and Stage 2, root nodes.
struct QueryPlan {
    const cac_graph *g;
    uint32_t seed, ranks, per_rank;
    uint32_t t;
    uint64_t trials;
    uint64_t *cuts;       // device, one per trial
    uint32_t query;       // engine bookkeeping id
    uint32_t groups = 0;  // > 0: the high-concurrency group variant (trials = groups)
};

int admit_groups(cac_ctx *ctx, KsEngine &eng, const QueryPlan &q);

int admit_stage1(cac_ctx *ctx, KsEngine &eng, const std::vector<const QueryPlan *> &qs);
int admit_big(cac_ctx *ctx, KsEngine &eng, const QueryPlan &q);

// The sparse root of one square_root trial contracted to k vertices above the dense limit: the
// graph's edges relabelled by the trial's Stage 1 labels, sorted and merged on the device (the
// reference's WeightedIteratedSparseSampling::reduce, .cpp:26-234). The list's buffer carries
// the node's reference.
int sparse_root(cac_ctx *ctx, KsEngine &eng, const QueryPlan &q, uint64_t *cut, uint32_t k0, uint32_t idx,
                const uint32_t *lab, uint32_t k, SparseNode *out) {
    const cac_graph *g = q.g;
    const uint64_t cap = std::max<uint64_t>(g->m, 1);
    MatBuf *list = nullptr;
    CAC_TRY(eng.alloc(align_up(cap * 4) * 2 + align_up(cap * 8), &list));
    list->refs++;
    char *p = static_cast<char *>(list->p);
    uint32_t *oa = reinterpret_cast<uint32_t *>(p), *ob = reinterpret_cast<uint32_t *>(p + align_up(cap * 4));
    uint64_t *ow = reinterpret_cast<uint64_t *>(p + 2 * align_up(cap * 4));
    DevBuf &scr = scratch(ctx, kSlotSparse), &cnt = scratch(ctx, kSlotSparseCount);
    int st = scr.ensure(merge_edges_scratch(cap));
    if (st == CAC_OK) st = cnt.ensure(4);
    if (st == CAC_OK)
        st = merge_edges<uint32_t>(ctx, g->u, g->v, g->w, g->m, lab, k, oa, ob, ow, cnt.as<uint32_t>(), scr.p);
    uint32_t mm = 0;
    if (st == CAC_OK && (cudaMemcpyAsync(&mm, cnt.p, 4, cudaMemcpyDeviceToHost, ctx->stream) != cudaSuccess ||
                         cudaStreamSynchronize(ctx->stream) != cudaSuccess)) {
        set_error("square_root: reading the sparse root's edge count failed");
        st = CAC_ERR_CUDA;
    }
    if (st != CAC_OK) {
        eng.release(list);
        return st;
    }
    *out = SparseNode{cut, k0, idx, 1, k, k >= 2 ? mm : 0, oa, ob, ow, true, true,
                      g->total_weight < (1ull << 32) ? 1u : 0u, q.query, list};
    return CAC_OK;
}

int admit(cac_ctx *ctx, KsEngine &eng, const QueryPlan &q) {
    cudaStream_t s = ctx->stream;
    const cac_graph *g = q.g;
    const uint32_t n = g->n;
    const uint64_t m = g->m;
    const uint32_t small = g->total_weight < (1ull << 32) ? 1u : 0u;
    if (q.trials == 0) return CAC_OK;
    if (q.t >= n && !ks_is_dense(ctx, n, m)) {
        // No pre-contraction and a sparse graph: every trial starts from the input edge list. The
        // dense levels below the sparse ones hold about n^2 entries per level and trial, so the
        // trials run in groups that keep two such levels within the bound, each group to its end.
        const uint64_t per_trial = 2ull * n * n * (small ? 4 : 8);
        const uint64_t bound = ctx->budget ? ctx->budget / 2 : (32ull << 30);
        const uint64_t group = std::max<uint64_t>(1, std::min<uint64_t>(q.trials, bound / per_trial));
        for (uint64_t g0 = 0; g0 < q.trials; g0 += group) {
            std::vector<SparseNode> roots;
            for (uint64_t i = g0; i < std::min(q.trials, g0 + group); i++) {
                const uint32_t r = (uint32_t)(i / q.per_rank), idx = (uint32_t)(i % q.per_rank);
                roots.push_back(SparseNode{q.cuts + i, q.seed + r, idx, 1, n, m, g->u, g->v, g->w, false, true, small,
                                           q.query, nullptr});
            }
            CAC_TRY(sparse_phase(ctx, eng, std::move(roots)));
            if (g0 + group < q.trials)
                while (!eng.idle()) CAC_TRY(eng.step());
        }
        return CAC_OK;
    }
    if (q.t >= n) {
        // no pre-contraction: every trial starts from the same dense matrix, built once
        Held root(eng);
        const size_t bytes = (size_t)n * ld_of(n) * (small ? 4 : 8);
        CAC_TRY(root.alloc(bytes));
        CAC_CUDA_TRY(cudaMemsetAsync(root.at(0), 0, bytes, s));
        if (m) {
            DevBuf &d = scratch(ctx, kSlotDd);
            std::vector<DenseDesc> dd{DenseDesc{g->u, g->v, g->w, nullptr, root.at(0), m, n, small}};
            CAC_TRY(upload(ctx, d, dd));
            dim3 grid((unsigned)std::max<uint64_t>(1, std::min<uint64_t>((m + 255) / 256, (uint64_t)ctx->num_sms * 8)), 1);
            dense_build_kernel<<<grid, 256, 0, s>>>(d.as<DenseDesc>());
            CAC_CUDA_TRY(cudaGetLastError());
            CAC_CUDA_TRY(cudaStreamSynchronize(s));  // the descriptor buffer goes out of scope
        }
        for (uint64_t i = 0; i < q.trials; i++) {
            const uint32_t r = (uint32_t)(i / q.per_rank), idx = (uint32_t)(i % q.per_rank);
            eng.add(KNode{q.cuts + i, q.seed + r, idx, 1, n, 1, small, q.query, root.at(0), root.buf});
        }
        return CAC_OK;
    }
    // Stage 1: the global-memory rounds of shrink_big.cu above 16384 vertices, else the
    // shared-memory kernel, batched with other queries' trials where the caller has several
    if (n > kMaxSmemVertices) return admit_big(ctx, eng, q);
    std::vector<const QueryPlan *> one{&q};
    return admit_stage1(ctx, eng, one);
}

// Stage 1 and Stage 2 of every trial of the given queries (t < n <= 16384), the trials of all of
// them together: one Stage 1 launch, one read-back of the contracted sizes and one dense build
// per chunk, whose scratch stays within 4 GB. Admitting the queries of a batch one by one costs a
// launch and two host synchronisations per query.
int admit_stage1(cac_ctx *ctx, KsEngine &eng, const std::vector<const QueryPlan *> &qs) {
    cudaStream_t s = ctx->stream;
    auto pre_words_of = [](uint64_t m) { return std::max<uint64_t>((m + 3) / 4, 1); };
    struct Item {
        const QueryPlan *q;
        uint64_t i;
    };
    std::vector<Item> items;
    for (const QueryPlan *q : qs)
        for (uint64_t i = 0; i < q->trials; i++) items.push_back({q, i});
    DevBuf &d_pre = scratch(ctx, kSlotPre), &d_lab = scratch(ctx, kSlotLab), &d_k = scratch(ctx, kSlotK),
           &d_sd = scratch(ctx, kSlotSd), &d_dd = scratch(ctx, kSlotDd);
    CAC_TRY(smem_optin(ctx, iss_shrink_kernel<kNT>));
    size_t c0 = 0;
    while (c0 < items.size()) {
        // a chunk: at most 65535 trials and 4 GB of prefix + label scratch
        size_t c1 = c0;
        uint64_t pre_words = 0, lab_words = 0;
        uint32_t nmax = 1;
        uint64_t mmax = 1;
        while (c1 < items.size() && c1 - c0 < 65535) {
            const cac_graph *g = items[c1].q->g;
            const uint64_t pw = pre_words_of(g->m), lw = g->n;
            if (c1 > c0 && (pre_words + pw) * 8 + (lab_words + lw) * 4 > (4ull << 30)) break;
            pre_words += pw;
            lab_words += lw;
            nmax = std::max(nmax, g->n);
            mmax = std::max(mmax, g->m);
            c1++;
        }
        const uint32_t B = (uint32_t)(c1 - c0);
        CAC_TRY(d_pre.ensure(pre_words * 8));
        CAC_TRY(d_lab.ensure(lab_words * 4));
        CAC_TRY(d_k.ensure((size_t)B * 4));
        std::vector<ShrinkDesc> sd(B);
        uint64_t po = 0, lo = 0;
        for (uint32_t b = 0; b < B; b++) {
            const QueryPlan &q = *items[c0 + b].q;
            const uint64_t i = items[c0 + b].i;
            ShrinkDesc &D = sd[b];
            D.U = q.g->u;
            D.V = q.g->v;
            D.W = q.g->w;
            D.m = q.g->m;
            D.pre = d_pre.as<uint64_t>() + po;
            D.lab = d_lab.as<uint32_t>() + lo;
            D.k_out = d_k.as<uint32_t>() + b;
            D.n = q.g->n;
            D.target = q.t;
            D.k0 = q.seed + (uint32_t)(i / q.per_rank);
            D.idx = (uint32_t)(i % q.per_rank);
            po += pre_words_of(q.g->m);
            lo += q.g->n;
        }
        const size_t sm = kBatch * sizeof(uint2) + kCoarse * sizeof(uint64_t) + (size_t)nmax * 6;
        CAC_TRY(upload(ctx, d_sd, sd));
        // fewer trials than SMs: one trial per SM either way, so each trial gets 1024 threads
        if (B < (uint32_t)ctx->num_sms) {
            CAC_TRY(smem_optin(ctx, iss_shrink_kernel<2 * kNT>));
            iss_shrink_kernel<2 * kNT><<<B, 2 * kNT, sm, s>>>(d_sd.as<ShrinkDesc>());
        } else {
            iss_shrink_kernel<kNT><<<B, kNT, sm, s>>>(d_sd.as<ShrinkDesc>());
        }
        CAC_CUDA_TRY(cudaGetLastError());
        // the contracted sizes: read back, or (planning ahead, no sparse root in the chunk) taken to
        // be the targets, which the dense build checks against Stage 1's counts on the device
        bool sparse_roots = false;
        for (uint32_t b = 0; b < B; b++) sparse_roots = sparse_roots || items[c0 + b].q->t > ctx->dense_limit;
        const bool planned = eng.plan_ahead() && !sparse_roots;
        std::vector<uint32_t> kdim(B);
        if (planned) {
            for (uint32_t b = 0; b < B; b++) kdim[b] = items[c0 + b].q->t;
        } else {
            CAC_CUDA_TRY(cudaMemcpyAsync(kdim.data(), d_k.p, (size_t)B * 4, cudaMemcpyDeviceToHost, s));
            CAC_CUDA_TRY(cudaStreamSynchronize(s));
        }
        // trials contracted to more than the dense limit: sparse roots (sorted, merged edge lists)
        SparseRoots sparse(eng);
        for (uint32_t b = 0; b < B; b++) {
            const QueryPlan &q = *items[c0 + b].q;
            if (q.t <= ctx->dense_limit) continue;
            SparseNode nd;
            CAC_TRY(sparse_root(ctx, eng, q, q.cuts + items[c0 + b].i, sd[b].k0, sd[b].idx, sd[b].lab, kdim[b], &nd));
            sparse.nodes.push_back(nd);
            kdim[b] = 0;  // no dense matrix
        }
        uint64_t bytes = 0;
        for (uint32_t b = 0; b < B; b++) {
            const uint64_t esize = items[c0 + b].q->g->total_weight < (1ull << 32) ? 4 : 8;
            bytes += ((uint64_t)kdim[b] * ld_of(kdim[b]) * esize + 15) / 16 * 16;
        }
        Held roots(eng);
        CAC_TRY(roots.alloc(std::max<uint64_t>(bytes, 16)));
        CAC_CUDA_TRY(cudaMemsetAsync(roots.at(0), 0, bytes, s));
        std::vector<DenseDesc> dd(B);
        uint64_t off = 0;
        for (uint32_t b = 0; b < B; b++) {
            const cac_graph *g = items[c0 + b].q->g;
            const uint32_t small = g->total_weight < (1ull << 32) ? 1u : 0u;
            // no scatter for a trial without a matrix (its labels would index past the buffer)
            dd[b] = DenseDesc{g->u, g->v, g->w, sd[b].lab, roots.at(off),
                              kdim[b] >= 2 ? g->m : 0, kdim[b], small};
            if (planned) {
                dd[b].k_act = sd[b].k_out;
                dd[b].err = eng.err_word();
            }
            off += ((uint64_t)kdim[b] * ld_of(kdim[b]) * (small ? 4 : 8) + 15) / 16 * 16;
        }
        CAC_TRY(upload(ctx, d_dd, dd));
        dim3 grid((unsigned)std::max<uint64_t>(
                      1, std::min<uint64_t>((mmax + 255) / 256, std::max<uint64_t>(1, (uint64_t)ctx->num_sms * 8 / B))),
                  B);
        dense_build_kernel<<<grid, 256, 0, s>>>(d_dd.as<DenseDesc>());
        CAC_CUDA_TRY(cudaGetLastError());
        for (uint32_t b = 0; b < B; b++) {
            const QueryPlan &q = *items[c0 + b].q;
            const uint64_t i = items[c0 + b].i;
            if (q.t > ctx->dense_limit) continue;  // a sparse root
            if (kdim[b] < 2) {
                // a single vertex left, or only isolated vertices: no cut edge
                fill_u64<<<1, 32, 0, s>>>(q.cuts + i, 1, 0);
                continue;
            }
            eng.add(KNode{q.cuts + i, sd[b].k0, sd[b].idx, 1, kdim[b], 1, dd[b].small, q.query, dd[b].mat, roots.buf});
        }
        // the scratch is refilled from the host for the next chunk (later kernels on the stream
        // are ordered after these, so the last chunk needs no wait)
        if (c1 < items.size()) CAC_CUDA_TRY(cudaStreamSynchronize(s));
        if (!sparse.nodes.empty()) CAC_TRY(sparse_phase(ctx, eng, sparse.take()));
        c0 = c1;
    }
    return CAC_OK;
}

// Stage 1 of a query above 16384 vertices: the global-memory rounds of shrink_big.cu, in chunks
// of trials whose scratch stays within 4 GB.
int admit_big(cac_ctx *ctx, KsEngine &eng, const QueryPlan &q) {
    cudaStream_t s = ctx->stream;
    const cac_graph *g = q.g;
    const uint32_t n = g->n;
    const uint64_t m = g->m;
    const uint32_t small = g->total_weight < (1ull << 32) ? 1u : 0u;
    const uint64_t per_trial = shrink_big_scratch(n, m, 1) + 4ull * n;
    const uint64_t chunk = std::max<uint64_t>(1, std::min<uint64_t>({q.trials, (4ull << 30) / per_trial, (uint64_t)65535}));
    DevBuf &d_pre = scratch(ctx, kSlotPre), &d_lab = scratch(ctx, kSlotLab), &d_k = scratch(ctx, kSlotK),
           &d_dd = scratch(ctx, kSlotDd);
    for (uint64_t c0 = 0; c0 < q.trials; c0 += chunk) {
        const uint32_t B = (uint32_t)std::min<uint64_t>(chunk, q.trials - c0);
        CAC_TRY(d_pre.ensure(shrink_big_scratch(n, m, B)));
        CAC_TRY(d_lab.ensure((size_t)B * n * 4));
        CAC_TRY(d_k.ensure((size_t)B * 4));
        std::vector<uint32_t> k0(B), idx(B);
        for (uint32_t b = 0; b < B; b++) {
            const uint64_t i = c0 + b;
            k0[b] = q.seed + (uint32_t)(i / q.per_rank);
            idx[b] = (uint32_t)(i % q.per_rank);
        }
        CAC_TRY(shrink_big(ctx, g, q.t, B, k0.data(), idx.data(), d_lab.as<uint32_t>(), d_k.as<uint32_t>(), d_pre.p));
        std::vector<uint32_t> kdim(B);
        CAC_CUDA_TRY(cudaMemcpyAsync(kdim.data(), d_k.p, (size_t)B * 4, cudaMemcpyDeviceToHost, s));
        CAC_CUDA_TRY(cudaStreamSynchronize(s));
        // trials contracted above the dense limit become sparse roots; otherwise more than 16384
        // vertices are left only when Stage 1 stopped with no edge between them (a disconnected
        // graph): every vertex is isolated and the trial's cut is exactly 0
        SparseRoots sparse(eng);
        for (uint32_t b = 0; b < B; b++) {
            if (q.t > ctx->dense_limit) {
                SparseNode nd;
                CAC_TRY(sparse_root(ctx, eng, q, q.cuts + c0 + b, k0[b], idx[b], d_lab.as<uint32_t>() + (size_t)b * n,
                                    kdim[b], &nd));
                sparse.nodes.push_back(nd);
                kdim[b] = 0;
            } else if (kdim[b] > kMaxSmemVertices) {
                kdim[b] = 0;
            }
        }
        const uint64_t esize = small ? 4 : 8;
        uint64_t bytes = 0;
        for (uint32_t b = 0; b < B; b++) bytes += ((uint64_t)kdim[b] * ld_of(kdim[b]) * esize + 15) / 16 * 16;
        Held roots(eng);
        CAC_TRY(roots.alloc(std::max<uint64_t>(bytes, 16)));
        CAC_CUDA_TRY(cudaMemsetAsync(roots.at(0), 0, bytes, s));
        std::vector<DenseDesc> dd(B);
        uint64_t off = 0;
        for (uint32_t b = 0; b < B; b++) {
            // no scatter for a trial without a matrix (its labels would index past the buffer)
            dd[b] = DenseDesc{g->u, g->v, g->w, d_lab.as<uint32_t>() + (size_t)b * n,
                              roots.at(off), kdim[b] >= 2 ? m : 0, kdim[b], small};
            off += ((uint64_t)kdim[b] * ld_of(kdim[b]) * esize + 15) / 16 * 16;
        }
        CAC_TRY(upload(ctx, d_dd, dd));
        if (m) {
            dim3 grid((unsigned)std::max<uint64_t>(1, std::min<uint64_t>((m + 255) / 256, std::max<uint64_t>(1, (uint64_t)ctx->num_sms * 8 / B))), B);
            dense_build_kernel<<<grid, 256, 0, s>>>(d_dd.as<DenseDesc>());
            CAC_CUDA_TRY(cudaGetLastError());
        }
        for (uint32_t b = 0; b < B; b++) {
            const uint64_t i = c0 + b;
            if (q.t > ctx->dense_limit) continue;  // a sparse root
            if (kdim[b] < 2) {
                fill_u64<<<1, 32, 0, s>>>(q.cuts + i, 1, 0);
                continue;
            }
            eng.add(KNode{q.cuts + i, k0[b], idx[b], 1, kdim[b], 1, small, q.query, dd[b].mat, roots.buf});
        }
        if (c0 + chunk < q.trials) CAC_CUDA_TRY(cudaStreamSynchronize(s));  // the scratch is reused by the next chunk
        if (!sparse.nodes.empty()) CAC_TRY(sparse_phase(ctx, eng, sparse.take()));
    }
    return CAC_OK;
}

// The high-concurrency group variant (SquareRootCut::participateInGroup, SquareRootCut.cpp:188-298):
// group trial g runs WeightedIteratedSparseSampling::shrink (.cpp:4-24) as Stage 1 rounds of a
// fixed floor(n^1.05) weighted draws (edgesToSamplePerProcessor, .hpp:66-67) with key
// (seed + g, 0, 1, 0), builds the contracted graph (reduce, .cpp:26-234: dense, or a sorted and
// merged sparse root above the dense limit), and, as parallel_cut(.., 2, ..) runs two recursive
// contractions of it (recursive_contract.cpp:45-83), starts two Karger-Stein recursions from that
// root with keys (seed + g, 0 | 1, 1 + h, 0). All groups' Stage 1 runs in one grid per chunk
// (shrink_big.cu with a fixed draw count per round).
int admit_groups(cac_ctx *ctx, KsEngine &eng, const QueryPlan &q) {
    cudaStream_t s = ctx->stream;
    const cac_graph *g = q.g;
    const uint32_t n = g->n;
    const uint64_t m = g->m;
    const uint32_t small = g->total_weight < (1ull << 32) ? 1u : 0u;
    const bool stage1 = q.t < n;
    const uint32_t dpr = group_draws(n);
    const uint64_t tt = std::min<uint64_t>(q.t, n);
    const uint64_t per_group = (stage1 ? shrink_task_scratch(n, m, dpr) : 0) + 4ull * n +
                               (q.t > ctx->dense_limit ? 16ull * m : tt * ld_of((uint32_t)tt) * (small ? 4 : 8));
    const uint64_t chunk = std::max<uint64_t>(1, std::min<uint64_t>({q.trials, (4ull << 30) / per_group, (uint64_t)65535}));
    DevBuf &d_pre = scratch(ctx, kSlotPre), &d_lab = scratch(ctx, kSlotLab), &d_k = scratch(ctx, kSlotK),
           &d_dd = scratch(ctx, kSlotDd);
    for (uint64_t c0 = 0; c0 < q.trials; c0 += chunk) {
        const uint32_t B = (uint32_t)std::min<uint64_t>(chunk, q.trials - c0);
        std::vector<uint32_t> kdim(B, n);
        if (stage1) {
            std::vector<ShrinkTask> tasks(B);
            CAC_TRY(d_lab.ensure((size_t)B * n * 4));
            CAC_TRY(d_k.ensure((size_t)B * 4));
            for (uint32_t b = 0; b < B; b++)
                tasks[b] = ShrinkTask{g->u, g->v, g->w, false, m, n, q.t, q.seed + (uint32_t)(c0 + b), 0, 1,
                                      d_lab.as<uint32_t>() + (size_t)b * n, d_k.as<uint32_t>() + b, dpr};
            CAC_TRY(d_pre.ensure(shrink_tasks_scratch(tasks)));
            CAC_TRY(shrink_tasks(ctx, tasks, d_pre.p));
            CAC_CUDA_TRY(cudaMemcpyAsync(kdim.data(), d_k.p, (size_t)B * 4, cudaMemcpyDeviceToHost, s));
            CAC_CUDA_TRY(cudaStreamSynchronize(s));
        }
        auto lab_of = [&](uint32_t b) -> const uint32_t * {
            return stage1 ? d_lab.as<uint32_t>() + (size_t)b * n : nullptr;
        };
        if (q.t > ctx->dense_limit) {
            // sparse roots: the merged contracted graph, shared by the group's two recursions
            SparseRoots sparse(eng);
            for (uint32_t b = 0; b < B; b++) {
                SparseNode nd;
                CAC_TRY(sparse_root(ctx, eng, q, q.cuts + c0 + b, q.seed + (uint32_t)(c0 + b), 0, lab_of(b), kdim[b],
                                    &nd));
                sparse.nodes.push_back(nd);
                nd.idx = 1;
                if (nd.buf) nd.buf->refs++;
                sparse.nodes.push_back(nd);
            }
            CAC_TRY(sparse_phase(ctx, eng, sparse.take()));
            continue;
        }
        // dense roots (more than 16384 vertices left only when Stage 1 found no edge between
        // them: a disconnected graph, cut 0)
        for (uint32_t b = 0; b < B; b++)
            if (kdim[b] > kMaxSmemVertices) kdim[b] = 0;
        const uint64_t esize = small ? 4 : 8;
        uint64_t bytes = 0;
        for (uint32_t b = 0; b < B; b++) bytes += ((uint64_t)kdim[b] * ld_of(kdim[b]) * esize + 15) / 16 * 16;
        Held roots(eng);
        CAC_TRY(roots.alloc(std::max<uint64_t>(bytes, 16)));
        CAC_CUDA_TRY(cudaMemsetAsync(roots.at(0), 0, bytes, s));
        std::vector<DenseDesc> dd(B);
        uint64_t off = 0;
        for (uint32_t b = 0; b < B; b++) {
            dd[b] = DenseDesc{g->u, g->v, g->w, lab_of(b), roots.at(off),
                              kdim[b] >= 2 ? m : 0, kdim[b], small};
            off += ((uint64_t)kdim[b] * ld_of(kdim[b]) * esize + 15) / 16 * 16;
        }
        CAC_TRY(upload(ctx, d_dd, dd));
        if (m) {
            dim3 grid((unsigned)std::max<uint64_t>(
                          1, std::min<uint64_t>((m + 255) / 256, std::max<uint64_t>(1, (uint64_t)ctx->num_sms * 8 / B))),
                      B);
            dense_build_kernel<<<grid, 256, 0, s>>>(d_dd.as<DenseDesc>());
            CAC_CUDA_TRY(cudaGetLastError());
        }
        for (uint32_t b = 0; b < B; b++) {
            const uint64_t i = c0 + b;
            if (kdim[b] < 2) {
                fill_u64<<<1, 32, 0, s>>>(q.cuts + i, 1, 0);
                continue;
            }
            for (uint32_t j = 0; j < 2; j++)
                eng.add(KNode{q.cuts + i, q.seed + (uint32_t)i, j, 1, kdim[b], 1, small, q.query, dd[b].mat, roots.buf});
        }
        if (c0 + chunk < q.trials) CAC_CUDA_TRY(cudaStreamSynchronize(s));  // the scratch is reused
    }
    return CAC_OK;
}

// Admission of several queries: those with Stage 1 in shared memory go through admit_stage1
// together, the others one by one.
int admit_many(cac_ctx *ctx, KsEngine &eng, const std::vector<const QueryPlan *> &qs) {
    std::vector<const QueryPlan *> batched;
    for (const QueryPlan *q : qs) {
        if (q->trials == 0) continue;
        if (q->groups) CAC_TRY(admit_groups(ctx, eng, *q));
        else if (q->t < q->g->n && q->g->n <= kMaxSmemVertices) batched.push_back(q);
        else CAC_TRY(admit(ctx, eng, *q));
    }
    return batched.empty() ? CAC_OK : admit_stage1(ctx, eng, batched);
}

int check_graph(const cac_graph *g, uint32_t t_override) {
    if (g->total_weight >= (1ull << 55)) {
        set_error("total edge weight >= 2^55 is not supported by the Stoer-Wagner leaf kernel");
        return CAC_ERR_UNSUPPORTED;
    }
    (void)t_override;  // contracted sizes above the dense limit run as sparse roots
    return CAC_OK;
}

}  // namespace

int mincut_admit_queries(cac_ctx *ctx, KsEngine &eng, const std::vector<MincutQuery> &qs,
                         const std::vector<uint32_t> &ids, std::vector<int> &status, std::vector<std::string> &msgs) {
    status.assign(qs.size(), CAC_OK);
    msgs.assign(qs.size(), std::string());
    std::vector<QueryPlan> plans;
    plans.reserve(qs.size());
    std::vector<size_t> which;
    for (size_t i = 0; i < qs.size(); i++) {
        const MincutQuery &q = qs[i];
        const int st = check_graph(q.g, q.t);
        if (st != CAC_OK) {
            status[i] = st;
            msgs[i] = cac_last_error();
            continue;
        }
        plans.push_back(QueryPlan{q.g, q.seed, q.ranks, q.per_rank, q.t ? q.t : intermediate_size(q.g->n, q.g->m),
                                  q.groups ? (uint64_t)q.groups : (uint64_t)q.ranks * q.per_rank, q.d_cuts, ids[i],
                                  q.groups});
        which.push_back(i);
        const QueryPlan &p = plans.back();
        if (p.trials)
            fill_u64<<<(unsigned)std::max<uint64_t>(1, std::min<uint64_t>((p.trials + 255) / 256, 4096)), 256, 0,
                       ctx->stream>>>(p.cuts, p.trials, kU64Max);
    }
    if (cudaGetLastError() != cudaSuccess) {
        set_error("mincut_admit_queries: filling the trial slots failed");
        for (size_t i : which) {
            status[i] = CAC_ERR_CUDA;
            msgs[i] = cac_last_error();
        }
        return CAC_ERR_CUDA;
    }
    std::vector<const QueryPlan *> ptrs;
    for (const QueryPlan &p : plans) ptrs.push_back(&p);
    const int st = admit_many(ctx, eng, ptrs);
    if (st != CAC_OK)
        for (size_t i : which) {
            status[i] = st;
            msgs[i] = cac_last_error();
        }
    return st;
}

namespace {

// One run of the queries through one engine; *redo is set when a run that planned ahead met a child
// off its target (its cuts are then not valid, and the caller runs the queries again without).
int run_queries(cac_ctx *ctx, std::vector<MincutQuery> &queries, float *device_ms, bool plan_ahead, bool *redo) {
    cudaStream_t s = ctx->stream;
    CAC_CUDA_TRY(cudaEventRecord(ctx->ev[0], s));
    KsEngine eng(ctx);
    eng.set_plan_ahead(plan_ahead);
    CAC_TRY(eng.init_err());
    std::vector<QueryPlan> plans(queries.size());
    for (size_t i = 0; i < queries.size(); i++) {
        MincutQuery &q = queries[i];
        QueryPlan &p = plans[i];
        p.g = q.g;
        p.seed = q.seed;
        p.ranks = q.ranks;
        p.per_rank = q.per_rank;
        p.t = q.t ? q.t : intermediate_size(q.g->n, q.g->m);
        p.trials = q.groups ? (uint64_t)q.groups : (uint64_t)q.ranks * q.per_rank;
        p.groups = q.groups;
        p.cuts = q.d_cuts;
        p.query = (uint32_t)i;
        if (p.trials)
            fill_u64<<<(unsigned)std::max<uint64_t>(1, std::min<uint64_t>((p.trials + 255) / 256, 4096)), 256, 0, s>>>(
                p.cuts, p.trials, kU64Max);
    }
    // admission by memory: a query is admitted when the engine's buffers leave room for its
    // estimated footprint (roots and two more levels of matrices); otherwise the engine steps first
    const uint64_t budget = ctx->budget ? ctx->budget / 2 : (48ull << 30);
    size_t next = 0;
    while (next < plans.size() || !eng.idle()) {
        // the queries that fit are admitted together (one Stage 1 launch for all of them)
        std::vector<const QueryPlan *> wave;
        uint64_t wave_est = 0;
        while (next < plans.size()) {
            const QueryPlan &p = plans[next];
            const uint64_t t = std::min<uint64_t>(p.t, p.g->n);
            const uint64_t est = (p.t < p.g->n ? p.trials : 1) * t * t * 8 * 3;
            if ((!eng.idle() || !wave.empty()) && ctx->held + wave_est + est > budget) break;
            wave.push_back(&p);
            wave_est += est;
            next++;
        }
        if (!wave.empty()) CAC_TRY(admit_many(ctx, eng, wave));
        if (!eng.idle()) CAC_TRY(eng.step());
    }
    uint32_t err = 0;
    CAC_TRY(eng.read_err(&err));
    CAC_CUDA_TRY(cudaEventRecord(ctx->ev[1], s));
    CAC_CUDA_TRY(cudaStreamSynchronize(s));
    if (device_ms) CAC_CUDA_TRY(cudaEventElapsedTime(device_ms, ctx->ev[0], ctx->ev[1]));
    if (plan_ahead && (err & kErrPlan)) {
        *redo = true;
        return CAC_OK;
    }
    if (err) return engine_error(err);
    return CAC_OK;
}

}  // namespace

// Runs the queries planning ahead (no read-back of children's sizes between levels) when the ctx
// allows it; the rare run in which a child stops off its target is run again level by level. Both
// give the same cuts: every draw is addressed by its trial, node and round, not by the schedule.
int mincut_run_queries(cac_ctx *ctx, std::vector<MincutQuery> &queries, float *device_ms) {
    for (const MincutQuery &q : queries) CAC_TRY(check_graph(q.g, q.t));
    bool redo = false;
    float ms = 0;
    CAC_TRY(run_queries(ctx, queries, &ms, ctx->plan_ahead, &redo));
    if (redo) {
        float ms2 = 0;
        CAC_TRY(run_queries(ctx, queries, &ms2, false, &redo));
        ms += ms2;
        ctx->plan_redos++;
    }
    if (device_ms) *device_ms = ms;
    return CAC_OK;
}

int mincut_trials(cac_ctx *ctx, const cac_graph *g, uint32_t seed, uint32_t ranks, uint32_t per_rank,
                  uint64_t *d_cuts, float *device_ms) {
    std::vector<MincutQuery> q{MincutQuery{g, seed, ranks, per_rank, d_cuts}};
    return mincut_run_queries(ctx, q, device_ms);
}

// A dense host matrix for the device: checks the weight bound and, when the total weight is below
// 2^32 (and so every entry), narrows it to the u32 node storage.
int host_matrix(uint32_t n, const uint64_t *mat_host, uint32_t *small, std::vector<unsigned char> &dev) {
    uint64_t total = 0, top = 0;
    for (uint64_t i = 0; i < (uint64_t)n * n; i++) {
        total += mat_host[i];
        top = std::max(top, mat_host[i]);
    }
    if (total / 2 >= (1ull << 55)) {
        set_error("total edge weight >= 2^55 is not supported");
        return CAC_ERR_UNSUPPORTED;
    }
    *small = (total / 2 < (1ull << 32) && top < (1ull << 32)) ? 1u : 0u;
    // the device layout: rows padded to ld_of(n) entries of 4 or 8 bytes
    const uint64_t ld = ld_of(n), es = *small ? 4 : 8;
    dev.assign(n * ld * es, 0);
    for (uint64_t i = 0; i < n; i++)
        for (uint64_t j = 0; j < n; j++) {
            const uint64_t x = mat_host[i * n + j];
            if (*small) reinterpret_cast<uint32_t *>(dev.data())[i * ld + j] = (uint32_t)x;
            else reinterpret_cast<uint64_t *>(dev.data())[i * ld + j] = x;
        }
    return CAC_OK;
}

int ks_dense_one(cac_ctx *ctx, uint32_t n, const uint64_t *mat_host, uint32_t seed, uint32_t rank, uint32_t trial,
                 uint64_t *cut) {
    if (n > kMaxSmemVertices) {
        set_error("dense Karger-Stein supports at most 16384 vertices");
        return CAC_ERR_UNSUPPORTED;
    }
    std::vector<unsigned char> dev;
    uint32_t small = 0;
    CAC_TRY(host_matrix(n, mat_host, &small, dev));
    cudaStream_t s = ctx->stream;
    DevBuf &d_cut = scratch(ctx, kSlotProbe0);
    CAC_TRY(d_cut.ensure(8));
    {
        KsEngine eng(ctx);
        CAC_TRY(eng.init_err());
        MatBuf *root = nullptr;
        CAC_TRY(eng.alloc(dev.size(), &root));
        CAC_CUDA_TRY(cudaMemcpyAsync(root->p, dev.data(), dev.size(), cudaMemcpyHostToDevice, s));
        CAC_CUDA_TRY(cudaStreamSynchronize(s));  // `dev` is pageable and goes out of scope
        fill_u64<<<1, 32, 0, s>>>(d_cut.as<uint64_t>(), 1, kU64Max);
        eng.add(KNode{d_cut.as<uint64_t>(), seed + rank, trial, 1, n, 1, small, 0, root->p, root});
        while (!eng.idle()) CAC_TRY(eng.step());
        uint32_t err = 0;
        CAC_TRY(eng.read_err(&err));
        if (err) {
            return engine_error(err);
        }
    }
    CAC_CUDA_TRY(cudaMemcpyAsync(cut, d_cut.p, 8, cudaMemcpyDeviceToHost, s));
    CAC_CUDA_TRY(cudaStreamSynchronize(s));
    return CAC_OK;
}

int exact_small(cac_ctx *ctx, uint32_t n, const uint64_t *mat_host, uint64_t *cut) {
    std::vector<unsigned char> dev;
    uint32_t small = 0;
    CAC_TRY(host_matrix(n, mat_host, &small, dev));
    cudaStream_t s = ctx->stream;
    DevBuf &buf = scratch(ctx, kSlotProbe0), &d_cuts = scratch(ctx, kSlotProbe1), &d_leaf = scratch(ctx, kSlotProbe2);
    CAC_TRY(buf.ensure(dev.size()));
    CAC_TRY(d_cuts.ensure(8));
    CAC_CUDA_TRY(cudaMemcpyAsync(buf.p, dev.data(), dev.size(), cudaMemcpyHostToDevice, s));
    fill_u64<<<1, 32, 0, s>>>(d_cuts.as<uint64_t>(), 1, kU64Max);
    std::vector<LeafDesc> leaves{LeafDesc{buf.p, d_cuts.as<uint64_t>(), nullptr, n, small}};
    CAC_TRY(upload(ctx, d_leaf, leaves));
    if (small) {
        const size_t sm = leaf_smem(n, true);
        CAC_TRY(smem_optin(ctx, sw_leaf_kernel<uint32_t>));
        sw_leaf_kernel<uint32_t><<<1, kLeafThreads, sm, s>>>(d_leaf.as<LeafDesc>());
    } else {
        const size_t sm = leaf_smem(n, false);
        CAC_TRY(smem_optin(ctx, sw_leaf_kernel<uint64_t>));
        sw_leaf_kernel<uint64_t><<<1, kLeafThreads, sm, s>>>(d_leaf.as<LeafDesc>());
    }
    CAC_CUDA_TRY(cudaGetLastError());
    CAC_CUDA_TRY(cudaMemcpyAsync(cut, d_cuts.p, 8, cudaMemcpyDeviceToHost, s));
    CAC_CUDA_TRY(cudaStreamSynchronize(s));
    return CAC_OK;
}

}  // namespace cac
