// vc_ub.cu -- the reference's two upper-bound heuristics on the GPU
// (vc_remove_max_ub / vc_remove_edge_ub in include/vcgpu.h).
//
// RemoveMaxApproximateMVC (src/auxFunctions.cpp:211-256) and
// RemoveEdgeApproximateMVC (:258-306) are greedy and order dependent: their
// results depend on the exact sequence of deletions, on the order in which the
// leaf and triangle rules visit the vertices (:44-127), and on the row order that
// CSRGraph::deleteVertex (CSRGraphRep.cpp:44-62) leaves behind, since it compacts
// each neighbour's row by copying the last live entry over the deleted one and
// the triangle test binary-searches those unsorted rows.  This kernel keeps that
// exact sequence and parallelises each step instead: one CTA per graph; a
// deletion updates all neighbours' rows at once (the rows are disjoint); the
// rules find "the next vertex in index order" with block-wide searches over
// bitmaps instead of full sweeps.
//
// Incremental bookkeeping that leaves the sequence unchanged:
//  * deg1: the vertices of degree 1 (bitmap, a summary bit per word, count).  A
//    leaf-rule pass visits them in index order from where the pass stands, exactly
//    the vertices the reference's sweep would act on; with none left no pass can act.
//  * mates: every entry (w in row x) knows where its mate (x in row w) is, so that a
//    deletion finds x in its neighbours' rows without reading them.
//  * two, dirty, moved: the vertices of degree 2 (bitmap); those of them that have
//    become so, and the vertices whose rows have changed, since the last pass that
//    found no triangle.  The test of vertex i reads deg(i), i's live prefix, the
//    degrees of its two live neighbours and the second neighbour's row.  i's prefix
//    changes only with its degree; falling degrees of its neighbours never let a
//    failed test succeed; so a test that failed can only succeed once i is dirty or
//    its second neighbour's row has moved.  The first firing vertex in index order
//    is the one the reference's restart-from-zero sweep would reach first.
//  * the largest degree (RemoveMax): an upper bound per block of vertices, made exact
//    only where it is the largest of all -- degrees only fall.
// The reference's binary search (auxFunctions.cpp:25-42) steps an unsigned
// index below zero (and reads out of bounds) in one corner case; there this
// search stops with "not found".
//
// What bounds it is one deletion's chain, whatever the size: find the vertex, read
// its row, the last entries of its neighbours' rows, move them -- three dependent
// reads from L2.  The rest is kept off it: bitmaps, degrees, offsets and the records
// of the last deletions sit in shared memory where they fit (graphs of up to some
// 14,000 vertices; the bitmaps alone above), and the leaf rule, most deletions of a
// sparse graph, is one warp's without a barrier of the block.  RemoveMax and
// RemoveEdge on a power-law graph of 12,000 vertices: 18.5 -> 5.3 and 21.6 -> 5.4 ms;
// of 100,000: 208 -> 72 and 236 -> 72 ms (before: 1024 threads, rows read and their
// neighbours of neighbours marked at every deletion, state in global memory; with
// the block's barriers in the leaf rule 6.3 ms on the smaller).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cstring>
#include <vector>

#include "vc_host.h"
#include "vc_types.h"
#include "vcgpu.h"

using namespace vcg;

namespace vch {
extern std::atomic<uint64_t> g_launches;
}
using namespace vch;

namespace {

constexpr unsigned kUbThreads = 512;
constexpr unsigned kUbWarps = kUbThreads / 32;
constexpr uint32_t kInf = 0xffffffffu;

struct UbParams {
    const InstDesc *inst;      // [count] n, offsets (row_off also into deg)
    const uint32_t *bad;       // [count] the CSR check failed
    const uint64_t *bits_off;  // [count] into bits: this graph's bitmaps where shared memory does not hold them
    const uint32_t *row_ptr;
    const uint32_t *col;
    uint32_t *dst;     // working copy of col, compacted by deletions
    uint32_t *mate;    // per entry of dst the place of its mate in the neighbour's row
    uint2 *gone;       // per vertex (as row_off): the deletion that last took an entry from its row, and from where
    int32_t *deg;      // working degrees, -1 = in the cover
    uint32_t *bits;
    uint32_t *ub;      // [count] results
    uint32_t smem;     // bytes of dynamic shared memory
    uint32_t mode;     // 0 RemoveMax, 1 RemoveEdge
    uint32_t r;        // RemoveEdge: the value of rand() the reference's draws used
};

constexpr int kShortRow = 8;          // entries of a moved row that one thread looks through
constexpr int kWarpDelete = 96;       // neighbours up to which one warp deletes a leaf's neighbour

// deg1, two, dirty, moved and deg1's summary, in words; then the cached maxima (two
// words each), then degrees and offsets where they fit too.
__host__ __device__ inline uint64_t ub_bitmap_words(uint32_t n)
{
    const uint64_t nw = (n + 31) / 32;
    return (4 * nw + (nw + 31) / 32 + 1) / 2 * 2;
}
// A cached maximum is of 2^shift vertices.  Graphs of up to 8192 vertices have as many
// blocks as the CTA has warps, at most, and each warp makes its block's maximum anew;
// above, about as many blocks as vertices in one, which one warp looks through.  (1024
// each: RemoveMax on 3-regular graphs of 1000 and 16,000 vertices 1.90 and 40.1 ms; with
// this and the moved rows' vertices marked 1.35 and 28.6.)
__host__ __device__ inline uint32_t ub_max_shift(uint32_t n)
{
    uint32_t s = 7;
    while (s < 9 && ((uint64_t)kUbWarps << s) < n) ++s;
    if (((uint64_t)kUbWarps << s) >= n) return s;
    for (s = 7; s < 16 && (1ull << (2 * s)) < n;) ++s;
    return s;
}
__host__ __device__ inline uint32_t ub_max_blocks(uint32_t n) { return (uint32_t)(((uint64_t)n + (1u << ub_max_shift(n)) - 1) >> ub_max_shift(n)); }
__host__ __device__ inline uint64_t ub_set_words(uint32_t n) { return ub_bitmap_words(n) + 2ull * ub_max_blocks(n); }
__host__ __device__ inline uint64_t ub_all_words(uint32_t n) { return ub_set_words(n) + 4ull * n + 1; }

struct UbShared {
    uint32_t x;          // the vertex to delete, or kInf
    uint32_t minimum, stamp;  // the block's, while one warp deletes
    uint32_t found;      // block search result
    uint32_t cnt1;       // vertices of degree 1
    uint32_t any;        // dirty or moved not empty
    unsigned long long amax;  // argmax key: degree << 32 | ~index
};

// The graph a CTA works on.
struct Ub {
    const uint32_t *rp;
    uint32_t *dst, *mate;
    uint2 *gone;
    int32_t *deg;
    uint32_t *d1, *s1, *d2, *dt, *mv;  // deg1, its summary, two, dirty, moved
    unsigned long long *bmax;          // per 2^shift vertices: at least the largest key
    uint32_t n, nw, shift;
};

__device__ __forceinline__ unsigned lane_of() { return threadIdx.x & 31u; }
__device__ __forceinline__ unsigned warp_of() { return threadIdx.x >> 5; }
__device__ __forceinline__ void ub_put(uint32_t *bm, uint32_t v) { atomicOr(&bm[v >> 5], 1u << (v & 31u)); }
__device__ __forceinline__ void ub_drop(uint32_t *bm, uint32_t v) { atomicAnd(&bm[v >> 5], ~(1u << (v & 31u))); }
__device__ __forceinline__ bool ub_has(const uint32_t *bm, uint32_t v) { return (bm[v >> 5] >> (v & 31u)) & 1u; }

__device__ __forceinline__ void ub_set1(const Ub &g, UbShared &sh, uint32_t v)
{
    ub_put(g.d1, v);
    ub_put(g.s1, v >> 5);
    atomicAdd(&sh.cnt1, 1u);
}

// Deletes live vertex x (CSRGraph::deleteVertex): each live neighbour w takes x
// out of its live prefix by moving its last live entry over it.  A thread per
// neighbour, kUbThreads of them at a time: the rows are disjoint, and only the
// mates cross.  The entry z that w moves from `last` to `pos` has its mate in z's
// row; if z loses x too and that mate is what z moves, it is found where z's x was
// (both ends of such a pair then write the same).  `stamp` numbers these steps of a
// graph from 1.  The block has passed a barrier since x was chosen, and passes one
// after this before it reads what this changed.  With Warp it is one warp's work,
// and its barriers are the warp's.
template <bool Warp>
__device__ __forceinline__ void ub_delete(const Ub &g, UbShared &sh, uint32_t x, uint32_t &stamp)
{
    constexpr int kStep = Warp ? 32 : (int)kUbThreads;
    const int me = Warp ? (int)lane_of() : (int)threadIdx.x;
    auto barrier = [] {
        if constexpr (Warp) __syncwarp();
        else __syncthreads();
    };
    const int dx = g.deg[x];
    const uint32_t bx = g.rp[x];
    for (int base = 0; base < dx; base += kStep) {
        ++stamp;
        const int t = base + me;
        const bool mine = t < dx;
        uint32_t w = 0, pos = 0, z = x, zm = 0;
        int dw = 0;
        if (mine) {
            w = g.dst[bx + (uint32_t)t];
            pos = g.mate[bx + (uint32_t)t];
            dw = g.deg[w];
            const uint32_t last = g.rp[w] + (uint32_t)dw - 1u;
            z = g.dst[last];
            zm = g.mate[last];
            g.gone[w] = make_uint2(stamp, pos);
        }
        barrier();
        if (mine && z != x) {
            const uint2 gz = g.gone[z];
            if (gz.x == stamp && zm == g.rp[z] + (uint32_t)g.deg[z] - 1u) zm = gz.y;
            g.dst[pos] = z;
            g.mate[pos] = zm;
            g.mate[zm] = pos;
        }
        barrier();
        if (mine) {
            g.deg[w] = dw - 1;
            if (dw == 3) {
                ub_put(g.d2, w);
                ub_put(g.dt, w);
            } else if (dw == 2) {
                ub_drop(g.d2, w);
                ub_set1(g, sh, w);
            } else if (dw == 1) {
                ub_drop(g.d1, w);
                atomicSub(&sh.cnt1, 1u);
            }
            ub_put(g.mv, w);
        }
        if (base + kStep < dx) barrier();
    }
    if (me == 0) {
        if (dx == 1) {
            ub_drop(g.d1, x);
            atomicSub(&sh.cnt1, 1u);
        } else if (dx == 2) {
            ub_drop(g.d2, x);
        }
        g.deg[x] = -1;
        sh.any = 1u;
    }
}

// The first vertex of degree 1 at index >= p, or kInf (one warp).  A summary bit
// may be set over an empty word: it is cleared when met.
__device__ uint32_t ub_next_leaf(const Ub &g, uint32_t p)
{
    const unsigned lane = lane_of();
    if (p >= g.n) return kInf;
    uint32_t x = *(volatile uint32_t *)&g.d1[p >> 5] & (~0u << (p & 31u));
    if (x) return (p & ~31u) + (uint32_t)(__ffs(x) - 1);
    const uint32_t sw = (g.nw + 31) / 32;
    uint32_t from = (p >> 5) + 1;  // words from here on
    for (uint32_t base = from >> 5; base < sw; base += 32) {
        const uint32_t i = base + lane;
        for (;;) {
            uint32_t m = i < sw ? *(volatile uint32_t *)&g.s1[i] : 0u;
            if (i == from >> 5) m &= ~0u << (from & 31u);
            const uint32_t bal = __ballot_sync(0xffffffffu, m != 0u);
            if (!bal) break;
            const uint32_t src = __ffs(bal) - 1;
            const uint32_t w = 32u * (base + src) + (uint32_t)(__ffs(__shfl_sync(0xffffffffu, m, src)) - 1);
            x = *(volatile uint32_t *)&g.d1[w];
            if (x) return 32u * w + (uint32_t)(__ffs(x) - 1);
            __syncwarp();
            if (lane == 0) atomicAnd(&g.s1[w >> 5], ~(1u << (w & 31u)));
            __syncwarp();
        }
    }
    return kInf;
}

// The largest key (degree << 32 | ~index) of block `i`, by one warp.
__device__ unsigned long long ub_block_max(const Ub &g, uint32_t i)
{
    unsigned long long best = 0;
    const uint32_t lo = i << g.shift, hi = min(g.n, lo + (1u << g.shift));
    for (uint32_t v = lo + lane_of(); v < hi; v += 32) {
        const int d = g.deg[v];
        const unsigned long long key = d > 0 ? ((unsigned long long)(uint32_t)d << 32) | (uint32_t)(~v) : 0ull;
        best = key > best ? key : best;
    }
#pragma unroll
    for (int k = 16; k; k >>= 1) {
        const unsigned long long o = __shfl_xor_sync(0xffffffffu, best, k);
        best = o > best ? o : best;
    }
    return best;
}

// auxBinarySearch over a (compacted, possibly unsorted) row, stopping where
// the reference's unsigned index would go below zero.
__device__ bool ub_search(const uint32_t *arr, long l, long r, uint32_t x)
{
    while (l <= r) {
        const long m = l + (r - l) / 2;
        const uint32_t a = arr[m];
        if (a == x) return true;
        if (a < x) l = m + 1;
        else r = m - 1;
    }
    return false;
}

// The triangle test of vertex i (auxFunctions.cpp:79-121): its two live
// neighbours are the first two entries of its compacted row.
__device__ bool ub_fires(const uint32_t *rp, const uint32_t *dst, const int32_t *deg, uint32_t i, uint32_t *n1,
                         uint32_t *n2)
{
    if (deg[i] != 2) return false;
    const uint32_t a = dst[rp[i]], b = dst[rp[i] + 1];
    const int da = deg[a], db = deg[b];
    if (da == 1 || (da == 2 && a < i)) return false;
    if (db == 1 || (db == 2 && b < i)) return false;
    if (!ub_search(dst, (long)rp[b], (long)rp[b + 1] - 1, a)) return false;
    *n1 = a;
    *n2 = b;
    return true;
}

__global__ void __launch_bounds__(kUbThreads) k_ub(UbParams P)
{
    __shared__ UbShared sh;
    extern __shared__ __align__(16) uint32_t ub_smem[];
    const uint32_t gi = blockIdx.x;
    if (P.bad[gi]) return;
    const uint32_t n = P.inst[gi].n;
    const uint64_t row_off = P.inst[gi].row_off, col_off = P.inst[gi].col_off;
    const uint32_t *rp0 = P.row_ptr + row_off;
    const uint32_t *col = P.col + col_off;
    int32_t *deg0 = P.deg + row_off;
    const bool set_in = 4ull * ub_set_words(n) <= P.smem, all_in = 4ull * ub_all_words(n) <= P.smem;
    uint32_t *sets = set_in ? ub_smem : P.bits + P.bits_off[gi];
    Ub g;
    g.n = n;
    g.nw = (n + 31) / 32;
    g.shift = ub_max_shift(n);
    g.dst = P.dst + col_off;
    g.mate = P.mate + col_off;
    g.gone = P.gone + row_off;
    g.d1 = sets;
    g.d2 = sets + g.nw;
    g.dt = sets + 2 * g.nw;
    g.mv = sets + 3 * g.nw;
    g.s1 = sets + 4 * g.nw;
    g.bmax = reinterpret_cast<unsigned long long *>(sets + ub_bitmap_words(n));
    uint32_t *rp_in = ub_smem + ub_set_words(n) + 2ull * n;
    if (all_in) g.gone = reinterpret_cast<uint2 *>(ub_smem + ub_set_words(n));
    g.deg = all_in ? reinterpret_cast<int32_t *>(rp_in + n + 1) : deg0;
    g.rp = all_in ? rp_in : rp0;
    const uint32_t m2 = n ? rp0[n] : 0u;
    if (threadIdx.x == 0) {
        sh.cnt1 = 0;
        sh.any = 1;
    }
    for (uint32_t e = threadIdx.x; e < m2; e += kUbThreads) g.dst[e] = col[e];
    for (uint32_t w = threadIdx.x; w < g.nw; w += kUbThreads) {
        g.d1[w] = 0;
        g.d2[w] = 0;
        g.dt[w] = ~0u;
        g.mv[w] = 0;
    }
    for (uint32_t w = threadIdx.x; w < (g.nw + 31) / 32; w += kUbThreads) g.s1[w] = 0;
    if (all_in)
        for (uint32_t v = threadIdx.x; v <= n; v += kUbThreads) rp_in[v] = rp0[v];
    __syncthreads();
    // With no row of more than kShortRow entries the triangle rule marks the degree-2
    // vertices of the rows that have moved; else every degree-2 vertex looks at its second
    // neighbour, as deletions beside long rows move too many of them (G(2000, 0.5) 12.5
    // ms, marked 17.3; but on a 3-regular graph of 4000 vertices RemoveMax and RemoveEdge
    // took 6.2 and 5.1, marked 5.2 and 4.5).
    bool is_long = false;
    for (uint32_t v = threadIdx.x; v < n; v += kUbThreads) {
        const int d = (int)(g.rp[v + 1] - g.rp[v]);
        is_long = is_long || d > kShortRow;
        g.deg[v] = d;
        g.gone[v] = make_uint2(0u, 0u);
        if (d == 1) ub_set1(g, sh, v);
        if (d == 2) ub_put(g.d2, v);
    }
    const bool all_short = !__syncthreads_or(is_long);
    const uint32_t blocks = ub_max_blocks(n);
    if (P.mode == 0)
        for (uint32_t i = warp_of(); i < blocks; i += kUbWarps) {
            const unsigned long long k = ub_block_max(g, i);
            if (lane_of() == 0) g.bmax[i] = k;
        }
    __syncthreads();
    uint32_t minimum = 0;           // uniform across the block
    uint32_t stamp = 0;             // steps of ub_delete so far
    uint32_t remaining = m2 / 2;    // RemoveEdge's edge count
    uint32_t vertex = 0;            // RemoveEdge's loop index
    for (;;) {
        if (P.mode == 1 && !(vertex < n && remaining > 0)) break;
        const uint32_t before = minimum;
        // leaf rule to its fixpoint: passes in index order while a pass acts.  One
        // warp runs it, with no barrier of the block, until a vertex of many
        // neighbours is due.
        {
            uint32_t p = 0;  // (in warp 0; so is `changed`)
            bool changed = false;
            for (;;) {
                __syncthreads();  // the deletion before this is complete
                if (warp_of() == 0) {
                    uint32_t x = kInf;
                    while (*(volatile uint32_t *)&sh.cnt1 != 0) {  // else no pass can act any more
                        uint32_t i = ub_next_leaf(g, p);
                        if (i == kInf && changed) {
                            changed = false;
                            i = ub_next_leaf(g, 0);
                        }
                        if (i == kInf) break;
                        changed = true;
                        p = i + 1;
                        const uint32_t only = *(volatile uint32_t *)&g.dst[g.rp[i]];  // its only live neighbour
                        if (g.deg[only] > kWarpDelete) {
                            x = only;
                            break;
                        }
                        ub_delete<true>(g, sh, only, stamp);
                        minimum += 1;
                        __syncwarp();
                    }
                    if (lane_of() == 0) {
                        sh.x = x;
                        sh.minimum = minimum;
                        sh.stamp = stamp;
                    }
                }
                __syncthreads();
                const uint32_t x = sh.x;
                minimum = sh.minimum;
                stamp = sh.stamp;
                if (x == kInf) break;
                ub_delete<false>(g, sh, x, stamp);
                minimum += 1;
            }
        }
        // triangle rule to its fixpoint: the first firing vertex, then restart
        for (;;) {
            __syncthreads();
            if (!sh.any) break;
            if (all_short) {  // the degree-2 vertices of moved rows are due, and no others
                for (uint32_t wi = threadIdx.x; wi < g.nw; wi += kUbThreads) {
                    uint32_t m = g.mv[wi];
                    if (m) g.mv[wi] = 0;
                    while (m) {
                        const uint32_t v = 32u * wi + (uint32_t)(__ffs(m) - 1);
                        m &= m - 1;
                        const int d = g.deg[v];
                        uint32_t y[kShortRow];
#pragma unroll
                        for (int k = 0; k < kShortRow; ++k) y[k] = k < d ? g.dst[g.rp[v] + k] : v;
#pragma unroll
                        for (int k = 0; k < kShortRow; ++k)
                            if (k < d && ub_has(g.d2, y[k])) ub_put(g.dt, y[k]);
                    }
                }
                __syncthreads();
            }
            uint32_t fire = kInf;
            for (uint32_t base = 0; base < g.nw && fire == kInf; base += kUbThreads) {
                __syncthreads();
                if (threadIdx.x == 0) sh.found = kInf;
                __syncthreads();
                const uint32_t wi = base + threadIdx.x;
                if (wi < g.nw) {
                    uint32_t x = g.d2[wi];
                    const uint32_t fresh = g.dt[wi];
                    if (all_short) x &= fresh;
                    while (x) {
                        const uint32_t i = 32u * wi + (uint32_t)(__ffs(x) - 1);
                        x &= x - 1;
                        if (!((fresh >> (i & 31u)) & 1u) && !ub_has(g.mv, g.dst[g.rp[i] + 1])) continue;
                        uint32_t a, b;
                        if (ub_fires(g.rp, g.dst, g.deg, i, &a, &b)) {
                            atomicMin(&sh.found, i);
                            break;
                        }
                    }
                }
                __syncthreads();
                fire = sh.found;
            }
            if (fire == kInf) {  // a full pass without a triangle: every test fails as things are
                __syncthreads();
                for (uint32_t w = threadIdx.x; w < g.nw; w += kUbThreads) {
                    g.dt[w] = 0;
                    g.mv[w] = 0;
                }
                if (threadIdx.x == 0) sh.any = 0;
                __syncthreads();
                break;
            }
            uint32_t a = 0, b = 0;
            ub_fires(g.rp, g.dst, g.deg, fire, &a, &b);
            __syncthreads();  // every thread has both
            ub_delete<false>(g, sh, a, stamp);
            __syncthreads();
            ub_delete<false>(g, sh, b, stamp);
            minimum += 2;
        }
        if (P.mode == 0) {
            // the lowest-index vertex of maximum degree
            unsigned long long k = 0;
            if (blocks <= kUbWarps) {
                __syncthreads();
                if (warp_of() < blocks) {
                    const unsigned long long now = ub_block_max(g, warp_of());
                    if (lane_of() == 0) g.bmax[warp_of()] = now;
                }
                __syncthreads();
                k = lane_of() < blocks ? g.bmax[lane_of()] : 0ull;
#pragma unroll
                for (int j = 16; j; j >>= 1) {
                    const unsigned long long o = __shfl_xor_sync(0xffffffffu, k, j);
                    k = o > k ? o : k;
                }
            }
            // the largest cached maximum that is still exact
            else for (;;) {
                __syncthreads();
                if (warp_of() == 0) {
                    unsigned long long best = 0;
                    uint32_t at = 0;
                    for (uint32_t i = lane_of(); i < blocks; i += 32) {
                        const unsigned long long k = g.bmax[i];
                        if (k > best) { best = k; at = i; }
                    }
#pragma unroll
                    for (int k = 16; k; k >>= 1) {
                        const unsigned long long o = __shfl_xor_sync(0xffffffffu, best, k);
                        const uint32_t oa = __shfl_xor_sync(0xffffffffu, at, k);
                        if (o > best) { best = o; at = oa; }
                    }
                    const unsigned long long now = best ? ub_block_max(g, at) : 0ull;
                    if (lane_of() == 0) {
                        if (best) g.bmax[at] = now;
                        sh.amax = now;
                        sh.found = now == best;
                    }
                }
                __syncthreads();
                k = sh.amax;
                if (sh.found) break;
            }
            if (k == 0) break;
            ub_delete<false>(g, sh, ~(uint32_t)k, stamp);
            minimum += 1;
        } else {
            // on to the next live vertex at once if the rules had nothing to do: they
            // would have nothing to do before each dead one either
            __syncthreads();
            for (bool live = minimum != before; !live && vertex < n;) {
                const uint32_t v = vertex + lane_of();
                const uint32_t m = __ballot_sync(0xffffffffu, v < n && g.deg[v] > 0);
                live = m != 0u;
                vertex = live ? vertex + (uint32_t)(__ffs(m) - 1) : min(n, vertex + 32u);
            }
            const int dv = vertex < n ? g.deg[vertex] : 0;
            if (dv > 0) {
                const uint32_t u = g.dst[g.rp[vertex] + P.r % (uint32_t)dv];
                remaining -= (uint32_t)dv;
                remaining -= (uint32_t)g.deg[u];
                ++remaining;
                __syncthreads();  // every thread has them
                ub_delete<false>(g, sh, vertex, stamp);
                __syncthreads();
                ub_delete<false>(g, sh, u, stamp);
                minimum += 2;
            }
            ++vertex;
        }
    }
    if (all_in) {
        __syncthreads();
        for (uint32_t v = threadIdx.x; v < n; v += kUbThreads) deg0[v] = g.deg[v];
    }
    if (threadIdx.x == 0) P.ub[gi] = minimum;
}

vc_status ub_run(const vc_csr_arena *a, uint32_t mode, uint32_t r, int32_t device, uint32_t *ub, uint8_t *cover,
                 float *kernel_ms)
{
    if (!a || !ub || (a->count && (!a->n || !a->row_off || !a->col_off || !a->row_ptr))) return VC_ERR_INVALID;
    const uint32_t count = a->count;
    if (count == 0) return VC_OK;
    uint64_t rows = 0, cols = 0, bits = 0;
    uint32_t nmax = 0;
    std::vector<uint64_t> boff(count);
    std::vector<InstDesc> desc(count);
    auto graph = [&](uint32_t i) {
        const uint32_t *rp = a->row_ptr + a->row_off[i];
        vc_csr g;
        g.n = a->n[i];
        g.m = rp[g.n] / 2;
        g.row_ptr = rp;
        g.col = a->col ? a->col + a->col_off[i] : nullptr;
        g.degree = nullptr;
        return g;
    };
    for (uint32_t i = 0; i < count; ++i) {
        if (a->n[i] > kMaxVertices) {  // unless a graph before it is invalid
            for (uint32_t j = 0; j < i; ++j) {
                const vc_csr g = graph(j);
                if (validate_csr(&g) != VC_OK) return VC_ERR_INVALID;
            }
            return VC_ERR_TOO_LARGE;
        }
        nmax = std::max(nmax, a->n[i]);
        rows = std::max<uint64_t>(rows, a->row_off[i] + a->n[i] + 1);
        boff[i] = bits;
        bits += ub_set_words(a->n[i]);
    }
    for (uint32_t i = 0; i < count; ++i) {
        const vc_csr g = graph(i);
        const vc_status v = check_head(&g);
        if (v != VC_OK) return v;
        cols = std::max<uint64_t>(cols, a->col_off[i] + 2ull * g.m);
        InstDesc d{};
        d.n = g.n;
        d.row_off = a->row_off[i];
        d.col_off = a->col_off[i];
        d.m2 = 2 * g.m;
        desc[i] = d;
    }
    vc_status err;
    Ctx *c = get_ctx(device, &err);
    if (!c) {
        for (uint32_t i = 0; i < count; ++i) {
            const vc_csr g = graph(i);
            if (validate_csr(&g) != VC_OK) return VC_ERR_INVALID;
        }
        return err;
    }
    std::lock_guard<std::mutex> lk(c->mu);
    cudaStream_t st = c->stream;
    // one piece of device memory, kept between calls up to a bound: descriptors,
    // offsets of the bitmaps, bounds, check results, offsets, ids (the graphs' and
    // the working copy), mates, degrees, last deletions, bitmaps
    uint64_t bytes = 0;
    auto piece = [&](uint64_t b) {
        const uint64_t at = bytes;
        bytes += (b + 255) / 256 * 256;
        return at;
    };
    const uint64_t o_desc = piece(sizeof(InstDesc) * (uint64_t)count), o_bo = piece(8ull * count), o_ub = piece(4ull * count),
                   o_bad = piece(4ull * count), o_rp = piece(4 * rows), o_col = piece(4 * cols), o_dst = piece(4 * cols),
                   o_mate = piece(4 * cols), o_deg = piece(4 * rows), o_gone = piece(8 * rows), o_bits = piece(4 * bits);
    struct Slab {
        Ctx *c;
        ~Slab()
        {
            if (c->ub.cap > kUbBytesKept) c->ub.release();
        }
    } slab{c};
    if (c->ub.ensure(bytes)) return VC_ERR_NOMEM;
    uint8_t *base = (uint8_t *)c->ub.p;
    bool ok = cudaMemcpyAsync(base + o_desc, desc.data(), sizeof(InstDesc) * count, cudaMemcpyHostToDevice, st) == cudaSuccess &&
              cudaMemcpyAsync(base + o_bo, boff.data(), 8ull * count, cudaMemcpyHostToDevice, st) == cudaSuccess &&
              cudaMemsetAsync(base + o_bad, 0, 4ull * count, st) == cudaSuccess &&
              cudaMemcpyAsync(base + o_rp, a->row_ptr, 4 * rows, cudaMemcpyHostToDevice, st) == cudaSuccess &&
              (cols == 0 || cudaMemcpyAsync(base + o_col, a->col, 4 * cols, cudaMemcpyHostToDevice, st) == cudaSuccess);
    if (!ok) {
        cudaStreamSynchronize(st);
        return VC_ERR_CUDA;
    }
    UbParams P;
    P.inst = (const InstDesc *)(base + o_desc);
    P.bad = (const uint32_t *)(base + o_bad);
    P.bits_off = (const uint64_t *)(base + o_bo);
    P.row_ptr = (const uint32_t *)(base + o_rp);
    P.col = (const uint32_t *)(base + o_col);
    P.dst = (uint32_t *)(base + o_dst);
    P.mate = (uint32_t *)(base + o_mate);
    P.gone = (uint2 *)(base + o_gone);
    P.deg = (int32_t *)(base + o_deg);
    P.bits = (uint32_t *)(base + o_bits);
    P.ub = (uint32_t *)(base + o_ub);
    P.mode = mode;
    P.r = r;
    // shared memory for the largest graph that fits whole; graphs above keep what fits of theirs
    const uint64_t room = (uint64_t)c->smem_optin - sizeof(UbShared) - 256;
    uint64_t need = 0;
    for (uint32_t i = 0; i < count; ++i)
        for (const uint64_t w : {ub_set_words(a->n[i]), ub_all_words(a->n[i])})
            if (4 * w <= room) need = std::max<uint64_t>(need, 4 * w);
    P.smem = (uint32_t)need;
    cudaEventRecord(c->ev0, st);
    void *args[] = {&P};
    // checked by their own return codes: an error the caller left pending is neither reported nor cleared
    bool good = launch_check(true, P.row_ptr, P.col, P.inst, (uint32_t *)(base + o_bad), 1, 1u, count, nmax, st, P.mate) == cudaSuccess &&
                cudaFuncSetAttribute(k_ub, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)need) == cudaSuccess &&
                cudaLaunchKernel((const void *)k_ub, dim3(count), dim3(kUbThreads), args, need, st) == cudaSuccess;
    cudaEventRecord(c->ev1, st);
    g_launches += 2;
    std::vector<uint32_t> res(2 * (size_t)count);  // bounds, check results
    std::vector<int32_t> deg(cover ? rows : 0);
    good = good && cudaMemcpyAsync(res.data(), base + o_ub, 4ull * count, cudaMemcpyDeviceToHost, st) == cudaSuccess &&
           cudaMemcpyAsync(res.data() + count, base + o_bad, 4ull * count, cudaMemcpyDeviceToHost, st) == cudaSuccess &&
           (!cover || cudaMemcpyAsync(deg.data(), base + o_deg, 4 * rows, cudaMemcpyDeviceToHost, st) == cudaSuccess);
    if (cudaStreamSynchronize(st) != cudaSuccess || !good) return VC_ERR_CUDA;
    for (uint32_t i = 0; i < count; ++i)
        if (res[count + i]) return VC_ERR_INVALID;
    if (kernel_ms) cudaEventElapsedTime(kernel_ms, c->ev0, c->ev1);
    std::copy(res.begin(), res.begin() + count, ub);
    if (cover) {
        uint64_t k = 0;
        for (uint32_t i = 0; i < count; ++i)
            for (uint32_t v = 0; v < a->n[i]; ++v) cover[k++] = deg[a->row_off[i] + v] == -1;
    }
    return VC_OK;
}

}  // namespace

extern "C" vc_status vc_remove_max_ub(const vc_csr_arena *a, int32_t device, uint32_t *ub, uint8_t *cover,
                                     float *kernel_ms)
{
    vch::DeviceGuard dg;
    return ub_run(a, 0u, 0u, device, ub, cover, kernel_ms);
}

extern "C" vc_status vc_remove_edge_ub(const vc_csr_arena *a, uint32_t r, int32_t device, uint32_t *ub,
                                      uint8_t *cover, float *kernel_ms)
{
    vch::DeviceGuard dg;
    return ub_run(a, 1u, r, device, ub, cover, kernel_ms);
}
