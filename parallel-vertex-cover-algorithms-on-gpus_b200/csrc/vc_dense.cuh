// vc_dense.cuh -- the search for graphs of at most 255 vertices (the batched
// workload's G(n, p) instances, n in [30, 200], and the 60-vertex case), and,
// with 20-word rows, for graphs of up to 640 vertices whose degrees all fit a
// byte (at most 254); with 16- and 32-word rows and 16-bit degrees (two to a
// word, see "Half" below), for graphs of up to 512 and 1024 vertices of any
// degree -- the dense DIMACS-style graphs the CSR walks handle worst.
//
// Same search as vc_search.cuh (the reference's degree-one, triangle and
// high-degree rules, the E > b^2 prune and max-degree branching), with dense
// bitsets instead of CSR walks:
//
//  * a CTA works on one graph at a time: its adjacency is staged once into
//    shared memory as one NW-word bitmap per vertex (NW = 8: 8 KB) and shared
//    by the CTA's warps, which split the graph's search tree among themselves
//    through the CTA pool (vc_search.cuh);
//  * one warp is one search unit; its node state is the live-vertex set L (NW
//    words in shared memory, word w kept by lane w; copied into registers
//    where a whole row is masked with it); a vertex taken into the cover
//    leaves L, so del = n - |L| and the cover is the complement of L;
//  * deg(v) = popc(adj[v] & L), kept as bytes (0 = removed or isolated), four
//    to a 32-bit word: lane l holds words l and l + 32 in registers, so the
//    rule tests of a pass look at four vertices per instruction (SWAR byte
//    arithmetic).  When a set M leaves L, only the rows of M are read: each
//    lane subtracts the 4-bit slices of those rows that cover its vertices
//    (the adjacency is symmetric).  After a backtrack the degrees are
//    recounted, one vertex per lane;
//  * the triangle test of a degree-2 vertex is one bit test and the leaf
//    rule's neighbour one find-first-set: no serial CSR row walks;
//  * a node's children are bounded by a clique packing before either is entered
//    ("the packing bound" below): a closed child costs no node, and with one
//    left the node is no branch;
//  * backtracking: an undo trail of removed ids (u16) and frames of (trail
//    position, branching vertex); restoring ORs bits back into L.
//
// Records exchanged through the CTA pool and the global ring are live bitmaps.
#pragma once
#include "vc_search.cuh"

namespace vcg {

__device__ __forceinline__ unsigned lane_id() { return threadIdx.x & 31u; }

template <int NW>
struct Rows {
    static constexpr bool kHalf = NW == 16 || NW == 32;  // 16-bit degrees (dense_half)
    static constexpr int kStride = NW == 8 ? 12 : (NW == 16 ? 20 : NW);  // dense_row_words
    static constexpr bool kSwz = NW == 32;  // 16-byte chunks of a row XOR-swizzled by the row's low 3 bits
    // Index of word w of row v.
    static __device__ __forceinline__ uint32_t at(uint32_t v, uint32_t w)
    {
        return v * kStride + (kSwz ? ((((w >> 2) ^ (v & 7u)) << 2) | (w & 3u)) : w);
    }
    static constexpr int kPer = kHalf ? 2 : 4;                             // degrees per word
    static constexpr int kJ = kHalf ? NW / 2 : (NW >= 8 ? NW / 4 : 1);     // degree words per lane
    // bits of a lane's candidate count (at most kPer * kJ)
    static constexpr int kCandBits = kPer * kJ >= 32 ? 6 : (kPer * kJ >= 16 ? 5 : (kPer * kJ >= 8 ? 4 : 3));
    static constexpr int kTri = 32 * NW * kStride;          // offset of the triangle bitmap
};

// 0x80 in every byte of x that is zero, 0 elsewhere.
__device__ __forceinline__ uint32_t bytes_zero(uint32_t x)
{
    return ~(((x & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | x | 0x7F7F7F7Fu);
}

// 4 bits -> the low bit of each of 4 bytes (bit b to bit 8b).
__device__ __forceinline__ uint32_t spread4(uint32_t nib) { return (nib * 0x00204081u) & 0x01010101u; }

// The top bits of 4 bytes (bit 8b+7) -> 4 bits (bit b).
__device__ __forceinline__ uint32_t gather4(uint32_t hb) { return ((hb >> 7) * 0x01020408u) >> 24; }

// Half: the same tests on two 16-bit degrees per word (values below 2^15).
// 0x8000 in every halfword of x that is zero, 0 elsewhere.
__device__ __forceinline__ uint32_t halves_zero(uint32_t x)
{
    return ~(((x & 0x7FFF7FFFu) + 0x7FFF7FFFu) | x | 0x7FFF7FFFu);
}

// 2 bits -> the low bit of each halfword.
__device__ __forceinline__ uint32_t spread2(uint32_t b) { return (b & 1u) | ((b & 2u) << 15); }

// The top bits of 2 halfwords (bits 15, 31) -> 2 bits.
__device__ __forceinline__ uint32_t gather2(uint32_t hb) { return ((hb >> 15) & 1u) | ((hb >> 30) & 2u); }

// extra CTA header words used by the dense kernel
enum : uint32_t { kCpStaged = 5, kCpCursorClosed = 6 };

// Per-phase cycle counters of the statistics mode (vc_debug_stats) cost a
// clock read and a branch per phase even when off, so they are compiled in
// only with VC_PHASE_TIMERS=1.
#ifndef VC_PHASE_TIMERS
#define VC_PHASE_TIMERS 0
#endif
constexpr bool kPhaseTimers = VC_PHASE_TIMERS != 0;

struct PhaseCycles {
    unsigned long long scan, apply, pop, branch;
};

template <int NW>
struct DSU {
    SUStat stat;
    PhaseCycles cyc;
    bool timed;
    const uint32_t *adj;  // CTA-shared [32*NW][kStride] rows, then the triangle bitmap
    uint8_t *ws;          // this warp's workspace; the arrays below sit at fixed offsets
    __device__ __forceinline__ uint32_t *frames() const { return reinterpret_cast<uint32_t *>(ws); }  // [32*NW] (trail position << 16) | vertex
    __device__ __forceinline__ uint32_t *marks() const { return frames() + 32 * NW; }  // [NW]
    __device__ __forceinline__ uint32_t *bits() const { return marks() + NW; }         // [NW] record / scratch
    __device__ __forceinline__ uint32_t *lsm() const { return bits() + NW; }           // [NW] the live set L
    __device__ __forceinline__ uint16_t *trail() const { return reinterpret_cast<uint16_t *>(lsm() + NW); }  // [32*NW]
    __device__ __forceinline__ uint16_t *cand() const { return trail() + 32 * NW; }   // [32*NW] pass candidates
    __device__ __forceinline__ uint8_t *degs() const { return reinterpret_cast<uint8_t *>(cand() + 32 * NW); }  // [32*NW] staging copy of D
    __device__ __forceinline__ uint16_t *degs16() const { return reinterpret_cast<uint16_t *>(cand() + 32 * NW); }  // the same, Half
    uint32_t D[Rows<NW>::kJ];   // degree bytes of vertices 4q..4q+3, q = 32j + lane (Half: 16-bit degrees of 2q, 2q+1)
    uint32_t Ln[Rows<NW>::kJ];  // their live bits (4 per word; Half: 2)
    const uint32_t *rp, *cl;
    uint32_t inst, n, nw, mode, k, cover_off;
    unsigned long long node_limit;
    uint32_t base_del, top;
    uint32_t c_best;
    uint32_t fr_bot, fr_top;
    uint32_t pending;  // how the next node starts: kPendApply / kPendRecount with the set in marks
    unsigned long long local_nodes;
    unsigned long long deadline;
};

enum : uint32_t { kPendApply = 1, kPendRecount = 2 };


template <int NW>
__device__ __forceinline__ void dsu_bind(DSU<NW> &s, uint8_t *ws, const uint32_t *adj)
{
    s.adj = adj;
    s.ws = ws;
}

template <int NW>
__device__ __forceinline__ uint32_t *rec_bits(DSU<NW> &s) { return s.bits(); }

// Loads the first nw (runtime, uniform) words of a row; the rest read as 0.
template <int NW>
__device__ __forceinline__ void load_row(const uint32_t *row, uint32_t (&r)[NW], uint32_t nw)
{
    if constexpr (NW % 4 == 0) {
#pragma unroll
        for (int w = 0; w < NW; w += 4) {
            if ((uint32_t)w < nw) {
                const uint4 q = *reinterpret_cast<const uint4 *>(row + w);
                r[w] = q.x; r[w + 1] = q.y; r[w + 2] = q.z; r[w + 3] = q.w;
            } else {
                r[w] = r[w + 1] = r[w + 2] = r[w + 3] = 0u;
            }
        }
    } else {
#pragma unroll
        for (int w = 0; w < NW; w += 2) {
            const uint2 q = *reinterpret_cast<const uint2 *>(row + w);
            r[w] = q.x; r[w + 1] = q.y;
        }
    }
}

// Row v of the adjacency (logical word order) into registers.
template <int NW>
__device__ __forceinline__ void load_row_at(const uint32_t *adj, uint32_t v, uint32_t (&r)[NW])
{
    if constexpr (Rows<NW>::kSwz) {
        const uint32_t sw = v & 7u;
#pragma unroll
        for (int c = 0; c < NW / 4; ++c) {
            const uint4 q = *reinterpret_cast<const uint4 *>(adj + v * Rows<NW>::kStride + 4u * ((uint32_t)c ^ sw));
            r[4 * c] = q.x; r[4 * c + 1] = q.y; r[4 * c + 2] = q.z; r[4 * c + 3] = q.w;
        }
    } else {
        load_row<NW>(adj + v * Rows<NW>::kStride, r, NW);
    }
}

// All NW words of L into registers.
template <int NW>
__device__ __forceinline__ void load_L(const DSU<NW> &s, uint32_t (&L)[NW])
{
    load_row<NW>(s.lsm(), L, NW);
}

// The live bits of this lane's degree words (from the mirror of L).
template <int NW>
__device__ __forceinline__ void live_nibbles(DSU<NW> &s)
{
    const unsigned lane = lane_id();
#pragma unroll
    for (int j = 0; j < Rows<NW>::kJ; ++j) {
        const uint32_t q = 32u * j + lane;
        if constexpr (Rows<NW>::kHalf)
            s.Ln[j] = q < 16u * s.nw ? (s.lsm()[q >> 4] >> (2u * (lane & 15u))) & 0x3u : 0u;
        else
            s.Ln[j] = q < 8u * s.nw ? (s.lsm()[q >> 3] >> (4u * (lane & 7u))) & 0xFu : 0u;
    }
}

// Degrees from scratch into the staging array, then each lane picks up its
// words.  With 4-word row chunks (NW = 8, 16, 20, 32) only the live vertices
// are counted -- listed by a prefix sum over the words of L, then one per lane
// -- and only over the chunks of L that hold a live vertex; the staging array
// is zeroed first, so removed and padding vertices read 0.  Deep in a dense
// graph's tree most vertices are gone, and this is most of a node's work.
template <int NW>
__device__ __forceinline__ void dense_degrees(DSU<NW> &s)
{
    const unsigned lane = lane_id();
    uint32_t L[NW];
    load_L(s, L);
    if constexpr (NW % 4 == 0) {
        constexpr int C = NW / 4;
        uint32_t nzc = 0;  // chunks of L with a live vertex (the same in every lane)
#pragma unroll
        for (int c = 0; c < C; ++c) nzc |= (uint32_t)((L[4 * c] | L[4 * c + 1] | L[4 * c + 2] | L[4 * c + 3]) != 0u) << c;
        uint32_t *d32 = reinterpret_cast<uint32_t *>(s.degs());
        constexpr uint32_t kStageWords = 32u * NW / Rows<NW>::kPer;
        for (uint32_t i = lane; i < kStageWords; i += 32) d32[i] = 0u;
        const uint32_t x = lane < (uint32_t)NW ? s.lsm()[lane] : 0u;
        const uint32_t cnt = __popc(x);
        uint32_t off = cnt;  // inclusive prefix over the words of L
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, off, d);
            if (lane >= (unsigned)d) off += t;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, off, 31);
        uint16_t *list = s.cand();  // free while the degrees are recounted
        uint32_t pos = off - cnt, m = x;
        while (m) {
            list[pos++] = (uint16_t)(32u * lane + (__ffs(m) - 1));
            m &= m - 1;
        }
        __syncwarp();
        for (uint32_t i = lane; i < total; i += 32) {
            const uint32_t v = list[i];
            const uint4 *row = reinterpret_cast<const uint4 *>(s.adj + v * Rows<NW>::kStride);
            const uint32_t sw = Rows<NW>::kSwz ? (v & 7u) : 0u;
            uint32_t c = 0;
#pragma unroll
            for (int k = 0; k < C; ++k) {
                if ((nzc >> k) & 1u) {
                    const uint4 r = row[(uint32_t)k ^ sw];
                    c += __popc(r.x & L[4 * k]) + __popc(r.y & L[4 * k + 1]) + __popc(r.z & L[4 * k + 2]) +
                         __popc(r.w & L[4 * k + 3]);
                }
            }
            if constexpr (Rows<NW>::kHalf) s.degs16()[v] = (uint16_t)c;
            else s.degs()[v] = (uint8_t)c;
        }
    } else {  // 2- and 4-word graphs: one vertex per lane
        const int kmax = (int)s.nw;
#pragma unroll 1
        for (int k = 0; k < kmax; ++k) {
            const uint32_t v = lane + 32u * k;
            uint32_t c = 0;
            if (v < s.n && ((s.lsm()[k] >> lane) & 1u)) {
                uint32_t r[NW];
                load_row<NW>(s.adj + v * Rows<NW>::kStride, r, NW);
#pragma unroll
                for (int w = 0; w < NW; ++w) c += __popc(r[w] & L[w]);
            }
            s.degs()[v] = (uint8_t)c;
        }
    }
    __syncwarp();
    const uint32_t *d32 = reinterpret_cast<const uint32_t *>(s.degs());
    constexpr uint32_t kWordsPerLsm = 32u / Rows<NW>::kPer;  // degree words per word of L
#pragma unroll
    for (int j = 0; j < Rows<NW>::kJ; ++j) {
        const uint32_t q = 32u * j + lane;
        s.D[j] = q < kWordsPerLsm * s.nw ? d32[q] : 0u;
    }
    live_nibbles(s);
}

// Log the vertices of the set in s.marks() on the trail (ascending) and drop
// them from L; lane w handles word w.
template <int NW>
__device__ __forceinline__ void dense_push(DSU<NW> &s)
{
    const unsigned lane = lane_id();
    const uint32_t mw = lane < NW ? s.marks()[lane] : 0u;
    const uint32_t c = __popc(mw);
    uint32_t off = c;  // inclusive prefix over the words
#pragma unroll
    for (int d = 1; d < NW; d <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, off, d);
        if (lane >= (unsigned)d) off += t;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, off, NW - 1);
    uint32_t pos = s.top + off - c, m = mw;
    while (m) {
        s.trail()[pos++] = (uint16_t)(32u * lane + (__ffs(m) - 1));
        m &= m - 1;
    }
    if (lane < NW) s.lsm()[lane] &= ~mw;
    s.top += total;
    __syncwarp();
}

// Put the trail above `pos` back into L.
template <int NW>
__device__ __forceinline__ void dense_restore(DSU<NW> &s, uint32_t pos)
{
    const unsigned lane = lane_id();
    if (lane < NW) s.bits()[lane] = 0;
    __syncwarp();
    for (uint32_t i = pos + lane; i < s.top; i += 32) {
        uint32_t u = s.trail()[i];
        atomicOr(&s.bits()[u >> 5], 1u << (u & 31u));
    }
    __syncwarp();
    if (lane < NW) s.lsm()[lane] |= s.bits()[lane];
    s.stat.restored += s.top - pos;
    s.top = pos;
    __syncwarp();
}

// ---- the packing bound
// What a node still needs is bounded from below by vertex-disjoint cliques of its
// live graph, of which any cover takes all vertices but one.  They are picked
// greedily: a vertex of least degree among the unpicked, its neighbour of least
// degree, and common neighbours of all picked so far while there are any.
// The degrees among the unpicked are held bit-sliced, plane B[k] having bit k of
// each degree and lane w the 32 vertices of word w, so that a row is taken off
// all degrees by one borrow chain.  Graphs of up to 512 vertices fill half a warp
// at most, so a warp bounds two nodes in step, one per group of 16 lanes.
// A step is a chain of four ballots, two shuffles and two row loads, about a
// hundred instructions, and a bound takes some forty of them: it is what a node
// now spends most of its time on, bound by issue with the SM full and by that
// chain's latency without.  (Two picks per step, and all vertices of degree 1 at
// once, both made batches slower: 15.0 -> 16.8 and 15.3 -> 18.5 ms.)  It pays for
// itself many times over: 512 graphs of 30 to 160 vertices and average degree 3 to
// 12 in one batch take 1.6 M nodes and 15.3 ms instead of 161 M and 470 ms; one of
// 197 vertices and 648 edges 30 k and 0.88 ms instead of 3.6 M and 22 ms.  When the
// bound went in, bit-slicing the degrees rather than holding them in bytes (four to
// a word, a word per lane) took the 512 graphs from 66 to 49 ms, and bounding both
// children of a node instead of each node as it is reached to 32; the rest came with
// the launch shapes and the hand-over of work.
constexpr int kPackPlanes = 5;  // degrees below 32
constexpr uint32_t kPackNow = 1u << 31;  // beside InstState's flags in a unit's copy: the bound's time has come

template <int NW>
struct PackGroup {
    static constexpr uint32_t kLanes = NW <= 16 ? 16 : 32;
    static constexpr uint32_t kGroups = 32 / kLanes;
    // This group's bits of a ballot, and its share of a warp-wide sum (below 2^16 per group).
    static __device__ __forceinline__ uint32_t of(uint32_t bal)
    {
        return kGroups == 1 ? bal : (bal >> (lane_id() & 16u)) & 0xffffu;
    }
    static __device__ __forceinline__ uint32_t sum(uint32_t x)
    {
        if constexpr (kGroups == 1) return __reduce_add_sync(0xffffffffu, x);
        else return (__reduce_add_sync(0xffffffffu, x << (lane_id() & 16u)) >> (lane_id() & 16u)) & 0xffffu;
    }
};

// The lowest vertex of the sets e (a word per lane, at least one bit in this
// lane's group unless the group is done): adds it to `picked` and returns its
// row's word among the live.
template <int NW>
__device__ __forceinline__ uint32_t pack_pick(const uint32_t *adj, uint32_t e, uint32_t bal, uint32_t word, uint32_t live,
                                              uint32_t &picked)
{
    using PG = PackGroup<NW>;
    // the lowest vertex of each word, found while the ballot is under way
    const uint32_t bit = e & (0u - e), low = 32u * word + (31u - __clz(bit | 1u));
    const uint32_t src = bal ? __ffs(bal) - 1 : 0u;  // the word it is in
    if (word == src) picked |= bit;
    const uint32_t v = __shfl_sync(0xffffffffu, low, PG::kGroups == 1 ? src : src + (lane_id() & 16u));
    return adj[Rows<NW>::at(v, word < (uint32_t)NW ? word : 0u)] & live;
}

// Takes the rows of the set bits `br` off the degrees.
__device__ __forceinline__ void pack_subtract(uint32_t (&B)[kPackPlanes], uint32_t br)
{
#pragma unroll
    for (int k = 0; k < kPackPlanes; ++k) {
        const uint32_t t = B[k];
        B[k] = t ^ br;
        br &= ~t;
    }
}

// True for the lanes of a group whose graph (planes B, this lane's word of its
// vertices) needs more than `b` vertices (b < 0: always).  Stops as soon as the
// packing says so, or as soon as that looks out of reach: a vertex of degree d is
// in a clique of at most d + 1 vertices and only one on a triangle of the staged
// graph in one of more than two, so what is left is taken to be worth half a
// vertex to each, two thirds if it is in tri, and then five sixths from degree 3
// and one from degree 6.
template <int NW>
__device__ __forceinline__ bool packing_exceeds(const uint32_t *adj, uint32_t (&B)[kPackPlanes], int32_t b, uint32_t tri)
{
    using PG = PackGroup<NW>;
    constexpr int K = kPackPlanes;
    const uint32_t word = lane_id() & (PG::kLanes - 1u);
    const int32_t need = 6 * (b + 1);
    int32_t have = 0;
    bool over = b < 0, go = !over;
    uint32_t live = B[0] | B[1] | B[2] | B[3] | B[4];  // unpicked with an unpicked neighbour
    for (int it = 0; it < 16 * NW; ++it) {  // a group's step picks two vertices at least
        uint32_t bal4 = PG::of(__ballot_sync(0xffffffffu, live != 0u));
        go = go && bal4 != 0u;
        if ((it & 3) == 0) {
            const uint32_t t = live & tri, three = B[2] | B[3] | B[4] | (B[1] & B[0]), six = B[3] | B[4] | (B[2] & B[1]);
            const int32_t left =
                (int32_t)PG::sum(3u * __popc(live) + __popc(t) + __popc(t & three) + __popc(t & six));
            go = go && have + left >= need;
        }
        if (!__any_sync(0xffffffffu, go)) break;
        // degrees 1, 2, 3 and the rest
        const uint32_t hi = B[2] | B[3] | B[4];
        const uint32_t c1 = B[0] & ~(B[1] | hi), c2 = B[1] & ~(B[0] | hi), c3 = B[0] & B[1] & ~hi;
        const uint32_t bal1 = PG::of(__ballot_sync(0xffffffffu, c1 != 0u));
        uint32_t bal2 = PG::of(__ballot_sync(0xffffffffu, c2 != 0u));
        uint32_t bal3 = PG::of(__ballot_sync(0xffffffffu, c3 != 0u));
        uint32_t picked = 0u;
        const uint32_t nu = pack_pick<NW>(adj, bal1 ? c1 : (bal2 ? c2 : (bal3 ? c3 : live)),
                                          bal1 ? bal1 : (bal2 ? bal2 : (bal3 ? bal3 : bal4)), word, live, picked);
        // its neighbour of the lowest class
        bal2 = PG::of(__ballot_sync(0xffffffffu, (nu & c2) != 0u));
        bal3 = PG::of(__ballot_sync(0xffffffffu, (nu & c3) != 0u));
        bal4 = PG::of(__ballot_sync(0xffffffffu, nu != 0u));
        const uint32_t np = pack_pick<NW>(adj, nu & (bal2 ? c2 : (bal3 ? c3 : ~0u)), bal2 ? bal2 : (bal3 ? bal3 : bal4), word,
                                          live, picked);
        have += 6;
        // common neighbours, as long as there are any
        const uint32_t unpicked = live;
        uint32_t common = nu & np;
        for (int more = 0; more < 32; ++more) {
            const uint32_t any = __ballot_sync(0xffffffffu, common != 0u);
            if (!any) break;
            const uint32_t bal = PG::of(any);
            const uint32_t row = pack_pick<NW>(adj, common, bal, word, bal ? unpicked : 0u, picked);
            pack_subtract(B, row);
            common &= row;
            have += bal ? 6 : 0;
        }
        if (go && have >= need) { over = true; go = false; }
        // the degrees less the first two rows (their sum in two bits, then a borrow chain)
        const uint32_t s0 = nu ^ np, s1 = nu & np;
        uint32_t br = ~B[0] & s0;
        B[0] = (B[0] ^ s0) & ~picked;
        const uint32_t b1 = B[1];
        B[1] = (b1 ^ s1 ^ br) & ~picked;
        br = (~b1 & (s1 | br)) | (s1 & br);
        live = B[0] | B[1];
#pragma unroll
        for (int k = 2; k < K; ++k) {
            const uint32_t bk = B[k];
            B[k] = (bk ^ br) & ~picked;
            br &= ~bk;
            live |= B[k];
        }
        if (!go) live = 0u;  // this group is done: its lanes only keep the other one company
    }
    return over;
}

// Which children of a settled node on vertex v the packing bound leaves open,
// when b more vertices may be taken: bit 0 "take v", bit 1 "take N(v)".  The
// children are bounded before their own reductions (picking vertices of degree 1
// first does for the bound what the leaf rule does for the node), so a child
// that is closed costs no settling, and a node with one open child is not a
// branch.  Needs degrees below 2^kPackPlanes.
template <int NW>
__device__ __forceinline__ uint32_t open_children(DSU<NW> &s, uint32_t v, uint32_t maxd, uint32_t b)
{
    using PG = PackGroup<NW>;
    constexpr int J = Rows<NW>::kJ;
    constexpr bool H = Rows<NW>::kHalf;
    constexpr int K = kPackPlanes;
    const unsigned lane = lane_id();
    const uint32_t word = lane & (PG::kLanes - 1u);
    uint32_t *d32 = reinterpret_cast<uint32_t *>(s.degs());
#pragma unroll
    for (int j = 0; j < J; ++j) {
        const uint32_t q = 32u * j + lane;
        if (q < (H ? 16u : 8u) * s.nw) d32[q] = s.D[j];
    }
    __syncwarp();
    uint32_t A[K];
#pragma unroll
    for (int k = 0; k < K; ++k) A[k] = 0u;
#pragma unroll 1
    for (uint32_t w = 0; w < s.nw; ++w) {
        const uint32_t d = H ? s.degs16()[32u * w + lane] : s.degs()[32u * w + lane];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const uint32_t x = __ballot_sync(0xffffffffu, (d >> k) & 1u);
            if (word == w) A[k] = x;
        }
    }
    const uint32_t live = A[0] | A[1] | A[2] | A[3] | A[4];
    const uint32_t at = word < (uint32_t)NW ? word : 0u;
    const uint32_t tri = word < (uint32_t)NW ? s.adj[Rows<NW>::kTri + at] : 0u;
    const uint32_t nv = s.adj[Rows<NW>::at(v, at)] & live;
    const uint32_t vbit = word == (v >> 5) ? 1u << (v & 31u) : 0u;
    uint32_t open = 0;
#pragma unroll 1
    for (uint32_t side = 0; side < 2; side += PG::kGroups) {
        const bool right = PG::kGroups == 2 ? lane >= 16u : side != 0u;  // this group's child takes N(v)
        uint32_t B[K];
#pragma unroll
        for (int k = 0; k < K; ++k) B[k] = A[k];
        const uint32_t gone = right ? nv | vbit : vbit;
        if (PG::kGroups == 2 || !right) {  // v's row comes off in the left child
            pack_subtract(B, right ? 0u : nv);
        }
        if (PG::kGroups == 2 || right) {  // the rows of v's neighbours in the right child
            uint32_t wm = PG::of(__ballot_sync(0xffffffffu, nv != 0u));
            while (wm) {
                const uint32_t w = __ffs(wm) - 1;
                wm &= wm - 1;
                uint32_t m = __shfl_sync(0xffffffffu, nv, w);
                while (m) {
                    const uint32_t u = 32u * w + (__ffs(m) - 1);
                    m &= m - 1;
                    pack_subtract(B, right ? s.adj[Rows<NW>::at(u, at)] & live : 0u);
                }
            }
        }
#pragma unroll
        for (int k = 0; k < K; ++k) B[k] &= ~gone;
        const int32_t bc = (int32_t)b - (right ? (int32_t)maxd : 1);
        const uint32_t closed = __ballot_sync(0xffffffffu, packing_exceeds<NW>(s.adj, B, bc, tri));
        if constexpr (PG::kGroups == 2) open = ((closed & 1u) ^ 1u) | (((closed >> 16) & 1u) ^ 1u) << 1;
        else open |= ((closed & 1u) ^ 1u) << side;
    }
    return open;
}

// The set in s.marks() has just left L (trail, L and its mirror already
// updated): subtract its edges from the degrees of the live vertices and zero
// the bytes of the removed ones.
template <int NW>
__device__ __forceinline__ void dense_apply_half(DSU<NW> &s)
{
    constexpr int J = Rows<NW>::kJ;
    const unsigned lane = lane_id();
    live_nibbles(s);
    {
        // word 2j + lane/16 of a row holds the bits of this lane's vertices 2q, 2q+1
        const uint32_t sh = 2u * (lane & 15u);
        const uint32_t hl = lane >> 4;
        const uint32_t mw = lane < s.nw ? s.marks()[lane] : 0u;
        uint32_t wm = __ballot_sync(0xffffffffu, mw != 0u);
        uint32_t acc[J];
#pragma unroll
        for (int j = 0; j < J; ++j) acc[j] = 0u;
        while (wm) {
            const uint32_t w = __ffs(wm) - 1;
            wm &= wm - 1;
            uint32_t m = __shfl_sync(0xffffffffu, mw, w);
            while (m) {
                const uint32_t u = 32u * w + (__ffs(m) - 1);
                m &= m - 1;
#pragma unroll
                for (int j = 0; j < J; ++j) acc[j] += spread2((s.adj[Rows<NW>::at(u, 2u * j + hl)] >> sh) & s.Ln[j]);
            }
        }
#pragma unroll
        for (int j = 0; j < J; ++j) s.D[j] = (s.D[j] - acc[j]) & (spread2(s.Ln[j]) * 0xFFFFu);
    }
}

template <int NW>
__device__ __forceinline__ void dense_apply(DSU<NW> &s)
{
    if constexpr (Rows<NW>::kHalf) {
        dense_apply_half(s);
        return;
    } else {
    constexpr int J = Rows<NW>::kJ;
    const unsigned lane = lane_id();
    live_nibbles(s);
    const uint32_t sh = 4u * (lane & 7u);
    const uint32_t *rows = s.adj + (lane >> 3);  // word 4j + lane/8 of a row holds this lane's bits
    const uint32_t mw = lane < s.nw ? s.marks()[lane] : 0u;  // lane w holds word w of the set
    uint32_t wm = __ballot_sync(0xffffffffu, mw != 0u);
    uint32_t acc[J];  // per-byte decrements (at most the degree, so no byte overflows)
#pragma unroll
    for (int j = 0; j < J; ++j) acc[j] = 0u;
    while (wm) {
        const uint32_t w = __ffs(wm) - 1;
        wm &= wm - 1;
        uint32_t m = __shfl_sync(0xffffffffu, mw, w);
        while (m) {  // two removed vertices per step
            const uint32_t u1 = 32u * w + (__ffs(m) - 1);
            m &= m - 1;
            const uint32_t *r1 = rows + u1 * Rows<NW>::kStride;
            if (m) {
                const uint32_t u2 = 32u * w + (__ffs(m) - 1);
                m &= m - 1;
                const uint32_t *r2 = rows + u2 * Rows<NW>::kStride;
#pragma unroll
                for (int j = 0; j < J; ++j)
                    acc[j] += spread4((r1[4 * j] >> sh) & s.Ln[j]) + spread4((r2[4 * j] >> sh) & s.Ln[j]);
            } else {
#pragma unroll
                for (int j = 0; j < J; ++j) acc[j] += spread4((r1[4 * j] >> sh) & s.Ln[j]);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < J; ++j) s.D[j] = (s.D[j] - acc[j]) & (spread4(s.Ln[j]) * 0xFFu);
    }
}

// One reduction pass (same rules and semantics as reduce_pass in vc_search.cuh)
// on current degrees.  Byte tests over each lane's degree words find the
// high-degree vertices (marked at once) and the degree-1 ones and degree-2 ones
// on a triangle of the graph, which are gathered into a list and worked one
// vertex per lane.  Returns true if marks
// were made (left in s.marks()); otherwise fills o with the degree sum, the
// maximum degree and its lowest vertex.
template <int NW>
__device__ __forceinline__ bool dense_pass_byte(DSU<NW> &s, uint32_t del, uint32_t bound, ScanOut &o)
{
    constexpr int J = Rows<NW>::kJ;
    const unsigned lane = lane_id();
    const uint32_t sh = 4u * (lane & 7u);
    const int tt = (int)bound - (int)del;  // the high-degree rule takes deg >= tt
    const uint32_t tl = (uint32_t)(tt & 0x7F) * 0x01010101u;
    const uint32_t *tri = s.adj + Rows<NW>::kTri;
    bool marked = false;
    uint32_t cn[J], ctot = 0;
#pragma unroll
    for (int j = 0; j < J; ++j) {
        const uint32_t d = s.D[j];
        const uint32_t nz = ~bytes_zero(d) & 0x80808080u;
        const uint32_t lo = ((d | 0x80808080u) - tl) & 0x80808080u;  // low 7 bits >= tt's
        const uint32_t mid = tt < 128 ? ((d & 0x80808080u) | lo) : (d & lo);
        const uint32_t ge = tt <= 1 ? nz : (tt > 255 ? 0u : mid);
        // degree 1, or degree 2 on a triangle of the graph
        const uint32_t tn = (tri[(32u * j + lane) >> 3] >> sh) & 0xFu;
        const uint32_t d12 = bytes_zero(d ^ 0x01010101u) | (bytes_zero(d ^ 0x02020202u) & (spread4(tn) << 7));
        const uint32_t hn = gather4(ge);
        if (hn) {
            atomicOr(&s.marks()[(32u * j + lane) >> 3], hn << sh);
            marked = true;
        }
        cn[j] = gather4(d12 & ~ge);
        ctot += __popc(cn[j]);
    }
    // compact the degree-1/2 candidates (at most 4J per lane) into s.cand()
    // (one vote first: many passes have none)
    const uint32_t lt = (1u << lane) - 1u;
    uint32_t pre = 0, total = 0;
    if (__any_sync(0xffffffffu, ctot != 0u)) {
#pragma unroll
        for (int b = 0; b < Rows<NW>::kCandBits; ++b) {
            const uint32_t bal = __ballot_sync(0xffffffffu, (ctot >> b) & 1u);
            pre += __popc(bal & lt) << b;
            total += __popc(bal) << b;
        }
    }
    if (total) {
        uint32_t *d32 = reinterpret_cast<uint32_t *>(s.degs());
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const uint32_t q = 32u * j + lane;
            if (q < 8u * s.nw) d32[q] = s.D[j];
            uint32_t m = cn[j];
            while (m) {
                const uint32_t b = __ffs(m) - 1;
                m &= m - 1;
                s.cand()[pre++] = (uint16_t)(4u * q + b);
            }
        }
        uint32_t L[NW];
        load_L(s, L);
        __syncwarp();
        for (uint32_t i = lane; i < total; i += 32) {  // degree-one / degree-two triangle rules
            const uint32_t v = s.cand()[i];
            const uint32_t dv = s.degs()[v];
            uint32_t r[NW];
            load_row<NW>(s.adj + v * Rows<NW>::kStride, r, NW);
            // v has exactly dv (1 or 2) live neighbours: the lowest and the
            // highest set bit of row & L
            uint32_t n1 = kNone, hi = kNone;
#pragma unroll
            for (int w = NW - 1; w >= 0; --w) {
                const uint32_t x = r[w] & L[w];
                n1 = x ? 32u * w + (__ffs(x) - 1) : n1;
            }
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                const uint32_t x = r[w] & L[w];
                hi = x ? 32u * w + (31u - __clz(x)) : hi;
            }
            const uint32_t n2 = dv == 2 ? hi : kNone;
            if (dv == 1) {
                const uint32_t du = s.degs()[n1];
                if (du > 1 || n1 < v) {
                    atomicOr(&s.marks()[n1 >> 5], 1u << (n1 & 31u));
                    marked = true;
                }
            } else if (n2 != kNone) {
                const uint32_t d1 = s.degs()[n1], d2 = s.degs()[n2];
                const bool keep = d1 == 1 || d2 == 1 || (d1 == 2 && n1 < v) || (d2 == 2 && n2 < v);
                if (!keep && ((s.adj[n2 * Rows<NW>::kStride + (n1 >> 5)] >> (n1 & 31u)) & 1u)) {
                    atomicOr(&s.marks()[n1 >> 5], 1u << (n1 & 31u));
                    atomicOr(&s.marks()[n2 >> 5], 1u << (n2 & 31u));
                    marked = true;
                }
            }
        }
    }
    s.stat.passes += 1;
    if (__any_sync(0xffffffffu, marked)) {
        __syncwarp();
        return true;
    }
    uint32_t acc = 0, mx = 0;
#pragma unroll
    for (int j = 0; j < J; ++j) {
        const uint32_t d = s.D[j];
        acc += (d & 0x00FF00FFu) + ((d >> 8) & 0x00FF00FFu);
        mx = max(mx, max(max(d & 0xFFu, (d >> 8) & 0xFFu), max((d >> 16) & 0xFFu, d >> 24)));
    }
    o.sum = __reduce_add_sync(0xffffffffu, (acc & 0xFFFFu) + (acc >> 16));
    o.maxd = __reduce_max_sync(0xffffffffu, mx);
    uint32_t first = kNone;
    if (o.maxd > 0) {
#pragma unroll
        for (int j = J - 1; j >= 0; --j) {
            const uint32_t e = bytes_zero(s.D[j] ^ (o.maxd * 0x01010101u));
            if (e) first = 4u * (32u * j + lane) + ((__ffs(e) >> 3) - 1);
        }
    }
    o.amax = __reduce_min_sync(0xffffffffu, first);
    return false;
}

// dense_pass on 16-bit degrees (Half): the same rules and results.
template <int NW>
__device__ __forceinline__ bool dense_pass_half(DSU<NW> &s, uint32_t del, uint32_t bound, ScanOut &o)
{
    constexpr int J = Rows<NW>::kJ;
    const unsigned lane = lane_id();
    const uint32_t sh = 2u * (lane & 15u);  // this lane's 2 bits in words of L, marks and tri
    const int tt = (int)bound - (int)del;  // the high-degree rule takes deg >= tt
    const uint32_t tl = (uint32_t)(tt > 0 ? min(tt, 0x7FFF) : 0) * 0x00010001u;
    const uint32_t *tri = s.adj + Rows<NW>::kTri;
    bool marked = false;
    uint32_t cn[J], ctot = 0;
#pragma unroll
    for (int j = 0; j < J; ++j) {
        const uint32_t d = s.D[j];
        const uint32_t q = 32u * j + lane;  // vertices 2q, 2q + 1
        const uint32_t nz = ~halves_zero(d) & 0x80008000u;
        // degrees are below 2^15, so 0x8000 + d - tt keeps its top bit iff d >= tt
        const uint32_t ge = tt <= 1 ? nz : (tt >= 0x7FFF ? 0u : ((d | 0x80008000u) - tl) & 0x80008000u);
        const uint32_t tn = (tri[q >> 4] >> sh) & 0x3u;
        const uint32_t d12 = halves_zero(d ^ 0x00010001u) | (halves_zero(d ^ 0x00020002u) & (spread2(tn) << 15));
        const uint32_t hn = gather2(ge);
        if (hn) {
            atomicOr(&s.marks()[q >> 4], hn << sh);
            marked = true;
        }
        cn[j] = gather2(d12 & ~ge);
        ctot += __popc(cn[j]);
    }
    const uint32_t lt = (1u << lane) - 1u;
    uint32_t pre = 0, total = 0;
    if (__any_sync(0xffffffffu, ctot != 0u)) {
#pragma unroll
        for (int b = 0; b < Rows<NW>::kCandBits; ++b) {
            const uint32_t bal = __ballot_sync(0xffffffffu, (ctot >> b) & 1u);
            pre += __popc(bal & lt) << b;
            total += __popc(bal) << b;
        }
    }
    if (total) {
        uint32_t *d32 = reinterpret_cast<uint32_t *>(s.degs16());
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const uint32_t q = 32u * j + lane;
            if (q < 16u * s.nw) d32[q] = s.D[j];
            uint32_t m = cn[j];
            while (m) {
                const uint32_t b = __ffs(m) - 1;
                m &= m - 1;
                s.cand()[pre++] = (uint16_t)(2u * q + b);
            }
        }
        uint32_t L[NW];
        load_L(s, L);
        __syncwarp();
        for (uint32_t i = lane; i < total; i += 32) {  // degree-one / degree-two triangle rules
            const uint32_t v = s.cand()[i];
            const uint32_t dv = s.degs16()[v];
            uint32_t r[NW];
            load_row_at<NW>(s.adj, v, r);
            uint32_t n1 = kNone, hi = kNone;  // lowest and highest live neighbour
#pragma unroll
            for (int w = NW - 1; w >= 0; --w) {
                const uint32_t x = r[w] & L[w];
                n1 = x ? 32u * w + (__ffs(x) - 1) : n1;
            }
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                const uint32_t x = r[w] & L[w];
                hi = x ? 32u * w + (31u - __clz(x)) : hi;
            }
            const uint32_t n2 = dv == 2 ? hi : kNone;
            if (dv == 1) {
                const uint32_t du = s.degs16()[n1];
                if (du > 1 || n1 < v) {
                    atomicOr(&s.marks()[n1 >> 5], 1u << (n1 & 31u));
                    marked = true;
                }
            } else if (n2 != kNone) {
                const uint32_t d1 = s.degs16()[n1], d2 = s.degs16()[n2];
                const bool keep = d1 == 1 || d2 == 1 || (d1 == 2 && n1 < v) || (d2 == 2 && n2 < v);
                if (!keep && ((s.adj[Rows<NW>::at(n2, n1 >> 5)] >> (n1 & 31u)) & 1u)) {
                    atomicOr(&s.marks()[n1 >> 5], 1u << (n1 & 31u));
                    atomicOr(&s.marks()[n2 >> 5], 1u << (n2 & 31u));
                    marked = true;
                }
            }
        }
    }
    s.stat.passes += 1;
    if (__any_sync(0xffffffffu, marked)) {
        __syncwarp();
        return true;
    }
    uint32_t acc = 0, mx = 0;
#pragma unroll
    for (int j = 0; j < J; ++j) {
        const uint32_t d = s.D[j];
        acc += (d & 0xFFFFu) + (d >> 16);
        mx = max(mx, max(d & 0xFFFFu, d >> 16));
    }
    o.sum = __reduce_add_sync(0xffffffffu, acc);
    o.maxd = __reduce_max_sync(0xffffffffu, mx);
    uint32_t first = kNone;
    if (o.maxd > 0) {
#pragma unroll
        for (int j = J - 1; j >= 0; --j) {
            const uint32_t e = halves_zero(s.D[j] ^ (o.maxd * 0x00010001u));
            if (e) first = 2u * (32u * j + lane) + ((__ffs(e) >> 4) - 1);
        }
    }
    o.amax = __reduce_min_sync(0xffffffffu, first);
    return false;
}

template <int NW>
__device__ __forceinline__ bool dense_pass(DSU<NW> &s, uint32_t del, uint32_t bound, ScanOut &o)
{
    if constexpr (Rows<NW>::kHalf) return dense_pass_half(s, del, bound, o);
    else return dense_pass_byte(s, del, bound, o);
}

// A node's settling: the pending set in s.marks() leaves L and the degrees are
// brought up to date (subtracted, or recounted after a backtrack or a new
// record), then reduction passes run to a fixpoint, each pass's marks taking the
// same path.  One copy of the push / update code serves every caller.
template <int NW>
__device__ __forceinline__ void dense_settle(DSU<NW> &s, uint32_t bound, ScanOut &o)
{
    const unsigned lane = lane_id();
    uint32_t how = s.pending;
    s.pending = 0;
#pragma unroll 1
    for (int pass = 0; pass < 4 * 32 * NW; ++pass) {
        if (how) {
            const long long t0 = (kPhaseTimers && s.timed) ? clock64() : 0;
            dense_push(s);
            if (how == kPendRecount) dense_degrees(s);
            else dense_apply(s);
            __syncwarp();
            if (lane < NW) s.marks()[lane] = 0;
            __syncwarp();
            if (kPhaseTimers && s.timed) s.cyc.apply += (unsigned long long)(clock64() - t0);
        }
        if (!dense_pass(s, s.base_del + s.top, bound, o)) break;
        how = kPendApply;
    }
}

// ---- the overloads the shared work-sharing code (vc_search.cuh) calls
template <class G, int NW>
__device__ __forceinline__ void bind_graph(DSU<NW> &s, const Params &P, uint32_t inst)
{
    const InstDesc d = load_desc(&P.inst[inst]);
    s.inst = inst;
    s.n = d.n;
    s.nw = d.nw;
    s.mode = d.mode;
    s.k = d.k;
    s.cover_off = d.cover_off;
    s.node_limit = d.node_limit;
    s.rp = P.row_ptr + d.row_off;
    s.cl = P.col + d.col_off;
    s.fr_bot = s.fr_top = 0;
    s.local_nodes = 0;
}

template <class G, int NW>
__device__ __forceinline__ void load_root(DSU<NW> &s)
{
    const unsigned w = lane_id();
    if (w < NW) {
        const uint32_t lo = 32u * w;
        s.lsm()[w] = lo + 32u <= s.n ? 0xffffffffu : (lo < s.n ? (1u << (s.n - lo)) - 1u : 0u);
        s.marks()[w] = 0;
    }
    s.top = 0;
    s.base_del = 0;
    __syncwarp();
    s.pending = kPendRecount;  // the node's settling counts the degrees
}

// Root `v` of a split graph: the vertices of larger degree (then of lower index) are
// in the cover and v is not, so its neighbours are too.  The n roots part the covers
// by their first vertex in that order that stays out.  From the single root of a
// dense graph the search goes down a spine of nearly n nodes, "take v" each, before
// its first leaf, one after another (300 vertices of density 0.75: 279 nodes and
// most of the solve's 1.7 ms); the children that it would leave behind are these
// roots, and all CTAs take them up at once.
template <int NW>
__device__ __forceinline__ void load_split_root(DSU<NW> &s, uint32_t v)
{
    const unsigned lane = lane_id();
    auto degree = [&](uint32_t u) {
        uint32_t r[NW], d = 0;
        load_row_at<NW>(s.adj, u, r);
#pragma unroll
        for (int i = 0; i < NW; ++i) d += __popc(r[i]);
        return d;
    };
    const uint32_t dv = degree(v);
    uint32_t keep = 0;
    for (uint32_t w = 0; w < s.nw; ++w) {
        const uint32_t u = 32u * w + lane;
        bool in = false;
        if (u < s.n) {
            const uint32_t du = degree(u);
            in = du < dv || (du == dv && u >= v);
        }
        const uint32_t x = __ballot_sync(0xffffffffu, in);
        if (lane == w) keep = x;
    }
    if (lane < (uint32_t)NW) {
        keep &= ~s.adj[Rows<NW>::at(v, lane)];
        s.lsm()[lane] = keep;
        s.marks()[lane] = 0;
    }
    const uint32_t live = __reduce_add_sync(0xffffffffu, __popc(keep));
    s.top = 0;
    s.base_del = s.n - live;
    __syncwarp();
    s.pending = kPendRecount;
}

// From a received live bitmap in s.bits().
template <class G, int NW>
__device__ __forceinline__ void rebuild(DSU<NW> &s)
{
    const unsigned w = lane_id();
    const uint32_t x = w < s.nw ? s.bits()[w] : 0u;
    if (w < NW) {
        s.lsm()[w] = x;
        s.marks()[w] = 0;
    }
    const uint32_t live = __reduce_add_sync(0xffffffffu, __popc(x));
    s.top = 0;
    s.base_del = s.n - live;
    __syncwarp();
    s.pending = kPendRecount;  // the node's settling counts the degrees
}

// The bottom frame's pending child as a live bitmap in s.bits(): L at that frame
// (L now plus the trail above the frame) minus N(v).
template <class G, int NW>
__device__ __forceinline__ void donation_bits(DSU<NW> &s)
{
    const unsigned lane = lane_id();
    const uint32_t f = s.frames()[s.fr_bot];
    const uint32_t pos = f >> 16, v = f & 0xffffu;
    if (lane < NW) s.bits()[lane] = s.lsm()[lane];
    __syncwarp();
    for (uint32_t i = pos + lane; i < s.top; i += 32) {
        uint32_t u = s.trail()[i];
        atomicOr(&s.bits()[u >> 5], 1u << (u & 31u));
    }
    __syncwarp();
    if (lane < NW) s.bits()[lane] &= ~s.adj[Rows<NW>::at(v, lane)];
    __syncwarp();
}

template <class G, int NW>
__device__ __forceinline__ void cover_bits(DSU<NW> &s, uint32_t *dst)
{
    const unsigned lane = lane_id();
    if (lane < s.nw) {
        const uint32_t lo = 32u * lane;
        const uint32_t valid = lo + 32u <= s.n ? 0xffffffffu : (1u << (s.n - lo)) - 1u;
        dst[lane] = ~s.lsm()[lane] & valid;
    }
}

// One warp makes row v of a graph's bitmap adjacency in `row` (NW words of its
// own shared memory) and writes it to `out` as stage_graph copies it: kStride
// words, chunks swizzled where the kernel's rows are.  The row's own bit, always
// clear in a graph without self loops, carries whether v lies on a triangle.
// Entries that break the CSR layout (a row past row_ptr[n], an id out of range, a
// self loop) are skipped, so no read or write leaves its array; device-resident
// input is also checked by k_check_csr, which drops a graph it flags.
constexpr uint32_t kPrepareLong = 32;  // entries of a neighbour's row that one lane walks
template <int NW>
__device__ __forceinline__ void prepare_row(const uint32_t *rp, const uint32_t *cl, uint32_t n, uint32_t m2, uint32_t v,
                                            uint32_t *row, uint32_t *out)
{
    const unsigned lane = lane_id();
    for (uint32_t w = lane; w < (uint32_t)NW; w += 32) row[w] = 0u;
    __syncwarp();
    const uint32_t e0 = rp[v], e1 = min(rp[v + 1], m2);
    for (uint32_t e = e0 + lane; e < e1; e += 32) {
        const uint32_t u = cl[e];
        if (u < n && u != v) atomicOr(&row[u >> 5], 1u << (u & 31u));
    }
    __syncwarp();
    // A neighbour of a neighbour that is a neighbour: a lane per neighbour, until one of
    // them finds it, and the warp for a neighbour whose row is long -- a lane alone took
    // 0.5 us an entry, and so did every leaf of a star along the hub's row (1000 vertices:
    // this kernel 537 us, now 25).  A vertex of degree 1 is on no triangle.
    bool tri = false;
    auto closes = [&](uint32_t x, uint32_t u) { return x < n && x != u && ((row[x >> 5] >> (x & 31u)) & 1u); };
    for (uint32_t eb = e0; e1 - e0 > 1u && eb < e1 && !tri; eb += 32) {
        const uint32_t u = eb + lane < e1 ? cl[eb + lane] : n;
        uint32_t f = u < n && u != v ? rp[u] : 1u;
        uint32_t f1 = u < n && u != v ? min(rp[u + 1], m2) : 0u;
        uint32_t todo = __ballot_sync(0xffffffffu, f < f1 && f1 - f > kPrepareLong);
        const uint32_t g0 = f, g1 = f1;
        if ((todo >> lane) & 1u) f = f1;
        while (__any_sync(0xffffffffu, f < f1)) {
            if (f < f1) tri = closes(cl[f++], u);
            tri = __any_sync(0xffffffffu, tri);
            if (tri) break;
        }
        while (todo && !tri) {
            const uint32_t src = __ffs(todo) - 1;
            todo &= todo - 1;
            const uint32_t w = __shfl_sync(0xffffffffu, u, src), h1 = __shfl_sync(0xffffffffu, g1, src);
            for (uint32_t h = __shfl_sync(0xffffffffu, g0, src); h < h1 && !tri; h += 128) {
                uint32_t x[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) x[k] = h + 32u * k + lane < h1 ? cl[h + 32u * k + lane] : n;
#pragma unroll
                for (int k = 0; k < 4; ++k) tri = tri || closes(x[k], w);
                tri = __any_sync(0xffffffffu, tri);
            }
        }
    }
    if (lane == 0 && tri) row[v >> 5] |= 1u << (v & 31u);
    __syncwarp();
    for (uint32_t w = lane; w < (uint32_t)Rows<NW>::kStride; w += 32)
        out[Rows<NW>::at(v, w)] = w < (uint32_t)NW ? row[w] : 0u;
    __syncwarp();
}

// Stage a graph's adjacency into the CTA's bitmaps (one warp; the CTA has no
// other active warp when this runs).  Not inlined: it is called from two rare
// places of the search loop, which has no registers to spare for it.
// From the rows k_prepare made: four 16-byte loads in flight per lane.
template <int NW>
__device__ __noinline__ void stage_rows(uint32_t *adj, const uint32_t *rows, uint32_t n)
{
    const unsigned lane = lane_id();
    const uint4 *src = reinterpret_cast<const uint4 *>(rows);
    uint4 *dst = reinterpret_cast<uint4 *>(adj);
    const uint32_t total = (n * Rows<NW>::kStride + 3u) / 4u;
    for (uint32_t i = lane; i < total; i += 128u) {
        uint4 q[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (i + 32u * k < total) q[k] = __ldcg(&src[i + 32u * k]);
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (i + 32u * k < total) dst[i + 32u * k] = q[k];
    }
    __syncwarp();
    for (uint32_t w = 0; w < (uint32_t)NW; ++w) {  // the rows' own bits are the tri bitmap
        const uint32_t v = 32u * w + lane;
        uint32_t own = 0u;
        if (v < n) {
            uint32_t *x = &adj[Rows<NW>::at(v, w)];
            own = (*x >> lane) & 1u;
            *x &= ~(1u << lane);
        }
        const uint32_t t = __ballot_sync(0xffffffffu, own != 0u);
        if (lane == 0) adj[Rows<NW>::kTri + w] = t;
    }
    __threadfence_block();
    __syncwarp();
}

// From the CSR, where no rows were made (servers, the allocation-free entry
// point, batches above the bound on their memory).  Eight loads of a row are in
// flight, and the bitmaps are known to be shared memory: without either, each entry's
// load waited for the store before it (through a generic pointer it may be the same
// word), and a complete graph of 255 vertices took the allocation-free call 0.60 ms,
// against 0.34 with both.
template <int NW>
__device__ __noinline__ void stage_csr(uint32_t *adj, const uint32_t *rp, const uint32_t *cl, uint32_t n, uint32_t m2)
{
    __builtin_assume(__isShared(adj));
    const unsigned lane = lane_id();
    for (uint32_t i = lane; i < Rows<NW>::kTri + (uint32_t)NW; i += 32) adj[i] = 0;
    __syncwarp();
    // Entries that break the CSR layout (a row past row_ptr[n], an id out of
    // range, a self loop) are skipped, so no read or write leaves its array;
    // device-resident input is checked by k_check_csr before the search, which
    // drops a graph it flags.
    for (uint32_t v = lane; v < n; v += 32) {  // row v belongs to lane v % 32
        const uint32_t e1 = min(__ldcg(&rp[v + 1]), m2);
        for (uint32_t e = __ldcg(&rp[v]); e < e1; e += 8) {
            uint32_t u[8];  // loads in flight
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k) u[k] = k < e1 - e ? __ldcg(&cl[e + k]) : n;
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k)
                if (u[k] < n && u[k] != v) adj[Rows<NW>::at(v, u[k] >> 5)] |= 1u << (u[k] & 31u);
        }
    }
    __syncwarp();
    // tri: v has a neighbour u with a common neighbour.  Only such a vertex can
    // ever meet the triangle rule (its two live neighbours adjacent), so the
    // passes look at degree-2 vertices in tri only.
    for (uint32_t v = lane; v < n; v += 32) {
        uint32_t r[NW];
        load_row_at<NW>(adj, v, r);
        bool t = false;
#pragma unroll 1
        for (uint32_t w = 0; w < (uint32_t)NW && !t; ++w) {
            uint32_t x = adj[Rows<NW>::at(v, w)];
            while (x && !t) {
                const uint32_t u = 32u * w + (__ffs(x) - 1);
                x &= x - 1;
                uint32_t c = 0;
#pragma unroll
                for (int k = 0; k < NW; ++k) c |= adj[Rows<NW>::at(u, k)] & r[k];
                t = c != 0u;
            }
        }
        if (t) atomicOr(&adj[Rows<NW>::kTri + (v >> 5)], 1u << (v & 31u));
    }
    __threadfence_block();
    __syncwarp();
}

template <int NW>
__device__ __forceinline__ void stage_graph(uint32_t *adj, const Params &P, uint32_t inst)
{
    const InstDesc *d = &P.inst[inst];
    const uint32_t n = __ldcg(&d->n);
    if (P.adj) {
        stage_rows<NW>(adj, P.adj + __ldcg(&d->adj_off), n);
    } else {
        const uint32_t *rp = P.row_ptr + __ldcg(&d->row_off);
        const uint32_t stated = __ldcg(&d->m2), m2 = __ldcg(&rp[n]);
        stage_csr<NW>(adj, rp, P.col + __ldcg(&d->col_off), n, stated != kNone ? min(m2, stated) : m2);
    }
}

// ---- first covers
// A plain solve of a graph of 16 words or more whose average degree is at most 16
// starts with dives on the first blocks after the one that takes up the search: two
// graphs of 700 and 913 vertices and average degree 3.2 went from 1.9 to 1.0 ms, four
// of 327..584 vertices from 4.6 to 3.5.  Dense graphs gain nothing; and with smaller
// ones the nodes fall as much (175 vertices: 6,700 to 530) but not the time (0.39 to
// 0.59 ms): against a tight incumbent a node's bound runs its full course, and the
// chain of nodes to the first leaf is what such a tree's time is.
constexpr uint32_t kDiveBlocks = 37;
// One greedy dive: a vertex of least degree, at random among them, stays out of
// the cover and its neighbours go in, until no edge is left.  The cover is left in
// `cover` (NW words) and its size returned; a dive that reaches `limit` vertices
// gives up.  Search units that would wait for work make a dive each: on sparse random
// graphs the best of a hundred is usually a minimum cover, and a search that prunes
// against it from the start opens a third to a tenth of the nodes that it opens
// while its own first leaves come in.
template <int NW>
__device__ __noinline__ uint32_t dense_dive(const uint32_t *adj, uint32_t *cover, uint32_t n, uint32_t limit, uint32_t seed)
{
    constexpr int K = Rows<NW>::kHalf ? 10 : 8;  // planes: every degree of the kernel's graphs
    const unsigned lane = lane_id();
    const uint32_t at = lane < (uint32_t)NW ? lane : 0u;
    uint32_t B[K];
#pragma unroll
    for (int k = 0; k < K; ++k) B[k] = 0u;
    for (uint32_t w = 0; 32u * w < n; ++w) {
        const uint32_t v = 32u * w + lane;
        uint32_t d = 0;
        if (v < n) {
            uint32_t r[NW];
            load_row_at<NW>(adj, v, r);
#pragma unroll
            for (int i = 0; i < NW; ++i) d += __popc(r[i]);
        }
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const uint32_t x = __ballot_sync(0xffffffffu, (d >> k) & 1u);
            if (lane == w) B[k] = x;
        }
    }
    uint32_t live = 0u, cov = 0u, size = 0u;
#pragma unroll
    for (int k = 0; k < K; ++k) live |= B[k];
    for (uint32_t it = 0; it < n; ++it) {
        uint32_t c = live;  // the vertices of least degree
#pragma unroll
        for (int k = K - 1; k >= 0; --k) {
            const uint32_t t = c & ~B[k];
            if (__any_sync(0xffffffffu, t != 0u)) c = t;
        }
        const uint32_t bal = __ballot_sync(0xffffffffu, c != 0u);
        if (!bal) break;
        seed = seed * 1664525u + 1013904223u;
        const uint32_t r1 = seed >> 27, r2 = (seed >> 22) & 31u;
        const uint32_t src = (__ffs(__funnelshift_r(bal, bal, r1)) - 1 + r1) & 31u;
        c = __shfl_sync(0xffffffffu, c, src);
        const uint32_t b = (__ffs(__funnelshift_r(c, c, r2)) - 1 + r2) & 31u;
        const uint32_t nb = adj[Rows<NW>::at(32u * src + b, at)] & live;
        cov |= nb;
        size += __reduce_add_sync(0xffffffffu, __popc(nb));
        if (size >= limit) return size;
        uint32_t wm = __ballot_sync(0xffffffffu, nb != 0u);
        while (wm) {
            const uint32_t w = __ffs(wm) - 1;
            wm &= wm - 1;
            uint32_t m = __shfl_sync(0xffffffffu, nb, w);
            while (m) {
                const uint32_t u = 32u * w + (__ffs(m) - 1);
                m &= m - 1;
                uint32_t br = adj[Rows<NW>::at(u, at)] & live;
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    const uint32_t t = B[k];
                    B[k] = t ^ br;
                    br &= ~t;
                }
            }
        }
        const uint32_t gone = nb | (lane == src ? 1u << b : 0u);
        live = 0u;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            B[k] &= ~gone;
            live |= B[k];
        }
    }
    if (lane < (uint32_t)NW) cover[lane] = cov;
    __syncwarp();
    return size;
}

// A dive on the CTA's staged graph `inst` by a unit without work; a cover that
// betters the incumbent (PVC: answers the question) is reported.  The unit holds no
// token of the graph: its CTA is not idle meanwhile, so the launch outlasts it.
template <int NW>
__device__ __forceinline__ void dive_on(DSU<NW> &s, const Params &P, uint32_t inst)
{
    using S = DSU<NW>;
    const unsigned lane = lane_id();
    const uint32_t n = __ldcg(&P.inst[inst].n), mode = __ldcg(&P.inst[inst].mode);
    const uint32_t limit = mode == kModePVC ? __ldcg(&P.inst[inst].k) + 1u
                                            : WarpG::bcast(ld_relaxed_u32(&P.st[inst].best));
    const uint32_t size = dense_dive<NW>(s.adj, s.bits(), n, limit, 2654435761u * (WarpG::su_global() + 1u) + inst);
    if (size >= limit) return;
    if (lane < NW) {
        const uint32_t lo = 32u * lane;
        s.lsm()[lane] = ~s.bits()[lane] & (lo + 32u <= n ? 0xffffffffu : (lo < n ? (1u << (n - lo)) - 1u : 0u));
    }
    __syncwarp();
    bind_graph<WarpG>(s, P, inst);
    report_leaf<WarpG, S>(s, P, size);
    s.inst = kNone;
}

// Acquire work for a dense search unit.  Local records always belong to the
// CTA's staged graph.  Only when the whole CTA is idle may the poller switch
// graphs: first to the next root from the cursor, then to records of any graph
// from the global ring.  Returns false when the launch is over.
template <int NW>
__device__ bool acquire_cta(DSU<NW> &s, const Params &P, CtaPool &cp, uint32_t *adj)
{
    using G = WarpG;
    using S = DSU<NW>;
    const unsigned lane = lane_id();
    if (lane == 0) {
        __threadfence_block();
        atomicAdd(&cp.hdr[kCpIdle], 1u);
    }
    bool poller = false;
    uint32_t nap = 64;
    for (;;) {
        s.stat.polls += 1;
        // 0 wait, 1 local slot, 2 global record, 3 exit, 4 new root
        uint32_t res = 0, slot = 0;
        unsigned long long qpos = 0;
        if (lane == 0) {
            if (vld(&cp.hdr[kCpExit])) {
                res = 3;
            } else if (vld(&cp.hdr[kCpCount]) > 0) {
                if (poller) { atomicExch(&cp.hdr[kCpPoller], 0u); poller = false; }
                atomicSub(&cp.hdr[kCpIdle], 1u);
                __threadfence_block();
                for (uint32_t i = 0; i < cp.lp; ++i)
                    if (atomicCAS(&cp.state[i], 2u, 3u) == 2u) { slot = i; res = 1; break; }
                if (res == 0) {
                    __threadfence_block();
                    atomicAdd(&cp.hdr[kCpIdle], 1u);
                }
            } else if (poller || atomicCAS(&cp.hdr[kCpPoller], 0u, 1u) == 0u) {
                poller = true;
                const uint32_t cnt = vld(&cp.hdr[kCpCount]);
                __threadfence_block();
                const bool cta_idle = cnt == 0 && vld(&cp.hdr[kCpIdle]) == cp.su;
                if (ld_relaxed_u64(&P.ctl[kAbort]) || ld_relaxed_u64(&P.ctl[kFinish])) {
                    atomicExch(&cp.hdr[kCpExit], 1u);
                    res = 3;
                } else if (cta_idle && !vld(&cp.hdr[kCpCursorClosed])) {
                    uint32_t i = kNone;
                    if (claim_root(P, i)) {
                        if (vld(&cp.hdr[kCpRegistered])) {
                            atomicAdd(&P.ctl[kState], 0xffffffffffffffffull);  // idle CTAs-1
                            cp.hdr[kCpRegistered] = 0u;
                        }
                        atomicSub(&cp.hdr[kCpIdle], 1u);
                        slot = i;
                        res = 4;
                    } else if (!P.server) {
                        cp.hdr[kCpCursorClosed] = 1u;
                    }
                }
                // one graph in the launch (a plain solve): every record is for the
                // graph this CTA already staged, so idle warps of a busy CTA may
                // take records from the ring too
                const bool single = P.count == 1 && !P.server;
                if (res == 0 && (P.server || single || vld(&cp.hdr[kCpCursorClosed]))) {
                    unsigned long long stw = ld_relaxed_u64(&P.ctl[kState]);
                    if (!vld(&cp.hdr[kCpRegistered]) && cta_idle) {
                        stw = atomicAdd(&P.ctl[kState], 1ull) + 1ull;
                        cp.hdr[kCpRegistered] = 1u;
                    }
                    const bool reg = vld(&cp.hdr[kCpRegistered]) != 0;
                    const bool staged = vld(&cp.hdr[kCpStaged]) != kNone;
                    // a registered CTA is fully idle, so the poller may switch graphs
                    if ((reg || (single && staged)) && (stw >> 32) > 0 && ring_claim_deq(P, qpos)) {
                        if (reg) {
                            atomicAdd(&P.ctl[kState], 0xfffffffeffffffffull);  // pending-1, idle CTAs-1
                            cp.hdr[kCpRegistered] = 0u;
                        } else {
                            atomicAdd(&P.ctl[kState], 0xffffffff00000000ull);  // pending-1
                        }
                        atomicSub(&cp.hdr[kCpIdle], 1u);
                        res = 2;
                    } else if (reg && (uint32_t)stw == gridDim.x && (stw >> 32) == 0 &&
                               (!P.server || server_may_stop(P))) {
                        atomicExch(&P.ctl[kFinish], 1ull);
                        atomicExch(&cp.hdr[kCpExit], 1u);
                        res = 3;
                    } else if (globaltimer() > s.deadline) {
                        stop_launch(P, kStopTime);
                        atomicExch(&cp.hdr[kCpExit], 1u);
                        res = 3;
                    }
                }
                if (res != 0) { atomicExch(&cp.hdr[kCpPoller], 0u); poller = false; }
            }
        }
        res = G::bcast(res);
        if (res == 3) return false;
        if (res == 4) {  // a new graph root for the whole CTA
            slot = G::bcast(slot);
            const uint32_t inst = P.split ? 0u : slot;
            const uint32_t key = __ldcg(&P.inst[inst].key);
            if (vld(&cp.hdr[kCpStaged]) != key) {
                stage_graph<NW>(adj, P, inst);
                if (lane == 0) cp.hdr[kCpStaged] = key;
            }
            bind_graph<G>(s, P, inst);
            if (P.split) load_split_root<NW>(s, slot);
            else load_root<G>(s);
            s.stat.roots += 1;
            return true;
        }
        if (res == 1) {
            slot = G::bcast(slot);
            const uint32_t *d = cp.data + (size_t)slot * P.stride;
            __threadfence_block();
            const uint32_t inst = vld(&d[0]);
            bind_graph<G>(s, P, inst);
            for (uint32_t w = lane; w < s.nw; w += 32) s.bits()[w] = vld(&d[4 + w]);
            __syncwarp();
            if (lane == 0) {
                atomicSub(&cp.hdr[kCpCount], 1u);
                __threadfence_block();
                atomicExch(&cp.state[slot], 0u);
            }
            if (start_record<G, S>(s, P)) return true;
            if (lane == 0) { __threadfence_block(); atomicAdd(&cp.hdr[kCpIdle], 1u); }
            continue;
        }
        if (res == 2) {
            qpos = G::bcast64(qpos);
            const uint32_t slot_i = (uint32_t)(qpos & P.q_mask);
            const uint32_t *g = P.pool_data + (size_t)slot_i * P.stride;
            __syncwarp();
            __threadfence();
            const uint32_t inst = __ldcg(&g[0]);
            const uint32_t key = __ldcg(&P.inst[inst].key);
            if (vld(&cp.hdr[kCpStaged]) != key) {
                stage_graph<NW>(adj, P, inst);
                if (lane == 0) cp.hdr[kCpStaged] = key;
            }
            bind_graph<G>(s, P, inst);
            for (uint32_t w = lane; w < s.nw; w += 32) s.bits()[w] = __ldcg(&g[4 + w]);
            __syncwarp();
            if (lane == 0) {
                __threadfence();
                ring_release(P, qpos);
            }
            if (start_record<G, S>(s, P)) return true;
            if (lane == 0) { __threadfence_block(); atomicAdd(&cp.hdr[kCpIdle], 1u); }
            continue;
        }
        if (lane == 0) __nanosleep(nap);
        const uint32_t most = P.count == 1 ? kPlainNapMax : (poller ? 4096u : kIdleNapMax);
        nap = nap < most ? nap * 2 : most;
        __syncwarp();
    }
}

template <int NW>
__device__ void su_main_dense(const Params &P, uint8_t *ws, uint32_t *adj, CtaPool &cp)
{
    using G = WarpG;
    using S = DSU<NW>;
    S s;
    dsu_bind(s, ws, adj);
    s.inst = kNone;
    s.fr_bot = s.fr_top = 0;
    s.pending = 0;
    s.local_nodes = 0;
    s.c_best = 0;
    s.top = 0;
    s.deadline = globaltimer() + P.time_limit_ns;
    if (lane_id() == 0) atomicCAS(&P.ctl[kT0], 0ull, globaltimer());
    s.stat = SUStat{0, 0, 0, 0, 0, 0, 0, 0, 0};
    s.cyc = PhaseCycles{0, 0, 0, 0};
    s.timed = P.stats != nullptr;
    unsigned long long nodes_total = 0;
    long long t_mark = clock64();
    bool have = false;
    uint32_t ticks = 0, c_flags = 0;
    unsigned long long c_state = 0;
    const unsigned lane = lane_id();
    // How often the incumbent and the idle units are looked up: a plain solve's
    // tree is over in a few hundred nodes per unit, so every other node (against
    // every eighth: graphs of 175 and 197 vertices 0.65 and 1.62 -> 0.62 and 1.43 ms);
    // a batch loses by it (1024 graphs 151 -> 162 ms).
    const uint32_t tick_mask = P.count == 1 ? 1u : 7u;
    bool packing = P.pack_after_ns == 0;
    const unsigned long long t_pack = globaltimer() + P.pack_after_ns;
    if (NW >= 16 && P.dives && blockIdx.x - 1u < kDiveBlocks) {  // block 0 takes up the search
        if (WarpG::su_local() == 0) {
            stage_graph<NW>(adj, P, 0);
            if (lane == 0) cp.hdr[kCpStaged] = __ldcg(&P.inst[0].key);
        }
        __syncthreads();
        const bool refused = (ld_relaxed_u32(&P.st[0].flags) & kBadGraph) || ld_relaxed_u64(&P.ctl[kAbort]) == kStopInput;
        if (!G::bcast((uint32_t)refused)) dive_on<NW>(s, P, 0);
    }

    for (;;) {
        if (!have) {
            if (s.inst != kNone && s.fr_top > s.fr_bot) {
                const long long t_pop = (kPhaseTimers && s.timed) ? clock64() : 0;
                s.fr_top -= 1;
                const uint32_t f = s.frames()[s.fr_top];
                const uint32_t v = f & 0xffffu;
                dense_restore(s, f >> 16);
                if (lane < NW) s.marks()[lane] = s.adj[Rows<NW>::at(v, lane)] & s.lsm()[lane];
                __syncwarp();
                s.pending = kPendRecount;  // take N(v), then recount
                have = true;
                if (kPhaseTimers && s.timed) s.cyc.pop += (unsigned long long)(clock64() - t_pop);
            } else {
                if (s.inst != kNone) finish_stint<G, S>(s, P);
                long long t0 = clock64();
                s.stat.busy += (unsigned long long)(t0 - t_mark);
                bool got = acquire_cta<NW>(s, P, cp, adj);
                t_mark = clock64();
                s.stat.idle += (unsigned long long)(t_mark - t0);
                if (!got) break;
                have = true;  // load_root / rebuild counted the degrees
                ticks = 0;
            }
        }
        InstState &st = P.st[s.inst];
        if ((ticks & tick_mask) == 0u) {
            uint32_t b = 0, f = 0;
            unsigned long long w = 0;
            if (lane == 0) {
                b = ld_relaxed_u32(&st.best);
                f = ld_relaxed_u32(&st.flags);
                w = ld_relaxed_u64(&P.ctl[kState]);
                // (every 32 nodes: with the packing bound 256 of the wide kernels' took 30 ms beyond the limit)
                if ((ticks & 31u) == 0u) {
                    if (ld_relaxed_u64(&P.ctl[kAbort])) f |= kError;
                    else if (globaltimer() > s.deadline) { stop_launch(P, kStopTime); f |= kError; }
                }
                if (!packing && globaltimer() > t_pack) f |= kPackNow;
            }
            s.c_best = G::bcast(b);
            c_flags = G::bcast(f);
            c_state = G::bcast64(w);
            packing = packing || (c_flags & kPackNow);
        }
        ++ticks;
        if (c_flags & (kFound | kBudget | kError | kBadGraph)) {
            if (lane == 0 && !(c_flags & (kFound | kBudget | kBadGraph))) atomicOr(&st.flags, kCut);
            s.fr_bot = s.fr_top = 0;
            s.pending = 0;
            if (lane < NW) s.marks()[lane] = 0;
            __syncwarp();
            have = false;
            continue;
        }
        s.local_nodes += 1;
        nodes_total += 1;
        if ((s.local_nodes & 127ull) == 0ull) {
            if (lane == 0) {
                unsigned long long tot = atomicAdd(&st.nodes, s.local_nodes) + s.local_nodes;
                if (s.node_limit && tot >= s.node_limit) atomicOr(&st.flags, kBudget);
            }
            s.local_nodes = 0;
        }
        const uint32_t best = s.c_best;
        const uint32_t bound = s.mode == kModeMVC ? best : s.k + 1;
        ScanOut o = {0u, 0u, kNone};
        const long long t_scan = (kPhaseTimers && s.timed) ? clock64() : 0;
        const unsigned long long apply0 = s.cyc.apply;
        dense_settle(s, bound, o);
        if (kPhaseTimers && s.timed) s.cyc.scan += (unsigned long long)(clock64() - t_scan) - (s.cyc.apply - apply0);
        const uint32_t del = s.base_del + s.top;
        const uint64_t edges = o.sum / 2;
        // b more vertices may be taken below this node
        const uint32_t limit = s.mode == kModeMVC ? best - 1u : s.k;
        bool prune = s.mode == kModeMVC ? del >= best : del > s.k;
        if (!prune) {
            const uint64_t b = (uint64_t)(limit - del);
            prune = edges >= b * b + 1 || edges > b * o.maxd;
        }
        if (prune) { have = false; continue; }
        if (o.maxd == 0) {
            report_leaf<G, S>(s, P, del);
            have = false;
            continue;
        }
        const uint32_t v = o.amax;
        // Degrees of at most 2 leave disjoint cycles (the leaf rule took the paths),
        // and every vertex of a cycle is in one of its minimum covers: no branch.  Before
        // there is an incumbent (or a k below n) as many vertices may be taken as there
        // are, and no packing needs that many: the bound is left out on the first descent
        // (three graphs of 33 vertices and density 0.95 in a batch: kernel 171 -> 143 us, 112
        // before there was the bound; G(60, 0.1) alone 100 -> 83).
        const uint32_t open = o.maxd == 2u ? 1u
                              : packing && limit < s.n && o.maxd < (1u << kPackPlanes)
                                  ? open_children(s, v, o.maxd, limit - del)
                                  : 3u;
        if (open == 0u) { have = false; continue; }
        const long long t_br = (kPhaseTimers && s.timed) ? clock64() : 0;
        if (open == 3u) {  // a branch: "take N(v)" waits in a frame
            if (lane == 0) s.frames()[s.fr_top] = (s.top << 16) | v;
            s.fr_top += 1;
            __syncwarp();
        }
        if (s.fr_top > s.fr_bot) {  // a waiting child to give away, at a node that does not branch too
            uint32_t want = 0;
            if (lane == 0) {
                uint32_t li = vld(&cp.hdr[kCpIdle]), lc = vld(&cp.hdr[kCpCount]);
                const bool local_need = li > lc;
                const bool ring_need = (long long)(uint32_t)c_state - (long long)(c_state >> 32) > (long long)P.ring_bias;
                // both a sibling warp and another CTA wait: the policy decides (local
                // first, ring first, or alternating)
                if (local_need && ring_need)
                    want = (P.ring_first == 1 || (P.ring_first == 2 && (s.stat.donations & 1ull))) ? 2 : 1;
                else if (local_need) want = 1;
                else if (ring_need) want = 2;
            }
            want = G::bcast(want);
            if (want == 1) donate_local<G, S>(s, P, cp);
            else if (want == 2 && donate_global<G, S>(s, P)) c_state += 1ull << 32;
        }
        // the child takes v, or N(v) where only that is left (marks are clear after a settled node)
        if (open == 2u) {
            if (lane < NW) s.marks()[lane] = s.adj[Rows<NW>::at(v, lane)] & s.lsm()[lane];
        } else if (lane == 0) {
            s.marks()[v >> 5] = 1u << (v & 31u);
        }
        __syncwarp();
        s.pending = kPendApply;
        if (kPhaseTimers && s.timed) s.cyc.branch += (unsigned long long)(clock64() - t_br);
    }
    if (P.stats && lane == 0) {
        unsigned long long *o = P.stats + (size_t)G::su_global() * kStatWords;
        uint32_t smid;
        asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
        o[kStNodes] = nodes_total;
        o[kStPasses] = s.stat.passes;
        o[kStDonations] = s.stat.donations;
        o[kStDonateFail] = s.stat.donate_fail;
        o[kStReceives] = s.stat.receives;
        o[kStRoots] = s.stat.roots;
        o[kStBusyCycles] = s.stat.busy;
        o[kStIdleCycles] = s.stat.idle;
        o[kStPolls] = s.stat.polls;
        o[kStRestored] = s.stat.restored;
        o[kStSmid] = smid;
        o[kStCycScan] = s.cyc.scan;
        o[kStCycApply] = s.cyc.apply;
        o[kStCycPop] = s.cyc.pop;
        o[kStCycBranch] = s.cyc.branch;
        o[kStCycOther] = s.stat.busy - s.cyc.scan - s.cyc.apply - s.cyc.pop - s.cyc.branch;
    }
}

}  // namespace vcg
