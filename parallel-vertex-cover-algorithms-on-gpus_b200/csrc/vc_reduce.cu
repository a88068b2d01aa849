// vc_reduce.cu -- the roots of large graphs, reduced before the search.
//
// A graph of more than kHalfMaxN vertices used to be reduced at the root of its
// search by the one search unit that holds it: a 512-thread CTA walked all its
// vertices once per reduction pass while 147 SMs waited (a power-law graph of
// 100,000 vertices, whose whole tree is that one node: 8.4 ms, now 0.22 with its
// checks; a planted cover of 2221 vertices 0.12, now 0.04).  Here the same rules run
// on their own: by the whole chip with a thread per vertex in one cooperative launch,
// by a cluster of CTAs for each of many graphs in one launch, or by one CTA each with
// the graph's degrees in shared memory (csrc/vc_solver.cu says which and why).  What
// bounds them is the chain of passes: on several CTAs two grid or cluster barriers
// and four dependent reads from L2 each (2.9 us on the chip), on one CTA three
// barriers of its own and the reads of the rows that the rules look at (0.75 us at
// 1500 vertices and 1.3 at 5000, where the search's CTA took 1.1 and 2.7).  What is
// left is written out as a graph of its own, rows in the old order, and goes to the
// kernel for its size.  The optimum is the number of vertices taken here plus the
// rest's.
//
// A caller's device memory has been checked for its layout only: where an edge is in
// one direction alone, a degree and the entries that are left of its row can part.
// The write-out keeps to the entries whose vertex is left and to the row's own
// places, and a row that it does not fill exactly marks the graph as uneven: its rest
// is not searched, the graph itself is.
//
// A pass decides the degree-one, degree-two/triangle and high-degree rules from
// one snapshot, as the search units do (vc_search.cuh, reduce_pass; the
// reference's helperFunctions.cuh:229-447): degrees change only in the pass's second
// half.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "vc_host.h"
#include "vc_search.cuh"

namespace cg = cooperative_groups;

namespace vcg {

constexpr uint32_t kLongRow = 64;        // longer rows are walked by a whole warp
constexpr uint32_t kReducePasses = 1024;  // of the chip or a cluster; what is left then goes to the search as it is

using vch::ReduceArgs;
using vch::ReduceHead;

// The CTAs that reduce one graph: the whole launch, a cluster of a launch over many
// graphs, or one CTA of such a launch (csrc/vc_solver.cu says which).
struct Chip {
    static constexpr bool kNear = false;
    static constexpr unsigned kThreads = 512;
    static __device__ __forceinline__ uint32_t cta() { return blockIdx.x; }
    static __device__ __forceinline__ uint32_t ctas() { return gridDim.x; }
    static __device__ __forceinline__ void sync() { cg::this_grid().sync(); }
};
struct Cluster {
    static constexpr bool kNear = false;
    static constexpr unsigned kThreads = 512;
    static __device__ __forceinline__ uint32_t cta() { return cg::this_cluster().block_rank(); }
    static __device__ __forceinline__ uint32_t ctas() { return cg::this_cluster().num_blocks(); }
    static __device__ __forceinline__ void sync() { cg::this_cluster().sync(); }
};
struct Block {
    static constexpr bool kNear = true;
    static constexpr unsigned kThreads = 1024;
    static __device__ __forceinline__ uint32_t cta() { return 0u; }
    static __device__ __forceinline__ uint32_t ctas() { return 1u; }
    static __device__ __forceinline__ void sync() { __syncthreads(); }
};

// The state of a graph on several CTAs, in global memory: taken[v] holds the pass that
// took v, so a vertex marked in the current pass still counts as live.
struct FarState {
    int32_t *deg_;
    uint32_t *taken;
    uint32_t pass;
    bool marked;
    __device__ __forceinline__ int32_t deg(uint32_t v) const { return __ldcg(&deg_[v]); }
    __device__ __forceinline__ int32_t unmarked_deg(uint32_t v) const { return __ldcg(&taken[v]) == 0u ? deg(v) : 0; }
    __device__ __forceinline__ bool live(uint32_t v) const
    {
        const uint32_t t = __ldcg(&taken[v]);
        return (t == 0u || t == pass) && deg(v) > 0;
    }
    __device__ __forceinline__ void mark(uint32_t v)
    {
        __stcg(&taken[v], pass);
        marked = true;
    }
    __device__ __forceinline__ void drop_edge(uint32_t u)
    {
        if (__ldcg(&taken[u]) == 0u) atomicSub(&deg_[u], 1);
    }
};

// On one CTA, in shared memory: a vertex that a pass marks goes on that pass's list
// and into the bitmap of all that were taken; its degree is set aside in the pass's
// second half, so the first half's are one snapshot.
struct NearState {
    int32_t *deg_;
    uint32_t *marks;
    uint16_t *list;
    uint32_t *count;  // of the pass
    __device__ __forceinline__ int32_t deg(uint32_t v) const { return *(volatile int32_t *)&deg_[v]; }
    __device__ __forceinline__ int32_t unmarked_deg(uint32_t v) const { return deg(v); }
    __device__ __forceinline__ bool live(uint32_t v) const { return deg(v) > 0; }
    __device__ __forceinline__ void mark(uint32_t v)
    {
        const uint32_t bit = 1u << (v & 31u);
        if (!(atomicOr(&marks[v >> 5], bit) & bit)) list[atomicAdd(count, 1u)] = (uint16_t)v;
    }
    __device__ __forceinline__ void drop_edge(uint32_t u)
    {
        if (deg(u) > 0) atomicSub(&deg_[u], 1);
    }
};

// The degree-one and triangle rules on v of degree d with live neighbours a (and b).
template <class S>
__device__ __forceinline__ void red_rules(const ReduceArgs &A, S &s, uint32_t v, int32_t d, uint32_t a, uint32_t b)
{
    if (a == kNone) return;
    const int32_t da = s.deg(a);
    if (d == 1) {
        if (da > 1 || a < v) s.mark(a);
        return;
    }
    if (b == kNone) return;
    const int32_t db = s.deg(b);
    if (da == 1 || db == 1 || (da == 2 && a < v) || (db == 2 && b < v)) return;
    if (!row_contains(false, A.rp, A.cl, b, a)) return;
    s.mark(a);
    s.mark(b);
}

// The first half of a pass: the three rules on vertices t0, t0 + step, ...
template <class S>
__device__ __forceinline__ void red_mark(const ReduceArgs &A, S &s, uint32_t t0, uint32_t step, uint32_t del)
{
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t base = 0; base < A.n; base += step) {  // the same for every thread: the warps stay whole
        const uint32_t v = t0 + base;
        const int32_t d = v < A.n ? s.unmarked_deg(v) : 0;
        uint32_t e0 = 0, e1 = 0;
        if (d > 0 && (uint64_t)d + del >= A.bound) {
            s.mark(v);
        } else if (d == 1 || d == 2) {
            e0 = __ldg(&A.rp[v]);
            e1 = __ldg(&A.rp[v + 1]);
        }
        const bool is_long = e1 - e0 > kLongRow;
        uint32_t a = kNone, b = kNone;
        if (!is_long) {
            for (uint32_t e = e0; e < e1; ++e) {
                const uint32_t u = __ldg(&A.cl[e]);
                if (!s.live(u)) continue;
                if (a == kNone) a = u; else { b = u; break; }
                if (d == 1) break;
            }
        }
        uint32_t todo = __ballot_sync(0xffffffffu, is_long);
        while (todo) {  // a warp per long row: its first live entries
            const uint32_t src = __ffs(todo) - 1;
            todo &= todo - 1;
            const uint32_t f0 = __shfl_sync(0xffffffffu, e0, src), f1 = __shfl_sync(0xffffffffu, e1, src);
            const uint32_t want = (uint32_t)__shfl_sync(0xffffffffu, d, src);
            uint32_t got = 0, x = kNone, y = kNone;
            for (uint32_t eb = f0; eb < f1 && got < want; eb += 32) {
                const uint32_t u = eb + lane < f1 ? __ldg(&A.cl[eb + lane]) : kNone;
                uint32_t m = __ballot_sync(0xffffffffu, u != kNone && s.live(u));
                while (m && got < want) {
                    const uint32_t w = __shfl_sync(0xffffffffu, u, __ffs(m) - 1);
                    m &= m - 1;
                    if (got == 0) x = w; else y = w;
                    ++got;
                }
            }
            if (lane == src) { a = x; b = y; }
        }
        if (d == 1 || d == 2) red_rules(A, s, v, d, a, b);
    }
}

// A warp takes a vertex per lane (v = kNone: none): their edges come off the degrees.
template <class S>
__device__ __forceinline__ void red_take(const ReduceArgs &A, S &s, uint32_t v)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t e0 = v != kNone ? __ldg(&A.rp[v]) : 0u, e1 = v != kNone ? __ldg(&A.rp[v + 1]) : 0u;
    const bool is_long = e1 - e0 > kLongRow;
    if (!is_long)
        for (uint32_t e = e0; e < e1; ++e) s.drop_edge(__ldg(&A.cl[e]));
    uint32_t todo = __ballot_sync(0xffffffffu, is_long);
    while (todo) {
        const uint32_t src = __ffs(todo) - 1;
        todo &= todo - 1;
        const uint32_t f0 = __shfl_sync(0xffffffffu, e0, src), f1 = __shfl_sync(0xffffffffu, e1, src);
        for (uint32_t e = f0 + lane; e < f1; e += 32) s.drop_edge(__ldg(&A.cl[e]));
    }
}

// The passes of a graph on several CTAs, to their fixpoint or limit.
template <class Grp>
__device__ __forceinline__ void red_passes_far(const ReduceArgs &A, uint32_t t0, uint32_t step)
{
    ReduceHead *H = A.head;
    FarState s{A.deg, A.taken, 0u, false};
    for (uint32_t v = t0; v < A.n; v += step) {
        A.deg[v] = (int32_t)(__ldg(&A.rp[v + 1]) - __ldg(&A.rp[v]));
        A.taken[v] = 0u;
    }
    Grp::sync();
    for (s.pass = 1; s.pass <= kReducePasses; ++s.pass) {
        s.marked = false;
        red_mark(A, s, t0, step, __ldcg(&H->taken));
        if (__syncthreads_or(s.marked) && threadIdx.x == 0) atomicMax(&H->last_pass, s.pass);
        Grp::sync();
        if (__ldcg(&H->last_pass) != s.pass) break;  // nothing marked: the fixpoint
        uint32_t mine = 0;
        for (uint32_t base = 0; base < A.n; base += step) {
            const uint32_t v = t0 + base;
            const bool take = v < A.n && __ldcg(&A.taken[v]) == s.pass;
            mine += take;
            red_take(A, s, take ? v : kNone);
        }
        mine = __reduce_add_sync(0xffffffffu, mine);
        if ((threadIdx.x & 31u) == 0 && mine) atomicAdd(&H->taken, mine);
        Grp::sync();
    }
}

// The same by one CTA.  A pass that marks takes a vertex, so n passes are enough.
__device__ __forceinline__ void red_passes_near(const ReduceArgs &A, NearState s, uint32_t *counts)
{
    for (uint32_t v = threadIdx.x; v < A.n; v += Block::kThreads) s.deg_[v] = (int32_t)(__ldg(&A.rp[v + 1]) - __ldg(&A.rp[v]));
    for (uint32_t w = threadIdx.x; w < (A.n + 31) / 32; w += Block::kThreads) s.marks[w] = 0u;
    if (threadIdx.x < 2) counts[threadIdx.x] = 0u;
    __syncthreads();
    uint32_t taken = 0;
    for (uint32_t pass = 0; pass < A.n; ++pass) {
        s.count = &counts[pass & 1u];
        red_mark(A, s, threadIdx.x, Block::kThreads, taken);
        __syncthreads();
        const uint32_t k = *(volatile uint32_t *)s.count;
        if (k == 0u) break;
        for (uint32_t base = 0; base < k; base += Block::kThreads) {
            const uint32_t i = base + threadIdx.x, v = i < k ? s.list[i] : kNone;
            if (v != kNone) s.deg_[v] = kDead;
            red_take(A, s, v);
        }
        if (threadIdx.x == 0) counts[~pass & 1u] = 0u;  // the next pass's
        taken += k;
        __syncthreads();
    }
    if (threadIdx.x == 0) A.head->taken = taken;
}

template <class Grp>
__device__ __forceinline__ void reduce_graph(const ReduceArgs &A)
{
    constexpr bool kNear = Grp::kNear;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t cta = Grp::cta(), ctas = Grp::ctas();
    const uint32_t t0 = cta * Grp::kThreads + threadIdx.x, step = ctas * Grp::kThreads;
    ReduceHead *H = A.head;
    if (H->bad) return;  // the check before this launch: the same for every CTA
    extern __shared__ int32_t red_smem[];
    __shared__ uint32_t s_counts[2];
    int32_t *deg = A.deg;
    uint32_t *map = A.map, *marks = nullptr;
    if constexpr (kNear) {
        deg = red_smem;
        marks = reinterpret_cast<uint32_t *>(red_smem + A.n);
        map = reinterpret_cast<uint32_t *>(red_smem);  // a vertex's new id takes the place of its degree
        red_passes_near(A, NearState{deg, marks, reinterpret_cast<uint16_t *>(marks + (A.n + 31) / 32), nullptr}, s_counts);
    } else {
        red_passes_far<Grp>(A, t0, step);
    }
    auto is_taken = [&](uint32_t v) {
        if constexpr (kNear) return ((marks[v >> 5] >> (v & 31u)) & 1u) != 0u;
        else return __ldcg(&A.taken[v]) != 0u;
    };
    auto degree = [&](uint32_t v) {
        if constexpr (kNear) return deg[v];
        else return __ldcg(&deg[v]);
    };

    // What is left: CTA i numbers the vertices of the i-th part of the old ids.
    __shared__ uint32_t s_cnt[Grp::kThreads / 32], s_sum[Grp::kThreads / 32];
    const uint32_t per = (A.n + ctas - 1) / ctas;
    const uint32_t lo = min(A.n, cta * per), hi = min(A.n, lo + per);
    auto left = [&](uint32_t v) -> uint32_t {
        const int32_t d = v < hi && !is_taken(v) ? degree(v) : 0;
        return d > 0 ? (uint32_t)d : 0u;
    };
    auto block_sums = [&](uint32_t c, uint32_t s) {  // per warp, into shared memory
        c = __reduce_add_sync(0xffffffffu, c);
        s = __reduce_add_sync(0xffffffffu, s);
        if (lane == 0) { s_cnt[threadIdx.x >> 5] = c; s_sum[threadIdx.x >> 5] = s; }
        __syncthreads();
    };
    uint32_t c = 0, s = 0, mx = 0;
    for (uint32_t v = lo + threadIdx.x; v < lo + per; v += Grp::kThreads) {
        const uint32_t d = left(v);
        if (v < hi) A.cover[v] = is_taken(v);
        c += d > 0u;
        s += d;
        mx = max(mx, d);
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0 && mx) atomicMax(&H->maxd, mx);
    block_sums(c, s);
    if (threadIdx.x == 0) {
        uint32_t tc = 0, ts = 0;
        for (uint32_t w = 0; w < Grp::kThreads / 32; ++w) { tc += s_cnt[w]; ts += s_sum[w]; }
        A.part[2 * cta] = tc;
        A.part[2 * cta + 1] = ts;
        atomicAdd(&H->n, tc);
        atomicAdd(&H->m2, ts);
    }
    Grp::sync();
    if (__ldcg(&H->n) == 0u) return;
    uint32_t base_c = 0, base_s = 0;  // the parts before this one
    for (uint32_t i = lane; i < cta; i += 32) {
        base_c += __ldcg(&A.part[2 * i]);
        base_s += __ldcg(&A.part[2 * i + 1]);
    }
    base_c = __reduce_add_sync(0xffffffffu, base_c);
    base_s = __reduce_add_sync(0xffffffffu, base_s);
    for (uint32_t vb = lo; vb < hi; vb += Grp::kThreads) {
        const uint32_t v = vb + threadIdx.x;
        const uint32_t d = left(v);
        uint32_t pc = d > 0u, ps = d;  // inclusive prefix over the warp
#pragma unroll
        for (int k = 1; k < 32; k <<= 1) {
            const uint32_t x = __shfl_up_sync(0xffffffffu, pc, k), y = __shfl_up_sync(0xffffffffu, ps, k);
            if (lane >= (uint32_t)k) { pc += x; ps += y; }
        }
        __syncthreads();  // the sums of the round before have been read
        if (lane == 31) { s_cnt[threadIdx.x >> 5] = pc; s_sum[threadIdx.x >> 5] = ps; }
        __syncthreads();
        uint32_t wc = 0, wsum = 0, tc = 0, ts = 0;
        for (uint32_t w = 0; w < Grp::kThreads / 32; ++w) {
            if (w < threadIdx.x >> 5) { wc += s_cnt[w]; wsum += s_sum[w]; }
            tc += s_cnt[w];
            ts += s_sum[w];
        }
        const uint32_t id = base_c + wc + pc - 1u;
        if (v < hi) map[v] = d > 0u ? id : kNone;
        if (d > 0u) {
            __stcg(&A.inv[id], v);
            __stcg(&A.rrp[id], base_s + wsum + ps - d);
        }
        base_c += tc;
        base_s += ts;
    }
    if (cta == ctas - 1 && threadIdx.x == 0) A.rrp[H->n] = H->m2;
    Grp::sync();
    auto new_id = [&](uint32_t u) {
        if constexpr (kNear) return map[u];
        else return __ldcg(&map[u]);
    };
    // a warp per row that is left, its entries that are left in the old order
    const uint32_t rows = __ldcg(&H->n);
    for (uint32_t id = t0 >> 5; id < rows; id += step >> 5) {
        const uint32_t v = __ldcg(&A.inv[id]);
        uint32_t out = __ldcg(&A.rrp[id]);
        const uint32_t end = __ldcg(&A.rrp[id + 1]);
        const uint32_t e1 = __ldg(&A.rp[v + 1]);
        for (uint32_t eb = __ldg(&A.rp[v]); eb < e1; eb += 32) {
            const uint32_t x = eb + lane < e1 ? new_id(__ldg(&A.cl[eb + lane])) : kNone;
            const uint32_t m = __ballot_sync(0xffffffffu, x != kNone);
            const uint32_t at = out + __popc(m & ((1u << lane) - 1u));
            if (x != kNone && at < end) A.rcl[at] = x;
            out += __popc(m);
        }
        if (out != end && lane == 0) __stcg(&H->uneven, 1u);
    }
}

__global__ void __launch_bounds__(Chip::kThreads, 2) k_reduce(ReduceArgs A) { reduce_graph<Chip>(A); }

__global__ void __launch_bounds__(Cluster::kThreads, 2) k_reduce_many(const ReduceArgs *list)
{
    const ReduceArgs A = list[blockIdx.x / Cluster::ctas()];
    reduce_graph<Cluster>(A);
}

__global__ void __launch_bounds__(Block::kThreads, 1) k_reduce_each(const ReduceArgs *list)
{
    const ReduceArgs A = list[blockIdx.x];
    reduce_graph<Block>(A);
}

}  // namespace vcg

using namespace vcg;

namespace vch {

cudaError_t launch_reduce(const ReduceArgs &r, uint32_t ctas, cudaStream_t stream)
{
    ReduceArgs A = r;
    const uint32_t grid = std::max<uint32_t>(1, std::min<uint32_t>((r.n + Chip::kThreads - 1) / Chip::kThreads, ctas));
    void *args[] = {&A};
    return cudaLaunchCooperativeKernel((const void *)k_reduce, dim3(grid), dim3(Chip::kThreads), args, 0, stream);
}

// `count` graphs side by side, a cluster each.
cudaError_t launch_reduce_many(const ReduceArgs *list, uint32_t count, cudaStream_t stream)
{
    constexpr uint32_t ctas = 8;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = ctas;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(count * ctas);
    cfg.blockDim = dim3(Cluster::kThreads);
    cfg.stream = stream;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    void *args[] = {&list};
    return cudaLaunchKernelExC(&cfg, (const void *)k_reduce_many, args);
}

// `count` graphs of at most nmax vertices, a CTA each: per vertex a degree, a place on
// the list and a mark.
cudaError_t launch_reduce_each(const ReduceArgs *list, uint32_t count, uint32_t nmax, cudaStream_t stream)
{
    const uint32_t smem = 6u * nmax + (nmax + 31) / 32 * 4 + 16;
    const cudaError_t e = cudaFuncSetAttribute(k_reduce_each, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    void *args[] = {&list};
    return cudaLaunchKernel((const void *)k_reduce_each, dim3(count), dim3(Block::kThreads), args, smem, stream);
}

// CTAs of a reduction: two per SM (the launch bounds leave room for them).
uint32_t reduce_ctas(const Ctx &c) { return 2u * (uint32_t)c.sms; }

}  // namespace vch
