// vc_reduce.cu -- the roots of large graphs, reduced by the whole chip.
//
// A graph of more than kHalfMaxN vertices used to be reduced at the root of its
// search by the one search unit that holds it: a 512-thread CTA walked all its
// vertices once per reduction pass while 147 SMs waited (a power-law graph of
// 100,000 vertices, whose whole tree is that one node: 8.4 ms, now 0.36 with its
// checks; a planted cover of 2262 vertices 0.11 and 0.07).  What bounds it is the
// chain of passes: two grid barriers and two rounds of dependent loads from L2
// each, whatever the size up to a vertex per thread.  Here the same
// rules run over the whole graph with a thread per vertex on every SM, one
// cooperative launch, two grid barriers per pass; or, where a batch has many such
// graphs, a cluster of CTAs and its barrier for each, all in one launch (a launch
// after another had left the chip idle but for the few CTAs of one graph: 1000 graphs
// of 1100 to 4000 vertices 69 ms, now 1.4).  What is left is written out as
// a graph of its own, rows in the old order, and goes to the kernel for its size
// (csrc/vc_solver.cu).  The optimum is the number of vertices taken here plus the
// rest's.  A caller's device memory has been checked for its layout only: where an
// edge is in one direction alone, a degree and the entries that are left of its row
// can part.  The write-out keeps to the entries whose vertex is left and to the row's
// own places, and a row that it does not fill exactly marks the graph as uneven:
// its rest is not searched, the graph itself is.
//
// A pass decides the degree-one, degree-two/triangle and high-degree rules from
// one snapshot, as the search units do (vc_search.cuh, reduce_pass; the
// reference's helperFunctions.cuh:229-447): taken[v] holds the pass that took v,
// so a vertex marked in the current pass still counts as live, and a vertex's
// degree changes only in the pass's second half.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "vc_host.h"
#include "vc_search.cuh"

namespace cg = cooperative_groups;

namespace vcg {

constexpr unsigned kReduceThreads = 512;
constexpr uint32_t kLongRow = 64;        // longer rows are walked by a whole warp
constexpr uint32_t kReducePasses = 1024;  // what is left after these goes to the search as it is

using vch::ReduceArgs;

// The CTAs that reduce one graph: the whole launch, or a cluster of a launch over
// many graphs (csrc/vc_solver.cu says which).
struct Chip {
    static __device__ __forceinline__ uint32_t cta() { return blockIdx.x; }
    static __device__ __forceinline__ uint32_t ctas() { return gridDim.x; }
    static __device__ __forceinline__ void sync() { cg::this_grid().sync(); }
};
struct Cluster {
    static __device__ __forceinline__ uint32_t cta() { return cg::this_cluster().block_rank(); }
    static __device__ __forceinline__ uint32_t ctas() { return cg::this_cluster().num_blocks(); }
    static __device__ __forceinline__ void sync() { cg::this_cluster().sync(); }
};

__device__ __forceinline__ bool red_live(const ReduceArgs &A, uint32_t u, uint32_t pass)
{
    const uint32_t t = __ldcg(&A.taken[u]);
    return (t == 0u || t == pass) && __ldcg(&A.deg[u]) > 0;
}

// The degree-one and triangle rules on v of degree d with live neighbours a (and b).
__device__ __forceinline__ bool red_rules(const ReduceArgs &A, uint32_t v, int32_t d, uint32_t a, uint32_t b, uint32_t pass)
{
    if (a == kNone) return false;
    const int32_t da = __ldcg(&A.deg[a]);
    if (d == 1) {
        if (da > 1 || a < v) {
            __stcg(&A.taken[a], pass);
            return true;
        }
        return false;
    }
    if (b == kNone) return false;
    const int32_t db = __ldcg(&A.deg[b]);
    if (da == 1 || db == 1 || (da == 2 && a < v) || (db == 2 && b < v)) return false;
    if (!row_contains(false, A.rp, A.cl, b, a)) return false;
    __stcg(&A.taken[a], pass);
    __stcg(&A.taken[b], pass);
    return true;
}

template <class Grp>
__device__ __forceinline__ void reduce_graph(const ReduceArgs &A)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t cta = Grp::cta(), ctas = Grp::ctas();
    const uint32_t t0 = cta * kReduceThreads + threadIdx.x, step = ctas * kReduceThreads;
    const uint32_t rounds = (A.n + step - 1) / step;  // the same for every thread: the warps stay whole
    vch::ReduceHead *H = A.head;
    if (*A.bad) return;  // the check before this launch: the same for every CTA
    for (uint32_t v = t0; v < A.n; v += step) {
        A.deg[v] = (int32_t)(__ldg(&A.rp[v + 1]) - __ldg(&A.rp[v]));
        A.taken[v] = 0u;
    }
    Grp::sync();
    for (uint32_t pass = 1; pass <= kReducePasses; ++pass) {
        const uint32_t del = __ldcg(&H->taken);
        bool marked = false;
        for (uint32_t r = 0; r < rounds; ++r) {
            const uint32_t v = t0 + r * step;
            int32_t d = 0;
            if (v < A.n && __ldcg(&A.taken[v]) == 0u) d = __ldcg(&A.deg[v]);
            uint32_t e0 = 0, e1 = 0;
            if (d > 0 && (uint64_t)d + del >= A.bound) {
                __stcg(&A.taken[v], pass);
                marked = true;
            } else if (d == 1 || d == 2) {
                e0 = __ldg(&A.rp[v]);
                e1 = __ldg(&A.rp[v + 1]);
            }
            const bool is_long = e1 - e0 > kLongRow;
            uint32_t a = kNone, b = kNone;
            if (!is_long) {
                for (uint32_t e = e0; e < e1; ++e) {
                    const uint32_t u = __ldg(&A.cl[e]);
                    if (!red_live(A, u, pass)) continue;
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
                    uint32_t m = __ballot_sync(0xffffffffu, u != kNone && red_live(A, u, pass));
                    while (m && got < want) {
                        const uint32_t w = __shfl_sync(0xffffffffu, u, __ffs(m) - 1);
                        m &= m - 1;
                        if (got == 0) x = w; else y = w;
                        ++got;
                    }
                }
                if (lane == src) { a = x; b = y; }
            }
            if (d == 1 || d == 2) marked |= red_rules(A, v, d, a, b, pass);
        }
        if (__syncthreads_or(marked) && threadIdx.x == 0) atomicMax(&H->last_pass, pass);
        Grp::sync();
        if (__ldcg(&H->last_pass) != pass) break;  // nothing marked: the fixpoint
        uint32_t mine = 0;
        for (uint32_t r = 0; r < rounds; ++r) {
            const uint32_t v = t0 + r * step;
            uint32_t e0 = 0, e1 = 0;
            if (v < A.n && __ldcg(&A.taken[v]) == pass) {
                e0 = __ldg(&A.rp[v]);
                e1 = __ldg(&A.rp[v + 1]);
                mine += 1;
            }
            const bool is_long = e1 - e0 > kLongRow;
            if (!is_long)
                for (uint32_t e = e0; e < e1; ++e) {
                    const uint32_t u = __ldg(&A.cl[e]);
                    if (__ldcg(&A.taken[u]) == 0u) atomicSub(&A.deg[u], 1);
                }
            uint32_t todo = __ballot_sync(0xffffffffu, is_long);
            while (todo) {
                const uint32_t src = __ffs(todo) - 1;
                todo &= todo - 1;
                const uint32_t f0 = __shfl_sync(0xffffffffu, e0, src), f1 = __shfl_sync(0xffffffffu, e1, src);
                for (uint32_t e = f0 + lane; e < f1; e += 32) {
                    const uint32_t u = __ldg(&A.cl[e]);
                    if (__ldcg(&A.taken[u]) == 0u) atomicSub(&A.deg[u], 1);
                }
            }
        }
        mine = __reduce_add_sync(0xffffffffu, mine);
        if (lane == 0 && mine) atomicAdd(&H->taken, mine);
        Grp::sync();
    }

    // What is left: CTA i numbers the vertices of the i-th part of the old ids.
    __shared__ uint32_t s_cnt[kReduceThreads / 32], s_sum[kReduceThreads / 32];
    const uint32_t per = (A.n + ctas - 1) / ctas;
    const uint32_t lo = min(A.n, cta * per), hi = min(A.n, lo + per);
    auto left = [&](uint32_t v) -> uint32_t {
        const int32_t d = v < hi && __ldcg(&A.taken[v]) == 0u ? __ldcg(&A.deg[v]) : 0;
        return d > 0 ? (uint32_t)d : 0u;
    };
    auto block_sums = [&](uint32_t c, uint32_t s) {  // per warp, into shared memory
        c = __reduce_add_sync(0xffffffffu, c);
        s = __reduce_add_sync(0xffffffffu, s);
        if (lane == 0) { s_cnt[threadIdx.x >> 5] = c; s_sum[threadIdx.x >> 5] = s; }
        __syncthreads();
    };
    uint32_t c = 0, s = 0, mx = 0;
    for (uint32_t v = lo + threadIdx.x; v < lo + per; v += kReduceThreads) {
        const uint32_t d = left(v);
        if (v < hi) A.cover[v] = __ldcg(&A.taken[v]) != 0u;
        c += d > 0u;
        s += d;
        mx = max(mx, d);
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0 && mx) atomicMax(&H->maxd, mx);
    block_sums(c, s);
    if (threadIdx.x == 0) {
        uint32_t tc = 0, ts = 0;
        for (uint32_t w = 0; w < kReduceThreads / 32; ++w) { tc += s_cnt[w]; ts += s_sum[w]; }
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
    for (uint32_t vb = lo; vb < hi; vb += kReduceThreads) {
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
        for (uint32_t w = 0; w < kReduceThreads / 32; ++w) {
            if (w < threadIdx.x >> 5) { wc += s_cnt[w]; wsum += s_sum[w]; }
            tc += s_cnt[w];
            ts += s_sum[w];
        }
        const uint32_t id = base_c + wc + pc - 1u;
        if (v < hi) __stcg(&A.map[v], d > 0u ? id : kNone);
        if (d > 0u) {
            __stcg(&A.inv[id], v);
            __stcg(&A.rrp[id], base_s + wsum + ps - d);
        }
        base_c += tc;
        base_s += ts;
    }
    if (cta == ctas - 1 && threadIdx.x == 0) A.rrp[H->n] = H->m2;
    Grp::sync();
    // a warp per row that is left, its entries that are left in the old order
    const uint32_t rows = __ldcg(&H->n);
    for (uint32_t id = t0 >> 5; id < rows; id += step >> 5) {
        const uint32_t v = __ldcg(&A.inv[id]);
        uint32_t out = __ldcg(&A.rrp[id]);
        const uint32_t end = __ldcg(&A.rrp[id + 1]);
        const uint32_t e1 = __ldg(&A.rp[v + 1]);
        for (uint32_t eb = __ldg(&A.rp[v]); eb < e1; eb += 32) {
            const uint32_t x = eb + lane < e1 ? __ldcg(&A.map[__ldg(&A.cl[eb + lane])]) : kNone;
            const uint32_t m = __ballot_sync(0xffffffffu, x != kNone);
            const uint32_t at = out + __popc(m & ((1u << lane) - 1u));
            if (x != kNone && at < end) A.rcl[at] = x;
            out += __popc(m);
        }
        if (out != end && lane == 0) __stcg(&H->uneven, 1u);
    }
}

__global__ void __launch_bounds__(kReduceThreads, 2) k_reduce(ReduceArgs A) { reduce_graph<Chip>(A); }

__global__ void __launch_bounds__(kReduceThreads, 2) k_reduce_many(const ReduceArgs *list)
{
    const ReduceArgs A = list[blockIdx.x / Cluster::ctas()];
    reduce_graph<Cluster>(A);
}

}  // namespace vcg

using namespace vcg;

namespace vch {

cudaError_t launch_reduce(const ReduceArgs &r, uint32_t ctas, cudaStream_t stream)
{
    ReduceArgs A = r;
    const uint32_t grid = std::max<uint32_t>(1, std::min<uint32_t>((r.n + kReduceThreads - 1) / kReduceThreads, ctas));
    void *args[] = {&A};
    return cudaLaunchCooperativeKernel((const void *)k_reduce, dim3(grid), dim3(kReduceThreads), args, 0, stream);
}

// `count` graphs side by side, a cluster of `ctas` CTAs each.
cudaError_t launch_reduce_many(const ReduceArgs *list, uint32_t count, uint32_t ctas, cudaStream_t stream)
{
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = ctas;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(count * ctas);
    cfg.blockDim = dim3(kReduceThreads);
    cfg.stream = stream;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    void *args[] = {&list};
    return cudaLaunchKernelExC(&cfg, (const void *)k_reduce_many, args);
}

// CTAs of a reduction: two per SM (the launch bounds leave room for them).
uint32_t reduce_ctas(const Ctx &c) { return 2u * (uint32_t)c.sms; }

}  // namespace vch
