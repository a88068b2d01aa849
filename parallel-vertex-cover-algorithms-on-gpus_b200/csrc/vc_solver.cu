// vc_solver.cu -- host side of libvcgpu.so: the C ABI (include/vcgpu.h), per-device
// contexts with grow-only device buffers, graph validation, launch sizing and
// result collection.  The search itself is vc_search.cuh.
//
// Replaces the host path of the reference's src/main.cu:101-359: device query
// (:101-121), sizing (:122, auxFunctions.cpp:469-578), allocations (:219-269),
// the kernel launch (:300-344) and the read-back (:348-359).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>

#include "vc_search.cuh"
#include "vc_dense.cuh"
#include "vc_lanes.cuh"
#include "vc_host.h"
#include "vcgpu.h"

using namespace vcg;

namespace vch {

std::atomic<uint64_t> g_launches{0};

// Resident threads per SM the search kernels are register-limited for
// (1024 -> at most 64 registers per thread, 32 warps per SM).
// Team-walk kernels also come with 768 (80 registers), taken where the extra
// registers cost no resident CTAs (see plan_variant).
#ifndef VC_MIN_THREADS_PER_SM
#define VC_MIN_THREADS_PER_SM 1024
#endif
constexpr unsigned kRoomyThreadsPerSM = 768;

// ---------------------------------------------------------------- kernels
template <class G, unsigned NT, unsigned MinThreads = VC_MIN_THREADS_PER_SM>
__global__ void __launch_bounds__(NT, MinThreads / NT) k_search(Params P)
{
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ uint32_t cp_hdr[kCpHdrWords];
    if (P.server && threadIdx.x == 0) atomicAdd(&P.ctl[kStarted], 1ull);  // residency check of server lanes
    const uint32_t su_per_cta = NT / G::kSize;
    CtaPool cp;
    cp.su = su_per_cta;
    cp.lp = P.cta_slots;
    cp.hdr = cp_hdr;
    cp.state = reinterpret_cast<uint32_t *>(smem + (P.gws ? 0 : (size_t)su_per_cta * P.su_bytes));
    cp.data = cp.state + ((P.cta_slots + 3) / 4 * 4);
    for (uint32_t i = threadIdx.x; i < kCpHdrWords; i += blockDim.x) cp_hdr[i] = 0;
    for (uint32_t i = threadIdx.x; i < P.cta_slots; i += blockDim.x) cp.state[i] = 0;
    __syncthreads();
    uint8_t *ws = P.gws ? P.gws + (size_t)G::su_global() * P.su_bytes : smem + (size_t)G::su_local() * P.su_bytes;
    su_main<G>(P, ws, cp);
}

// Register budget of the dense search units (resident threads per SM).  Graphs of
// at most 255 vertices: 1024 (64 registers).  The packing bound keeps some twenty
// words in registers and spills a tenth as much as with 1280 (48 registers): 1024
// graphs of up to 200 vertices 125 -> 118 ms; 768 (80 registers): 121, 512: 130.  A
// plain solve has idle units and waits for its longest chain of nodes: 512 (128
// registers, no spills), eight calls on G(60, 0.1) 1.07 -> 0.91 ms, one of 197
// vertices 0.99 -> 0.84.
#ifndef VC_DENSE_THREADS
#define VC_DENSE_THREADS 1024
#endif
#ifndef VC_DENSE_WARPS
#define VC_DENSE_WARPS 4
#endif
constexpr unsigned kPlainThreads = 512;
constexpr unsigned kLaneThreads = 1280;  // a server's 8-word lane: three CTAs per SM beside the other lanes' kernels
template <int NW>
struct DenseOcc {
    // 20-word graphs: three 256-thread CTAs' worth of registers (80 per thread),
    // so that a server lane of them fits beside three 8-word CTAs per SM;
    // 16- and 32-word graphs (16-bit degrees, rows and L in registers): two and
    // one CTA per SM, as many as their staged adjacency leaves room for
    static constexpr unsigned kThreads =
        NW == 32 ? 256u : (NW == 16 ? 512u : (NW >= 16 ? 768u : VC_DENSE_THREADS));
};

template <int NW, unsigned NT, unsigned Threads = DenseOcc<NW>::kThreads>
__global__ void __launch_bounds__(NT, (Threads / NT < 32 ? Threads / NT : 32)) k_dense(Params P)  // 32 CTAs/SM at most
{
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ uint32_t cp_hdr[kCpHdrWords];
    if (P.server && threadIdx.x == 0) atomicAdd(&P.ctl[kStarted], 1ull);  // residency check of server lanes
    const uint32_t su_per_cta = NT / 32;
    uint32_t *adj = reinterpret_cast<uint32_t *>(smem);
    uint8_t *ws0 = smem + dense_adj_bytes(NW);
    CtaPool cp;
    cp.su = su_per_cta;
    cp.lp = P.cta_slots;
    cp.hdr = cp_hdr;
    cp.state = reinterpret_cast<uint32_t *>(ws0 + (size_t)su_per_cta * P.su_bytes);
    cp.data = cp.state + ((P.cta_slots + 3) / 4 * 4);
    for (uint32_t i = threadIdx.x; i < kCpHdrWords; i += blockDim.x) cp_hdr[i] = (i == kCpStaged) ? kNone : 0u;
    for (uint32_t i = threadIdx.x; i < P.cta_slots; i += blockDim.x) cp.state[i] = 0;
    __syncthreads();
    su_main_dense<NW>(P, ws0 + (size_t)WarpG::su_local() * P.su_bytes, adj, cp);
}

// One thread per search unit (vc_lanes.cuh); NT lanes per CTA.
#ifndef VC_LANE_THREADS
#define VC_LANE_THREADS 128
#endif
template <int NW, unsigned NT>
__global__ void __launch_bounds__(NT, 1) k_lanes(Params P)
{
    extern __shared__ __align__(16) uint32_t lsm[];
    __shared__ uint32_t hdr[kLhWords];
    const LaneLayout lo(P.np / 32u, NW, NT, P.cta_slots);
    if (threadIdx.x < kLhWords) {
        const uint32_t i = threadIdx.x;
        hdr[i] = i == kLhIdle ? NT : ((i == kLhGraph || i == kLhKey) ? kNone : 0u);
    }
    for (uint32_t i = threadIdx.x; i < P.cta_slots; i += NT) lsm[lo.sstate + i] = 0;
    __syncthreads();
    lanes_main<NW, NT>(P, lsm, hdr);
}

// What a launch needs before the search: control words, covers and counters
// cleared, the ring's sequence numbers, the graphs' states and, for the dense
// kernels, their adjacency as bitmap rows (A.adj; NW = 0: none), a warp per row
// and block (x, y) the rows 32y.. of graph x.  With the rows made once by the
// whole chip, a CTA that changes graphs copies 16-byte words instead of walking
// CSR rows one lane per row: the first staging of a 450-vertex graph of average
// degree 315 took over a millisecond.
struct PrepareArgs {
    unsigned long long *ctl, *seq;
    uint32_t q;
    uint32_t *covers;
    uint32_t cover_words;
    InstState *st;
    const InstDesc *inst;
    uint32_t count;
    uint32_t roots;  // per graph
    const uint32_t *row_ptr, *col;
    uint32_t *adj;
};

constexpr unsigned kPrepareThreads = 256;
constexpr unsigned kPrepareRows = 32;  // per block

template <int NW>
__global__ void __launch_bounds__(kPrepareThreads) k_prepare(PrepareArgs A)
{
    const uint32_t block = blockIdx.x + gridDim.x * blockIdx.y;
    const uint32_t t0 = block * kPrepareThreads + threadIdx.x, step = gridDim.x * gridDim.y * kPrepareThreads;
    for (uint32_t i = t0; i < A.q; i += step) A.seq[i] = i;
    for (uint32_t i = t0; i < A.cover_words; i += step) A.covers[i] = 0u;
    for (uint32_t i = t0; i < kCtlWords; i += step) A.ctl[i] = 0ull;
    for (uint32_t i = t0; i < A.count; i += step) {
        InstState s;
        s.best = A.inst[i].init_best;
        s.act = A.roots;
        s.flags = 0;
        s.lock = 0;
        s.cover_size = kNone;
        s.pad = 0;
        s.nodes = 0;
        s.t_done = 0;
        A.st[i] = s;
    }
    if constexpr (NW > 0) {
        __shared__ uint32_t rows[kPrepareThreads / 32][NW];
        for (uint32_t g = blockIdx.x; g < A.count; g += gridDim.x) {
            const InstDesc &d = A.inst[g];
            const uint32_t *rp = A.row_ptr + d.row_off, *cl = A.col + d.col_off;
            const uint32_t m2 = d.m2 != kNone ? min(rp[d.n], d.m2) : rp[d.n];
            const uint32_t lo = kPrepareRows * blockIdx.y, hi = min(d.n, lo + kPrepareRows);
            for (uint32_t v = lo + threadIdx.x / 32; v < hi; v += kPrepareThreads / 32)
                prepare_row<NW>(rp, cl, d.n, m2, v, rows[threadIdx.x / 32], A.adj + d.adj_off);
        }
    }
}

// ---------------------------------------------------------------- buffers
cudaError_t DevBuf::ensure(size_t bytes)
{
    if (bytes <= cap) return cudaSuccess;
    if (p) cudaFree(p);
    p = nullptr;
    cap = 0;
    size_t want = std::max<size_t>(bytes, 256);
    want = want + want / 4;
    cudaError_t e = cudaMalloc(&p, want);
    if (e != cudaSuccess) { p = nullptr; return e; }
    cap = want;
    return cudaSuccess;
}

void DevBuf::release()
{
    if (p) cudaFree(p);
    p = nullptr;
    cap = 0;
}

cudaError_t PinBuf::ensure(size_t bytes)
{
    if (bytes <= cap) return cudaSuccess;
    if (p) cudaFreeHost(p);
    p = nullptr;
    cap = 0;
    size_t want = std::max<size_t>(bytes, 4096);
    want = want + want / 4;
    cudaError_t e = cudaMallocHost(&p, want);
    if (e != cudaSuccess) { p = nullptr; return e; }
    cap = want;
    return cudaSuccess;
}

void PinBuf::release()
{
    if (p) cudaFreeHost(p);
    p = nullptr;
    cap = 0;
}

static std::mutex g_ctx_mu;
static Ctx *g_ctx[64];

Ctx *get_ctx(int dev, vc_status *err)
{
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) { *err = VC_ERR_NO_DEVICE; return nullptr; }
    if (dev < 0) {
        if (cudaGetDevice(&dev) != cudaSuccess) { *err = VC_ERR_CUDA; return nullptr; }
    }
    if (dev >= ndev || dev >= 64) { *err = VC_ERR_INVALID; return nullptr; }
    std::lock_guard<std::mutex> lk(g_ctx_mu);
    if (!g_ctx[dev]) {
        Ctx *c = new Ctx();
        c->dev = dev;
        if (cudaSetDevice(dev) != cudaSuccess) { delete c; *err = VC_ERR_CUDA; return nullptr; }
        cudaDeviceProp prop;
        if (cudaGetDeviceProperties(&prop, dev) != cudaSuccess) { delete c; *err = VC_ERR_CUDA; return nullptr; }
        c->sms = prop.multiProcessorCount;
        c->smem_optin = (int)prop.sharedMemPerBlockOptin;
        c->coop = prop.cooperativeLaunch;
        // VC_LANES=1 selects lane search units for graphs of at most 255 vertices
        if (const char *e = getenv("VC_LANES")) c->lanes_mode = atoi(e) ? 1 : 0;
        if (cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess ||
            cudaEventCreate(&c->ev0) != cudaSuccess || cudaEventCreate(&c->ev1) != cudaSuccess) {
            delete c;
            *err = VC_ERR_CUDA;
            return nullptr;
        }
        g_ctx[dev] = c;
    }
    if (cudaSetDevice(dev) != cudaSuccess) { *err = VC_ERR_CUDA; return nullptr; }
    *err = VC_OK;
    return g_ctx[dev];
}

// ---------------------------------------------------------------- sizing
// Resident CTAs per SM of `fn` with `smem` bytes of dynamic shared memory (0 on
// error).  The answer is a property of the kernel and the device: it is kept; the
// attribute is set every time, since a launch elsewhere may have lowered it.
template <unsigned NT, class F>
static int ctas_per_sm(Ctx &c, F fn, uint32_t smem)
{
    int per_sm = 0;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 0;
    std::lock_guard<std::mutex> lk(c.occ_mu);
    for (const Ctx::Occ &o : c.occ)
        if (o.fn == (const void *)fn && o.smem == smem) return o.per_sm;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, (int)NT, smem) != cudaSuccess) return 0;
    if (c.occ.size() < 256) c.occ.push_back({(const void *)fn, smem, per_sm});
    return per_sm;
}

template <unsigned NT, class F>
static cudaError_t plan_variant_fn(Ctx &c, Plan &pl, uint32_t smem_per_block, F fn)
{
    const int per_sm = ctas_per_sm<NT>(c, fn, smem_per_block);
    if (per_sm <= 0) return cudaErrorInvalidConfiguration;
    pl.fn = (const void *)fn;
    pl.block = NT;
    pl.grid = (uint32_t)per_sm * (uint32_t)c.sms;
    pl.smem = smem_per_block;
    return cudaSuccess;
}

// The CSR kernel for group G: team-walk kernels take the 80-register build
// when shared memory already holds the SM to as few CTAs (their row walks
// keep more values live than the lane walks).
template <class G, unsigned NT>
static cudaError_t plan_variant(Ctx &c, Plan &pl, uint32_t smem_per_block)
{
    if constexpr (G::kTeam) {
        auto roomy = k_search<G, NT, kRoomyThreadsPerSM>;
        const int r = ctas_per_sm<NT>(c, roomy, smem_per_block);
        if (r > 0 && r >= ctas_per_sm<NT>(c, k_search<G, NT>, smem_per_block))
            return plan_variant_fn<NT>(c, pl, smem_per_block, roomy);
    }
    return plan_variant_fn<NT>(c, pl, smem_per_block, k_search<G, NT>);
}

static uint32_t cta_pool_bytes(uint32_t slots, uint32_t stride)
{
    return slots ? 4u * ((slots + 3) / 4 * 4) + 4u * slots * stride : 0u;
}

// Chooses the search-unit shape for a vertex capacity np: one warp per SU with
// its workspace in shared memory for np <= kWarpMaxNP (up to 8 warps per CTA,
// sharing a CTA pool of 2 slots per warp), else one 512-thread CTA per SU, in
// shared memory while it fits, else in a global workspace.

template <int NW>
static cudaError_t plan_dense(Ctx &c, Plan &pl, const PlanOpts &o)
{
    const Tune *t = o.tune;
    pl.np = 32 * NW;
    pl.su_bytes = dense_workspace_bytes(NW);
    pl.stride = (4 + NW + 3) / 4 * 4;
    const uint32_t budget = (uint32_t)c.smem_optin - 1024;
    // search units sharing one staged graph: 8, and 4 for graphs of at most 255
    // vertices in a launch of their own, where a second copy of the rows leaves room
    // for as many units -- a CTA can go to another graph once all its units are idle
    // (512 graphs of 30..160 vertices 17.5 -> 15.5 ms; 2 units: 14.7, but 1024 graphs of
    // up to 200 vertices 121 -> 125 ms)
    uint32_t warps = (t && t->set) ? t->warps : (NW <= 8 && !o.lane ? VC_DENSE_WARPS : 8);
    const uint32_t per_warp = (t && t->set) ? t->pool : 2;
    // 32-word graphs (a 147 KB adjacency) step 8 -> 6 -> 4 warps, the others halve
    while (warps > 1 && dense_adj_bytes(NW) + warps * pl.su_bytes + cta_pool_bytes(per_warp * warps, pl.stride) > budget)
        warps = (NW == 32 && warps == 8) ? 6 : (warps == 6 ? 4 : warps >> 1);
    pl.cta_slots = warps > 1 ? per_warp * warps : 0;
    uint32_t smem = dense_adj_bytes(NW) + warps * pl.su_bytes + cta_pool_bytes(pl.cta_slots, pl.stride);
    cudaError_t e;
    switch (warps) {
    case 8:
        if constexpr (NW == 8) {
            e = o.lane ? plan_variant_fn<256>(c, pl, smem, k_dense<NW, 256, kLaneThreads>)
                       : plan_variant_fn<256>(c, pl, smem, k_dense<NW, 256>);
        } else {
            e = plan_variant_fn<256>(c, pl, smem, k_dense<NW, 256>);
        }
        break;
    case 6:
        if constexpr (NW == 32) e = plan_variant_fn<192>(c, pl, smem, k_dense<NW, 192>);
        else e = cudaErrorInvalidConfiguration;
        break;
    case 4:
        if constexpr (NW <= 8) {
            e = o.plain ? plan_variant_fn<128>(c, pl, smem, k_dense<NW, 128, kPlainThreads>)
                        : plan_variant_fn<128>(c, pl, smem, k_dense<NW, 128>);
        } else {
            e = plan_variant_fn<128>(c, pl, smem, k_dense<NW, 128>);
        }
        break;
    case 2: e = plan_variant_fn<64>(c, pl, smem, k_dense<NW, 64>); break;
    default: e = plan_variant_fn<32>(c, pl, smem, k_dense<NW, 32>); break;
    }
    if (e != cudaSuccess) return e;
    pl.num_su = pl.grid * (pl.block / 32);
    pl.global_ws = false;
    pl.dense = true;
    return cudaSuccess;
}

template <int NW>
static cudaError_t plan_lanes(Ctx &c, Plan &pl, uint32_t nmax)
{
    constexpr unsigned NT = VC_LANE_THREADS;
    const uint32_t nwc = std::max<uint32_t>(1, (nmax + 31) / 32);
    pl.np = 32 * nwc;
    pl.stride = (4 + NW + 3) / 4 * 4;
    pl.cta_slots = kLanePoolSlots;
    const LaneLayout lo(nwc, NW, NT, pl.cta_slots);
    pl.su_bytes = 4u * (17u * nwc);  // degree bytes, trail bytes, flag words per lane
    cudaError_t e = plan_variant_fn<NT>(c, pl, 4u * lo.words, k_lanes<NW, NT>);
    if (e != cudaSuccess) return e;
    pl.num_su = pl.grid * NT;
    pl.global_ws = false;
    pl.dense = true;
    pl.lanes = true;
    return cudaSuccess;
}

// Warp units, `warps` to a CTA.
template <class G>
static cudaError_t plan_warps(Ctx &c, Plan &pl, uint32_t warps, uint32_t smem)
{
    switch (warps) {
    case 8: return plan_variant<G, 256>(c, pl, smem);
    case 4: return plan_variant<G, 128>(c, pl, smem);
    case 2: return plan_variant<G, 64>(c, pl, smem);
    default: return plan_variant<G, 32>(c, pl, smem);
    }
}

cudaError_t make_plan(Ctx &c, uint32_t np, uint32_t nmax, Plan &pl, const PlanOpts &o)
{
    pl.dense = false;
    pl.lanes = false;
    if (o.lanes && !c.force_sparse && nmax <= 255) {
        if (nmax <= 64) return plan_lanes<2>(c, pl, nmax);
        if (nmax <= 128) return plan_lanes<4>(c, pl, nmax);
        return plan_lanes<8>(c, pl, nmax);
    }
    const uint32_t smem_budget = o.smem_budget, warp_max_np = o.warp_max_np;
    // dense bitsets up to 255 vertices, and up to 640 when every degree fits a
    // byte (degrees are bytes; 0 = removed or isolated)
    if (nmax <= 64 && !c.force_sparse) return plan_dense<2>(c, pl, o);
    if (nmax <= 128 && !c.force_sparse) return plan_dense<4>(c, pl, o);
    if (nmax <= 255 && !c.force_sparse) return plan_dense<8>(c, pl, o);
    if (nmax <= kWideMaxN && o.wide && !c.force_sparse) return plan_dense<20>(c, pl, o);
    if (nmax <= kHalfMaxN && o.half && !c.force_sparse)
        return nmax <= 512 ? plan_dense<16>(c, pl, o) : plan_dense<32>(c, pl, o);
    const Tune *t = (o.tune && o.tune->set && !c.force_sparse) ? o.tune : nullptr;
    pl.np = np;
    pl.su_bytes = su_workspace_bytes(np);
    pl.stride = (4 + np / 32 + 3) / 4 * 4;
    const uint32_t static_smem = 1024;  // reductions / broadcasts / CTA pool header
    uint32_t budget = (uint32_t)c.smem_optin - static_smem;
    if (smem_budget) budget = std::min(budget, smem_budget > static_smem ? smem_budget - static_smem : 0u);
    // a tuned choice: warp units (in shared memory where their workspaces fit,
    // else in global memory) or CTA units
    const bool tuned_warps = t && !t->cta_units;
    const bool tuned_cta = t && t->cta_units;
    const uint32_t per_warp = t ? t->pool : 2;
    const bool warp_gws = o.warp_gws || (tuned_warps && np > kWarpMaxNP);
    if (!tuned_cta && np <= (warp_max_np ? warp_max_np : (tuned_warps ? (1u << 16) : kWarpMaxNP)) && warp_gws) {
        // warp units with their workspaces in global memory: the CTA holds
        // only its pool
        uint32_t warps = t ? t->warps : (o.warps ? o.warps : 8);
        pl.cta_slots = warps > 1 ? per_warp * warps : 0;
        const uint32_t smem = cta_pool_bytes(pl.cta_slots, pl.stride);
        cudaError_t e = o.team ? plan_warps<TeamG<WarpG>>(c, pl, warps, smem) : plan_warps<WarpG>(c, pl, warps, smem);
        if (e != cudaSuccess) return e;
        pl.num_su = pl.grid * (pl.block / 32);
        pl.global_ws = true;
        return cudaSuccess;
    }
    if (!tuned_cta && np <= (warp_max_np ? warp_max_np : kWarpMaxNP)) {
        uint32_t warps = t ? t->warps : 8;
        while (warps > 1 && warps * pl.su_bytes + cta_pool_bytes(per_warp * warps, pl.stride) > budget) warps >>= 1;
        if (warps * pl.su_bytes + cta_pool_bytes(warps > 1 ? per_warp * warps : 0, pl.stride) <= budget) {
            pl.cta_slots = warps > 1 ? per_warp * warps : 0;
            uint32_t smem = warps * pl.su_bytes + cta_pool_bytes(pl.cta_slots, pl.stride);
            cudaError_t e = o.team ? plan_warps<TeamG<WarpG>>(c, pl, warps, smem) : plan_warps<WarpG>(c, pl, warps, smem);
            if (e != cudaSuccess) return e;
            pl.num_su = pl.grid * (pl.block / 32);
            pl.global_ws = false;
            return cudaSuccess;
        }
    }
    pl.cta_slots = 0;
    {
        const uint32_t smem = pl.su_bytes <= budget ? pl.su_bytes : 0u;
        cudaError_t e = o.team ? plan_variant<TeamG<BlockG<512>>, 512>(c, pl, smem)
                               : plan_variant<BlockG<512>, 512>(c, pl, smem);
        if (e != cudaSuccess) return e;
        pl.global_ws = smem == 0;
    }
    pl.num_su = pl.grid;
    return cudaSuccess;
}

// Caps a plan's persistent grid at `per_sm` CTAs per SM (a server lane that
// shares the device with another lane's kernel).
void cap_plan(const Ctx &c, Plan &pl, uint32_t per_sm)
{
    const uint32_t su_per_cta = pl.grid ? pl.num_su / pl.grid : 1;
    pl.grid = std::min(pl.grid, per_sm * (uint32_t)c.sms);
    pl.num_su = pl.grid * su_per_cta;
}

// k_check_csr over `count` graphs of at most nmax vertices.
cudaError_t launch_check(bool full, const uint32_t *rp, const uint32_t *cl, const InstDesc *inst, uint32_t *bad,
                                uint32_t stride, uint32_t value, uint32_t count, uint32_t nmax, cudaStream_t stream, uint32_t *mate)
{
    const uint32_t x = std::min<uint32_t>(count, 4096);
    const dim3 grid(x, std::max<uint32_t>(1, std::min<uint32_t>((nmax + 7) / 8, 4096 / x)));
    void *args[] = {&rp, &cl, &inst, &bad, &stride, &value, &count, &mate};
    return cudaLaunchKernel(full ? (const void *)k_check_csr<true> : (const void *)k_check_csr<false>, grid, dim3(256), args, 0,
                            stream);
}

// The kernel that readies a launch (k_prepare) for bitmap rows of nw words, 0 = none.
static cudaError_t launch_prepare(uint32_t nw, uint32_t nmax, const PrepareArgs &A, cudaStream_t stream)
{
    // rows: 32 per block, a column of blocks per graph; and blocks for the longest list
    const uint32_t longest = std::max(std::max(A.q, A.cover_words), std::max<uint32_t>(A.count, kCtlWords));
    const uint32_t lists = std::min<uint32_t>((longest + kPrepareThreads - 1) / kPrepareThreads, 64u);
    const dim3 grid =
        nw ? dim3(std::min<uint32_t>(A.count, 1u << 20), std::max((nmax + kPrepareRows - 1) / kPrepareRows, lists / A.count))
           : dim3(lists);
    const void *fn = nullptr;
    switch (nw) {
    case 0: fn = (const void *)k_prepare<0>; break;
    case 2: fn = (const void *)k_prepare<2>; break;
    case 4: fn = (const void *)k_prepare<4>; break;
    case 8: fn = (const void *)k_prepare<8>; break;
    case 16: fn = (const void *)k_prepare<16>; break;
    case 20: fn = (const void *)k_prepare<20>; break;
    case 32: fn = (const void *)k_prepare<32>; break;
    default: return cudaErrorInvalidValue;
    }
    void *args[] = {const_cast<PrepareArgs *>(&A)};
    return cudaLaunchKernel(fn, grid, dim3(kPrepareThreads), args, 0, stream);
}

// When a plain solve's units take up the packing bound (vc_dense.cuh): at once,
// except on the graphs of 129 to 255 vertices with 768 edges or more, after 25 ms.
// Without the bound those trees take tens of ms to minutes and with it they take
// milliseconds (the batched workload's graph of 166 vertices and 865 edges: 77 and
// 5.7 ms), but a solve of that graph limited to 20 ms has to run out of time --
// the suite holds the time limit to that -- so what such a graph costs is 25 ms
// more than it could.  Batches and servers use the bound from the start.
static unsigned long long pack_after(const InstDesc &d)
{
    return d.n > 128 && d.n <= 255 && d.m2 != kNone && d.m2 >= 2 * 768 ? 25000000ull : 0ull;
}

// ---------------------------------------------------------------- one launch
// Runs every graph of `job` (arena already on the device) to completion and
// copies back the per-graph state and cover bitmaps.
vc_status run_job(Ctx &c, Job &job, cudaStream_t stream)
{
    const uint32_t count = (uint32_t)job.desc.size();
    if (count == 0) return VC_OK;
    uint32_t nmax = 0, cover_words = 0;
    uint64_t sum_n = 0, sum_m2 = 0;
    for (auto &d : job.desc) {
        nmax = std::max(nmax, d.n);
        d.cover_off = cover_words;
        cover_words += d.nw;
        if (d.m2 != kNone) { sum_n += d.n; sum_m2 += d.m2; }
    }
    uint32_t np = std::max<uint32_t>(32, (nmax + 31) / 32 * 32);
    Plan pl;
    PlanOpts po;
    po.wide = job.wide;
    po.half = job.half;
    po.plain = count == 1;
    po.team = sum_m2 >= 4 * sum_n && sum_n > 0;  // average degree 4 or more: rows walked by teams
    // Lane units (one thread per search unit, vc_lanes.cuh) are opt-in: they
    // execute half the instructions per tree node of warp units but, at 12
    // resident warps per SM, issue on a fifth of the cycles (ncu, batched
    // workload) and reach a quarter of the warp units' node rate.
    po.lanes = c.lanes_mode == 1;
    const Tune *tn = job.tune ? job.tune : &c.tune[tune_class(nmax, job.wide)];
    po.tune = tn->set ? tn : nullptr;
    if (make_plan(c, np, nmax, pl, po) != cudaSuccess) return VC_ERR_CUDA;
    const uint32_t stride = pl.stride;
    uint32_t q = 1024;
    const uint32_t ring_units = pl.lanes ? pl.grid : pl.num_su;  // lane CTAs poll the ring as a whole
    while (q < 2 * ring_units) q <<= 1;
    const size_t ring_cap_bytes = (size_t)512 << 20;
    while (q > 64 && (size_t)q * stride * 4 > ring_cap_bytes) q >>= 1;

    size_t gws_bytes = pl.global_ws ? (size_t)pl.num_su * pl.su_bytes : 0;
    // One piece in (the descriptors, with a small host-resident graph) and one out
    // (control words, states, covers), each mirrored in pinned memory: one copy each.
    const size_t also_at = sizeof(InstDesc) * (size_t)count, rp_at = also_at + sizeof(InstDesc) * job.others.size();
    const size_t col_at = rp_at + (job.h_rp ? 4ull * (job.desc[0].n + 1) : 0);
    const size_t in_bytes = col_at + (job.h_rp ? 4ull * job.desc[0].m2 : 0);
    const size_t st_at = sizeof(unsigned long long) * kCtlWords, covers_at = st_at + sizeof(InstState) * (size_t)count;
    const size_t out_bytes = covers_at + sizeof(uint32_t) * (size_t)cover_words;
    if (c.in.ensure(in_bytes) || c.out.ensure(out_bytes) || c.seq.ensure(sizeof(unsigned long long) * q) ||
        c.data.ensure((size_t)q * stride * 4) || (gws_bytes && c.gws.ensure(gws_bytes)))
        return VC_ERR_NOMEM;
    if (c.h_in.ensure(in_bytes) || c.h_out.ensure(out_bytes)) return VC_ERR_NOMEM;
    uint8_t *d_in = (uint8_t *)c.in.p, *d_out = (uint8_t *)c.out.p;
    if (job.h_rp) {
        job.d_rp = (const uint32_t *)(d_in + rp_at);
        job.d_col = (const uint32_t *)(d_in + col_at);
    }

    // bitmap rows for the dense kernels, up to a bound on what they take (above it
    // the search units make them from the CSR when they stage a graph)
    const uint32_t nw = pl.dense && !pl.lanes ? pl.np / 32 : 0;
    uint64_t adj_words = 0;
    if (nw) {
        for (auto &d : job.desc) {
            d.adj_off = adj_words;
            adj_words += ((uint64_t)d.n * dense_row_words(nw) + 3) / 4 * 4;
        }
        if (4 * adj_words > kAdjBytesMax || c.adj.ensure(4 * adj_words)) adj_words = 0;
    }
    {
        uint8_t *h = (uint8_t *)c.h_in.p;
        memcpy(h, job.desc.data(), sizeof(InstDesc) * count);
        memcpy(h + also_at, job.others.data(), rp_at - also_at);
        if (job.h_rp) {
            memcpy(h + rp_at, job.h_rp, col_at - rp_at);
            if (in_bytes > col_at) memcpy(h + col_at, job.h_col, in_bytes - col_at);
        }
        cudaMemcpyAsync(d_in, h, in_bytes, cudaMemcpyHostToDevice, stream);
    }
    PrepareArgs A;
    A.ctl = (unsigned long long *)d_out;
    A.seq = (unsigned long long *)c.seq.p;
    A.q = q;
    A.covers = (uint32_t *)(d_out + covers_at);
    A.cover_words = cover_words;
    A.st = (InstState *)(d_out + st_at);
    A.inst = (const InstDesc *)d_in;
    A.count = count;
    const uint32_t split = count == 1 && nw ? split_roots(job.desc[0].n, job.desc[0].m2) : 0u;
    A.roots = split ? split : 1u;
    A.row_ptr = job.d_rp;
    A.col = job.d_col;
    A.adj = adj_words ? (uint32_t *)c.adj.p : nullptr;
    cudaEventRecord(c.ev0, stream);
    if (launch_prepare(adj_words ? nw : 0, nmax, A, stream) != cudaSuccess) return VC_ERR_CUDA;
    g_launches += 1;
    if (job.check) {
        const bool all = job.check == 2;
        uint32_t most = nmax;
        for (const auto &d : job.others) most = std::max(most, d.n);
        if (launch_check(all, job.d_rp, job.d_col, A.inst, all ? (uint32_t *)&A.ctl[kAbort] : &A.st->flags,
                         all ? 0u : sizeof(InstState) / 4, all ? (uint32_t)kStopInput : kBadGraph,
                         count + (uint32_t)job.others.size(), most, stream) != cudaSuccess)
            return VC_ERR_CUDA;
        g_launches += 1;
    }

    Params P;
    memset(&P, 0, sizeof(P));
    P.row_ptr = job.d_rp;
    P.col = job.d_col;
    P.inst = A.inst;
    P.st = A.st;
    P.covers = A.covers;
    P.adj = A.adj;
    P.count = count;
    P.num_su = pl.num_su;
    P.ctl = A.ctl;
    P.pool_seq = (unsigned long long *)c.seq.p;
    P.pool_data = (uint32_t *)c.data.p;
    P.q_mask = q - 1;
    P.stride = stride;
    P.np = np;
    P.su_bytes = pl.su_bytes;
    P.cta_slots = pl.cta_slots;
    P.gws = pl.global_ws ? (uint8_t *)c.gws.p : nullptr;
    P.stats = nullptr;
    if (c.stats_on) {
        if (c.stats.ensure(sizeof(unsigned long long) * kStatWords * pl.num_su)) return VC_ERR_NOMEM;
        cudaMemsetAsync(c.stats.p, 0, sizeof(unsigned long long) * kStatWords * pl.num_su, stream);
        P.stats = (unsigned long long *)c.stats.p;
    }
    double tl = job.time_limit_s > 0 ? job.time_limit_s : 300.0;
    P.time_limit_ns = (unsigned long long)(tl * 1e9);
    P.pack_after_ns = count == 1 ? pack_after(job.desc[0]) : 0ull;
    P.split = split;
    P.dives = !split && count == 1 && job.desc[0].m2 / 16 <= job.desc[0].n;
    P.ring_bias = po.tune ? po.tune->ring_bias : 0;
    P.ring_first = po.tune ? po.tune->ring_first : 0u;

    void *args[] = {&P};
    cudaError_t e = c.coop ? cudaLaunchCooperativeKernel(pl.fn, dim3(pl.grid), dim3(pl.block), args, pl.smem, stream)
                           : cudaErrorNotSupported;
    if (e != cudaSuccess) return VC_ERR_CUDA;
    g_launches += 1;
    cudaEventRecord(c.ev1, stream);
    cudaMemcpyAsync(c.h_out.p, d_out, out_bytes, cudaMemcpyDeviceToHost, stream);
    if (cudaStreamSynchronize(stream) != cudaSuccess) return VC_ERR_CUDA;
    const uint8_t *h_out = (const uint8_t *)c.h_out.p;
    const unsigned long long *h_ctl = (const unsigned long long *)h_out;
    job.t0 = h_ctl[kT0];
    cudaEventElapsedTime(&job.kernel_ms, c.ev0, c.ev1);
    job.stopped = h_ctl[kAbort];
    if (job.stopped == kStopInput) return VC_ERR_INVALID;
    job.st.assign((const InstState *)(h_out + st_at), (const InstState *)(h_out + st_at) + count);
    job.covers.assign((const uint32_t *)(h_out + covers_at), (const uint32_t *)(h_out + covers_at) + cover_words);
    job.plan = pl;
    if (c.stats_on) {
        c.last_stats.resize((size_t)kStatWords * pl.num_su);
        cudaMemcpy(c.last_stats.data(), c.stats.p, sizeof(unsigned long long) * kStatWords * pl.num_su,
                   cudaMemcpyDeviceToHost);
        c.last_num_su = pl.num_su;
    }
    c.last_plan = pl;
    return VC_OK;
}

// The bound a request's search starts from: covers smaller than this.
static uint32_t init_best_for(const vc_request *r, uint32_t n)
{
    if (r->instance == VC_PVC) return n + 1;
    uint32_t ub = r->ub ? std::min<uint32_t>(r->ub, n) : n;
    return ub + 1;
}

// Size, decision and cover of a graph of n vertices: `found` is the size of the
// cover found (kNone: none), `mask` writes it.
template <class F>
static void fill_answer(const vc_request *req, uint32_t n, uint32_t found, vc_result *out, F mask)
{
    if (req->instance == VC_PVC) {
        out->decision = found != kNone ? 1u : 0u;
        out->size = found != kNone ? found : 0u;
    } else {
        out->decision = 1;
        out->size = found != kNone ? found : (req->ub ? req->ub : n);  // none below the bound: min(ub, OPT) = ub
    }
    out->has_cover = found != kNone ? 1u : 0u;
    if (out->cover_mask) {
        if (found != kNone) mask(out->cover_mask);
        else memset(out->cover_mask, 0, n);
    }
}

// Fills one vc_result, of a graph of n vertices, from the collected state of
// graph i of a job: that graph, or the rest of its reduction.
vc_status fill_result(const Job &job, uint32_t i, const vc_request *req, uint32_t n, vc_result *out)
{
    const InstDesc &d = job.desc[i];
    const InstState &s = job.st[i];
    const Reduce *red = job.rest.empty() ? nullptr : job.rest[i];
    const uint32_t taken = red ? red->h.taken : 0u;
    vc_status st;
    if (s.flags & kBadGraph) st = VC_ERR_INVALID;
    else if (s.flags & kError) st = VC_ERR_INTERNAL;
    else if (s.flags & kBudget) st = VC_BUDGET;
    else if ((s.flags & kCut) || !(s.flags & kDone)) st = stopped_status(job.stopped);
    else st = VC_OK;
    out->status = st;
    out->tree_nodes = s.nodes;
    out->kernel_ms = job.kernel_ms;
    out->done_ms = (s.t_done && job.t0 && s.t_done >= job.t0) ? (float)((s.t_done - job.t0) * 1e-6) : 0.0f;
    const uint32_t found = s.cover_size != kNone ? taken + s.cover_size : kNone;
    fill_answer(req, n, found, out, [&](uint8_t *mask) {
        const uint32_t *w = job.covers.data() + d.cover_off;
        if (red) {
            memcpy(mask, red->h_cover, n);
            for (uint32_t v = 0; v < d.n; ++v)
                if ((w[v >> 5] >> (v & 31u)) & 1u) mask[red->h_inv[v]] = 1;
        } else {
            for (uint32_t v = 0; v < d.n; ++v) mask[v] = (uint8_t)((w[v >> 5] >> (v & 31u)) & 1u);
        }
    });
    return st;
}

// ---------------------------------------------------------------- large graphs
// How large graphs (largest first) are reduced: the first `chip` by the whole chip, one
// after another, those up to `near` by a cluster of CTAs each in one launch, the others
// by one CTA each in another.  Kernel times of one power-law graph, its check included
// (us; a pass takes the same share of each):
//   vertices            1,500  3,000  6,000  12,000  24,000  100,000
//   whole chip            125    116    136     154     167      220
//   a cluster of 8                              270     380     1330
//   one CTA                78     82    126     228     416
// A pass of the chip is two grid barriers and four dependent reads from L2 whatever the
// size; one CTA's are barriers of its own and shared memory, but it walks all vertices;
// and 148 CTAs, or 37 clusters, run side by side.  The line between the chip and one
// CTA for a graph by itself is at 7,400 vertices.  The chip alone (and launches one after
// another in a batch) had made cascades and batches slower than the search's own units
// are at a root: a path of 1500 vertices 0.87 -> 2.3 ms, now 0.60; 1000 graphs of 1100
// to 4000 vertices on the device, planted and power-law, 2.4 -> 69 and 125 ms, now 0.86
// and 1.3; one of 100,000 vertices beside 256 of them 12 -> 17, now 0.48.
constexpr uint32_t kNearMax = 24576;  // vertices that one CTA's shared memory holds
struct ReduceSplit {
    uint32_t chip, near;
};
static ReduceSplit split_reductions(const std::vector<Reduce> &reds, uint32_t sms)
{
    const uint32_t count = (uint32_t)reds.size();
    uint32_t near = 0;
    while (near < count && reds[near].n > kNearMax) ++near;
    ReduceSplit best{count, count};
    auto on_chip = [](uint32_t n) { return 150.0 + 0.0007 * n; };
    double chip = 0;
    for (const Reduce &r : reds) chip += on_chip(r.n);
    double most[2] = {0, 0}, sum[2] = {0, 0}, least = chip;
    for (uint32_t k = count; k-- > 0;) {  // the first k get the chip
        const bool one = k >= near;
        const double t = one ? 30.0 + 0.0162 * reds[k].n : 110.0 + 0.0112 * reds[k].n;
        most[one] = std::max(most[one], t);
        sum[one] += t / (one ? sms : sms / 4);
        chip -= on_chip(reds[k].n);
        const double all = chip + std::max(most[0], sum[0]) + std::max(most[1], sum[1]);
        if (all < least) { least = all; best = {k, std::max(k, near)}; }
    }
    return best;
}

// Checks and reduces the graphs (largest first) at their roots; the answers come back
// in their heads and covers (one synchronisation).  Their rows are in rp and cl.  With
// check 2 the call's other graphs are checked too, and one that fails stops every
// reduction: VC_ERR_INVALID.
static vc_status run_reductions(Ctx &c, std::vector<Reduce> &reds, int check, const uint32_t *rp, const uint32_t *cl,
                                const std::vector<InstDesc> &others, cudaStream_t stream, float *ms)
{
    const uint32_t count = (uint32_t)reds.size(), ctas = reduce_ctas(c);
    const ReduceSplit split = split_reductions(reds, (uint32_t)c.sms);
    size_t words = 0;
    auto take = [&](size_t n) {  // 16-byte pieces
        const size_t at = words;
        words += (n + 3) / 4 * 4;
        return at;
    };
    // one piece that goes in, one that comes back (the new ids only where there is a
    // search to follow), and scratch
    const uint32_t checked = count + (check == 2 ? (uint32_t)others.size() : 0u);
    const size_t descs = take(checked * sizeof(InstDesc) / 4), list = take(count * sizeof(ReduceArgs) / 4), in_words = words;
    const size_t heads = take(count * sizeof(ReduceHead) / 4);
    std::vector<size_t> cover_at, inv_at, at;
    for (const Reduce &r : reds) cover_at.push_back(take((r.n + 3) / 4));
    const size_t back_words = words - heads;
    for (const Reduce &r : reds) inv_at.push_back(take(r.n));
    const size_t pinned = words;
    for (const Reduce &r : reds) {
        at.push_back(take(4ull * r.n + 1 + 2ull * ctas));
        at.push_back(take(r.m2));
    }
    if (c.red.ensure(4 * words) || c.h_red.ensure(4 * pinned)) return VC_ERR_NOMEM;
    uint32_t *base = (uint32_t *)c.red.p, *h = (uint32_t *)c.h_red.p;
    InstDesc *h_desc = (InstDesc *)(h + descs);
    ReduceArgs *h_list = (ReduceArgs *)(h + list);
    ReduceHead *d_head = (ReduceHead *)(base + heads), *h_head = (ReduceHead *)(h + heads);
    for (uint32_t i = 0; i < count; ++i) {
        Reduce &r = reds[i];
        uint32_t *p = base + at[2 * i];
        r.deg = (int32_t *)p;
        r.taken = p + r.n;
        r.map = p + 2ull * r.n;
        r.rrp = p + 3ull * r.n;
        r.part = p + 4ull * r.n + 1;
        r.rcl = base + at[2 * i + 1];
        r.inv = base + inv_at[i];
        r.cover = (uint8_t *)(base + cover_at[i]);
        r.head = d_head + i;
        r.bad = &d_head[check == 2 ? 0 : i].bad;
        r.h_inv = h + inv_at[i];
        r.h_cover = (const uint8_t *)(h + cover_at[i]);
        h_list[i] = r;
        InstDesc d{};
        d.n = r.n;
        d.m2 = r.m2;
        d.row_off = (uint64_t)(r.rp - rp);
        d.col_off = (uint64_t)(r.cl - cl);
        h_desc[i] = d;
    }
    uint32_t others_n = 0;
    for (uint32_t i = count; i < checked; ++i) {
        h_desc[i] = others[i - count];
        others_n = std::max(others_n, h_desc[i].n);
    }
    bool ok = cudaMemsetAsync(d_head, 0, count * sizeof(ReduceHead), stream) == cudaSuccess &&
              cudaMemcpyAsync(base, h, 4 * in_words, cudaMemcpyHostToDevice, stream) == cudaSuccess;
    cudaEventRecord(c.ev0, stream);
    auto check_from = [&](uint32_t i, uint32_t end, uint32_t nmax) {  // graphs i .. end - 1 of the list
        const uint32_t k = end - i;
        if (!check || k == 0) return;
        ok = ok && launch_check(check == 2, rp, cl, (const InstDesc *)(base + descs) + i, &d_head[check == 2 ? 0 : i].bad,
                                check == 2 ? 0u : sizeof(ReduceHead) / 4, 1u, k, nmax, stream) == cudaSuccess;
        g_launches += 1;
    };
    // (a launch's blocks are as many for each of its graphs)
    for (uint32_t i = 0; i < split.chip; ++i) check_from(i, i + 1, reds[i].n);
    if (split.chip < split.near) check_from(split.chip, split.near, reds[split.chip].n);
    if (split.near < count) check_from(split.near, count, reds[split.near].n);
    check_from(count, checked, others_n);
    for (uint32_t i = 0; ok && i < split.chip; ++i) {
        ok = launch_reduce(reds[i], ctas, stream) == cudaSuccess;
        g_launches += 1;
    }
    const ReduceArgs *d_list = (const ReduceArgs *)(base + list);
    if (split.chip < split.near) {
        ok = ok && launch_reduce_many(d_list + split.chip, split.near - split.chip, stream) == cudaSuccess;
        g_launches += 1;
    }
    if (split.near < count) {
        ok = ok && launch_reduce_each(d_list + split.near, count - split.near, reds[split.near].n, stream) == cudaSuccess;
        g_launches += 1;
    }
    cudaEventRecord(c.ev1, stream);
    ok = ok && cudaMemcpyAsync(h_head, d_head, 4 * back_words, cudaMemcpyDeviceToHost, stream) == cudaSuccess;
    if (cudaStreamSynchronize(stream) != cudaSuccess || !ok) return VC_ERR_CUDA;
    cudaEventElapsedTime(ms, c.ev0, c.ev1);
    for (uint32_t i = 0; i < count; ++i) reds[i].h = h_head[i];
    Plan pl;  // what vc_debug_stats reports if there is nothing left to search
    pl.block = 512;
    pl.grid = std::min<uint32_t>((reds[0].n + pl.block - 1) / pl.block, ctas);
    pl.np = (reds[0].n + 31) / 32 * 32;
    c.last_plan = pl;
    c.last_num_su = 0;
    c.last_stats.clear();
    return check == 2 && h_head[0].bad ? VC_ERR_INVALID : VC_OK;
}

// The new ids of the rests that are searched, for fill_result (part of the next
// synchronisation): a copy each, or one of all where they are many.
static void fetch_new_ids(const std::vector<Reduce> &reds, const std::vector<uint8_t> &searched, cudaStream_t stream)
{
    if (std::count(searched.begin(), searched.end(), 1) > 8) {
        const Reduce &a = reds.front(), &z = reds.back();
        cudaMemcpyAsync(a.h_inv, a.inv, 4ull * (z.inv - a.inv + z.n), cudaMemcpyDeviceToHost, stream);
        return;
    }
    for (size_t j = 0; j < reds.size(); ++j)
        if (searched[j]) cudaMemcpyAsync(reds[j].h_inv, reds[j].inv, 4ull * reds[j].h.n, cudaMemcpyDeviceToHost, stream);
}

// The search a reduction leaves to do: false if there is none (out's answer is
// filled in), else `d` describes the rest.
static bool rest_of(const Reduce &r, const vc_request *req, float ms, InstDesc &d, vc_result *out)
{
    const uint32_t limit = req->instance == VC_PVC ? std::min<uint32_t>(req->k, r.n) : init_best_for(req, r.n) - 1;
    if (r.h.n == 0 || r.h.taken > limit) {
        out->status = VC_OK;
        out->tree_nodes = 1;
        out->kernel_ms = ms;
        out->done_ms = ms;
        fill_answer(req, r.n, r.h.taken <= limit ? r.h.taken : kNone, out, [&](uint8_t *m) { memcpy(m, r.h_cover, r.n); });
        return false;
    }
    d.n = r.h.n;
    d.nw = (d.n + 31) / 32;
    d.mode = req->instance == VC_PVC ? kModePVC : kModeMVC;
    d.k = std::min(limit - r.h.taken, d.n);
    d.init_best = req->instance == VC_PVC ? d.n + 1 : d.k + 1;
    d.node_limit = req->node_limit;
    d.m2 = r.h.m2;
    return true;
}

// A context keeps the buffers of reductions up to these sizes.
static void trim_reductions(Ctx &c)
{
    if (c.red.cap > (1ull << 30)) c.red.release();
    if (c.h_red.cap > (256ull << 20)) c.h_red.release();
}

}  // namespace vch

// ---------------------------------------------------------------- C ABI
using namespace vch;

extern "C" const char *vc_status_string(vc_status s)
{
    switch (s) {
    case VC_OK: return "ok";
    case VC_ERR_INVALID: return "invalid argument";
    case VC_ERR_CUDA: return "CUDA error";
    case VC_ERR_NOMEM: return "out of device memory";
    case VC_ERR_TOO_LARGE: return "graph too large";
    case VC_TIMEOUT: return "time limit reached";
    case VC_BUDGET: return "node limit reached";
    case VC_ERR_INTERNAL: return "internal error";
    case VC_ERR_NO_DEVICE: return "no CUDA device";
    case VC_PENDING: return "pending";
    }
    return "unknown";
}

extern "C" uint64_t vc_kernel_launches(void) { return g_launches.load(); }

// Diagnostics (not part of the reference surface): enable (bit 0)
// per-search-unit counters on a device, force the CSR kernel (bit 1) or lane
// search units (bit 2) for graphs of at most 255 vertices, and read the last launch's counters as rows of
// kStatWords u64 (nodes, passes, donations, failed donations, receives, roots,
// busy cycles, idle cycles, polls, restored vertices, SM id).  Returns the
// number of search units; copies at most max_rows rows.
extern "C" uint32_t vc_debug_stats(int32_t device, int32_t enable, uint64_t *rows, uint32_t max_rows,
                                   uint32_t *launch_shape)
{
    vch::DeviceGuard dg;
    vc_status err;
    Ctx *c = get_ctx(device, &err);
    if (!c) return 0;
    std::lock_guard<std::mutex> lk(c->mu);
    if (enable >= 0) c->stats_on = (enable & 1) != 0;
    if (enable >= 0) c->force_sparse = (enable & 2) != 0;
    if (enable >= 0) c->lanes_mode = (enable & 4) ? 1 : 0;
    uint32_t nsu = c->last_num_su;
    if (rows) {
        // rows exist only for a launch that ran with the counters on
        uint32_t k = std::min(nsu, max_rows);
        k = std::min<uint32_t>(k, (uint32_t)(c->last_stats.size() / kStatWords));
        memcpy(rows, c->last_stats.data(), sizeof(uint64_t) * kStatWords * k);
    }
    if (launch_shape) {
        launch_shape[0] = c->last_plan.grid;
        launch_shape[1] = c->last_plan.block;
        launch_shape[2] = c->last_plan.smem;
        launch_shape[3] = c->last_plan.num_su;
        launch_shape[4] = c->last_plan.np | (c->last_plan.dense ? 0x80000000u : 0u);
    }
    return nsu;
}

// Host-resident graphs of more entries than this are checked on the device: a
// launch costs what the host takes for about so many.
constexpr uint64_t kHostCheckEntries = 2048;

extern "C" vc_status vc_solve(const vc_csr *g, const vc_request *req, vc_result *out)
{
    vch::DeviceGuard dg;
    auto t0 = std::chrono::steady_clock::now();
    if (!g || !req || !out) return VC_ERR_INVALID;
    if (req->instance != VC_MVC && req->instance != VC_PVC) return VC_ERR_INVALID;
    const bool dev_in = (req->flags & VC_FLAG_DEVICE_INPUT) != 0;
    const bool validate = !dev_in && !(req->flags & VC_FLAG_NO_VALIDATE);
    const bool on_device = validate && 2ull * g->m > kHostCheckEntries;  // the rest of the checks
    if (validate) {
        vc_status v = on_device ? check_head(g) : validate_csr(g);
        if (v != VC_OK) return v;
    } else if (!g->row_ptr || (g->m && !g->col)) {
        return VC_ERR_INVALID;
    }
    out->size = 0;
    out->decision = 0;
    out->has_cover = 0;
    out->tree_nodes = 0;
    out->kernel_ms = 0;
    if (g->n == 0) {
        out->status = VC_OK;
        out->decision = 1;
        out->has_cover = 1;
        out->total_ms = 0;
        return VC_OK;
    }
    if (g->n > kMaxVertices) return on_device && validate_csr(g) != VC_OK ? VC_ERR_INVALID : VC_ERR_TOO_LARGE;
    vc_status err;
    Ctx *c = get_ctx(req->device, &err);
    if (!c) return on_device && validate_csr(g) != VC_OK ? VC_ERR_INVALID : err;
    std::lock_guard<std::mutex> lk(c->mu);
    cudaStream_t stream = req->stream ? (cudaStream_t)req->stream : c->stream;

    // a large graph: its root is reduced by the whole chip, the search gets the rest
    const bool large = g->n > kHalfMaxN && !c->force_sparse && 2ull * g->m < kNone;
    const size_t rp_b = sizeof(uint32_t) * ((size_t)g->n + 1), col_b = sizeof(uint32_t) * 2 * (size_t)g->m;
    Job job;
    if (dev_in) {
        job.d_rp = g->row_ptr;
        job.d_col = g->col;
    } else if (!large && rp_b + col_b <= kSmallGraphBytes) {
        job.h_rp = g->row_ptr;
        job.h_col = g->col;
    } else {
        if (c->rp.ensure(rp_b) || c->col.ensure(std::max<size_t>(col_b, 4))) return VC_ERR_NOMEM;
        cudaMemcpyAsync(c->rp.p, g->row_ptr, rp_b, cudaMemcpyHostToDevice, stream);
        if (g->m) cudaMemcpyAsync(c->col.p, g->col, col_b, cudaMemcpyHostToDevice, stream);
        job.d_rp = (const uint32_t *)c->rp.p;
        job.d_col = (const uint32_t *)c->col.p;
    }
    job.check = dev_in ? 1 : (on_device ? 2 : 0);
    job.time_limit_s = req->time_limit_s;
    InstDesc d{};
    float reduce_ms = 0;
    std::vector<Reduce> red;
    if (large) {
        Reduce r;
        r.rp = job.d_rp;
        r.cl = job.d_col;
        r.n = g->n;
        r.m2 = 2 * g->m;
        r.bound = req->instance == VC_PVC ? std::min<uint32_t>(req->k, g->n) + 1 : init_best_for(req, g->n);
        red.push_back(r);
        const vc_status s = run_reductions(*c, red, job.check, r.rp, r.cl, {}, stream, &reduce_ms);
        if (s == VC_ERR_NOMEM || (s == VC_OK && red[0].h.uneven)) {
            red.clear();  // no room for it, or no graph: the search reduces the root itself
        } else {
            const bool bad = s == VC_OK && red[0].h.bad;
            if (s != VC_OK || bad) {
                out->status = bad ? VC_ERR_INVALID : s;
                trim_reductions(*c);
                return out->status;
            }
            if (!rest_of(red[0], req, reduce_ms, d, out)) {
                trim_reductions(*c);
                out->total_ms = std::chrono::duration<float, std::milli>(std::chrono::steady_clock::now() - t0).count();
                return VC_OK;
            }
            job.d_rp = red[0].rrp;
            job.d_col = red[0].rcl;
            job.check = 0;
            job.rest.push_back(&red[0]);
            fetch_new_ids(red, {1}, stream);
            job.wide = d.n <= kWideMaxN && red[0].h.maxd <= 254;
        }
    }
    if (red.empty()) {
        d.n = g->n;
        d.nw = (g->n + 31) / 32;
        d.mode = req->instance == VC_PVC ? kModePVC : kModeMVC;
        d.k = std::min<uint32_t>(req->k, g->n);
        d.init_best = init_best_for(req, g->n);
        d.node_limit = req->node_limit;
        d.m2 = 2ull * g->m < (uint64_t)kNone ? (uint32_t)(2ull * g->m) : kNone;
        job.wide = !dev_in && wide_ok(g->n, g->row_ptr);
    }
    job.half = !job.wide && half_ok(d.n);
    job.desc.push_back(d);
    vc_status s = run_job(*c, job, stream);
    if (s == VC_OK && (job.st[0].flags & kBadGraph)) s = VC_ERR_INVALID;
    if (s != VC_OK) { out->status = s; return s; }
    s = fill_result(job, 0, req, g->n, out);
    out->kernel_ms += reduce_ms;
    out->done_ms += reduce_ms;
    trim_reductions(*c);
    out->total_ms = std::chrono::duration<float, std::milli>(std::chrono::steady_clock::now() - t0).count();
    return s;
}

extern "C" vc_status vc_solve_batch(const vc_csr_arena *a, const vc_request *reqs, vc_result *out)
{
    vch::DeviceGuard dg;
    auto t0 = std::chrono::steady_clock::now();
    if (!a || !reqs || !out) return VC_ERR_INVALID;
    if (a->count == 0) return VC_OK;
    if (!a->n || !a->row_off || !a->col_off || !a->row_ptr) return VC_ERR_INVALID;
    const bool dev_in = (reqs[0].flags & VC_FLAG_DEVICE_INPUT) != 0;
    for (uint32_t i = 1; i < a->count; ++i)
        if (((reqs[i].flags & VC_FLAG_DEVICE_INPUT) != 0) != dev_in) return VC_ERR_INVALID;
    if (dev_in) return VC_ERR_INVALID;  // per-graph sizes are read on the host: use vc_solve_batch_device
    return vc_solve_batch_impl(a, reqs, out, nullptr, nullptr, t0);
}

namespace vch {
vc_status vc_solve_batch_impl(const vc_csr_arena *a, const vc_request *reqs, vc_result *out, const uint32_t *d_rp,
                              const uint32_t *d_col, std::chrono::steady_clock::time_point t0)
{
    const uint32_t count = a->count;
    // every early failure is reported in each graph's result too
    auto fail = [&](vc_status st) {
        for (uint32_t i = 0; i < count; ++i) {
            out[i].status = st;
            out[i].size = 0;
            out[i].decision = 0;
            out[i].has_cover = 0;
            out[i].tree_nodes = 0;
        }
        return st;
    };
    uint64_t rows = 0, cols = 0;
    for (uint32_t i = 0; i < count; ++i) {
        if (reqs[i].instance != VC_MVC && reqs[i].instance != VC_PVC) return fail(VC_ERR_INVALID);
        if (a->n[i] > kMaxVertices) return fail(VC_ERR_TOO_LARGE);
        rows = std::max<uint64_t>(rows, a->row_off[i] + a->n[i] + 1);
    }
    for (uint32_t i = 0; i < count; ++i) {
        const uint32_t *rp = a->row_ptr + a->row_off[i];
        cols = std::max<uint64_t>(cols, a->col_off[i] + rp[a->n[i]]);
    }
    const bool validate = !d_rp && !(reqs[0].flags & VC_FLAG_NO_VALIDATE);
    const bool on_device = validate && cols > kHostCheckEntries;
    auto host_checks = [&](bool all) {
        for (uint32_t i = 0; i < count; ++i) {
            vc_csr g;
            g.n = a->n[i];
            const uint32_t *rp = a->row_ptr + a->row_off[i];
            g.m = rp[g.n] / 2;
            g.row_ptr = rp;
            g.col = a->col ? a->col + a->col_off[i] : nullptr;
            g.degree = nullptr;
            const vc_status v = all ? validate_csr(&g) : check_head(&g);
            if (v != VC_OK) return v;
        }
        return VC_OK;
    };
    if (validate) {
        const vc_status v = host_checks(!on_device);
        if (v != VC_OK) return fail(v);
    }
    vc_status err;
    Ctx *c = get_ctx(reqs[0].device, &err);
    if (!c) return fail(on_device && host_checks(true) != VC_OK ? VC_ERR_INVALID : err);
    std::lock_guard<std::mutex> lk(c->mu);
    cudaStream_t stream = reqs[0].stream ? (cudaStream_t)reqs[0].stream : c->stream;
    Job job;
    if (d_rp) {
        job.d_rp = d_rp;
        job.d_col = d_col;
    } else {
        if (c->rp.ensure(sizeof(uint32_t) * rows) || c->col.ensure(sizeof(uint32_t) * std::max<uint64_t>(cols, 1)))
            return fail(VC_ERR_NOMEM);
        cudaMemcpyAsync(c->rp.p, a->row_ptr, sizeof(uint32_t) * rows, cudaMemcpyHostToDevice, stream);
        if (cols) cudaMemcpyAsync(c->col.p, a->col, sizeof(uint32_t) * cols, cudaMemcpyHostToDevice, stream);
        job.d_rp = (const uint32_t *)c->rp.p;
        job.d_col = (const uint32_t *)c->col.p;
    }
    int check = d_rp ? 1 : (on_device ? 2 : 0);
    float total_kernel = 0;
    // graph i as the checks and the searches read it
    auto desc_of = [&](uint32_t i) {
        InstDesc d{};
        d.n = a->n[i];
        d.nw = (d.n + 31) / 32;
        d.row_off = a->row_off[i];
        d.col_off = a->col_off[i];
        d.mode = reqs[i].instance == VC_PVC ? kModePVC : kModeMVC;
        d.k = std::min<uint32_t>(reqs[i].k, d.n);
        d.init_best = init_best_for(&reqs[i], d.n);
        d.node_limit = reqs[i].node_limit;
        d.m2 = a->row_ptr[a->row_off[i] + d.n];
        return d;
    };
    // Large graphs first: their roots are reduced (largest first) and the search gets
    // what is left of them.
    std::vector<Reduce> reds;
    std::vector<uint32_t> red_of;  // the graph each reduction is of
    if (!c->force_sparse) {
        for (uint32_t i = 0; i < count; ++i)
            if (a->n[i] > kHalfMaxN) red_of.push_back(i);
        std::stable_sort(red_of.begin(), red_of.end(), [&](uint32_t x, uint32_t y) { return a->n[x] > a->n[y]; });
        for (const uint32_t i : red_of) {
            const uint32_t *rp = a->row_ptr + a->row_off[i];
            Reduce r;
            r.rp = job.d_rp + a->row_off[i];
            r.cl = job.d_col + a->col_off[i];
            r.n = a->n[i];
            r.m2 = rp[r.n];
            r.bound = reqs[i].instance == VC_PVC ? std::min<uint32_t>(reqs[i].k, r.n) + 1 : init_best_for(&reqs[i], r.n);
            reds.push_back(r);
        }
    }
    struct Trim {
        Ctx *c;
        ~Trim() { trim_reductions(*c); }
    } trim{c};
    if (!reds.empty()) {
        std::vector<InstDesc> others;
        for (uint32_t i = 0; check == 2 && i < count; ++i)
            if (a->n[i] > 0 && a->n[i] <= kHalfMaxN) others.push_back(desc_of(i));
        const vc_status s = run_reductions(*c, reds, check, job.d_rp, job.d_col, others, stream, &total_kernel);
        if (s == VC_ERR_NOMEM) {
            reds.clear();  // no room: the search reduces the roots itself
            red_of.clear();
        } else if (s != VC_OK) {
            return fail(s);
        } else if (check == 2) {
            check = 0;  // every graph has passed
        }
    }
    std::vector<const Reduce *> red_at(count, nullptr);
    for (size_t j = 0; j < reds.size(); ++j)
        if (!reds[j].h.uneven) red_at[red_of[j]] = &reds[j];
    vc_status first = VC_OK;
    std::vector<vc_status> got(count, VC_OK);
    // One launch per kernel shape: dense bitsets (n <= 255), wide dense bitsets
    // (n <= 640, every degree <= 254), dense bitsets with 16-bit degrees (n <=
    // 1024), warp search units (n <= kWarpMaxNP), CTA search units (larger); the
    // shape is sized by the largest graph of its class, so small graphs never
    // run in a large graph's workspace.  The row offsets are host arrays on both
    // entry points.  The rests of reductions are classes 5 to 9, in launches of
    // their own: their rows are not in the arena.
    auto klass = [&](uint32_t n, bool wide) {
        if (n <= 255) return 0;
        if (wide) return 1;
        if (half_ok(n)) return 2;
        return n <= kWarpMaxNP ? 3 : 4;
    };
    std::vector<int> cls(count, -1);
    std::vector<InstDesc> rest(reds.size());
    std::vector<vc_result> early(reds.size());  // answers of graphs without a rest
    std::vector<uint8_t> searched(reds.size(), 0);
    for (size_t j = 0; j < reds.size(); ++j) {
        const uint32_t i = red_of[j];
        Reduce &r = reds[j];
        if (r.h.uneven) {  // searched as it is
            searched[j] = 1;
            continue;
        }
        early[j] = out[i];
        if (r.h.bad) {  // device-resident input: this graph only
            early[j].cover_mask = nullptr;
            fill_answer(&reqs[i], r.n, kNone, &early[j], [](uint8_t *) {});
            early[j].status = VC_ERR_INVALID;
            early[j].tree_nodes = 0;
            early[j].done_ms = 0;
            continue;
        }
        rest[j] = InstDesc{};
        early[j].cover_mask = nullptr;  // written below, when every launch has gone well
        if (!rest_of(r, &reqs[i], total_kernel, rest[j], &early[j])) continue;
        searched[j] = 1;
        cls[i] = 5 + klass(rest[j].n, rest[j].n <= kWideMaxN && r.h.maxd <= 254);
    }
    fetch_new_ids(reds, searched, stream);
    for (uint32_t i = 0; i < count; ++i)
        if (a->n[i] > 0 && !red_at[i]) cls[i] = klass(a->n[i], wide_ok(a->n[i], a->row_ptr + a->row_off[i]));
    std::vector<Job> jobs;
    std::vector<std::vector<uint32_t>> members;
    for (int cl = 0; cl < 10; ++cl) {
        std::vector<uint32_t> mem;
        for (uint32_t i = 0; i < count; ++i)
            if (cls[i] == cl) mem.push_back(i);
        if (mem.empty()) continue;
        Job cj;
        const bool rests = cl >= 5;
        cj.d_rp = rests ? (const uint32_t *)c->red.p : job.d_rp;
        cj.d_col = rests ? (const uint32_t *)c->red.p : job.d_col;
        cj.wide = cl % 5 == 1;
        cj.half = cl % 5 == 2;
        cj.check = rests ? 0 : check;
        if (check == 2) {  // the first launch's checks are for the whole call: no graph is searched before all have passed
            for (uint32_t i = 0; i < count; ++i)
                if (cls[i] >= 0 && cls[i] != cl) cj.others.push_back(desc_of(i));
            check = 0;
        }
        cj.desc.resize(mem.size());
        double tl = 0;
        for (size_t j = 0; j < mem.size(); ++j) {
            const uint32_t i = mem[j];
            InstDesc &d = cj.desc[j];
            if (rests) {
                const Reduce *r = red_at[i];
                d = rest[r - reds.data()];
                d.row_off = (uint64_t)(r->rrp - (const uint32_t *)c->red.p);
                d.col_off = (uint64_t)(r->rcl - (const uint32_t *)c->red.p);
                cj.rest.push_back(r);
            } else {
                d = desc_of(i);
            }
            d.key = (uint32_t)j;
            tl = std::max(tl, reqs[i].time_limit_s);
        }
        cj.time_limit_s = tl;
        vc_status s = run_job(*c, cj, stream);
        if (s == VC_ERR_INVALID) return fail(s);
        if (s != VC_OK) {
            for (uint32_t i = 0; i < count; ++i) out[i].status = s;
            return s;
        }
        total_kernel += cj.kernel_ms;
        jobs.push_back(std::move(cj));
        members.push_back(std::move(mem));
    }
    for (size_t q = 0; q < jobs.size(); ++q)
        for (size_t j = 0; j < members[q].size(); ++j) {
            const uint32_t i = members[q][j];
            got[i] = fill_result(jobs[q], (uint32_t)j, &reqs[i], a->n[i], &out[i]);
        }
    for (size_t j = 0; j < reds.size(); ++j) {
        if (searched[j]) continue;
        const uint32_t i = red_of[j];
        uint8_t *mask = out[i].cover_mask;
        out[i] = early[j];
        out[i].cover_mask = mask;
        if (mask) {
            if (out[i].has_cover) memcpy(mask, reds[j].h_cover, reds[j].n);
            else memset(mask, 0, reds[j].n);
        }
        got[i] = out[i].status;
    }
    for (uint32_t i = 0; i < count && first == VC_OK; ++i) first = got[i];
    float total = std::chrono::duration<float, std::milli>(std::chrono::steady_clock::now() - t0).count();
    for (uint32_t i = 0; i < count; ++i) {
        out[i].total_ms = total;
        out[i].kernel_ms = total_kernel;
        if (a->n[i] == 0) {
            out[i].status = VC_OK;
            out[i].size = 0;
            out[i].decision = 1;
            out[i].has_cover = 1;
            out[i].tree_nodes = 0;
            out[i].done_ms = 0;
        }
    }
    return first;
}
}  // namespace vch

// Batched solve over an arena already resident on the device: the per-graph
// sizes and offsets stay on the host (`a` holds host arrays for n, row_off,
// col_off and the row_ptr values), d_rp / d_col are the device copies.
extern "C" vc_status vc_solve_batch_device(const vc_csr_arena *a, const uint32_t *d_rp, const uint32_t *d_col,
                                           const vc_request *reqs, vc_result *out)
{
    vch::DeviceGuard dg;
    auto t0 = std::chrono::steady_clock::now();
    if (!a || !reqs || !out || !d_rp) return VC_ERR_INVALID;
    if (a->count == 0) return VC_OK;
    return vc_solve_batch_impl(a, reqs, out, d_rp, d_col, t0);
}
