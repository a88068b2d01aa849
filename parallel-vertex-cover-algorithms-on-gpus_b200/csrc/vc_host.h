// vc_host.h -- host-side types shared by the library's translation units.
#pragma once
#include <cuda_runtime.h>

#include <chrono>
#include <cstdint>
#include <mutex>
#include <vector>

#include "vcgpu.h"
#include "vc_types.h"

namespace vch {

// Search units are warps up to this vertex capacity, CTAs above it.
#ifndef VC_WARP_MAX_NP
#define VC_WARP_MAX_NP 1024
#endif
constexpr uint32_t kWarpMaxNP = VC_WARP_MAX_NP;
constexpr uint32_t kMaxVertices = 1u << 26;

// Puts the calling thread's current device back when an entry point returns:
// the library switches devices for its own work, never for its caller.
struct DeviceGuard {
    int prev = -1;
    DeviceGuard()
    {
        if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
    }
    ~DeviceGuard()
    {
        int cur = -1;
        if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev);
    }
    DeviceGuard(const DeviceGuard &) = delete;
    DeviceGuard &operator=(const DeviceGuard &) = delete;
};

struct DevBuf {
    void *p = nullptr;
    size_t cap = 0;
    cudaError_t ensure(size_t bytes);
    void release();
};

struct PinBuf {
    void *p = nullptr;
    size_t cap = 0;
    cudaError_t ensure(size_t bytes);
    void release();
};

// A launch-shape choice for one size class of graphs, set by vc_autotune (or
// vc_set_tuning); `set` = 0 keeps the built-in rules.
struct Tune {
    uint32_t set = 0;
    uint32_t cta_units = 0;   // CSR classes: 1 = one 512-thread CTA per search unit, 0 = warp units
    uint32_t warps = 8;       // warps (search units) per CTA: 2, 4 or 8
    uint32_t pool = 2;        // CTA pool slots (donated subtrees) per warp: 1, 2 or 4
    int32_t ring_bias = 0;    // global-ring donations while idle CTAs minus queued records exceed this
    uint32_t ring_first = 0;  // 1: when a sibling warp and another CTA both wait, the ring gets the subtree
    float nodes_per_s = 0;    // what the calibration measured with this choice
};

// Size classes of the tuner: dense bitsets of 2, 4 and 8 words (n <= 64, 128,
// 255), the wide dense kernel (n <= 640, degrees <= 254), CSR up to 1024
// vertices, CSR above.
constexpr int kTuneClasses = 6;
inline int tune_class(uint32_t nmax, bool wide)
{
    if (nmax <= 64) return 0;
    if (nmax <= 128) return 1;
    if (nmax <= 255) return 2;
    if (wide && nmax <= 640) return 3;
    return nmax <= 1024 ? 4 : 5;
}

struct Plan {
    const void *fn = nullptr;
    uint32_t block = 0, grid = 0, smem = 0;
    uint32_t np = 0, su_bytes = 0, num_su = 0, stride = 0, cta_slots = 0;
    bool global_ws = false;
    bool dense = false;
    bool lanes = false;  // one thread per search unit (vc_lanes.cuh)
};

// Per-device state: one stream, grow-only device and pinned buffers, a lock
// that serialises solves on the device.
struct Ctx {
    int dev = -1;
    int sms = 0;
    int smem_optin = 0;
    int coop = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    DevBuf rp, col, seq, data, gws, adj;
    DevBuf in, out;      // one launch's descriptors (and a small graph), its control words, states and covers
    PinBuf h_in, h_out;
    DevBuf ub;     // the upper-bound heuristics (vc_ub.cu)
    DevBuf red;    // reductions of large graphs (struct Reduce)
    PinBuf h_red;
    bool stats_on = false;
    bool force_sparse = false;
    Tune tune[kTuneClasses];
    int lanes_mode = 0;  // graphs <= 255 vertices: 0 warp search units (default), 1 lane search units
    DevBuf stats;
    std::vector<unsigned long long> last_stats;
    uint32_t last_num_su = 0;
    Plan last_plan;
    struct Occ {
        const void *fn;
        uint32_t smem;
        int per_sm;
    };
    std::vector<Occ> occ;  // resident CTAs per SM, as asked for once per kernel and shared-memory size
    std::mutex occ_mu;     // (a server is planned without `mu`)
    std::mutex mu;
};

// What k_reduce reports of a graph (zeroed before it, but for `bad`).
struct ReduceHead {
    uint32_t n, m2, maxd;  // what is left: vertices, entries, largest degree
    uint32_t taken;        // vertices taken into the cover
    uint32_t last_pass;
    uint32_t bad;          // the CSR check failed: nothing was reduced (a host-resident call: the first head's is for all)
    uint32_t uneven;       // rows and degrees part (edges in one direction only): the rest is no graph
    uint32_t pad;
};

// What the reduction of a graph's root (csrc/vc_reduce.cu) reads and leaves.
struct ReduceArgs {
    const uint32_t *rp = nullptr, *cl = nullptr;
    uint32_t n = 0, bound = 0;                   // high-degree rule: deg + taken >= bound
    int32_t *deg = nullptr;
    uint32_t *taken = nullptr;                   // the pass that took a vertex, 0 = live
    uint32_t *map = nullptr, *inv = nullptr;     // old id -> new id, new id -> old id
    uint32_t *rrp = nullptr, *rcl = nullptr;     // what is left
    uint8_t *cover = nullptr;                    // 1 = taken
    uint32_t *part = nullptr;                    // per CTA: vertices left, entries left
    ReduceHead *head = nullptr;
    const uint32_t *bad = nullptr;               // not 0: nothing is reduced
};

// A graph to reduce at its root, and the host's copies of what came of it.
struct Reduce : ReduceArgs {
    uint32_t m2 = 0;
    ReduceHead h = {};
    const uint8_t *h_cover = nullptr;
    uint32_t *h_inv = nullptr;
};

struct Job {
    const uint32_t *d_rp = nullptr;
    const uint32_t *d_col = nullptr;
    std::vector<vcg::InstDesc> desc;
    // a host-resident graph that run_job copies with its descriptor (instead of d_rp, d_col)
    const uint32_t *h_rp = nullptr, *h_col = nullptr;
    double time_limit_s = 0;
    // results
    std::vector<vcg::InstState> st;
    std::vector<uint32_t> covers;
    float kernel_ms = 0;
    unsigned long long t0 = 0;
    unsigned long long stopped = 0;  // the control word kAbort
    bool wide = false;  // every graph may take the 20-word dense kernel
    bool half = false;  // every graph may take the 16/32-word dense kernels (16-bit degrees)
    // k_check_csr before the search: 0 none, 1 the layout (caller's device memory; a graph that fails is flagged), 2
    // all of it (one that fails stops the launch: VC_ERR_INVALID), with 2 also of the graphs in `others`
    int check = 0;
    std::vector<vcg::InstDesc> others;
    std::vector<const Reduce *> rest;  // per graph: the reduction it is the rest of (empty: none are)
    const Tune *tune = nullptr;  // a shape to try instead of the context's table (the tuner's candidates)
    Plan plan;
};

// The most device memory a context keeps for bitmap rows (c.adj).
constexpr uint64_t kAdjBytesMax = 4ull << 30;

// The most device memory a context keeps for the upper-bound heuristics (c.ub).
constexpr uint64_t kUbBytesKept = 1ull << 30;

// Host-resident graphs up to this many bytes go to the device in one copy with
// their descriptor, from pinned memory; larger ones straight from the caller's.
constexpr size_t kSmallGraphBytes = 256u << 10;

// The largest graph of the wide dense kernel; it also needs every degree <= 254.
constexpr uint32_t kWideMaxN = 640;

// The largest graph of the dense kernels with 16-bit degrees (any degree).
constexpr uint32_t kHalfMaxN = 1024;

// True if a graph of n vertices takes a dense kernel with 16-bit degrees (when
// the byte kernels cannot take it).
inline bool half_ok(uint32_t n) { return n > 255 && n <= kHalfMaxN; }

// True if a graph of n vertices (host row offsets) fits the wide dense kernel.
inline bool wide_ok(uint32_t n, const uint32_t *row_ptr)
{
    if (n > kWideMaxN || !row_ptr) return false;
    for (uint32_t v = 0; v < n; ++v)
        if (row_ptr[v + 1] - row_ptr[v] > 254u) return false;
    return true;
}

// From how many roots the dense kernels search a graph that has a launch to itself: all
// n, or one (0), by its size and density (m2 / n^2).
// At two fifths and above, from 64 vertices, MVC and both PVC answers gain (plain
// kernel: 200 vertices of 0.5 0.94 -> 0.62 ms, 300 of 0.75 1.65 -> 0.41, 256 of 0.9
// 0.98 -> 0.09, 1000 of 0.8 6.6 -> 4.1).  Down to 0.15 they do for 16 to 192 vertices:
// the trees are a few hundred nodes, most of them the spine, and with the packing bound
// at its nodes they had become slower than without (allocation-free calls, without the
// bound, with it, and from n roots: 64 vertices of 0.3 0.27, 0.35 and 0.14 ms; of 0.7
// 0.20, 0.31 and 0.07; 180 vertices, bipartite, PVC no 0.33, 0.38 and 0.16).  Above that
// size the spine is a small part of the tree at 0.3 (200 vertices 6.2 -> 5.8) and a PVC
// "yes", which the first descent often finds, comes later (0.8 -> 1.6).
inline uint32_t split_roots(uint32_t n, uint32_t m2)
{
    const uint64_t n2 = (uint64_t)n * n;
    if (m2 == vcg::kNone) return 0u;
    return (n >= 64 && 5ull * m2 >= 2 * n2) || (n >= 16 && n <= 192 && 20ull * m2 >= 3 * n2) ? n : 0u;
}

struct PlanOpts {
    uint32_t smem_budget = 0;  // bytes per CTA for CSR workspaces, 0 = the device limit
    uint32_t warp_max_np = 0;  // largest capacity given warp units, 0 = kWarpMaxNP
    uint32_t warps = 0;        // warps per CTA with warp_gws, 0 = 8
    bool wide = false;         // graphs of 256..640 vertices may take the wide dense kernel
    bool warp_gws = false;     // warp units with global-memory workspaces
    bool lanes = false;        // graphs <= 255 vertices take the lane kernel
    bool half = false;         // graphs of 256..1024 vertices take the 16-bit-degree dense kernels
    bool team = false;         // CSR kernels walk rows with teams of lanes (average degree >= 4)
    bool plain = false;        // a launch of one graph
    bool lane = false;         // a server lane, which shares the SMs with other lanes' kernels
    const Tune *tune = nullptr; // the size class's tuned shape, if any
};

// The status of a graph whose search a launch left unfinished (its control word kAbort).
inline vc_status stopped_status(unsigned long long why) { return why == vcg::kStopTime ? VC_TIMEOUT : VC_ERR_INTERNAL; }

Ctx *get_ctx(int dev, vc_status *err);
cudaError_t make_plan(Ctx &c, uint32_t np, uint32_t nmax, Plan &pl, const PlanOpts &o = PlanOpts());
void cap_plan(const Ctx &c, Plan &pl, uint32_t per_sm);
cudaError_t launch_reduce(const ReduceArgs &r, uint32_t ctas, cudaStream_t stream);
cudaError_t launch_reduce_many(const ReduceArgs *list, uint32_t count, cudaStream_t stream);
cudaError_t launch_reduce_each(const ReduceArgs *list, uint32_t count, uint32_t nmax, cudaStream_t stream);
uint32_t reduce_ctas(const Ctx &c);
vc_status run_job(Ctx &c, Job &job, cudaStream_t stream);
vc_status fill_result(const Job &job, uint32_t i, const vc_request *req, uint32_t n, vc_result *out);
vc_status validate_csr(const vc_csr *g);
vc_status check_head(const vc_csr *g);
cudaError_t launch_check(bool full, const uint32_t *rp, const uint32_t *cl, const vcg::InstDesc *inst, uint32_t *bad,
                         uint32_t stride, uint32_t value, uint32_t count, uint32_t nmax, cudaStream_t stream,
                         uint32_t *mate = nullptr);
vc_status vc_solve_batch_impl(const vc_csr_arena *a, const vc_request *reqs, vc_result *out, const uint32_t *d_rp,
                              const uint32_t *d_col, std::chrono::steady_clock::time_point t0);

}  // namespace vch
