// cpd_runtime.cu -- the GPU side of the C ABI: contexts, per-pass slots (stream,
// pooled device buffers, pinned staging, captured CUDA graph), the ray-table cache,
// the synchronous entry points and the continuous-batching server.
#include <cuda_runtime.h>

#include <algorithm>
#include <iterator>
#include <array>
#include <atomic>
#include <chrono>
#include <cmath>
#include <condition_variable>
#include <cstddef>
#include <cstring>
#include <deque>
#include <map>
#include <memory>
#include <mutex>
#include <set>
#include <thread>
#include <tuple>
#include <vector>

#include "cpd_gpu.cuh"
#include "cpd_host.h"
#include "cpd_orders.h"

namespace cpd {
namespace {

struct DevBuf {
    void *p = nullptr;
    size_t cap = 0;
    cudaError_t ensure(size_t bytes)
    {
        if (bytes <= cap) return cudaSuccess;
        if (p) cudaFree(p);
        p = nullptr;
        cap = 0;
        size_t want = std::max<size_t>(bytes, 256);
        want = want + want / 4;
        cudaError_t e = cudaMalloc(&p, want);
        if (e == cudaSuccess) cap = want;
        return e;
    }
    void release()
    {
        if (p) cudaFree(p);
        p = nullptr;
        cap = 0;
    }
    template <class T>
    T *as() const
    {
        return reinterpret_cast<T *>(p);
    }
};

struct HostBuf {
    void *p = nullptr;
    void *dev = nullptr;  // the device's address of a mapped buffer
    size_t cap = 0;
    // mapped: the GPU reads and writes the buffer in place (over NVLink-C2C on this
    // machine), so a kernel can deliver results without a copy
    cudaError_t ensure(size_t bytes, bool mapped = false)
    {
        if (bytes <= cap) return cudaSuccess;
        if (p) cudaFreeHost(p);
        p = dev = nullptr;
        cap = 0;
        size_t want = std::max<size_t>(bytes, 256);
        want = want + want / 4;
        cudaError_t e = cudaHostAlloc(&p, want, mapped ? cudaHostAllocMapped : cudaHostAllocDefault);
        if (e == cudaSuccess && mapped) e = cudaHostGetDevicePointer(&dev, p, 0);
        if (e == cudaSuccess) cap = want;
        return e;
    }
    void release()
    {
        if (p) cudaFreeHost(p);
        p = nullptr;
        cap = 0;
    }
    template <class T>
    T *as() const
    {
        return reinterpret_cast<T *>(p);
    }
};

struct RayKey {
    uint64_t seed_bits;
    uint32_t R;
    bool operator<(const RayKey &o) const { return seed_bits != o.seed_bits ? seed_bits < o.seed_bits : R < o.R; }
};

// The sampling flags a trace mode may carry.
constexpr uint32_t kSamplingBits = CPD_SAMPLING_ADAPTIVE | CPD_SAMPLING_EXACT;
// Most rows of a pass whose trace takes equal shares of span slots: every warp scans the
// blocks' spans (32 per step) to find its share.
constexpr uint64_t kBalancedMaxRows = 16384;

// The kernel node of `fn` in a captured graph (nullptr if none).
cudaGraphNode_t find_kernel_node(cudaGraph_t g, const void *fn)
{
    size_t n = 0;
    if (cudaGraphGetNodes(g, nullptr, &n) != cudaSuccess || n == 0) return nullptr;
    std::vector<cudaGraphNode_t> nodes(n);
    if (cudaGraphGetNodes(g, nodes.data(), &n) != cudaSuccess) return nullptr;
    for (cudaGraphNode_t nd : nodes) {
        cudaGraphNodeType t;
        if (cudaGraphNodeGetType(nd, &t) != cudaSuccess || t != cudaGraphNodeTypeKernel) continue;
        cudaKernelNodeParams kp{};
        if (cudaGraphKernelNodeGetParams(nd, &kp) == cudaSuccess && kp.func == fn) return nd;
    }
    return nullptr;
}

// Everything one pass needs on the device, plus its staging and its captured graph.
// A context owns one slot (the synchronous calls); a server owns several, so that
// passes overlap on the device.
struct PassSlot {
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr, done = nullptr;
    cudaEvent_t kev[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
    // inputs (tables, designs, jobs) in one arena, uploaded with one copy; results
    // (DesignOut[n] then HostStatus) written by the kernels into mapped host memory;
    // `in` ends with the device-side Control words
    DevBuf in, lp, lx, hist, S1, S2, acc, queue, pout, perm;
    HostBuf h_in, h_outs;
    size_t ctl_off = 0;
    bool hist_dirty = true;
    uint32_t qcap = 1u << 18;
    // Captured passes, most recently used first: a caller that alternates between a few
    // launch signatures (designs of different detector sizes, say) replays each one's
    // graph instead of capturing anew. The key holds every pointer and size the graph
    // bakes in, plus buf_gen, which changes whenever a buffer of the slot is reallocated.
    struct CachedGraph {
        std::vector<uint8_t> key;
        cudaGraphExec_t exec;
        int launches;
        // a single-design pass: the captured graph (kept: its node handle addresses the
        // exec's node), the trace node, and the launch arguments it holds, whose design
        // constants (fc, fl) change from call to call while the key stays the same
        cudaGraph_t graph = nullptr;
        cudaGraphNode_t trace_node = nullptr;
        LaunchArgs args{};
    };
    std::vector<CachedGraph> graphs;
    static constexpr size_t kGraphCache = 8;
    uint64_t buf_gen = 0;
    // The wavelength-point and ray tables (the arena after the designs and jobs) of the
    // last pass, when they came from the context's caches: identity of each table in
    // upload order, and references that keep those tables (and so their addresses)
    // alive. A pass with the same key leaves them in place and uploads the designs and
    // jobs only.
    std::vector<const void *> tables_key;
    std::vector<std::shared_ptr<const void>> tables_refs;
    // the pass in flight / last finished
    uint32_t n = 0;
    uint64_t hist_cells = 0;
    double *p_out_host = nullptr;
    bool profiled = false, timed = true;
    int launches = 0;
    double last_ms = 0.0;
    uint64_t h2d = 0, d2h = 0;
    double kernel_ms[4] = {0, 0, 0, 0};

    cudaError_t create()
    {
        cudaError_t e = cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking);
        if (e == cudaSuccess) e = cudaEventCreate(&ev0);
        if (e == cudaSuccess) e = cudaEventCreate(&ev1);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&done, cudaEventDisableTiming);
        for (int i = 0; i < 5 && e == cudaSuccess; i++) e = cudaEventCreate(&kev[i]);
        return e;
    }
    void destroy()
    {
        if (stream) cudaStreamSynchronize(stream);
        for (CachedGraph &c : graphs) {
            cudaGraphExecDestroy(c.exec);
            if (c.graph) cudaGraphDestroy(c.graph);
        }
        graphs.clear();
        for (DevBuf *b : {&in, &lp, &lx, &hist, &S1, &S2, &acc, &queue, &pout, &perm}) b->release();
        for (HostBuf *b : {&h_in, &h_outs}) b->release();
        for (cudaEvent_t *ev : {&ev0, &ev1, &done, &kev[0], &kev[1], &kev[2], &kev[3], &kev[4]})
            if (*ev) cudaEventDestroy(*ev), *ev = nullptr;
        if (stream) cudaStreamDestroy(stream);
        stream = nullptr;
    }
};

}  // namespace
}  // namespace cpd

using namespace cpd;

struct cpd_context {
    int device = 0;
    int num_sms = 0;
    std::mutex mu;        // serialises the synchronous entry points (main slot)
    std::mutex cache_mu;  // ray-table cache
    PassSlot main;
    DevBuf pair_design, pair_lam, pair_z, pair_bins, pair_ts, pair_flags, peak, logtab;
    DevBuf bld_params, bld_out, bld_status;  // cpd_design_build_device
    // cpd_transmission_probability: the design, the wavelengths, the ray table of the
    // reference's ray points (kept while max_m stays the same), the results
    DevBuf tp_design, tp_lam, tp_z, tp_out, tp_rays, tp_tab, tp_lp, tp_t64;
    uint32_t tp_m = 0, tp_tab_m = 0, tp_rz = 0;
    uint32_t ray_tile = 32;
    uint32_t warps_per_cta = 8;
    bool profiling = false;
    std::atomic<bool> timed{false};  // single-design passes record events too: the caller asks for their times
    bool use_graphs = true;
    bool autotune = false;
    std::map<RayKey, RayTablePtr> ray_cache;
    PointOrders orders;
    std::set<RayKey> host_only;  // tables that a pass could not make on the device
    std::map<RayKey, std::shared_ptr<const std::vector<double>>> lam_cache;  // wavelength u-points per (seed, W)
    // launch shape picked by the autotuner per class of batch
    std::map<std::array<uint64_t, 6>, std::pair<uint32_t, uint32_t>> tune_cache;
};

namespace {

#define CPD_TRY(expr)                                 \
    do {                                              \
        cudaError_t _e = (expr);                      \
        if (_e != cudaSuccess) return CPD_CUDA_ERROR; \
    } while (0)

RayTablePtr ray_table_cached(cpd_context *ctx, double seed, uint32_t R)
{
    uint64_t bits;
    std::memcpy(&bits, &seed, 8);
    RayKey key{bits, R};
    {
        std::lock_guard<std::mutex> lk(ctx->cache_mu);
        auto it = ctx->ray_cache.find(key);
        if (it != ctx->ray_cache.end()) return it->second;
    }
    std::vector<double> u(R);
    seed_points(seed, 1, R, u.data());
    auto t = std::make_shared<RayTable>();
    ray_table(u.data(), R, t->z64, t->z32, &t->rank);
    std::lock_guard<std::mutex> lk(ctx->cache_mu);
    if (ctx->ray_cache.size() > 256) ctx->ray_cache.clear();
    return ctx->ray_cache.emplace(key, t).first->second;
}

// The wavelength u-points of the GPU seed policy, u_i = fract(fma(i, 1/phi, seed)),
// cached per seed like the ray tables (an optimizer reuses its seeds). The points of W
// wavelengths are the first W of any longer table of the same seed, so one table of
// max(1024, W rounded up to a power of two) points serves every W up to its length:
// the designs of a batch with mixed W share a few tables.
LamPtr lam_points_cached(cpd_context *ctx, double seed, uint32_t W)
{
    uint64_t bits;
    std::memcpy(&bits, &seed, 8);
    uint32_t L = 1024;
    while (L < W) L <<= 1;
    W = L;
    RayKey key{bits, W};
    {
        std::lock_guard<std::mutex> lk(ctx->cache_mu);
        auto it = ctx->lam_cache.find(key);
        if (it != ctx->lam_cache.end()) return it->second;
    }
    auto v = std::make_shared<std::vector<double>>(W);
    seed_points(seed, 0, W, v->data());
    std::lock_guard<std::mutex> lk(ctx->cache_mu);
    if (ctx->lam_cache.size() > 256) ctx->lam_cache.clear();
    return ctx->lam_cache.emplace(key, v).first->second;
}

// One design's sampling inputs for a pass: the points of a seed, or the caller's own.
struct PassDesign {
    const DevDesign *dev;      // host copy
    uint32_t W, R;
    bool seeded;
    double seed;
    const double *lam_u;       // !seeded: W wavelength u-points (host)
    const double *ray_u;       // !seeded: R ray u-points (host)
    // the ray table from the host; none: the pass makes it on the device from the points
    // (rays_keep: a table of the context's cache; its device copy may then stay resident)
    const RayTable *rays = nullptr;
    RayTablePtr rays_keep = nullptr, rays_own = nullptr;
    // set instead of dev: the design is built on the device from this record (detector
    // positioned first when acceptance > 0; the same acceptance for every design of a pass)
    const cpd_spectrometer_params *params = nullptr;
    double acceptance = 0.0;
};

struct PassResult {
    std::vector<DesignOut> outs;
    bool overflow = false;    // the re-trace queue was too small
    bool bad_table = false;   // a ray table could not be made on the device
};

// Whether points in (0, 1) crowd in table_sort_kernel's buckets, as far as 64 of them show it (that
// takes 0.3 us, all of 3000 points 3): a pass that finds a bucket too full is run again with the host's
// table, 340 instead of 250 us for 4000 points within 1e-9 of each other.
bool crowded(const double *u, uint32_t R)
{
    if (R <= kTableBucket) return false;
    uint32_t M = 1024u;
    while (M < R) M <<= 1;
    const uint32_t n = std::min(R, 64u);
    uint32_t b[64];
    for (uint32_t i = 0; i < n; i++) b[i] = (uint32_t)(u[(uint64_t)i * R / n] * M);
    std::sort(b, b + n);
    bool suspect = false;  // of 64 points spread evenly, four in one of 1024 buckets: 1 in 1600
    for (uint32_t i = 3; i < n; i++) suspect |= b[i] == b[i - 3];
    if (!suspect) return false;
    std::vector<uint32_t> count(M, 0u);
    for (uint32_t j = 0; j < R; j++)
        if (++count[(uint32_t)(u[j] * M)] > kTableBucket) return true;
    return false;
}

// Whether a pass may make the ray table on the device: its points lie in (0, 1) and do not crowd, it
// fits table_sort_kernel, and the trace does not read the f64 table.
bool device_table(cpd_context *ctx, const PassDesign &p, uint32_t mode)
{
    if (p.R > kTableRays || (mode & ~kSamplingBits) == CPD_TRACE_FP64) return false;
    if (p.seeded) {
        if (!(p.seed >= 0.0 && p.seed < 1.0)) return false;
        uint64_t bits;
        std::memcpy(&bits, &p.seed, 8);
        std::lock_guard<std::mutex> lk(ctx->cache_mu);
        return ctx->host_only.empty() || !ctx->host_only.count(RayKey{bits, p.R});
    }
    bool in = true;
    for (uint32_t j = 0; j < p.R; j++) in &= p.ray_u[j] > 0.0 && p.ray_u[j] < 1.0;
    return in && !crowded(p.ray_u, p.R);
}

// PointOrders' calls, on a slot's stream.
struct OrderDevice {
    cudaStream_t stream;
    uint32_t *alloc(uint32_t n)
    {
        uint32_t *p = nullptr;
        if (cudaMalloc(&p, sizeof(uint32_t) * n) == cudaSuccess) return p;
        cudaGetLastError();
        return nullptr;
    }
    bool upload(uint32_t *dst, const uint32_t *src, uint32_t n)
    {
        return cudaMemcpyAsync(dst, src, sizeof(uint32_t) * n, cudaMemcpyHostToDevice, stream) == cudaSuccess;
    }
    bool wait() { return cudaStreamSynchronize(stream) == cudaSuccess; }
    void free(uint32_t *p) { cudaFree(p); }
};

const uint32_t *point_order(cpd_context *ctx, cudaStream_t stream, uint32_t R, uint64_t seed_fixed, uint32_t &rot)
{
    std::lock_guard<std::mutex> lk(ctx->cache_mu);
    OrderDevice dev{stream};
    return ctx->orders.get(dev, R, seed_fixed, rot);
}

// The host's table for a design's points.
void host_table(cpd_context *ctx, PassDesign &p)
{
    if (p.seeded) {
        p.rays_keep = ray_table_cached(ctx, p.seed, p.R);
        p.rays = p.rays_keep.get();
    } else {
        auto t = std::make_shared<RayTable>();
        ray_table(p.ray_u, p.R, t->z64, t->z32, &t->rank);
        p.rays_own = t;
        p.rays = t.get();
    }
}

void choose_table(cpd_context *ctx, PassDesign &p, uint32_t mode)
{
    if (!device_table(ctx, p, mode)) host_table(ctx, p);
}

// After a pass that reported a table the device could not make: its seeds' tables come from
// the host from now on.
void mark_host_only(cpd_context *ctx, const std::vector<std::pair<double, uint32_t>> &seeds)
{
    std::lock_guard<std::mutex> lk(ctx->cache_mu);
    if (ctx->host_only.size() > 4096) ctx->host_only.clear();
    for (const auto &s : seeds) {
        uint64_t bits;
        std::memcpy(&bits, &s.first, 8);
        ctx->host_only.insert(RayKey{bits, s.second});
    }
}

// Whether a pass gives its coated designs to rows_kernel (by_rows), the rule for all of them: under
// the fixed-N hybrid trace, but for short tables on many rows, whose pieces of a few rays save less
// than their edges cost. The ray-by-ray kernels give the same numbers. us, rows_kernel / ray by ray: 64
// designs x 4096 rows, 16 bins, 64 rays 538 / 320, 128 496 / 397, 200 475 / 484; 64 bins, 64 rays 649 /
// 469, 200 691 / 638, 256 698 / 679, 320 692 / 740; 128 designs x 128 rows, 32 bins, 128 rays 243 / 231;
// 64 x 128 150 / 163; one design x 16384, 16 bins, 128 rays 64 / 57, 256 62 / 66; 64 bins, 128 rays 88 /
// 73; 100 bins 103 / 107, 256 bins 99 / 153 (a cell's histogram costs the ray-by-ray kernels more).
// Beside designs for the ray-by-ray kernels it is one more kernel in the chain (~20 us), which takes
// 8 M coated rays to win back: 4 coated and 4 uncoated designs of 128 rows, 2.1 M coated rays 119 / 110,
// 4.2 M 135 / 133, 8.4 M 157 / 175; 32 and 1, 4.2 M 156 / 138, 8.4 M 161 / 161, 16.8 M 177 / 201.
struct RowsRule {
    uint64_t rows = 0, coated_rows = 0, coated_rays = 0;
    uint32_t n = 0, others = 0, max_B = 0, max_R = 0;  // others: not coated; max_R: of the coated designs
    bool on = false;
};
bool coated(const PassDesign &p) { return p.params ? p.params->ar_coated != 0 : p.dev->fc.pieces != 0; }
RowsRule rows_rule(const std::vector<PassDesign> &ds, uint32_t mode)
{
    RowsRule r;
    r.n = (uint32_t)ds.size();
    for (const PassDesign &p : ds) {
        r.rows += p.W;
        r.max_B = std::max(r.max_B, p.params ? p.params->bin_count : p.dev->B);
        if (!coated(p)) {
            r.others++;
            continue;
        }
        r.coated_rows += p.W;
        r.coated_rays += (uint64_t)p.W * p.R;
        r.max_R = std::max(r.max_R, p.R);
    }
    const bool many = r.n > 1 ? r.rows >= 16384u : r.rows >= 8192u && r.max_B <= 80u;
    r.on = mode == CPD_TRACE_HYBRID && r.coated_rows && !(many && r.coated_rays <= 256u * r.coated_rows) &&
           (!r.others || r.coated_rays >= 1u << 23);
    return r;
}
// A coated design under that rule (a device build decides in its record whether the pieces apply;
// if not, its rays go through fast_ray there).
bool by_rows(const PassDesign &p, const RowsRule &r) { return r.on && coated(p); }

uint32_t tile_rows_for(uint32_t B, uint32_t n)
{
    return std::max<uint32_t>(1u, (n > 1 ? kTileCellsBatch : kTileCells) / B);
}

// Device bytes one design occupies in a pass (histogram, per-row tables, ray tables):
// the admission unit of the server.
uint64_t design_bytes(uint32_t W, uint32_t R, uint32_t B)
{
    return (uint64_t)W * (8ull * B + sizeof(LamParams) + sizeof(LamDF) + 8) + 16ull * R + 16ull * B +
           sizeof(DevDesign) + sizeof(DesignJob) + sizeof(DesignAcc) + sizeof(DesignOut);
}

// Plans, stages and issues one pass on slot `s` (asynchronously; `s.done` is recorded
// at the end). Accumulators are zeroed when `fresh`; they persist otherwise (the seeds
// of one call).
int pass_issue(cpd_context *ctx, PassSlot &S, const std::vector<PassDesign> &ds, uint32_t mode, bool fresh,
               double *p_out_host, bool use_graph, bool profile)
{
    const uint32_t n = (uint32_t)ds.size();
    const bool adaptive = (mode & CPD_SAMPLING_ADAPTIVE) != 0u;
    const bool all_exact = adaptive && (mode & CPD_SAMPLING_EXACT) != 0u;
    const bool on_device = n > 0 && ds[0].params != nullptr;  // every design of the pass, or none
    mode &= ~kSamplingBits;
    std::vector<DesignJob> jobs(n);
    std::vector<uint8_t> owns_rays(n, 1);  // designs that share a ray table share its copy
    std::vector<uint8_t> owns_lam(n, 1);   // likewise for the caller's wavelength points
    // a table's identity: the host table or points it comes from, or its seed and size
    using TableId = std::tuple<const void *, uint64_t, uint32_t>;
    std::map<TableId, std::pair<uint64_t, uint64_t>> ray_offs;
    std::map<std::pair<const double *, uint32_t>, uint64_t> lam_offs;
    std::vector<TableJob> tabs;
    // identity of the tables in upload order (null entries: not from a cache)
    std::vector<const void *> tables_key;
    bool cacheable = true, any_host = false;
    uint32_t table_max = 0;
    uint64_t rows = 0, groups = 0, hist = 0, cells = 0, lam = 0, upts = 0, ray = 0, rnk = 0, accc = 0, items = 0, tiles = 0;
    const RowsRule rule = rows_rule(ds, adaptive ? CPD_SAMPLING_ADAPTIVE : mode);
    const uint32_t max_B = rule.max_B;
    RowsPlan plan{1u, 1u};
    if (rule.on) plan = plan_rows(rule.coated_rows, rule.max_R, max_B, ctx->num_sms);
    for (uint32_t i = 0; i < n; i++) {
        const PassDesign &p = ds[i];
        DesignJob &J = jobs[i];
        std::memset(&J, 0, sizeof(J));
        J.W = p.W;
        J.R = p.R;
        J.Rz = p.rays ? (uint32_t)p.rays->z64.size() : p.R;
        J.seeded = p.seeded ? 1u : 0u;
        J.seed = p.seed;
        J.B = on_device ? p.params->bin_count : p.dev->B;
        J.row_off = rows;
        owns_lam[i] = 0;
        if (!p.seeded) {
            auto lo = lam_offs.emplace(std::make_pair(p.lam_u, p.W), lam);
            J.lam_off = lo.first->second;
            owns_lam[i] = lo.second;
            if (owns_lam[i]) lam += p.W;
            cacheable = false;  // the caller's points may change in place
        }
        uint64_t seed_bits = 0;
        if (p.seeded) std::memcpy(&seed_bits, &p.seed, 8);
        const TableId id = p.rays     ? TableId{p.rays, 0, 0}
                           : p.seeded ? TableId{nullptr, seed_bits, p.R}
                                      : TableId{p.ray_u, 1, p.R};
        auto ro = ray_offs.emplace(id, std::make_pair(ray, rnk));
        J.ray_off = ro.first->second.first;
        J.rank_off = ro.first->second.second;
        owns_rays[i] = ro.second;
        if (owns_rays[i]) {
            tables_key.push_back(p.rays);
            tables_key.push_back(reinterpret_cast<const void *>(seed_bits));
            tables_key.push_back(reinterpret_cast<const void *>((uintptr_t)p.R));
            cacheable = cacheable && (!p.rays || p.rays_keep);
            if (p.rays) {
                any_host = true;
            } else {
                TableJob t{};
                t.seed = p.seed;
                t.seed_fixed = p.seeded ? (uint64_t)(p.seed * 18446744073709551616.0) : 0;
                t.points = p.seeded ? 0u : 1u;
                t.u_off = upts;
                t.ray_off = ray;
                t.rank_off = rnk;
                t.R = p.R;
                if (p.seeded) t.order = point_order(ctx, S.stream, p.R, t.seed_fixed, t.rot);
                else upts += p.R;
                table_max = std::max(table_max, p.R);
                tabs.push_back(t);
            }
        }
        J.acc_off = accc;
        J.item_off = items;
        J.tile_off = tiles;
        J.nchunk = std::max<uint32_t>(1u, (J.Rz + ctx->ray_tile - 1) / ctx->ray_tile);
        J.pieces = by_rows(p, rule) ? 1u : 0u;
        J.hist_off = hist;
        J.grp_off = groups;
        J.grp_rows = std::min(plan.group, std::max(1u, kRowsCells / J.B));
        if (J.pieces) groups += (J.W + J.grp_rows - 1) / J.grp_rows;
        J.tile_rows = tile_rows_for(J.B, n);
        J.ntiles = (J.W + J.tile_rows - 1) / J.tile_rows;
        ff::split(kTScaleInv / (double)J.R, J.unit_hi, J.unit_lo);
        ff::split(-31.0 - std::log2((double)J.R), J.lu_hi, J.lu_lo);
        J.pscale = kTScaleInv / (double)J.R;
        rows += J.W;
        cells += (uint64_t)J.W * J.B;
        if (!J.pieces) hist += (uint64_t)J.W * J.B;  // rows_kernel keeps its cells in shared memory
        if (owns_rays[i]) {
            ray += (J.Rz + 1u) & ~1u;  // even: every table starts 16-byte aligned
            if (adaptive) rnk += J.R;
        }
        accc += J.B;
        if (!J.pieces) items += (uint64_t)((J.W + 31) / 32) * J.nchunk;
        if (!J.pieces) tiles += J.ntiles;
    }
    // one input arena: z64 (FP64 study mode) | z32 | ranks (adaptive sampling) | wavelength
    // points | ray points | designs | jobs | parameter records | table jobs | Control words, in
    // 256-byte sections. A pass uploads its tail: from the z tables on where the host made one,
    // from the points on where the caller gave them, else from the designs on; the tables that
    // it makes on the device, and those resident from the previous pass, are not uploaded.
    auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
    const bool f64 = mode == CPD_TRACE_FP64;
    const size_t o_z64 = 0;
    const size_t o_z32 = o_z64 + (f64 ? al(sizeof(double) * ray) : 0);
    const size_t o_rank = o_z32 + al(2 * sizeof(float) * ray);
    const size_t o_lam = o_rank + al(sizeof(uint32_t) * rnk);
    const size_t o_u = o_lam + al(sizeof(double) * lam);
    const size_t o_des = o_u + al(sizeof(double) * upts);
    const size_t o_job = o_des + al(sizeof(DevDesign) * n);
    const size_t o_par = o_job + al(sizeof(DesignJob) * n);  // parameter records (device builds)
    const size_t o_tab = o_par + (on_device ? al(sizeof(cpd_spectrometer_params) * n) : 0);
    // the pass's Control words close the arena: uploaded as zeros with the inputs (one copy
    // node instead of a copy and a memset ahead of the first kernel)
    const size_t o_ctl = o_tab + al(sizeof(TableJob) * tabs.size());
    const size_t in_bytes = o_ctl + sizeof(Control);
    const size_t ctl_off = al(sizeof(DesignOut) * n);
    const size_t out_bytes = ctl_off + sizeof(HostStatus);
    CPD_TRY(S.h_in.ensure(in_bytes));
    CPD_TRY(S.h_outs.ensure(out_bytes, true));
    const void *in_before = S.in.p;
    CPD_TRY(S.in.ensure(in_bytes));
    // the tables already on the device from the previous pass of this slot
    tables_key.push_back(adaptive ? &kSamplingBits : nullptr);  // the rank section
    tables_key.push_back(f64 ? &kSamplingBits : nullptr);       // the z64 section
    tables_key.push_back(S.in.p);
    const bool resident = cacheable && S.in.p == in_before && tables_key == S.tables_key;
    // a device build writes the design records itself: they are not uploaded
    const size_t up_off = any_host && !resident ? 0 : lam || upts ? o_lam : on_device ? o_job : o_des;
    const size_t up_bytes = in_bytes - up_off;
    char *hin = S.h_in.as<char>();
    std::memset(hin + o_ctl, 0, sizeof(Control));
    for (uint32_t i = 0; i < n; i++) {
        if (on_device) reinterpret_cast<cpd_spectrometer_params *>(hin + o_par)[i] = *ds[i].params;
        else reinterpret_cast<DevDesign *>(hin + o_des)[i] = *ds[i].dev;
        reinterpret_cast<DesignJob *>(hin + o_job)[i] = jobs[i];
        if (owns_lam[i])
            std::memcpy(reinterpret_cast<double *>(hin + o_lam) + jobs[i].lam_off, ds[i].lam_u, sizeof(double) * jobs[i].W);
        if (resident || !owns_rays[i]) continue;
        if (!ds[i].rays) continue;
        if (f64)
            std::memcpy(reinterpret_cast<double *>(hin + o_z64) + jobs[i].ray_off, ds[i].rays->z64.data(),
                        sizeof(double) * jobs[i].Rz);
        std::memcpy(reinterpret_cast<float *>(hin + o_z32) + 2 * jobs[i].ray_off, ds[i].rays->z32.data(),
                    2 * sizeof(float) * jobs[i].Rz);
        if (adaptive)
            std::memcpy(reinterpret_cast<uint32_t *>(hin + o_rank) + jobs[i].rank_off, ds[i].rays->rank.data(),
                        sizeof(uint32_t) * jobs[i].R);
    }
    if (resident) tabs.clear();
    const uint32_t nsort =
        (uint32_t)(std::stable_partition(tabs.begin(), tabs.end(), [](const TableJob &t) { return !t.order; }) - tabs.begin());
    if (!tabs.empty()) std::memcpy(hin + o_tab, tabs.data(), sizeof(TableJob) * tabs.size());
    for (uint32_t i = 0; i < n; i++)
        if (owns_rays[i] && !ds[i].rays && !ds[i].seeded)
            for (const TableJob &t : tabs)
                if (t.points && t.ray_off == jobs[i].ray_off)
                    std::memcpy(reinterpret_cast<double *>(hin + o_u) + t.u_off, ds[i].ray_u, sizeof(double) * t.R);
    if (cacheable) {
        S.tables_key = tables_key;
        S.tables_refs.clear();
        for (const PassDesign &p : ds)
            if (p.rays_keep) S.tables_refs.push_back(p.rays_keep);
    } else {
        S.tables_key.clear();
        S.tables_refs.clear();
    }
    // device buffers (a reallocation retires the captured graphs that hold the old addresses)
    const void *bufs_before[] = {S.lp.p, S.lx.p, S.hist.p, S.S1.p, S.S2.p, S.acc.p, S.queue.p, S.h_in.p, S.h_outs.p, S.perm.p, in_before};
    const size_t hist_bytes = sizeof(unsigned long long) * std::max<uint64_t>(hist, 1);
    const size_t old_hist = S.hist.cap;
    // the LamParams, then (single-design passes) one span per 32-row block
    // or, where rows_kernel's teams are small, a HeavyRow for each
    const bool heavy = groups && plan.team < kRowsWarps &&
                       (n > 1 || (uint64_t)plan.group * rule.max_R / plan.team >= kRowsHeavyGroup);
    CPD_TRY(S.lp.ensure(sizeof(LamParams) * std::max<uint64_t>(rows, 1) + sizeof(uint2) * ((rows + 31) / 32) +
                        (heavy ? 16u + sizeof(HeavyRow) * rows : 0)));
    CPD_TRY(S.lx.ensure(sizeof(LamDF) * std::max<uint64_t>(rows, 1)));
    CPD_TRY(S.hist.ensure(hist_bytes));
    if (S.hist.cap != old_hist) S.hist_dirty = true;
    CPD_TRY(S.S1.ensure(sizeof(unsigned long long) * std::max<uint64_t>(accc, 1)));
    CPD_TRY(S.S2.ensure(sizeof(unsigned long long) * std::max<uint64_t>(accc, 1)));
    CPD_TRY(S.acc.ensure(sizeof(DesignAcc) * n));
    CPD_TRY(S.queue.ensure(sizeof(QEntry) * S.qcap));
    if (p_out_host) CPD_TRY(S.pout.ensure(sizeof(double) * cells));
    CPD_TRY(S.perm.ensure(sizeof(uint32_t) * std::max<uint64_t>(nsort ? ray : 1, 1)));
    S.ctl_off = ctl_off;
    {
        const void *after[] = {S.lp.p, S.lx.p, S.hist.p, S.S1.p, S.S2.p, S.acc.p, S.queue.p, S.h_in.p, S.h_outs.p, S.perm.p, S.in.p};
        if (!std::equal(std::begin(after), std::end(after), std::begin(bufs_before))) S.buf_gen++;
    }

    cudaStream_t s = S.stream;
    if (S.hist_dirty) {
        CPD_TRY(cudaMemsetAsync(S.hist.p, 0, S.hist.cap, s));
        S.hist_dirty = false;
    }
    S.h2d += up_bytes;
    S.d2h += out_bytes + (p_out_host ? sizeof(double) * cells : 0);
    char *din = S.in.as<char>();

    LaunchArgs a;
    std::memset(&a, 0, sizeof(a));
    a.designs = reinterpret_cast<const DevDesign *>(din + o_des);
    a.jobs = reinterpret_cast<const DesignJob *>(din + o_job);
    a.njobs = n;
    a.total_rows = rows;
    a.total_items = items;
    a.total_groups = groups;
    a.team = plan.team;
    a.total_tiles = tiles;
    a.lam_u = reinterpret_cast<const double *>(din + o_lam);
    a.z64 = reinterpret_cast<const double *>(din + o_z64);
    a.z32 = reinterpret_cast<const float *>(din + o_z32);
    a.tables = reinterpret_cast<const TableJob *>(din + o_tab);
    a.ntables = (uint32_t)tabs.size();
    a.nsort = nsort;
    a.table_max = tabs.empty() ? 0u : table_max;
    a.ray_u = reinterpret_cast<const double *>(din + o_u);
    a.perm = S.perm.as<uint32_t>();
    a.rank = adaptive ? reinterpret_cast<const uint32_t *>(din + o_rank) : nullptr;
    a.adaptive = adaptive ? (all_exact ? 2u : 1u) : 0u;
    if (adaptive && !all_exact) {
        // (a device build decides in its record)
        uint32_t with = 0, maybe = 0;
        for (const PassDesign &p : ds) a.max_rounds = std::max(a.max_rounds, (p.R + kRoundRays - 1u) / kRoundRays);
        for (const PassDesign &p : ds) {
            with += p.dev && p.dev->fc.pieces;
            maybe += p.params && p.params->ar_coated;
        }
        a.adapt_pieces = with == n ? 1u : maybe == n ? 2u : with || maybe ? 3u : 0u;
    }
    a.max_B = max_B;
    a.lp = S.lp.as<LamParams>();
    a.lx = S.lx.as<LamDF>();
    if (heavy) a.heavy = reinterpret_cast<HeavyRow *>(S.lp.as<char>() + ((sizeof(LamParams) * rows + sizeof(uint2) * ((rows + 31) / 32) + 15u) & ~size_t(15)));
    a.hist = S.hist.as<unsigned long long>();
    a.S1 = S.S1.as<unsigned long long>();
    a.S2 = S.S2.as<unsigned long long>();
    a.acc = S.acc.as<DesignAcc>();
    a.out = reinterpret_cast<DesignOut *>(S.h_outs.dev);
    a.status = reinterpret_cast<HostStatus *>(reinterpret_cast<char *>(S.h_outs.dev) + ctl_off);
    a.ctl = reinterpret_cast<Control *>(din + o_ctl);
    a.clear_acc = fresh ? 1u : 0u;
    a.acc_cells = accc;
    a.queue = S.queue.as<QEntry>();
    a.qcap = S.qcap;
    a.ray_tile = ctx->ray_tile;
    for (uint32_t i = 0; i < n; i++)
        if (jobs[i].Rz <= kStageRays && jobs[i].Rz > a.stage_cap) a.stage_cap = jobs[i].Rz;
    a.mode = mode;
    if (mode == CPD_TRACE_FP32) {
        a.guards = no_guards();
        a.yguard_rel = 0.0;
    } else {
        a.guards = default_guards();
        a.yguard_rel = kYGuardRel;
    }
    // One host-built design with a fixed ray count: the trace splits its rays into equal
    // shares per warp (no work-item counter, no tail of unequal items) and reads the
    // design's constants as kernel parameters. The bound on rows x rays keeps each warp's
    // share arithmetic in range.
    if (n == 1 && !on_device && !adaptive && mode != CPD_TRACE_FP64 &&
        rows <= kBalancedMaxRows && rows * (uint64_t)jobs[0].Rz <= (1ull << 31)) {
        a.spans = reinterpret_cast<uint2 *>(S.lp.as<LamParams>() + rows);
        a.fc = ds[0].dev->fc;
        a.fl = fast_limits(a.fc, a.guards);
        a.one = jobs[0];
        a.one.seed = 0.0;  // not part of the graph: read from the uploaded job
    }
    // A pass of one design is short beside the events that would time it (two event nodes of the
    // graph: 6 us of a call of 38 to 50), so its kernels time it themselves, until the caller
    // asks for times.
    const bool timed = n > 1 || !use_graph || profile || ctx->timed.load();
    if (!timed)
        a.stamp = nsort ? STAMP_SORT : !tabs.empty() ? STAMP_Z : on_device ? STAMP_BUILD : STAMP_SETUP;
    a.p_out = p_out_host ? S.pout.as<double>() : nullptr;
    a.logtab = ctx->logtab.as<float>();
    if (on_device) {
        a.params = reinterpret_cast<const cpd_spectrometer_params *>(din + o_par);
        a.build_acceptance = ds[0].acceptance;
    }

    // The whole pass -- input upload, the kernels (which clear the accumulators and write the
    // results into mapped host memory) and, where it is timed, the two events around them -- is
    // one graph, captured once per signature and replayed.
    // The design constants of a single-design pass are not part of the key: the cached
    // graph's trace node gets them per call.
    std::vector<uint8_t> key(sizeof(a) + 9 * sizeof(uint64_t));
    {
        LaunchArgs ka = a;
        std::memset(&ka.fc, 0, sizeof(ka.fc));
        std::memset(&ka.fl, 0, sizeof(ka.fl));
        std::memcpy(key.data(), &ka, sizeof(ka));
    }
    const uint64_t extra[9] = {n, ctx->warps_per_cta, (uint64_t)ctx->num_sms, in_bytes, up_off,
                               out_bytes, fresh ? accc + 1 : 0, S.buf_gen, (uint64_t)(uintptr_t)S.h_in.p};
    std::memcpy(key.data() + sizeof(a), extra, sizeof(extra));
    auto record = [&](cudaStream_t st, bool capturing) -> int {
        const unsigned evf = capturing ? cudaEventRecordExternal : cudaEventRecordDefault;
        // the per-design accumulators are cleared by the setup kernel (clear_acc), the
        // Control words arrive zeroed with the inputs, and the results are written into
        // mapped host memory: one copy ahead of the kernels
        cudaMemcpyAsync(S.in.as<char>() + up_off, S.h_in.as<char>() + up_off, up_bytes, cudaMemcpyHostToDevice, st);
        // External: under stream capture these become event-record nodes of the graph
        if (timed) cudaEventRecordWithFlags(S.ev0, st, evf);
        const int l = launch_pass(a, ctx->num_sms, ctx->warps_per_cta, st, profile ? S.kev : nullptr, true);
        if (timed) cudaEventRecordWithFlags(S.ev1, st, evf);
        return l;
    };
    if (use_graph && !profile) {
        auto hit = std::find_if(S.graphs.begin(), S.graphs.end(),
                                [&](const PassSlot::CachedGraph &c) { return c.key == key; });
        if (hit == S.graphs.end()) {
            cudaGraph_t g = nullptr;
            CPD_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
            const int launches = record(s, true);
            CPD_TRY(cudaStreamEndCapture(s, &g));
            cudaGraphExec_t exec = nullptr;
            const cudaError_t e = cudaGraphInstantiate(&exec, g, 0);
            if (e != cudaSuccess) cudaGraphDestroy(g);
            CPD_TRY(e);
            PassSlot::CachedGraph c{key, exec, launches};
            c.args = a;
            if (a.spans) {
                c.graph = g;
                c.trace_node = find_kernel_node(g, single_trace_kernel_fn(a));
                if (!c.trace_node) {
                    cudaGraphExecDestroy(exec);
                    cudaGraphDestroy(g);
                    return CPD_CUDA_ERROR;
                }
            } else {
                cudaGraphDestroy(g);
            }
            if (S.graphs.size() >= PassSlot::kGraphCache) {
                cudaGraphExecDestroy(S.graphs.back().exec);
                if (S.graphs.back().graph) cudaGraphDestroy(S.graphs.back().graph);
                S.graphs.pop_back();
            }
            S.graphs.insert(S.graphs.begin(), c);
        } else if (hit != S.graphs.begin()) {
            std::rotate(S.graphs.begin(), hit, hit + 1);  // most recently used first
        }
        PassSlot::CachedGraph &cg = S.graphs.front();
        if (cg.trace_node && (std::memcmp(&cg.args.fc, &a.fc, sizeof(a.fc)) != 0 ||
                              std::memcmp(&cg.args.fl, &a.fl, sizeof(a.fl)) != 0)) {
            cudaKernelNodeParams kp{};
            CPD_TRY(cudaGraphKernelNodeGetParams(cg.trace_node, &kp));
            void *args[] = {&a};
            kp.kernelParams = args;
            kp.extra = nullptr;
            CPD_TRY(cudaGraphExecKernelNodeSetParams(cg.exec, cg.trace_node, &kp));
            cg.args = a;
        }
        CPD_TRY(cudaGraphLaunch(cg.exec, s));
        S.launches = cg.launches;
    } else {
        S.launches = record(s, false);
        CPD_TRY(cudaGetLastError());
    }
    if (p_out_host)
        CPD_TRY(cudaMemcpyAsync(p_out_host, S.pout.p, sizeof(double) * cells, cudaMemcpyDeviceToHost, s));
    CPD_TRY(cudaEventRecord(S.done, s));
    S.n = n;
    S.hist_cells = hist;
    S.p_out_host = p_out_host;
    S.profiled = profile;
    S.timed = timed;
    return CPD_OK;
}

// Collects the results of the pass issued on `S` (its `done` event has completed).
int pass_finish(PassSlot &S, PassResult &res)
{
    CPD_TRY(cudaEventSynchronize(S.done));
    const HostStatus *c = reinterpret_cast<const HostStatus *>(S.h_outs.as<char>() + S.ctl_off);
    float ms = 0.f;
    if (S.timed) cudaEventElapsedTime(&ms, S.ev0, S.ev1);
    S.last_ms = S.timed ? ms : c->t1 > c->t0 ? (double)(c->t1 - c->t0) * 1e-6 : 0.0;
    if (S.profiled)
        for (int i = 0; i < 4; i++) {
            float km = 0.f;
            cudaEventElapsedTime(&km, S.kev[i], S.kev[i + 1]);
            S.kernel_ms[i] = km;
        }
    res.overflow = (c->overflow & kOverflowQueue) != 0 || c->queue_count > S.qcap;
    res.bad_table = (c->overflow & kOverflowTable) != 0;
    if (res.overflow || res.bad_table) S.hist_dirty = true;
    if (res.bad_table) S.tables_key.clear();
    res.outs.assign(S.h_outs.as<DesignOut>(), S.h_outs.as<DesignOut>() + S.n);
    return CPD_OK;
}

// rays: the fixed-N estimator's ray count; under adaptive sampling the rays actually
// consumed (counted on the device) replace it.
void fill_fitness(const DesignOut &o, uint64_t rays, cpd_fitness &f, bool need_conv, bool adaptive = false)
{
    std::memset(&f, 0, sizeof(f));
    f.size = o.size;  // from the design record (built on the host or on the device)
    f.deviation = o.deviation;
    f.info = o.info;
    f.h_cond = o.h_cond;
    f.h_det = o.h_det;
    f.max_sem = o.max_sem;
    f.rays = adaptive ? o.fast : rays;
    f.hits = o.hits;
    f.retraced = o.retraced;
    f.fast_rays = adaptive ? o.fast - std::min(o.fast, o.retraced) : o.fast;
    f.wavelengths = (uint32_t)o.rows;
    f.status = o.status ? o.status : (need_conv && !o.converged) ? CPD_NOT_CONVERGED : CPD_OK;
}

bool valid_design(const cpd_design *d)
{
    return d && d->nglass >= 1 && d->nglass <= CPD_MAX_GLASS && d->bin_count >= 1 && d->bin_count <= CPD_MAX_BINS;
}

// A CPD_TRACE_* value, optionally with CPD_SAMPLING_ADAPTIVE (hybrid trace only) and
// then CPD_SAMPLING_EXACT.
bool valid_mode(uint32_t m)
{
    const uint32_t t = m & ~kSamplingBits, smp = m & kSamplingBits;
    if (t > CPD_TRACE_FP64) return false;
    return smp == 0u || (t == CPD_TRACE_HYBRID && (smp & CPD_SAMPLING_ADAPTIVE));
}

bool is_adaptive(uint32_t m) { return (m & CPD_SAMPLING_ADAPTIVE) != 0u; }

// What the pass needs of a parameter record before the device builds it (the build
// checks the rest and reports failures per design).
bool valid_params(const cpd_spectrometer_params &p)
{
    return p.nglass >= 1 && p.nglass <= CPD_MAX_GLASS && p.bin_count >= 1 && p.bin_count <= CPD_MAX_BINS;
}

bool valid_item(const cpd_batch_item &it)
{
    return it.max_n >= 1 && it.max_n <= CPD_MAX_WAVELENGTHS && it.max_eval >= 1 && it.max_eval <= CPD_MAX_RAYS;
}

// Takes back what a pass that is run again has counted: the ray counters of its designs return to
// those of the results before it (its trace adds to them as it goes; every other sum of such a pass
// is left out by the entropy and finalize kernels).
int restore_counters(PassSlot &S, const std::vector<DesignOut> &before)
{
    static_assert(offsetof(DesignAcc, hits) + 3 * sizeof(DesignAcc::hits) == sizeof(DesignAcc), "the counters end the record");
    for (size_t i = 0; i < before.size(); i++) {
        DesignAcc c{};
        c.hits[0] = before[i].hits;
        c.retraced[0] = before[i].retraced;
        c.fast[0] = before[i].fast;
        CPD_TRY(cudaMemcpyAsync(S.acc.as<DesignAcc>()[i].hits, c.hits, 3 * sizeof(c.hits), cudaMemcpyHostToDevice, S.stream));
    }
    CPD_TRY(cudaStreamSynchronize(S.stream));
    return CPD_OK;
}

// Runs one pass on `S` to completion, growing the re-trace queue and re-running the
// pass if it overflowed, or with the host's tables if the device could not make one. Such a
// pass leaves the persistent accumulators as they were: the entropy kernel skips it, and the
// ray counters are restored (unless the re-run clears them: fresh).
int run_pass_checked(cpd_context *ctx, PassSlot &S, const std::vector<PassDesign> &pds, uint32_t mode, bool fresh,
                     double *p_out, PassResult &res, bool use_graph)
{
    std::vector<PassDesign> by_host;  // the same designs with the host's tables
    std::vector<DesignOut> before;
    if (!fresh) before.assign(S.h_outs.as<DesignOut>(), S.h_outs.as<DesignOut>() + pds.size());
    for (int attempt = 0; attempt < 7; attempt++) {
        const std::vector<PassDesign> &ds = by_host.empty() ? pds : by_host;
        int e = attempt ? restore_counters(S, before) : (int)CPD_OK;
        if (!e) e = pass_issue(ctx, S, ds, mode, fresh, p_out, use_graph, ctx->profiling);
        if (!e) e = pass_finish(S, res);
        if (e) {
            S.hist_dirty = true;
            return e;
        }
        if (res.bad_table) {
            std::vector<std::pair<double, uint32_t>> seeds;
            by_host = pds;
            for (PassDesign &p : by_host) {
                if (p.rays) continue;
                if (p.seeded) seeds.emplace_back(p.seed, p.R);
                host_table(ctx, p);
            }
            mark_host_only(ctx, seeds);
            continue;
        }
        if (!res.overflow) return CPD_OK;
        S.qcap *= 4;
    }
    return CPD_NO_CAPACITY;
}

// Whether every design of a batch goes through rows_kernel, which has no launch shape to tune.
bool all_by_rows(const std::vector<PassDesign> &ds, uint32_t mode)
{
    return rows_rule(ds, mode).on && std::all_of(ds.begin(), ds.end(), coated);
}

// The class of a batch for the launch-shape cache: trace mode, whether it has a shape to tune, and
// the binary orders of magnitude of its design count, wavelength rows, rays and widest detector.
std::array<uint64_t, 6> tune_class(const std::vector<PassDesign> &ds, uint32_t mode)
{
    uint64_t rows = 0, rays = 0, maxB = 0;
    for (const PassDesign &p : ds) {
        rows += p.W;
        rays += (uint64_t)p.W * p.R;
        maxB = std::max<uint64_t>(maxB, p.params ? p.params->bin_count : p.dev->B);
    }
    auto lg = [](uint64_t v) {
        uint64_t b = 0;
        while ((1ull << b) < v && b < 63) b++;
        return b;
    };
    return {mode, all_by_rows(ds, mode), lg(ds.size()), lg(rows), lg(rays), lg(maxB)};
}

// The autotuner: times every (ray tile, warps per CTA) candidate on the batch itself
// (captured graph, two timed passes after one warm-up each, minimum device time) and
// keeps the fastest. Results do not depend on the launch shape (integer accumulation),
// so any candidate is safe to pick.
int tune_pass(cpd_context *ctx, const std::vector<PassDesign> &ds, uint32_t mode, double *best_ms)
{
    static const uint32_t kTiles[] = {4, 8, 16, 32, 64, 128, 256};
    static const uint32_t kWarps[] = {2, 4, 8};
    const uint32_t rt0 = ctx->ray_tile, w0 = ctx->warps_per_cta;
    const bool timed = ctx->timed.exchange(true);
    double best = 1e300;
    uint32_t brt = rt0, bw = w0;
    PassResult res;
    // Besides the powers of two: tiles that make the work items a whole number of rounds
    // of the resident warps (2..6 items per warp), so that the last round is not a tail.
    std::vector<std::pair<uint32_t, uint32_t>> cands;
    const bool pieces = all_by_rows(ds, mode);
    if (pieces) cands.push_back({rt0, w0});  // no work items: the caller's shape stays
    for (uint32_t w : kWarps) {
        if (pieces) break;
        for (uint32_t rt : kTiles) cands.push_back({rt, w});
        uint64_t blocks = 0, rays = 0;
        for (const PassDesign &p : ds) {
            blocks += (p.W + 31) / 32;
            rays += (uint64_t)((p.W + 31) / 32) * (p.rays ? p.rays->z64.size() : p.R);
        }
        const uint64_t warps = trace_resident_warps(ctx->num_sms, w);
        for (uint64_t k = 2; k <= 6 && blocks; k++) {
            const uint64_t per = (rays + k * warps - 1) / (k * warps);  // rays per item
            if (per >= 2 && per <= 4096) cands.push_back({(uint32_t)per, w});
        }
    }
    for (const auto &cw : cands) {
        const uint32_t rt = cw.first, w = cw.second;
        {
            ctx->ray_tile = rt;
            ctx->warps_per_cta = w;
            double m = 1e300;
            for (int k = 0; k < 3; k++) {
                const int e = run_pass_checked(ctx, ctx->main, ds, mode, true, nullptr, res, ctx->use_graphs);
                if (e) {
                    ctx->ray_tile = rt0;
                    ctx->warps_per_cta = w0;
                    ctx->timed = timed;
                    return e;
                }
                if (k) m = std::min(m, ctx->main.last_ms);
            }
            if (m < best) {
                best = m;
                brt = rt;
                bw = w;
            }
        }
    }
    ctx->ray_tile = brt;
    ctx->warps_per_cta = bw;
    ctx->timed = timed;
    ctx->tune_cache[tune_class(ds, mode)] = {brt, bw};
    if (best_ms) *best_ms = best;
    return CPD_OK;
}

// A pass's design under the seed policy.
PassDesign seeded_design(cpd_context *ctx, const DevDesign *dev, double seed, uint32_t W, uint32_t R, uint32_t mode)
{
    PassDesign p{};
    p.dev = dev;
    p.W = W;
    p.R = R;
    p.seeded = true;
    p.seed = seed;
    choose_table(ctx, p, mode);
    return p;
}

// Builds the pass inputs of a batch (host copies kept alive by the caller's vectors).
void batch_inputs(cpd_context *ctx, const cpd_design *designs, const cpd_batch_item *items, uint32_t n, uint32_t mode,
                  std::vector<DevDesign> &devs, std::vector<PassDesign> &ds)
{
    devs.resize(n);
    ds.reserve(n);
    for (uint32_t i = 0; i < n; i++) {
        design_to_dev(designs[i], devs[i]);
        ds.push_back(seeded_design(ctx, &devs[i], items[i].seed, items[i].max_n, items[i].max_eval, mode));
    }
}

}  // namespace

namespace cpd {
int context_device(const cpd_context *ctx) { return ctx->device; }
int context_sms(const cpd_context *ctx) { return ctx->num_sms; }
const float *context_logtab(const cpd_context *ctx) { return ctx->logtab.as<float>(); }
RayTablePtr context_ray_table(cpd_context *ctx, double seed, uint32_t R) { return ray_table_cached(ctx, seed, R); }
LamPtr context_lam_points(cpd_context *ctx, double seed, uint32_t W) { return lam_points_cached(ctx, seed, W); }
void fitness_from_out(const DesignOut &o, uint64_t rays, cpd_fitness &f) { fill_fitness(o, rays, f, true, false); }
}  // namespace cpd

// ------------------------------------------------------------------ the server

namespace {
struct SrvRequest {
    std::vector<cpd_design> designs;
    std::vector<cpd_spectrometer_params> params;  // instead of designs: built on the device
    double acceptance = 0.0;
    std::vector<cpd_batch_item> items;
    std::vector<cpd_fitness> outs;
    uint32_t remaining = 0;
    uint32_t mode = 0;
    int status = CPD_OK;
    bool done = false;
    std::chrono::steady_clock::time_point t_submit, t_done;
};
struct SrvWork {
    uint64_t req;
    uint32_t idx;
    uint64_t bytes;
};
}  // namespace

struct cpd_server {
    cpd_context *ctx = nullptr;
    std::vector<std::unique_ptr<PassSlot>> slots;
    std::vector<std::vector<SrvWork>> slot_work;
    std::vector<bool> busy;
    uint64_t budget = 0, in_use = 0;
    uint32_t max_designs_per_pass = 256;
    std::mutex mu;
    std::condition_variable cv_work, cv_done;
    std::deque<SrvWork> pending;
    std::map<uint64_t, SrvRequest> reqs;
    uint64_t next_id = 1;
    std::thread worker;
    bool stop = false;
    uint64_t designs_done = 0, passes = 0, max_in_flight = 0;
};

namespace {

// Completes the pass on slot i (called by the worker without the lock held for the
// device wait; the lock is taken to publish results).
void srv_complete(cpd_server *sv, size_t i)
{
    PassSlot &S = *sv->slots[i];
    PassResult res;
    int e = pass_finish(S, res);
    std::lock_guard<std::mutex> lk(sv->mu);
    auto &work = sv->slot_work[i];
    if (!e && (res.overflow || res.bad_table)) e = CPD_NO_CAPACITY;  // re-queued below
    if (e == CPD_NO_CAPACITY && (S.qcap < (1u << 26) || res.bad_table)) {
        // run the same designs again, with a larger re-trace queue (up to a limit) or the host's tables
        if (res.overflow && S.qcap < (1u << 26)) S.qcap *= 4;
        if (res.bad_table) {
            std::vector<std::pair<double, uint32_t>> seeds;
            for (const SrvWork &wk : work) {
                auto rit = sv->reqs.find(wk.req);
                if (rit != sv->reqs.end()) seeds.emplace_back(rit->second.items[wk.idx].seed, rit->second.items[wk.idx].max_eval);
            }
            mark_host_only(sv->ctx, seeds);
        }
        for (auto it = work.rbegin(); it != work.rend(); ++it) {
            sv->in_use -= it->bytes;
            sv->pending.push_front(*it);
        }
        e = CPD_OK;
        work.clear();
    }
    for (size_t k = 0; k < work.size(); k++) {
        auto rit = sv->reqs.find(work[k].req);
        if (rit == sv->reqs.end()) continue;
        SrvRequest &r = rit->second;
        if (e) r.status = e;
        else fill_fitness(res.outs[k], (uint64_t)r.items[work[k].idx].max_n * r.items[work[k].idx].max_eval,
                          r.outs[work[k].idx], true, is_adaptive(r.mode));
        if (--r.remaining == 0) {
            r.done = true;
            r.t_done = std::chrono::steady_clock::now();
        }
        sv->designs_done++;
    }
    for (auto &w : work) sv->in_use -= w.bytes;
    work.clear();
    sv->busy[i] = false;
    sv->passes++;
    sv->cv_done.notify_all();
}

void srv_loop(cpd_server *sv)
{
    cudaSetDevice(sv->ctx->device);
    for (;;) {
        bool progressed = false;
        // completions
        for (size_t i = 0; i < sv->slots.size(); i++) {
            bool b;
            {
                std::lock_guard<std::mutex> lk(sv->mu);
                b = sv->busy[i];
            }
            if (b && cudaEventQuery(sv->slots[i]->done) != cudaErrorNotReady) {
                srv_complete(sv, i);
                progressed = true;
            }
        }
        // admissions: each free slot takes the oldest pending designs of one trace mode
        // while they fit the device-memory budget
        for (size_t i = 0; i < sv->slots.size(); i++) {
            std::vector<SrvWork> take;
            std::vector<DevDesign> devs;
            uint32_t mode = 0;
            {
                std::lock_guard<std::mutex> lk(sv->mu);
                if (sv->busy[i] || sv->pending.empty()) continue;
                bool others = false;
                for (size_t j = 0; j < sv->slots.size(); j++) others |= sv->busy[j];
                const SrvRequest &r0 = sv->reqs[sv->pending.front().req];
                mode = r0.mode;
                const bool dev0 = !r0.params.empty();
                const double acc0 = r0.acceptance;
                while (!sv->pending.empty() && take.size() < sv->max_designs_per_pass) {
                    const SrvWork &w = sv->pending.front();
                    // a pass holds designs of one trace mode and one kind (built on the host,
                    // or on the device with one acceptance)
                    const SrvRequest &rw = sv->reqs[w.req];
                    if (rw.mode != mode || rw.params.empty() != !dev0 || rw.acceptance != acc0) break;
                    if (sv->in_use + w.bytes > sv->budget && (others || !take.empty())) break;
                    sv->in_use += w.bytes;
                    take.push_back(w);
                    sv->pending.pop_front();
                }
                if (take.empty()) continue;
                sv->busy[i] = true;
                sv->slot_work[i] = take;
                uint64_t nb = 0;
                for (size_t j = 0; j < sv->slots.size(); j++) nb += sv->busy[j];
                sv->max_in_flight = std::max<uint64_t>(sv->max_in_flight, nb);
            }
            // host preparation and issue without the lock (the slot belongs to the worker)
            std::vector<PassDesign> ds(take.size());
            devs.resize(take.size());
            for (size_t k = 0; k < take.size(); k++) {
                const SrvRequest *r;
                {
                    std::lock_guard<std::mutex> lk(sv->mu);
                    r = &sv->reqs[take[k].req];
                }
                const cpd_batch_item &it = r->items[take[k].idx];
                if (r->params.empty()) design_to_dev(r->designs[take[k].idx], devs[k]);
                ds[k] = seeded_design(sv->ctx, &devs[k], it.seed, it.max_n, it.max_eval, mode);
                if (!r->params.empty()) {
                    ds[k].dev = nullptr;
                    ds[k].params = &r->params[take[k].idx];
                    ds[k].acceptance = r->acceptance;
                }
            }
            int e = pass_issue(sv->ctx, *sv->slots[i], ds, mode, true, nullptr, false, false);
            if (e) {
                std::lock_guard<std::mutex> lk(sv->mu);
                sv->slots[i]->hist_dirty = true;
                for (auto &w : take) {
                    SrvRequest &r = sv->reqs[w.req];
                    r.status = e;
                    if (--r.remaining == 0) {
                        r.done = true;
                        r.t_done = std::chrono::steady_clock::now();
                    }
                    sv->in_use -= w.bytes;
                }
                sv->busy[i] = false;
                sv->slot_work[i].clear();
                sv->cv_done.notify_all();
            }
            progressed = true;
        }
        {
            std::unique_lock<std::mutex> lk(sv->mu);
            bool any_busy = false;
            for (bool b : sv->busy) any_busy |= b;
            if (sv->stop && !any_busy && sv->pending.empty()) return;
            if (!progressed) {
                if (any_busy) {
                    lk.unlock();
                    std::this_thread::sleep_for(std::chrono::microseconds(20));
                } else {
                    sv->cv_work.wait_for(lk, std::chrono::milliseconds(50));
                }
            }
        }
    }
}

}  // namespace

// ------------------------------------------------------------------ C ABI

extern "C" {

int cpd_context_create(int device, cpd_context **out)
{
    if (!out) return CPD_INVALID_ARGUMENT;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) return CPD_CUDA_ERROR;
    if (cudaSetDevice(device) != cudaSuccess) return CPD_CUDA_ERROR;
    cpd_context *ctx = new cpd_context();
    ctx->device = device;
    cudaDeviceGetAttribute(&ctx->num_sms, cudaDevAttrMultiProcessorCount, device);
    std::vector<float> tab(4 * ff::kLogTable);
    ff::make_log_table(tab.data());
    if (configure_kernels() != cudaSuccess || ctx->main.create() != cudaSuccess || ctx->logtab.ensure(sizeof(float) * tab.size()) != cudaSuccess ||
        cudaMemcpyAsync(ctx->logtab.p, tab.data(), sizeof(float) * tab.size(), cudaMemcpyHostToDevice, ctx->main.stream) !=
            cudaSuccess ||
        cudaStreamSynchronize(ctx->main.stream) != cudaSuccess) {  // every slot's stream reads it
        ctx->main.destroy();
        ctx->logtab.release();
        delete ctx;
        return CPD_CUDA_ERROR;
    }
    *out = ctx;
    return CPD_OK;
}

void cpd_context_destroy(cpd_context *ctx)
{
    if (!ctx) return;
    cudaSetDevice(ctx->device);
    ctx->main.destroy();
    {
        OrderDevice dev{nullptr};
        ctx->orders.release(dev);
    }
    for (DevBuf *b : {&ctx->tp_design, &ctx->tp_lam, &ctx->tp_z, &ctx->tp_out, &ctx->tp_rays, &ctx->tp_tab, &ctx->tp_lp,
                      &ctx->tp_t64})
        b->release();
    for (DevBuf *b : {&ctx->bld_params, &ctx->bld_out, &ctx->bld_status, &ctx->pair_design, &ctx->pair_lam,
                      &ctx->pair_z, &ctx->pair_bins, &ctx->pair_ts,
                      &ctx->pair_flags, &ctx->peak, &ctx->logtab})
        b->release();
    delete ctx;
}

int cpd_set_launch_shape(cpd_context *ctx, uint32_t ray_tile, uint32_t warps_per_cta)
{
    if (!ctx) return CPD_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> lk(ctx->mu);
    if (ray_tile) ctx->ray_tile = std::min<uint32_t>(ray_tile, CPD_MAX_RAYS);
    if (warps_per_cta) {
        if (warps_per_cta > 8) return CPD_INVALID_ARGUMENT;
        ctx->warps_per_cta = warps_per_cta;
    }
    return CPD_OK;
}

int cpd_get_launch_shape(cpd_context *ctx, uint32_t *ray_tile, uint32_t *warps_per_cta)
{
    if (!ctx) return CPD_INVALID_ARGUMENT;
    if (ray_tile) *ray_tile = ctx->ray_tile;
    if (warps_per_cta) *warps_per_cta = ctx->warps_per_cta;
    return CPD_OK;
}

int cpd_last_timing(cpd_context *ctx, double *kernel_ms, uint32_t *launches)
{
    if (!ctx) return CPD_INVALID_ARGUMENT;
    if (kernel_ms) *kernel_ms = ctx->main.last_ms;
    if (kernel_ms) ctx->timed = true;
    if (launches) *launches = (uint32_t)ctx->main.launches;
    return CPD_OK;
}

int cpd_set_profiling(cpd_context *ctx, int on)
{
    if (!ctx) return CPD_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> lk(ctx->mu);
    ctx->profiling = on != 0;
    return CPD_OK;
}

int cpd_last_kernel_times(cpd_context *ctx, double ms[4])
{
    if (!ctx || !ms) return CPD_INVALID_ARGUMENT;
    for (int i = 0; i < 4; i++) ms[i] = ctx->main.kernel_ms[i];
    return CPD_OK;
}

int cpd_last_transfer_bytes(cpd_context *ctx, uint64_t *h2d, uint64_t *d2h)
{
    if (!ctx) return CPD_INVALID_ARGUMENT;
    if (h2d) *h2d = ctx->main.h2d;
    if (d2h) *d2h = ctx->main.d2h;
    return CPD_OK;
}

#define CPD_SYNC_ENTRY(ctx)                                                 \
    std::lock_guard<std::mutex> lk((ctx)->mu);                              \
    if (cudaSetDevice((ctx)->device) != cudaSuccess) return CPD_CUDA_ERROR; \
    (ctx)->main.h2d = (ctx)->main.d2h = 0

int cpd_fitness_gpu_points(cpd_context *ctx, const cpd_design *d, const double *lam_u, uint32_t W,
                           const double *ray_u, uint32_t R, uint32_t trace_mode, cpd_fitness *out, double *p_out)
{
    if (!ctx || !valid_design(d) || !lam_u || !ray_u || !out) return CPD_INVALID_ARGUMENT;
    if (W == 0 || W > CPD_MAX_WAVELENGTHS || R == 0 || R > CPD_MAX_RAYS || !valid_mode(trace_mode))
        return CPD_INVALID_ARGUMENT;
    CPD_SYNC_ENTRY(ctx);
    DevDesign D;
    design_to_dev(*d, D);
    std::vector<PassDesign> ds(1);
    ds[0].dev = &D;
    ds[0].W = W;
    ds[0].R = R;
    ds[0].lam_u = lam_u;
    ds[0].ray_u = ray_u;
    choose_table(ctx, ds[0], trace_mode);
    PassResult res;
    int e = run_pass_checked(ctx, ctx->main, ds, trace_mode, true, p_out, res, ctx->use_graphs);
    if (e) return e;
    fill_fitness(res.outs[0], (uint64_t)W * R, *out, false, is_adaptive(trace_mode));
    return CPD_OK;
}

int cpd_fitness_gpu(cpd_context *ctx, const cpd_design *d, const double *seeds, uint32_t nseeds, uint32_t max_n,
                    uint32_t nwarp, uint32_t max_eval, cpd_fitness *out)
{
    return cpd_fitness_gpu_ex(ctx, d, seeds, nseeds, max_n, nwarp, max_eval, 0u, out);
}

int cpd_fitness_gpu_ex(cpd_context *ctx, const cpd_design *d, const double *seeds, uint32_t nseeds, uint32_t max_n,
                       uint32_t nwarp, uint32_t max_eval, uint32_t sampling, cpd_fitness *out)
{
    if (!ctx || !valid_design(d) || !seeds || !out || nseeds == 0) return CPD_INVALID_ARGUMENT;
    if (max_n == 0 || max_eval == 0 || max_eval > CPD_MAX_RAYS) return CPD_INVALID_ARGUMENT;
    if ((uint64_t)max_n * nseeds > CPD_MAX_WAVELENGTHS) return CPD_INVALID_ARGUMENT;
    const uint32_t mode = CPD_TRACE_HYBRID | sampling;
    if ((sampling & ~kSamplingBits) || !valid_mode(mode)) return CPD_INVALID_ARGUMENT;
    CPD_SYNC_ENTRY(ctx);
    // the adaptive kernels have no launch shape to tune
    const bool tune = ctx->autotune && !ctx->profiling && !is_adaptive(mode);
    if (!tune && nwarp >= 1 && nwarp <= 8) ctx->warps_per_cta = nwarp;
    DevDesign D;
    design_to_dev(*d, D);
    PassResult res;
    uint64_t rays = 0;
    for (uint32_t s = 0; s < nseeds; s++) {
        const std::vector<PassDesign> ds{seeded_design(ctx, &D, seeds[s], max_n, max_eval, mode)};
        if (tune && s == 0) {
            // the autotuner replaces the reference's nwarp hint
            auto it = ctx->tune_cache.find(tune_class(ds, mode));
            if (it != ctx->tune_cache.end()) {
                ctx->ray_tile = it->second.first;
                ctx->warps_per_cta = it->second.second;
            } else {
                const int te = tune_pass(ctx, ds, mode, nullptr);
                if (te) return te;
            }
        }
        int e = run_pass_checked(ctx, ctx->main, ds, mode, s == 0, nullptr, res, ctx->use_graphs);
        if (e) return e;
        rays += (uint64_t)max_n * max_eval;
        if (res.outs[0].converged) break;
    }
    fill_fitness(res.outs[0], rays, *out, true, is_adaptive(mode));
    return out->status;
}

int cpd_fitness_gpu_batch(cpd_context *ctx, const cpd_design *designs, const cpd_batch_item *items, uint32_t n,
                          uint32_t trace_mode, cpd_fitness *outs)
{
    if (!ctx || !designs || !items || !outs || n == 0 || !valid_mode(trace_mode)) return CPD_INVALID_ARGUMENT;
    for (uint32_t i = 0; i < n; i++)
        if (!valid_design(&designs[i]) || !valid_item(items[i])) return CPD_INVALID_ARGUMENT;
    CPD_SYNC_ENTRY(ctx);
    std::vector<DevDesign> devs;
    std::vector<PassDesign> ds;
    batch_inputs(ctx, designs, items, n, trace_mode, devs, ds);
    if (ctx->autotune && !ctx->profiling && !is_adaptive(trace_mode)) {
        auto it = ctx->tune_cache.find(tune_class(ds, trace_mode));
        if (it != ctx->tune_cache.end()) {
            ctx->ray_tile = it->second.first;
            ctx->warps_per_cta = it->second.second;
        } else {
            const int te = tune_pass(ctx, ds, trace_mode, nullptr);
            if (te) return te;
        }
    }
    PassResult res;
    int e = run_pass_checked(ctx, ctx->main, ds, trace_mode, true, nullptr, res, ctx->use_graphs);
    if (e) return e;
    for (uint32_t i = 0; i < n; i++)
        fill_fitness(res.outs[i], (uint64_t)items[i].max_n * items[i].max_eval, outs[i], true,
                     is_adaptive(trace_mode));
    return CPD_OK;
}

int cpd_fitness_gpu_batch_params(cpd_context *ctx, const cpd_spectrometer_params *params,
                                 const cpd_batch_item *items, uint32_t n, double acceptance, uint32_t trace_mode,
                                 cpd_fitness *outs)
{
    if (!ctx || !params || !items || !outs || n == 0 || !valid_mode(trace_mode)) return CPD_INVALID_ARGUMENT;
    if (acceptance != 0.0 && !(acceptance > 0.0 && acceptance <= 1.0)) return CPD_INVALID_ARGUMENT;
    for (uint32_t i = 0; i < n; i++)
        if (!valid_params(params[i]) || !valid_item(items[i])) return CPD_INVALID_ARGUMENT;
    CPD_SYNC_ENTRY(ctx);
    std::vector<PassDesign> ds;
    ds.reserve(n);
    for (uint32_t i = 0; i < n; i++) {
        ds.push_back(seeded_design(ctx, nullptr, items[i].seed, items[i].max_n, items[i].max_eval, trace_mode));
        ds[i].params = &params[i];
        ds[i].acceptance = acceptance;
    }
    if (ctx->autotune && !ctx->profiling && !is_adaptive(trace_mode)) {
        auto it = ctx->tune_cache.find(tune_class(ds, trace_mode));
        if (it != ctx->tune_cache.end()) {
            ctx->ray_tile = it->second.first;
            ctx->warps_per_cta = it->second.second;
        } else {
            const int te = tune_pass(ctx, ds, trace_mode, nullptr);
            if (te) return te;
        }
    }
    PassResult res;
    int e = run_pass_checked(ctx, ctx->main, ds, trace_mode, true, nullptr, res, ctx->use_graphs);
    if (e) return e;
    for (uint32_t i = 0; i < n; i++)
        fill_fitness(res.outs[i], (uint64_t)items[i].max_n * items[i].max_eval, outs[i], true,
                     is_adaptive(trace_mode));
    return CPD_OK;
}

int cpd_design_build_device(cpd_context *ctx, const cpd_spectrometer_params *params, uint32_t n, double acceptance,
                            cpd_design *out, int32_t *status)
{
    if (!ctx || ((!params || !out || !status) && n)) return CPD_INVALID_ARGUMENT;
    if (acceptance != 0.0 && !(acceptance > 0.0 && acceptance <= 1.0)) return CPD_INVALID_ARGUMENT;
    if (n == 0) return CPD_OK;
    CPD_SYNC_ENTRY(ctx);
    cudaStream_t s = ctx->main.stream;
    CPD_TRY(ctx->bld_params.ensure(sizeof(cpd_spectrometer_params) * n));
    CPD_TRY(ctx->bld_out.ensure(sizeof(cpd_design) * n));
    CPD_TRY(ctx->bld_status.ensure(sizeof(int32_t) * n));
    CPD_TRY(cudaMemcpyAsync(ctx->bld_params.p, params, sizeof(cpd_spectrometer_params) * n, cudaMemcpyHostToDevice, s));
    launch_build_records(ctx->bld_params.as<cpd_spectrometer_params>(), n, acceptance, ctx->bld_out.as<cpd_design>(),
                         ctx->bld_status.as<int32_t>(), s);
    CPD_TRY(cudaGetLastError());
    CPD_TRY(cudaMemcpyAsync(out, ctx->bld_out.p, sizeof(cpd_design) * n, cudaMemcpyDeviceToHost, s));
    CPD_TRY(cudaMemcpyAsync(status, ctx->bld_status.p, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, s));
    CPD_TRY(cudaStreamSynchronize(s));
    ctx->main.h2d += sizeof(cpd_spectrometer_params) * n;
    ctx->main.d2h += (sizeof(cpd_design) + sizeof(int32_t)) * n;
    return CPD_OK;
}

int cpd_autotune_batch(cpd_context *ctx, const cpd_design *designs, const cpd_batch_item *items, uint32_t n,
                       uint32_t trace_mode, uint32_t *ray_tile, uint32_t *warps_per_cta, double *best_ms)
{
    if (!ctx || !designs || !items || n == 0 || trace_mode > CPD_TRACE_FP64) return CPD_INVALID_ARGUMENT;  // fixed-N only
    for (uint32_t i = 0; i < n; i++)
        if (!valid_design(&designs[i]) || !valid_item(items[i])) return CPD_INVALID_ARGUMENT;
    CPD_SYNC_ENTRY(ctx);
    std::vector<DevDesign> devs;
    std::vector<PassDesign> ds;
    batch_inputs(ctx, designs, items, n, trace_mode, devs, ds);
    const int e = tune_pass(ctx, ds, trace_mode, best_ms);
    if (e) return e;
    if (ray_tile) *ray_tile = ctx->ray_tile;
    if (warps_per_cta) *warps_per_cta = ctx->warps_per_cta;
    return CPD_OK;
}

int cpd_set_autotune(cpd_context *ctx, int on)
{
    if (!ctx) return CPD_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> lk(ctx->mu);
    ctx->autotune = on != 0;
    return CPD_OK;
}

int cpd_transmission_probability(cpd_context *ctx, const cpd_design *d, const double *wavelengths, uint32_t n,
                                 uint32_t max_m, double *out)
{
    return cpd_transmission_probability_ex(ctx, d, wavelengths, n, max_m, 0u, out, nullptr);
}

int cpd_transmission_probability_ex(cpd_context *ctx, const cpd_design *d, const double *wavelengths, uint32_t n,
                                    uint32_t max_m, uint32_t flags, double *out, uint32_t *rays_out)
{
    if (!ctx || !valid_design(d) || !wavelengths || !out || n == 0 || n > CPD_MAX_WAVELENGTHS || max_m == 0 ||
        max_m > CPD_MAX_RAYS || (flags & ~(uint32_t)CPD_TP_FIXED_N))
        return CPD_INVALID_ARGUMENT;
    // the reference CPU ray points (fitness.rs:19): the incremental R1 sequence from 0.5
    auto ref_points = [](uint32_t m, double *u) {
        double st = 0.5;
        for (uint32_t j = 0; j < m; j++) {
            st = st + kAlpha;
            st = st - std::trunc(st);
            u[j] = st;
        }
    };
    if (flags & CPD_TP_FIXED_N) {
        // explicit wavelengths: bounds (0, 1) make wmin + (wmax - wmin)*u == u exactly
        cpd_design dd = *d;
        dd.wavelength_bounds[0] = 0.0;
        dd.wavelength_bounds[1] = 1.0;
        std::vector<double> ray_u(max_m);
        ref_points(max_m, ray_u.data());
        cpd_fitness f;
        const int e = cpd_fitness_gpu_points(ctx, &dd, wavelengths, n, ray_u.data(), max_m, CPD_TRACE_HYBRID, &f, out);
        if (!e && rays_out)
            for (uint32_t i = 0; i < n; i++) rays_out[i] = max_m;
        return e;
    }
    CPD_SYNC_ENTRY(ctx);
    PassSlot &S = ctx->main;
    cudaStream_t s = S.stream;
    DevDesign D;
    design_to_dev(*d, D);
    const bool pieces = D.fc.pieces && max_m <= kTpMaxRays;
    if (ctx->tp_m != max_m || (pieces && ctx->tp_tab_m != max_m)) {
        std::vector<double> z(max_m);
        ref_points(max_m, z.data());
        std::vector<uint32_t> order;
        if (pieces) {
            // the rays by point (spread evenly: a bucket each, then the few that share one)
            order.resize(max_m);
            std::vector<uint32_t> at(max_m + 1u, 0u);
            const auto bucket = [&](double u) { return std::min(max_m - 1u, (uint32_t)(u * max_m)); };
            for (uint32_t j = 0; j < max_m; j++) at[bucket(z[j]) + 1u]++;
            for (uint32_t b = 0; b < max_m; b++) at[b + 1u] += at[b];
            std::vector<uint32_t> next(at.begin(), at.end() - 1);
            for (uint32_t j = 0; j < max_m; j++) order[next[bucket(z[j])]++] = j;
            for (uint32_t b = 0; b < max_m; b++)
                if (at[b + 1u] - at[b] > 1u)
                    std::sort(order.begin() + at[b], order.begin() + at[b + 1u], [&](uint32_t i, uint32_t j) { return z[i] < z[j]; });
        }
        for (uint32_t j = 0; j < max_m; j++) z[j] = norminv(z[j]);
        if (ctx->tp_m != max_m) {
            ctx->tp_m = 0;
            CPD_TRY(ctx->tp_z.ensure(sizeof(double) * max_m));
            CPD_TRY(cudaMemcpyAsync(ctx->tp_z.p, z.data(), sizeof(double) * max_m, cudaMemcpyHostToDevice, s));
            CPD_TRY(cudaStreamSynchronize(s));  // z is about to go
            ctx->tp_m = max_m;
            S.h2d += sizeof(double) * max_m;
        }
        if (pieces) {
            // the counts' reciprocals, and the counts | sorted z | ranks
            ctx->tp_tab_m = 0;
            std::vector<double> tab(2u * (max_m + 2u) + (size_t)max_m + (max_m + 1u) / 2u);
            float *z32 = reinterpret_cast<float *>(tab.data() + 2u * (max_m + 2u));
            uint32_t *rank = reinterpret_cast<uint32_t *>(z32 + 2u * max_m);
            uint32_t rz = 0;
            for (uint32_t i = 0; i < max_m; i++) {
                const uint32_t j = order[i];
                rank[j] = 0xffffffffu;
                if (!std::isfinite(z[j])) continue;
                split_f32(z[j], z32[2 * rz], z32[2 * rz + 1]);
                rank[j] = rz++;
            }
            for (uint32_t c = 0; c < max_m + 2u; c++) {
                tab[2u * c] = 1.0 / (double)c;
                tab[2u * c + 1u] = (double)c;
            }
            CPD_TRY(ctx->tp_tab.ensure(sizeof(double) * tab.size()));
            CPD_TRY(cudaMemcpyAsync(ctx->tp_tab.p, tab.data(), sizeof(double) * tab.size(), cudaMemcpyHostToDevice, s));
            CPD_TRY(cudaStreamSynchronize(s));
            ctx->tp_rz = rz;
            ctx->tp_tab_m = max_m;
            S.h2d += sizeof(double) * tab.size();
        }
    }
    const size_t out_bytes = sizeof(double) * (size_t)n * D.B;
    // the design and the wavelengths in one copy
    const size_t lam_off = (sizeof(DevDesign) + 255) & ~size_t(255), in_bytes = lam_off + sizeof(double) * n;
    CPD_TRY(S.h_in.ensure(in_bytes));
    CPD_TRY(ctx->tp_design.ensure(in_bytes));
    CPD_TRY(ctx->tp_out.ensure(out_bytes));
    CPD_TRY(ctx->tp_rays.ensure(sizeof(uint32_t) * n));
    std::vector<uint32_t> rays(n);
    if (pieces) {
        D.wmin = 0.0;  // a point is its wavelength
        D.wmax = 1.0;
        D.dc.wmin = ff::F2{0.f, 0.f};
        D.dc.wspan = ff::F2{1.f, 0.f};
    }
    std::memcpy(S.h_in.p, &D, sizeof(DevDesign));
    std::memcpy(S.h_in.as<char>() + lam_off, wavelengths, sizeof(double) * n);
    CPD_TRY(cudaMemcpyAsync(ctx->tp_design.p, S.h_in.p, in_bytes, cudaMemcpyHostToDevice, s));
    const DevDesign *dd = ctx->tp_design.as<DevDesign>();
    const double *dl = reinterpret_cast<const double *>(ctx->tp_design.as<char>() + lam_off);
    CPD_TRY(cudaEventRecord(S.ev0, s));
    if (pieces) {
        CPD_TRY(ctx->tp_lp.ensure(sizeof(LamParams) * n));
        CPD_TRY(ctx->tp_t64.ensure(sizeof(double) * n));
        TpArgs a{};
        a.d = dd;
        a.lambdas = dl;
        a.n = n;
        a.max_m = max_m;
        a.z64 = ctx->tp_z.as<double>();
        a.cnt = ctx->tp_tab.as<double2>();
        a.z32 = reinterpret_cast<const float2 *>(a.cnt + max_m + 2u);
        a.rank = reinterpret_cast<const uint32_t *>(a.z32 + max_m);
        a.lp = ctx->tp_lp.as<LamParams>();
        a.t64 = ctx->tp_t64.as<double>();
        a.out = ctx->tp_out.as<double>();
        a.rays_out = ctx->tp_rays.as<uint32_t>();
        a.guards = default_guards();
        a.Rz = ctx->tp_rz;
        launch_tp_pieces(a, D.B, s);
    } else {
        launch_tp_adaptive(dd, D.B, dl, n, ctx->tp_z.as<double>(), max_m, ctx->tp_out.as<double>(),
                           ctx->tp_rays.as<uint32_t>(), false, s);
    }
    CPD_TRY(cudaGetLastError());
    CPD_TRY(cudaEventRecord(S.ev1, s));
    CPD_TRY(cudaMemcpyAsync(out, ctx->tp_out.p, out_bytes, cudaMemcpyDeviceToHost, s));
    CPD_TRY(cudaMemcpyAsync(rays.data(), ctx->tp_rays.p, sizeof(uint32_t) * n, cudaMemcpyDeviceToHost, s));
    CPD_TRY(cudaStreamSynchronize(s));
    S.launches = pieces ? 2 : 1;
    float ms = 0.f, left_ms = 0.f;
    cudaEventElapsedTime(&ms, S.ev0, S.ev1);
    // wavelengths with hits of more than one transmittance, by the general kernel (glass of an index
    // near 1 behind a steep exit face; then often every wavelength, so all in one launch)
    if (std::find(rays.begin(), rays.end(), 0u) != rays.end()) {
        CPD_TRY(cudaEventRecord(S.ev0, s));
        launch_tp_adaptive(dd, D.B, dl, n, ctx->tp_z.as<double>(), max_m, ctx->tp_out.as<double>(), ctx->tp_rays.as<uint32_t>(),
                           true, s);
        CPD_TRY(cudaGetLastError());
        CPD_TRY(cudaEventRecord(S.ev1, s));
        CPD_TRY(cudaMemcpyAsync(out, ctx->tp_out.p, out_bytes, cudaMemcpyDeviceToHost, s));
        CPD_TRY(cudaMemcpyAsync(rays.data(), ctx->tp_rays.p, sizeof(uint32_t) * n, cudaMemcpyDeviceToHost, s));
        CPD_TRY(cudaStreamSynchronize(s));
        cudaEventElapsedTime(&left_ms, S.ev0, S.ev1);
        S.d2h += out_bytes + sizeof(uint32_t) * n;
        S.launches++;
    }
    if (rays_out) std::memcpy(rays_out, rays.data(), sizeof(uint32_t) * n);
    S.last_ms = ms + left_ms;
    S.h2d += in_bytes;
    S.d2h += out_bytes + sizeof(uint32_t) * n;
    return CPD_OK;
}

int cpd_trace_rays(cpd_context *ctx, const cpd_design *d, const double *lam_u, const double *ray_u, uint32_t n,
                   uint32_t trace_mode, uint32_t *bins, double *ts, uint8_t *flags)
{
    if (!ctx || !valid_design(d) || !lam_u || !ray_u || !bins || !ts || trace_mode > CPD_TRACE_FP64)
        return CPD_INVALID_ARGUMENT;
    if (n == 0) return CPD_OK;
    CPD_SYNC_ENTRY(ctx);
    PassSlot &S = ctx->main;
    DevDesign D;
    design_to_dev(*d, D);
    std::vector<double> z(n);
    for (uint32_t i = 0; i < n; i++) z[i] = norminv(ray_u[i]);
    cudaStream_t s = S.stream;
    CPD_TRY(ctx->pair_design.ensure(sizeof(DevDesign)));
    CPD_TRY(ctx->pair_lam.ensure(sizeof(double) * n));
    CPD_TRY(ctx->pair_z.ensure(sizeof(double) * n));
    CPD_TRY(ctx->pair_bins.ensure(sizeof(uint32_t) * n));
    CPD_TRY(ctx->pair_ts.ensure(sizeof(double) * n));
    CPD_TRY(ctx->pair_flags.ensure(n));
    CPD_TRY(cudaMemcpyAsync(ctx->pair_design.p, &D, sizeof(DevDesign), cudaMemcpyHostToDevice, s));
    CPD_TRY(cudaMemcpyAsync(ctx->pair_lam.p, lam_u, sizeof(double) * n, cudaMemcpyHostToDevice, s));
    CPD_TRY(cudaMemcpyAsync(ctx->pair_z.p, z.data(), sizeof(double) * n, cudaMemcpyHostToDevice, s));
    CPD_TRY(cudaEventRecord(S.ev0, s));
    launch_trace_pairs(ctx->pair_design.as<DevDesign>(), ctx->pair_lam.as<double>(), ctx->pair_z.as<double>(), n,
                       trace_mode, ctx->pair_bins.as<uint32_t>(), ctx->pair_ts.as<double>(),
                       ctx->pair_flags.as<uint8_t>(), s);
    CPD_TRY(cudaGetLastError());
    CPD_TRY(cudaEventRecord(S.ev1, s));
    CPD_TRY(cudaMemcpyAsync(bins, ctx->pair_bins.p, sizeof(uint32_t) * n, cudaMemcpyDeviceToHost, s));
    CPD_TRY(cudaMemcpyAsync(ts, ctx->pair_ts.p, sizeof(double) * n, cudaMemcpyDeviceToHost, s));
    if (flags) CPD_TRY(cudaMemcpyAsync(flags, ctx->pair_flags.p, n, cudaMemcpyDeviceToHost, s));
    CPD_TRY(cudaStreamSynchronize(s));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, S.ev0, S.ev1);
    S.last_ms = ms;
    S.launches = 1;
    return CPD_OK;
}

int cpd_measure_fp32_peak(cpd_context *ctx, uint32_t iters, double *tflops)
{
    if (!ctx || !tflops || iters == 0) return CPD_INVALID_ARGUMENT;
    CPD_SYNC_ENTRY(ctx);
    PassSlot &S = ctx->main;
    const int threads = 256;
    const int blocks = ctx->num_sms * 8;
    CPD_TRY(ctx->peak.ensure(sizeof(float) * blocks));
    cudaStream_t s = S.stream;
    launch_fma_peak(ctx->peak.as<float>(), 16, blocks, threads, s);  // warm-up
    CPD_TRY(cudaEventRecord(S.ev0, s));
    launch_fma_peak(ctx->peak.as<float>(), iters, blocks, threads, s);
    CPD_TRY(cudaEventRecord(S.ev1, s));
    CPD_TRY(cudaStreamSynchronize(s));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, S.ev0, S.ev1);
    const double flops = 2.0 * 8.0 * 16.0 * (double)iters * threads * (double)blocks;
    *tflops = flops / (ms * 1e-3) / 1e12;
    S.last_ms = ms;
    S.launches = 2;
    return CPD_OK;
}

int cpd_measure_sfu_peak(cpd_context *ctx, uint32_t iters, double *gops)
{
    if (!ctx || !gops || iters == 0) return CPD_INVALID_ARGUMENT;
    CPD_SYNC_ENTRY(ctx);
    PassSlot &S = ctx->main;
    const int threads = 256;
    const int blocks = ctx->num_sms * 8;
    CPD_TRY(ctx->peak.ensure(sizeof(float) * blocks));
    cudaStream_t s = S.stream;
    launch_mufu_peak(ctx->peak.as<float>(), 16, blocks, threads, s);  // warm-up
    CPD_TRY(cudaEventRecord(S.ev0, s));
    launch_mufu_peak(ctx->peak.as<float>(), iters, blocks, threads, s);
    CPD_TRY(cudaEventRecord(S.ev1, s));
    CPD_TRY(cudaStreamSynchronize(s));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, S.ev0, S.ev1);
    const double ops = 8.0 * 16.0 * (double)iters * threads * (double)blocks;
    *gops = ops / (ms * 1e-3) / 1e9;
    S.last_ms = ms;
    S.launches = 2;
    return CPD_OK;
}

// ------------------------------------------------------------------ server ABI

int cpd_server_create(cpd_context *ctx, uint64_t mem_budget_bytes, uint32_t slots, uint32_t max_designs_per_pass,
                      cpd_server **out)
{
    if (!ctx || !out || slots == 0 || slots > 8 || mem_budget_bytes == 0) return CPD_INVALID_ARGUMENT;
    *out = nullptr;
    if (cudaSetDevice(ctx->device) != cudaSuccess) return CPD_CUDA_ERROR;
    cpd_server *sv = new cpd_server();
    sv->ctx = ctx;
    sv->budget = mem_budget_bytes;
    if (max_designs_per_pass) sv->max_designs_per_pass = max_designs_per_pass;
    for (uint32_t i = 0; i < slots; i++) {
        sv->slots.emplace_back(new PassSlot());
        if (sv->slots.back()->create() != cudaSuccess) {
            for (auto &s : sv->slots) s->destroy();
            delete sv;
            return CPD_CUDA_ERROR;
        }
    }
    sv->slot_work.resize(slots);
    sv->busy.assign(slots, false);
    sv->worker = std::thread(srv_loop, sv);
    *out = sv;
    return CPD_OK;
}

int cpd_server_submit(cpd_server *sv, const cpd_design *designs, const cpd_batch_item *items, uint32_t n,
                      uint32_t trace_mode, uint64_t *request_id)
{
    if (!sv || !designs || !items || !request_id || n == 0 || !valid_mode(trace_mode)) return CPD_INVALID_ARGUMENT;
    for (uint32_t i = 0; i < n; i++)
        if (!valid_design(&designs[i]) || !valid_item(items[i])) return CPD_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> lk(sv->mu);
    if (sv->stop) return CPD_INVALID_ARGUMENT;
    const uint64_t id = sv->next_id++;
    SrvRequest &r = sv->reqs[id];
    r.designs.assign(designs, designs + n);
    r.items.assign(items, items + n);
    r.outs.resize(n);
    r.remaining = n;
    r.mode = trace_mode;
    r.t_submit = std::chrono::steady_clock::now();
    for (uint32_t i = 0; i < n; i++)
        sv->pending.push_back(
            SrvWork{id, i, design_bytes(items[i].max_n, items[i].max_eval, designs[i].bin_count)});
    *request_id = id;
    sv->cv_work.notify_one();
    return CPD_OK;
}

int cpd_server_submit_params(cpd_server *sv, const cpd_spectrometer_params *params, const cpd_batch_item *items,
                             uint32_t n, double acceptance, uint32_t trace_mode, uint64_t *request_id)
{
    if (!sv || !params || !items || !request_id || n == 0 || !valid_mode(trace_mode)) return CPD_INVALID_ARGUMENT;
    if (acceptance != 0.0 && !(acceptance > 0.0 && acceptance <= 1.0)) return CPD_INVALID_ARGUMENT;
    for (uint32_t i = 0; i < n; i++)
        if (!valid_params(params[i]) || !valid_item(items[i])) return CPD_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> lk(sv->mu);
    if (sv->stop) return CPD_INVALID_ARGUMENT;
    const uint64_t id = sv->next_id++;
    SrvRequest &r = sv->reqs[id];
    r.params.assign(params, params + n);
    r.acceptance = acceptance;
    r.items.assign(items, items + n);
    r.outs.resize(n);
    r.remaining = n;
    r.mode = trace_mode;
    r.t_submit = std::chrono::steady_clock::now();
    for (uint32_t i = 0; i < n; i++)
        sv->pending.push_back(
            SrvWork{id, i, design_bytes(items[i].max_n, items[i].max_eval, params[i].bin_count)});
    *request_id = id;
    sv->cv_work.notify_one();
    return CPD_OK;
}

int cpd_server_wait(cpd_server *sv, uint64_t request_id, cpd_fitness *outs, double timeout_ms, double *latency_ms)
{
    if (!sv || !outs) return CPD_INVALID_ARGUMENT;
    std::unique_lock<std::mutex> lk(sv->mu);
    auto it = sv->reqs.find(request_id);
    if (it == sv->reqs.end()) return CPD_INVALID_ARGUMENT;
    const auto deadline = std::chrono::steady_clock::now() +
                          std::chrono::microseconds((int64_t)(std::max(0.0, timeout_ms) * 1000.0));
    while (!it->second.done) {
        if (sv->cv_done.wait_until(lk, deadline) == std::cv_status::timeout && !it->second.done) return CPD_TIMEOUT;
        it = sv->reqs.find(request_id);
        if (it == sv->reqs.end()) return CPD_INVALID_ARGUMENT;
    }
    SrvRequest &r = it->second;
    std::memcpy(outs, r.outs.data(), sizeof(cpd_fitness) * r.outs.size());
    if (latency_ms) *latency_ms = std::chrono::duration<double, std::milli>(r.t_done - r.t_submit).count();
    const int status = r.status;
    sv->reqs.erase(it);
    return status;
}

int cpd_server_stats(cpd_server *sv, uint64_t *designs_done, uint64_t *passes, uint64_t *max_in_flight,
                     uint64_t *pending)
{
    if (!sv) return CPD_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> lk(sv->mu);
    if (designs_done) *designs_done = sv->designs_done;
    if (passes) *passes = sv->passes;
    if (max_in_flight) *max_in_flight = sv->max_in_flight;
    if (pending) *pending = sv->pending.size();
    return CPD_OK;
}

void cpd_server_destroy(cpd_server *sv)
{
    if (!sv) return;
    {
        std::lock_guard<std::mutex> lk(sv->mu);
        sv->stop = true;
        sv->cv_work.notify_all();
    }
    if (sv->worker.joinable()) sv->worker.join();
    cudaSetDevice(sv->ctx->device);
    for (auto &s : sv->slots) s->destroy();
    delete sv;
}

}  // extern "C"
