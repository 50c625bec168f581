// cpd_kernels.cu -- the GB300 kernels of the fitness path.
//
// A pass over a set of designs runs on one stream:
//   tables   (passes whose ray tables are not resident) the points of each table sorted
//            (table_sort_kernel) and turned into start heights (table_z_kernel)
//   build    (designs given as parameter records) eight lanes per design, f64
//   setup    one thread per (design, wavelength): the flat-face chain in float-float
//            (cpd_df.h) -> LamParams for the fast path and LamDF for the re-trace
// and then, for designs whose coated exit face admits certified pieces (cpd_piece.h) under the
// fixed-N hybrid trace (but for short tables on many rows and a few such designs beside others),
//   rows     rows_kernel: a wavelength's trace, re-trace and entropy by one team of warps, its
//            cells in shared memory; ahead of it, in passes of many designs, rows_kernel<HEAVY>
//            for rows that are mostly re-traced;
// for all others (uncoated designs, the FP32 and FP64 study modes),
//   trace    persistent warps over work items (design, 32-wavelength block, ray
//            chunk); lane = wavelength; FP32 exit face + detector per ray; hits
//            accumulate per lane as run-length fixed-point sums (rays are sorted by
//            start height, so consecutive rays mostly share a bin) flushed with one
//            64-bit atomic per run; guard-band rays go to the warp's list, which the warp
//            re-traces itself (the global queue once the list is full)
//   retrace  every queued ray: float-float re-trace (exact f64 in the FP64 study mode,
//            bit-identical to the reference's f64 CPU trace)
//   entropy  one warp (many tiles) or one block (few) per (design, row tile): p = sum/R,
//            p log2 p, per-bin sums of p and p^2 in float-float with fixed-point
//            accumulation (order independent)
// and for both
//   finalize one warp per design: H(D), MI, SEM convergence (in a single-design pass the
//            block that completes the last rows or entropy tile runs it).
// A single-design pass with a fixed ray count (the plain call) runs setup_pair_kernel (two
// warps per 32 rows), and trace_spans_kernel (equal shares of the ray slots per warp) in place
// of trace; its design's constants are kernel parameters. Adaptive sampling replaces trace and
// retrace with adaptive1_pieces_kernel (many rows), adaptive_block_kernel or adaptive_equal_kernel
// (designs with pieces), adaptive1_kernel or adaptive_kernel (the others), adaptive_mixed_kernel (few
// rows of both) and adaptive_exact_kernel.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "cpd_build.h"
#include "cpd_df.h"
#include "cpd_gpu.cuh"
#include "cpd_piece.h"

namespace cpd {

namespace {

enum Field { F_ROW = 0, F_ITEM = 1, F_TILE = 2, F_GROUP = 3 };

template <int FIELD>
__device__ __forceinline__ uint64_t job_field(const DesignJob &j)
{
    return FIELD == F_ROW ? j.row_off : FIELD == F_ITEM ? j.item_off : FIELD == F_TILE ? j.tile_off : j.grp_off;
}

// Largest i with field(jobs[i]) <= v.
template <int FIELD>
__device__ __forceinline__ uint32_t find_job(const DesignJob *__restrict__ jobs, uint32_t n, uint64_t v)
{
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if (job_field<FIELD>(jobs[mid]) <= v) lo = mid;
        else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ void push_ray(const LaunchArgs &a, uint32_t d, uint32_t k, uint32_t j)
{
    unsigned long long pos = atomicAdd(&a.ctl->queue_count, 1ull);
    if (pos < a.qcap) a.queue[pos] = QEntry{d, k, j, 0u};
    else atomicOr(&a.ctl->overflow, kOverflowQueue);
}

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// The start of a pass that its kernels time themselves (its first kernel is `which`).
__device__ __forceinline__ void stamp_start(const LaunchArgs &a, uint32_t which)
{
    if (a.stamp == which && blockIdx.x == 0u && blockIdx.y == 0u && threadIdx.x == 0u) a.status->t0 = global_ns();
}

// The rays [j0, j1) and [j2, j3) of row k, queued with one atomic for the whole run (a row's
// guard bands can hold dozens of rays; one round trip to the queue counter per ray made a
// serial chain on the setup's critical path).
__device__ __forceinline__ void push_ranges(const LaunchArgs &a, uint32_t d, uint32_t k, uint32_t j0, uint32_t j1,
                                            uint32_t j2, uint32_t j3)
{
    const uint32_t na = j1 > j0 ? j1 - j0 : 0u, nb = j3 > j2 ? j3 - j2 : 0u;
    if (na + nb == 0u) return;
    const unsigned long long pos = atomicAdd(&a.ctl->queue_count, (unsigned long long)(na + nb));
    if (pos + na + nb > a.qcap) atomicOr(&a.ctl->overflow, kOverflowQueue);
    for (uint32_t i = 0; i < na + nb; i++) {
        if (pos + i >= a.qcap) break;
        a.queue[pos + i] = QEntry{d, k, i < na ? j0 + i : j2 + (i - na), 0u};
    }
}

// Designs built on the device from parameter records: the f64 construction of cpd_build.h, eight
// lanes to a design. FP64 bounds it: a warp instruction takes its scheduler ~64 cycles whatever its
// active lanes, so what counts is the length of one design's program. The lanes take a face's sine
// and cosine each, the positioning's two traces run on two of them, and the device record's ~95
// float splits are spread over all; the rest every lane does alike. (One thread per design, which
// also built the prism twice: build and setup of 512 designs took 356 us, now 76.)
constexpr uint32_t kBuildLanes = 8;
constexpr uint32_t kBuildPerWarp = 32 / kBuildLanes;
struct BuildScratch {
    cpd_design d;
    DevDesign D;
    double nx[kBuildLanes], ny[kBuildLanes], off[kBuildLanes];
};

__device__ __forceinline__ double shfl_d(double v, uint32_t src)
{
    return __longlong_as_double(__shfl_sync(0xffffffffu, __double_as_longlong(v), (int)src));
}

// build::design_positioned of record p into S.d (zero-filled on an error), by lane l of the
// design's eight. The operations and their order are those of build::prism, position and design.
__device__ __forceinline__ int build_design(const cpd_spectrometer_params &p, double acceptance, BuildScratch &S, uint32_t l,
                                            uint32_t lane)
{
    using build::V2;
    cpd_design &d = S.d;
    for (uint32_t i = l; i < sizeof(cpd_design) / 4; i += kBuildLanes) reinterpret_cast<uint32_t *>(&d)[i] = 0u;
    const int G0 = p.nglass, G = G0 < 1 ? 1 : G0 > CPD_MAX_GLASS ? CPD_MAX_GLASS : G0;
    const double height = p.height, h2 = x::mul(height, 0.5);
    // face l's normal and the length it takes; the last lane: the detector's normal
    const V2 nl = build::rot180(build::angled((int)l <= G && l < kBuildLanes - 1u ? p.angles[l] : p.det_angle));
    S.nx[l] = nl.x;
    S.ny[l] = nl.y;
    S.off[l] = x::mul(fabs(x::div(nl.y, nl.x)), h2);
    __syncwarp();
    int prism_err = G0 != G || !(height > 0.0) || !(fabs(p.curvature) > 0.0) || !(fabs(p.curvature) <= 1.0)
                        ? (int)CPD_INVALID_ARGUMENT : 0;
    // create_joined_trapezoids
    bool finite = true;
    double mx = S.off[0];
    for (int k = 0; k <= G; k++) {
        if (k) {
            const bool turn = build::sign_bit(S.ny[k - 1]) != build::sign_bit(S.ny[k]);
            const double d1 = S.off[k - 1], d2 = S.off[k];
            mx = x::add(mx, x::add(p.lengths[k - 1], turn ? x::add(d1, d2) : fabs(x::sub(d1, d2))));
        }
        if (k < G) {
            if (l == 0u) {
                d.face_point[k][0] = mx;
                d.face_point[k][1] = h2;
                d.face_normal[k][0] = S.nx[k];
                d.face_normal[k][1] = S.ny[k];
            }
            finite = finite && build::finite(mx) && build::finite(S.nx[k]);
        }
    }
    // CurvedPlane::from_hyperplane
    const V2 last_pt{mx, h2}, last_n{S.nx[G], S.ny[G]};
    const double kc = p.curvature;
    const double chord = fabs(x::div(height, last_n.x));
    const double radius = x::div(x::mul(chord, 0.5), fabs(kc));
    const double apothem = x::sqrt_(x::sub(x::mul(radius, radius), x::mul(x::mul(chord, chord), 0.25)));
    const double sagitta = x::sub(radius, apothem);
    const V2 c = build::vfma(last_n, copysign(apothem, kc), last_pt), m = build::vfma(last_n, -copysign(sagitta, kc), last_pt);
    const double r2 = x::add(x::mul(sagitta, sagitta), x::mul(x::mul(chord, chord), 0.25));
    if (!prism_err && (!finite || !build::finite(radius) || !build::finite(apothem))) prism_err = CPD_INVALID_ARGUMENT;
    if (l == 0u) {
        d.nglass = G;
        d.ar_coated = p.ar_coated ? 1 : 0;
        d.height = height;
        d.exit_center[0] = c.x;
        d.exit_center[1] = c.y;
        d.exit_radius = radius;
        d.exit_bound_center[0] = m.x;
        d.exit_bound_center[1] = m.y;
        d.exit_bound_r2 = r2;
        build::source(p, d);
    }
    for (uint32_t i = l; i < CPD_MAX_GLASS * 6u; i += kBuildLanes) (&d.glass[0][0])[i] = (&p.glass[0][0])[i];
    __syncwarp();
    int e = 0;
    double pos[2] = {p.det_position[0], p.det_position[1]};
    int32_t flipped = p.det_flipped;
    if (acceptance > 0.0) {
        // detector_array_positioning: the rays of the acceptance band's two ends, one lane each
        e = acceptance <= 1.0 ? prism_err : (int)CPD_INVALID_ARGUMENT;
        DevDesign &D = S.D;
        if (l == 0u) {
            D.G = G;
            D.ar = d.ar_coated;
            D.height = height;
            D.ccx = c.x;
            D.ccy = c.y;
            D.crad = radius;
            D.cbx = m.x;
            D.cby = m.y;
            D.cbr2 = r2;
            D.wmin = p.wavelength_bounds[0];
            D.wmax = p.wavelength_bounds[1];
            D.bym = p.beam_y_mean;
        }
        for (uint32_t i = l; i < CPD_MAX_GLASS * 6u; i += kBuildLanes) (&D.glass[0][0])[i] = (&d.glass[0][0])[i];
        for (uint32_t k = l; k < CPD_MAX_GLASS; k += kBuildLanes) {
            D.ppx[k] = d.face_point[k][0];
            D.ppy[k] = d.face_point[k][1];
            D.pnx[k] = d.face_normal[k][0];
            D.pny[k] = d.face_normal[k][1];
        }
        __syncwarp();
        const double uh = x::mul(fmax(x::sub(1.0, acceptance), 0.0), 0.5);
        x::Ray r{0.0, D.bym, 1.0, 0.0, 1.0, 1.0};
        int er = 0;
        if (l < 2u && !e) er = x::prism(D, x::wavelength(D, l ? x::sub(1.0, uh) : uh), r);
        __syncwarp();
        const uint32_t a0 = lane & ~(kBuildLanes - 1u);
        const int e0 = __shfl_sync(0xffffffffu, er, (int)a0), e1 = __shfl_sync(0xffffffffu, er, (int)a0 + 1);
        const double lox = shfl_d(r.ox, a0), loy = shfl_d(r.oy, a0), lodx = shfl_d(r.dx, a0), lody = shfl_d(r.dy, a0);
        const double upx = shfl_d(r.ox, a0 + 1u), upy = shfl_d(r.oy, a0 + 1u), updx = shfl_d(r.dx, a0 + 1u),
                     updy = shfl_d(r.dy, a0 + 1u);
        const double tm = x::mul(x::add(r.ts, r.tp), 0.5), t0 = shfl_d(tm, a0), t1 = shfl_d(tm, a0 + 1u);
        if (!e) e = e0 ? e0 : e1;
        if (!e && (t0 <= 1e-3 || t1 <= 1e-3)) e = CPD_RAYTRACE_ANGULAR_RESPONSE_TOO_WEAK;
        // rot90(angled(det_angle)); S.n? of the last lane is its rot180
        const V2 spec{x::mul(S.ny[kBuildLanes - 1], p.det_length), x::mul(-S.nx[kBuildLanes - 1], p.det_length)};
        const double ca = updx, cb = -lodx, cc = updy, dd = -lody;
        const double det = x::sub(x::mul(ca, dd), x::mul(cb, cc));
        if (!e && det == 0.0) e = CPD_RAYTRACE_NO_SURFACE_INTERSECTION;
        const double i10 = x::div(-cc, det), i11 = x::div(ca, det);
        double tx = x::add(x::sub(spec.x, upx), lox), ty = x::add(x::sub(spec.y, upy), loy);
        double d2 = x::add(x::mul(i10, tx), x::mul(i11, ty));
        int32_t fl = 0;
        if (!(d2 > 0.0)) {
            tx = x::add(x::sub(-spec.x, upx), lox);
            ty = x::add(x::sub(-spec.y, upy), loy);
            d2 = x::add(x::mul(i10, tx), x::mul(i11, ty));
            if (!e && d2 < 0.0) e = CPD_RAYTRACE_NO_SURFACE_INTERSECTION;
            fl = 1;
        }
        pos[0] = x::fma_(lodx, d2, lox);
        pos[1] = x::fma_(lody, d2, loy);
        flipped = fl;
    }
    if (!e) {
        if (p.bin_count == 0 || p.bin_count > CPD_MAX_BINS || !(p.linear_slope > 0.0) || !(p.bin_size > 0.0) ||
            !(p.det_length > 0.0) || !(p.wavelength_bounds[1] >= p.wavelength_bounds[0]))
            e = CPD_INVALID_ARGUMENT;
        else e = prism_err;
    }
    const double min_ci = build::cos_(p.max_incident_angle);
    const V2 n{S.nx[kBuildLanes - 1], S.ny[kBuildLanes - 1]};
    const V2 u = flipped ? build::rot90(n) : build::rot90ccw(n);
    const V2 mid = build::vfma(u, x::mul(p.det_length, 0.5), V2{pos[0], pos[1]});
    const double dx = mid.x, dy = x::sub(mid.y, p.beam_y_mean);
    const double size = x::sqrt_(x::add(x::mul(dx, dx), x::mul(dy, dy)));
    const double deviation = fabs(x::div(dy, size));
    __syncwarp();
    if (e) {
        for (uint32_t i = l; i < sizeof(cpd_design) / 4; i += kBuildLanes) reinterpret_cast<uint32_t *>(&d)[i] = 0u;
    } else if (l == 0u) {
        d.bin_count = p.bin_count;
        d.bin_size = p.bin_size;
        d.linear_slope = p.linear_slope;
        d.linear_intercept = p.linear_intercept;
        d.min_ci = min_ci;
        d.det_length = p.det_length;
        d.det_normal[0] = n.x;
        d.det_normal[1] = n.y;
        d.det_direction[0] = u.x;
        d.det_direction[1] = u.y;
        d.det_position[0] = pos[0];
        d.det_position[1] = pos[1];
        d.size = size;
        d.deviation = deviation;
    }
    __syncwarp();
    return e;
}

// build::to_dev of S.d into S.D, the float-float copies by all eight lanes.
__device__ __forceinline__ void build_to_dev(BuildScratch &S, uint32_t l)
{
    DevDesign &D = S.D;
    // the exact tables and the FP32 constants, then the values to split in DFConst's order
    if (l == 0u) build::to_dev_exact(S.d, D);
    __syncwarp();
    for (uint32_t i = l; i < sizeof(DFConst) / sizeof(ff::F2); i += kBuildLanes) {
        ff::F2 v;
        ff::split(build::dev_value(D, (int)i), v.hi, v.lo);
        reinterpret_cast<ff::F2 *>(&D.dc)[i] = v;
    }
    __syncwarp();
}

// Written straight into the pass's design records. A design whose construction fails keeps its
// status in the record; the setup then loses all its rays.
__global__ void __launch_bounds__(32) build_kernel(const LaunchArgs a)
{
    stamp_start(a, STAMP_BUILD);
    __shared__ __align__(16) BuildScratch S[kBuildPerWarp];
    const uint32_t lane = threadIdx.x, sub = lane / kBuildLanes, l = lane % kBuildLanes;
    const uint32_t i = min(blockIdx.x * kBuildPerWarp + sub, a.njobs - 1u);  // (a spare group repeats the last design)
    const int e = build_design(a.params[i], a.build_acceptance, S[sub], l, lane);
    build_to_dev(S[sub], l);
    if (l == 0u) {
        S[sub].D.status = e;
        if (e) S[sub].D.B = a.jobs[i].B;
    }
    __syncwarp();
    uint4 *out = reinterpret_cast<uint4 *>(const_cast<DevDesign *>(a.designs) + i);
    for (uint32_t w = l; w < sizeof(DevDesign) / 16; w += kBuildLanes) out[w] = reinterpret_cast<const uint4 *>(&S[sub].D)[w];
}

// cpd_design records from parameter records, for the host (cpd_design_build_device).
__global__ void __launch_bounds__(32) build_records_kernel(const cpd_spectrometer_params *p, uint32_t n,
                                                           double acceptance, cpd_design *out, int32_t *status)
{
    __shared__ __align__(16) BuildScratch S[kBuildPerWarp];
    const uint32_t lane = threadIdx.x, sub = lane / kBuildLanes, l = lane % kBuildLanes;
    const uint32_t i = min(blockIdx.x * kBuildPerWarp + sub, n - 1u);
    const int e = build_design(p[i], acceptance, S[sub], l, lane);
    if (l == 0u) status[i] = e;
    uint32_t *o = reinterpret_cast<uint32_t *>(out + i);
    for (uint32_t w = l; w < sizeof(cpd_design) / 4; w += kBuildLanes) o[w] = reinterpret_cast<const uint32_t *>(&S[sub].d)[w];
}


__device__ __forceinline__ void cp_async16(void *smem, const void *gmem)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}

// The u-point of wavelength k of a design.
__device__ __forceinline__ double lam_point(const LaunchArgs &a, const DesignJob &J, uint32_t k)
{
    return J.seeded ? x::seed_point(J.seed, k) : a.lam_u[J.lam_off + k];
}

// ------------------------------------------------------------------ ray tables on the device

constexpr uint32_t kTableThreads = 1024;
constexpr size_t table_smem_bytes(uint32_t buckets, uint32_t R) { return 4u * (size_t)buckets + 2u * (size_t)R; }

// One block per table without a known order (the caller's own points, and the first table of a
// size): the order of its points, perm[sorted position] = ray. The points go
// into at least R buckets of equal width by their leading bits (a shared-memory count, a scan,
// a scatter), and each bucket's few are put in order by one thread. The points of a seed are
// spread evenly (the R1 sequence: at most three share a bucket); the caller's own may not be,
// and a bucket of more than kTableBucket leaves the table to the host. Keys are integers (a
// seed's points as 64-bit fractions: no FP64 instruction). Latency bounds it: one block, ~10 us for
// 8192 points (the host's sort and f64 quantiles: 400 us; a call on 3001 own points 238 -> 102 us).
// That is why a size's order is kept from its second use on: a seed only turns it, and a call with
// a fresh seed, 128 x 8192 rays, takes 51 us with it, 61 sorted anew, 285 by the host's tables.
__global__ void __launch_bounds__(kTableThreads) table_sort_kernel(const LaunchArgs a)
{
    stamp_start(a, STAMP_SORT);
    cudaTriggerProgrammaticLaunchCompletion();
    extern __shared__ __align__(16) uint32_t table_smem[];
    __shared__ uint32_t warp_sum[kTableThreads / 32u];
    const TableJob t = a.tables[blockIdx.x];
    const uint32_t R = t.R, tid = threadIdx.x, lane = tid & 31u;
    const uint32_t bits = R > 1024u ? 32u - __clz(R - 1u) : 10u, M = 1u << bits;
    uint32_t *cnt = table_smem;
    uint16_t *slot = reinterpret_cast<uint16_t *>(table_smem + M);
    const uint64_t alpha = (uint64_t)(kAlpha * 18446744073709551616.0);
    const double *pts = a.ray_u + t.u_off;
    const auto bucket = [&](uint32_t j) -> uint32_t {
        if (!t.points) return (uint32_t)((t.seed_fixed + alpha * (j + 1u)) >> (64u - bits));
        const uint64_t b = (uint64_t)__double_as_longlong(pts[j]);  // in (0, 1): positive, exponent below 1023
        const int e = (int)(b >> 52) - 1011;                         // value 2^64 = significand 2^e
        const uint64_t m = (b & 0xfffffffffffffull) | 0x10000000000000ull;
        return (uint32_t)((e >= 0 ? m << e : e > -64 ? m >> -e : 0ull) >> (64u - bits));
    };
    const auto key = [&](uint32_t j) -> uint64_t {
        return t.points ? (uint64_t)__double_as_longlong(pts[j]) : t.seed_fixed + alpha * (j + 1u);
    };
    for (uint32_t i = tid; i < M; i += kTableThreads) cnt[i] = 0u;
    __syncthreads();
    for (uint32_t j = tid; j < R; j += kTableThreads) atomicAdd(cnt + bucket(j), 1u);
    __syncthreads();
    // exclusive scan of the counts: M / 1024 consecutive buckets per thread
    const uint32_t per = M / kTableThreads, b0 = tid * per;
    uint32_t sum = 0u, most = 0u;
    for (uint32_t i = 0; i < per; i++) {
        const uint32_t v = cnt[b0 + i];
        sum += v;
        most = max(most, v);
    }
    if (most > kTableBucket) atomicOr(&a.ctl->overflow, kOverflowTable);
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += v;
    }
    if (lane == 31u) warp_sum[tid >> 5] = incl;
    __syncthreads();
    uint32_t before = 0u;
    {
        const uint32_t v = lane < (tid >> 5) ? warp_sum[lane] : 0u;
        before = __reduce_add_sync(0xffffffffu, v);
    }
    uint32_t at = before + incl - sum;
    for (uint32_t i = 0; i < per; i++) {
        const uint32_t v = cnt[b0 + i];
        cnt[b0 + i] = at;
        at += v;
    }
    __syncthreads();
    for (uint32_t j = tid; j < R; j += kTableThreads) slot[atomicAdd(cnt + bucket(j), 1u)] = (uint16_t)j;
    __syncthreads();
    // cnt[b] is now the end of bucket b
    for (uint32_t b = tid; b < M; b += kTableThreads) {
        const uint32_t s = b ? cnt[b - 1u] : 0u, e = cnt[b];
        if (e - s < 2u || e - s > kTableBucket) continue;
        for (uint32_t i = s + 1u; i < e; i++) {
            const uint16_t v = slot[i];
            const uint64_t kv = key(v);
            uint32_t q = i;
            for (; q > s; q--) {
                const uint16_t w = slot[q - 1u];
                const uint64_t kw = key(w);
                if (kw < kv || (kw == kv && w < v)) break;
                slot[q] = w;
            }
            slot[q] = v;
        }
    }
    __syncthreads();
    uint32_t *perm = a.perm + t.ray_off;
    for (uint32_t i = tid; i < R; i += kTableThreads) perm[i] = slot[i];
}

// One thread per sorted position: its z in f64 (the host's own operations but for CUDA's log),
// split into floats, and the ray's rank. blockIdx.x is the table (a pass may have more than 65535).
// A warp's f64 instruction takes its scheduler ~64 cycles, so the positions are spread two warps to
// a block; with a known order this kernel is all a new seed costs, beside the setup's face loop
// (FP64 issue bounds it).
__global__ void __launch_bounds__(64) table_z_kernel(const LaunchArgs a)
{
    stamp_start(a, STAMP_Z);
    cudaTriggerProgrammaticLaunchCompletion();
    if (a.nsort) cudaGridDependencySynchronize();  // the order
    const TableJob t = a.tables[blockIdx.x];
    const uint32_t i = blockIdx.y * blockDim.x + threadIdx.x;
    if (i >= t.R) return;
    const uint32_t at = i + t.rot;
    const uint32_t j = t.order ? t.order[at < t.R ? at : at - t.R] : a.perm[t.ray_off + i];
    double z = x::norminv(t.points ? a.ray_u[t.u_off + j] : x::seed_point(t.seed, j + 1u));
    if (!isfinite(z)) {
        // a point that rounds to 0: its start height is not finite, and the host's table leaves it out
        atomicOr(&a.ctl->overflow, kOverflowTable);
        z = 0.0;
    }
    float hi, lo;
    split_f32(z, hi, lo);
    reinterpret_cast<float2 *>(const_cast<float *>(a.z32))[t.ray_off + i] = make_float2(hi, lo);
    if (a.rank) const_cast<uint32_t *>(a.rank)[t.rank_off + j] = i;
}

// The setup of one wavelength row (below): LamParams and LamDF, and the row's guard-band
// rays queued. Returns the row's fast-path range [core_lo, core_hi) (empty: hi <= lo).
// A row whose design failed its device build: every ray of it is lost.
__device__ __forceinline__ uint2 setup_failed_row(const LaunchArgs &a, uint64_t row)
{
    LamParams P;
    zero_lam_params(P);
    LamDF *E = a.lx + row;
    memset(E, 0, sizeof(LamDF));
    E->lost = 1u;
    a.lp[row] = P;
    return make_uint2(0u, 0u);
}

// A row with this many rays for the float-float trace goes to rows_kernel<HEAVY>. Almost all such
// rows have no reference ray (their rays miss the exit face or are reflected) and are traced whole.
constexpr uint32_t kRowsHeavy = 256;
constexpr uint32_t kNotHere = 0xffffffffu;  // such a row's ranges in its LamParams: empty

// A row's LamParams after lambda_setup_df: its guard-band rays queued as the mode asks, the
// record written. Returns the row's fast-path range [core_lo, core_hi) (empty: hi <= lo).
__device__ __forceinline__ uint2 setup_finish(const LaunchArgs &a, uint32_t d, uint32_t k, uint64_t row, LamParams &P,
                                              bool pieces)
{
    if (a.adaptive) {
        // the adaptive rounds trace every ray of the band themselves
    } else if (pieces) {
        // rows_kernel re-traces the guard bands itself; without a reference ray, all of the band
        if (P.all_exact) P.core_lo = P.core_hi = P.band_hi;
        if (a.heavy && P.band_hi - P.band_lo >= P.core_hi - P.core_lo + kRowsHeavy) {
            a.heavy[atomicAdd(&a.ctl->heavy_count, 1u)] = HeavyRow{row, 0u, {P.core_lo, P.core_hi, P.band_lo, P.band_hi}};
            P.core_lo = P.core_hi = P.band_lo = P.band_hi = kNotHere;
        }
    } else if (a.mode == CPD_TRACE_FP64 || (P.all_exact && a.mode == CPD_TRACE_HYBRID)) {
        push_ranges(a, d, k, P.band_lo, P.band_hi, 0u, 0u);
        P.core_lo = P.core_hi = 0;
    } else if (P.all_exact) {
        // FP32-only study mode without a reference ray: these rays are counted as lost
        P.core_lo = P.core_hi = 0;
    } else {
        push_ranges(a, d, k, P.band_lo, P.core_lo, P.core_hi, P.band_hi);
    }
    a.lp[row] = P;
    return make_uint2(P.core_lo, P.core_hi);
}

// The setup of one wavelength row (below): LamParams and LamDF, and the row's guard-band
// rays queued. Returns the row's fast-path range [core_lo, core_hi) (empty: hi <= lo).
__device__ __forceinline__ void setup_row(const LaunchArgs &a, uint64_t row, uint32_t d, double u,
                                          const DevDesign &sD, uint32_t d0, bool stage_z, const float *sz)
{
    const DesignJob &J = a.jobs[d];
    const uint32_t k = (uint32_t)(row - J.row_off);
    const bool staged = d == d0;
    const DevDesign &D = staged ? sD : a.designs[d];
    const float *z32 = staged && stage_z ? sz : a.z32 + 2 * J.ray_off;
    if (D.status) {
        setup_failed_row(a, row);
        return;
    }
    LamParams P;
    lambda_setup_df(D, u, z32, J.Rz, P, a.yguard_rel, a.lx + row, a.adaptive != 0);
    setup_finish(a, d, k, row, P, J.pieces != 0u);
}

// One thread per row; kSetupThreads per block where that leaves every SM as many warps as it holds
// (below, a warp per block spreads the rows over more SMs). A block's warps run the same code on
// one design's tables: 2.3 M rows of 1024 designs take 534 us in blocks of 128 at 96 registers (20
// warps per SM; 528 at 80, which spills), 538 at the compiler's 107, 613 in blocks of 32, where one
// issue slot in five waits for instructions. FP32 issue bounds it (5400 instructions per warp: 335 us).
// The block first copies its design record and, for
// tables of up to a.stage_cap rays, its sorted z table into shared memory with
// asynchronous 16-byte copies that are all in flight at once (one memory latency
// instead of a chain of dependent loads), so the per-wavelength program and its binary
// searches run on shared-memory operands. Ray tables start 16-byte aligned (the host
// pads each to an even number of rays).
// STAMPED: the pass's first stamp (a branch of its own in front of the trigger below costs passes of
// several designs 2 to 4 us, though none of them takes it: 8 x 128 rows, adaptive, 66.6 -> 71.1).
constexpr uint32_t kSetupThreads = 128;
template <bool STAMPED>
__global__ void __maxnreg__(96) setup_kernel(const LaunchArgs a)
{
    if (STAMPED) stamp_start(a, STAMP_SETUP);
    // lets the trace kernel's blocks become resident now; they wait for this grid's
    // results in cudaGridDependencySynchronize
    cudaTriggerProgrammaticLaunchCompletion();
    if (a.clear_acc) {
        // a fresh pass: zero the per-bin and per-design accumulators (the kernels that add
        // to them wait for this grid to complete)
        const uint64_t gt = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
        const uint64_t nt = (uint64_t)gridDim.x * blockDim.x;
        for (uint64_t i = gt; i < a.acc_cells; i += nt) a.S1[i] = a.S2[i] = 0ull;
        unsigned long long *acc = reinterpret_cast<unsigned long long *>(a.acc);
        const uint64_t words = (uint64_t)a.njobs * (sizeof(DesignAcc) / sizeof(unsigned long long));
        for (uint64_t i = gt; i < words; i += nt) acc[i] = 0ull;
    }
    __shared__ __align__(16) DevDesign sD;
    extern __shared__ __align__(16) float sz[];  // 2 even(stage_cap) floats
    if (a.ntables) cudaGridDependencySynchronize();  // the ray tables
    const uint64_t row0 = blockIdx.x * (uint64_t)blockDim.x;
    const uint64_t row = row0 + threadIdx.x;
    const uint32_t d0 = find_job<F_ROW>(a.jobs, a.njobs, row0);
    const DesignJob &J0 = a.jobs[d0];
    const bool stage_z = J0.Rz <= a.stage_cap;
    // the row's design and wavelength point, loaded while the copies below are in flight
    // (the point is not in L2 when the previous pass's tables were evicted)
    uint32_t d = 0;
    double u = 0.0;
    if (row < a.total_rows) {
        d = find_job<F_ROW>(a.jobs, a.njobs, row);
        const DesignJob &J = a.jobs[d];
        u = lam_point(a, J, (uint32_t)(row - J.row_off));
    }
    {
        const char *src = reinterpret_cast<const char *>(a.designs + d0);
        char *dst = reinterpret_cast<char *>(&sD);
        for (uint32_t i = threadIdx.x; i < sizeof(DevDesign) / 16; i += blockDim.x) cp_async16(dst + 16 * i, src + 16 * i);
        if (stage_z) {
            const char *zs = reinterpret_cast<const char *>(a.z32 + 2 * J0.ray_off);
            char *zd = reinterpret_cast<char *>(sz);
            const uint32_t n16 = (J0.Rz + 1u) / 2u;  // 16-byte chunks (two rays each)
            for (uint32_t i = threadIdx.x; i < n16; i += blockDim.x) cp_async16(zd + 16 * i, zs + 16 * i);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    __syncthreads();
    if (row < a.total_rows) setup_row(a, row, d, u, sD, d0, stage_z, sz);
}


// The rays [j0, j1) of the 32-row block blk of design d (lane = row), each lane clamped
// to its row's fast-path range: FP32 fast path, hits as run-length fixed-point sums
// flushed with one 64-bit atomic per run, guard-band rays queued for the re-trace.
// The setup of a single-design pass (a.spans set) by two warps per block of 32 rows. Each
// row's flat-face chain splits into two halves that depend on each other only through the
// direction entering each face: warp 0 runs the direction part of every face (the glass
// index, the refraction, the Fresnel factors), warp 1 the position part (the distance to
// the face, the bounds it puts on y, the point on it), face by face in step: at face k warp
// 1 reads the direction d_k that warp 0 published at face k - 1, one block barrier per face.
// Each warp stops where lambda_setup_df's loop would stop (a face parallel to the ray, which
// both see from the same cosine; total internal reflection, which warp 0 reports; a bound
// independent of y, which warp 1 reports), and warp 0 then finishes the row alone (y
// interval, ray ranges, reference ray). The functions are lambda_setup_df's own, so every
// output is bit-identical to the one-warp setup; the chain that is one warp per SM in the
// plain call is about half as long.
__global__ void __launch_bounds__(64) setup_pair_kernel(const LaunchArgs a)
{
    stamp_start(a, STAMP_SETUP);
    cudaTriggerProgrammaticLaunchCompletion();
    if (a.clear_acc) {
        const uint64_t gt = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
        const uint64_t nt = (uint64_t)gridDim.x * blockDim.x;
        for (uint64_t i = gt; i < a.acc_cells; i += nt) a.S1[i] = a.S2[i] = 0ull;
        unsigned long long *acc = reinterpret_cast<unsigned long long *>(a.acc);
        const uint64_t words = (uint64_t)a.njobs * (sizeof(DesignAcc) / sizeof(unsigned long long));
        for (uint64_t i = gt; i < words; i += nt) acc[i] = 0ull;
    }
    __shared__ __align__(16) DevDesign sD;
    extern __shared__ __align__(16) float sz[];  // 2 even(stage_cap) floats
    __shared__ ff::F2 s_dir[CPD_MAX_GLASS + 1][2][32];  // direction entering face k (x, y)
    __shared__ uint32_t s_tir[32], s_bound[32];          // stops reported at the last face
    __shared__ SetupPos s_pos[32];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint64_t row = blockIdx.x * 32ull + lane;
    const DesignJob &J = a.one;
    const bool have = row < a.total_rows;
    const bool stage_z = J.Rz <= a.stage_cap;
    // the seed from the uploaded job: the parameter's is left out (it would make every seed a
    // graph of its own)
    const double u = have && warp == 0 ? lam_point(a, a.jobs[0], (uint32_t)row) : 0.0;
    {
        // two groups of copies: the design record, which the face loop needs, and the z
        // table, which only the ray ranges after the loop read (its copies land while the
        // faces run)
        const char *src = reinterpret_cast<const char *>(a.designs);
        char *dst = reinterpret_cast<char *>(&sD);
        for (uint32_t i = threadIdx.x; i < sizeof(DevDesign) / 16; i += blockDim.x) cp_async16(dst + 16 * i, src + 16 * i);
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (stage_z && !a.ntables) {
            const char *zs = reinterpret_cast<const char *>(a.z32 + 2 * J.ray_off);
            char *zd = reinterpret_cast<char *>(sz);
            const uint32_t n16 = (J.Rz + 1u) / 2u;  // 16-byte chunks (two rays each)
            for (uint32_t i = threadIdx.x; i < n16; i += blockDim.x) cp_async16(zd + 16 * i, zs + 16 * i);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
    }
    __syncthreads();
    const DevDesign &D = sD;
    const int G = D.G;
    const float yg = (float)a.yguard_rel;
    SetupDir Sd = setup_dir_init();
    SetupPos Sp = setup_pos_init();
    const ff::F2 lambda = warp == 0 ? setup_lambda(D, u) : ff::F2{0.f, 0.f};
    bool stop = !have || D.status != 0;
    bool lost = false;  // warp 0: a face parallel to the ray, or total internal reflection
#pragma unroll 1
    for (int k = 0; k < G; k++) {
        bool tir = false;
        if (!stop) {
            if (warp == 0) {
                const ff::F2 ci = face_cos(D, k, Sd.dx, Sd.dy);
                if (ci.hi == 0.f) {
                    lost = stop = true;
                } else if (!face_direction(D, k, lambda, ci, Sd, false)) {
                    lost = stop = tir = true;
                } else {
                    s_dir[k + 1][0][lane] = Sd.dx;
                    s_dir[k + 1][1][lane] = Sd.dy;
                }
            } else {
                const ff::F2 dx = k == 0 ? df::c(1.f) : s_dir[k][0][lane];
                const ff::F2 dy = k == 0 ? df::c(0.f) : s_dir[k][1][lane];
                const ff::F2 ci = face_cos(D, k, dx, dy);
                if (ci.hi == 0.f) stop = true;  // warp 0 sees the same cosine
                else face_position(D, k, ci, dx, dy, Sp, yg);
                if (Sp.lost) stop = true;
            }
        }
        if (warp == 0) s_tir[lane] = tir ? 1u : 0u;
        else s_bound[lane] = Sp.lost ? 1u : 0u;
        __syncthreads();
        // lambda_setup_df breaks after a face's direction part that found total internal
        // reflection, and before the face after one whose position part found a bound
        // independent of y
        if (warp == 0 && s_bound[lane]) stop = true;
        if (warp == 1 && s_tir[lane]) stop = true;
        __syncthreads();  // the flags are written again at the next face
    }
    if (warp == 1) s_pos[lane] = Sp;
    if (a.ntables) {
        // tables made in this pass, beside the face loop
        cudaGridDependencySynchronize();
        if (stage_z) {
            const char *zs = reinterpret_cast<const char *>(a.z32 + 2 * J.ray_off);
            char *zd = reinterpret_cast<char *>(sz);
            const uint32_t n16 = (J.Rz + 1u) / 2u;
            for (uint32_t i = threadIdx.x; i < n16; i += blockDim.x) cp_async16(zd + 16 * i, zs + 16 * i);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");  // this thread's share of the z table
    __syncthreads();
    if (warp == 1) return;
    uint2 core = make_uint2(0u, 0u);
    if (have) {
        if (D.status) {
            core = setup_failed_row(a, row);
        } else {
            Sp = s_pos[lane];
            const float *z32 = stage_z ? sz : a.z32 + 2 * J.ray_off;
            LamParams P;
            zero_lam_params(P);
            setup_tail(D, z32, J.Rz, P, a.lx + row, Sd, Sp, lost || Sp.lost);
            core = setup_finish(a, 0u, (uint32_t)row, row, P, J.pieces != 0u);
        }
    }
    // this block's 32 rows are the trace's block blockIdx.x
    const bool any = core.y > core.x;
    const uint32_t lo = __reduce_min_sync(0xffffffffu, any ? core.x : 0xffffffffu);
    const uint32_t hi = __reduce_max_sync(0xffffffffu, any ? core.y : 0u);
    if (lane == 0) {
        const uint2 sp = hi > lo ? make_uint2(lo, hi) : make_uint2(0u, 0u);
        a.spans[blockIdx.x] = sp;
        if (sp.y > sp.x) atomicAdd(&a.ctl->item_counter, (unsigned long long)(sp.y - sp.x));
    }
}

// Flagged rays a warp of the single-design trace keeps for its own re-trace.
constexpr uint32_t kWarpFlags = 32;

// The float-float re-trace of one queued ray (k, j) of design d, counted in copy sp of
// the design's counters.
__device__ __forceinline__ void retrace_ray(const LaunchArgs &a, uint32_t d, uint32_t k, uint32_t j, uint32_t sp)
{
    const DesignJob &J = a.jobs[d];
    const float *z = a.z32 + 2 * (J.ray_off + j);
    uint32_t bin = 0;
    float t = 0.f;
    if (trace_df(a.designs[d], a.lx[J.row_off + k], z[0], z[1], bin, t)) {
        atomicAdd(a.hist + J.hist_off + (uint64_t)k * J.B + bin, (unsigned long long)t_fixed(t));
        atomicAdd(&a.acc[d].hits[sp], 1ull);
    }
    atomicAdd(&a.acc[d].retraced[sp], 1ull);
}

// PARAM_FC: the single-design trace, whose constants are kernel parameters. Flagged rays
// go to the warp's list (wlist, *wcount: design, row, ray), the global queue once it is full.
template <bool PARAM_FC>
__device__ __forceinline__ void trace_block_rays(const LaunchArgs &a, uint32_t d, const DesignJob &J, uint32_t blk,
                                                 uint32_t j0, uint32_t j1, uint32_t lane, uint3 *wlist,
                                                 uint32_t *wcount)
{
    const uint32_t k = blk * 32u + lane;
    // the design's constants: kernel parameters (constant-bank operands, no registers)
    // for a single-design pass, else a copy in registers
    const FastConst Cd = PARAM_FC ? FastConst{} : a.designs[d].fc;
    const FastConst &C = PARAM_FC ? a.fc : Cd;
    const FastLimits Ld = PARAM_FC ? FastLimits{} : fast_limits(Cd, a.guards);
    const FastLimits &Lm = PARAM_FC ? a.fl : Ld;
    LamParams P;
    uint32_t lo = 0, hi = 0;
    if (k < J.W) {
        P = a.lp[J.row_off + k];
        lo = max(j0, P.core_lo);
        hi = min(j1, P.core_hi);
    }
    const float2 *__restrict__ zt = reinterpret_cast<const float2 *>(a.z32) + J.ray_off;
    unsigned long long *hrow = a.hist + J.hist_off + (uint64_t)k * J.B;
    uint32_t cur = 0xffffffffu;
    unsigned long long sum = 0ull;
    uint32_t nhit = 0;
    for (uint32_t j = lo; j < hi; ++j) {
        const float2 z = __ldg(zt + j);
        uint32_t bin = 0;
        float t = 0.f;
        const int r = fast_ray(C, Lm, P, a.guards, z.x, z.y, bin, t);
        if (r == RAY_HIT) {
            if (bin != cur) {
                if (sum) atomicAdd(hrow + cur, sum);
                cur = bin;
                sum = 0ull;
            }
            sum += t_fixed(t);
            nhit++;
        } else if (r == RAY_FLAG) {
            const uint32_t pos = atomicAdd(wcount, 1u);
            if (pos < kWarpFlags) wlist[pos] = make_uint3(d, k, j);
            else push_ray(a, d, k, j);
        }
    }
    if (sum) atomicAdd(hrow + cur, sum);
    nhit = __reduce_add_sync(0xffffffffu, nhit);
    const uint32_t nfast = __reduce_add_sync(0xffffffffu, hi > lo ? hi - lo : 0u);
    const uint32_t sp = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) % (uint32_t)kSpread;
    if (lane == 0 && nhit) atomicAdd(&a.acc[d].hits[sp], (unsigned long long)nhit);
    if (lane == 0 && nfast) atomicAdd(&a.acc[d].fast[sp], (unsigned long long)nfast);
}

// The trace of a single-design pass whose setup wrote the blocks' spans (a.spans). Its
// design constants are kernel parameters (constant-bank operands), which frees the ~17
// registers a copy of them takes (75 registers with the re-trace list, no spill). Measured
// on the 4096 x 1024 plain pass: at 64 registers
// (4 blocks of 256 per SM, 32 warps, no spill) the trace issues 68% of the slots against
// 62%, but fills the register file, so the re-trace and entropy blocks can no longer
// become resident while it runs, and the pass is ~1.5 us slower than at 3 blocks per SM.
#ifndef CPD_TRACE_SPANS_MIN_BLOCKS
#define CPD_TRACE_SPANS_MIN_BLOCKS 3
#endif
__global__ void __launch_bounds__(256, CPD_TRACE_SPANS_MIN_BLOCKS) trace_spans_kernel(const LaunchArgs a)
{
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();  // setup's LamParams and queue
    const uint32_t lane = threadIdx.x & 31u;
    // Equal shares of the design's fast-path ray slots: the blocks' spans laid end to
    // end (U slots in all), warp w taking [U w / nw, U (w + 1) / nw). A warp's lanes
    // step through a block's span together, so a span costs its length whatever the
    // rows' own ranges; every warp gets the same work and no warp waits on a counter.
    // Nothing stays live in registers across a segment's ray loop (which needs every
    // register it can get): the cursor waits in shared memory, and the share's end and the
    // prefix over the spans are found again from the pass's words for each segment.
    // A warp's flagged rays wait in its list and are re-traced by the warp after its share
    // (rays past kWarpFlags go to the global queue and the re-trace kernel): the re-trace
    // of the pass then overlaps the trace instead of following it.
    __shared__ volatile unsigned long long s_cur[8];  // per warp of the block (<= 256 threads)
    __shared__ uint3 s_flags[8][kWarpFlags];
    __shared__ uint32_t s_nflags[8];
    const uint32_t wib = threadIdx.x >> 5;
    {
        const uint64_t w = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
        const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
        s_cur[wib] = a.ctl->item_counter * w / nw;  // the next slot of this warp's share
        if (lane == 0) s_nflags[wib] = 0u;
    }
    for (;;) {
        __syncwarp();
        uint64_t cur = s_cur[threadIdx.x >> 5];
        const uint64_t end = a.ctl->item_counter * (((blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5) + 1u) /
                             (((uint64_t)gridDim.x * blockDim.x) >> 5);
        if (cur >= end) break;
        const uint32_t nb = (a.jobs[0].W + 31u) / 32u;
        uint64_t pre = 0;  // slots of the blocks before group c
        uint32_t c = 0, sx, len, incl;
        for (;;) {
            const uint32_t b = c + lane;
            const uint2 s = b < nb ? a.spans[b] : make_uint2(0u, 0u);
            sx = s.x;
            len = s.y - s.x;
            incl = len;  // inclusive scan over the group
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= (uint32_t)o) incl += v;
            }
            const uint32_t tot = __shfl_sync(0xffffffffu, incl, 31);
            if (pre + tot > cur) break;
            pre += tot;
            c += 32u;
        }
        // the block holding the cursor: the first whose end lies past it (nonempty)
        const int l = __ffs(__ballot_sync(0xffffffffu, pre + incl > cur)) - 1;
        const uint32_t bx = __shfl_sync(0xffffffffu, sx, l);
        const uint32_t ln = __shfl_sync(0xffffffffu, len, l);
        const uint64_t e0 = pre + __shfl_sync(0xffffffffu, incl, l) - ln;
        const uint64_t rem = end - e0;
        const uint32_t stop = rem < ln ? (uint32_t)rem : ln;
        const uint32_t r0 = bx + (uint32_t)(cur - e0);
        __syncwarp();
        s_cur[threadIdx.x >> 5] = e0 + stop;
        const DesignJob J = a.jobs[0];
        trace_block_rays<true>(a, 0u, J, c + (uint32_t)l, r0, bx + stop, lane, s_flags[wib], &s_nflags[wib]);
    }
    __syncwarp();
    const uint32_t nf = min(s_nflags[wib], kWarpFlags);
    const uint32_t sp = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) % (uint32_t)kSpread;
    for (uint32_t i = lane; i < nf; i += 32u) retrace_ray(a, 0u, s_flags[wib][i].y, s_flags[wib][i].z, sp);
}

// 72 registers: 28 resident warps per SM (blocks of 2 or 4 warps) against 24 at 80, for a
// 24-byte spill; measured on the 1024-design batched pass: 12.82 -> 12.33 ms (64 registers
// spill 88 bytes: 16.4 ms)
#ifndef CPD_TRACE_MAXNREG
#define CPD_TRACE_MAXNREG 72
#endif
__global__ void __maxnreg__(CPD_TRACE_MAXNREG) trace_kernel(const LaunchArgs a)
{
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();  // setup's LamParams and queue
    const uint32_t lane = threadIdx.x & 31u;
    // a warp's flagged rays wait in its list; the warp re-traces them once half of the
    // list is taken, and at its end (rays past kWarpFlags go to the global queue)
    __shared__ uint3 s_flags[8][kWarpFlags];
    __shared__ uint32_t s_nflags[8];
    const uint32_t wib = threadIdx.x >> 5;
    const uint32_t sp = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) % (uint32_t)kSpread;
    if (lane == 0) s_nflags[wib] = 0u;
    for (;;) {
        unsigned long long item = 0;
        if (lane == 0) item = atomicAdd(&a.ctl->item_counter, 1ull);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= a.total_items) break;
        const uint32_t d = find_job<F_ITEM>(a.jobs, a.njobs, item);
        const DesignJob J = a.jobs[d];
        const uint64_t local = item - J.item_off;
        const uint32_t blk = (uint32_t)(local / J.nchunk);
        const uint32_t chunk = (uint32_t)(local - (uint64_t)blk * J.nchunk);
        const uint32_t j0 = chunk * a.ray_tile;
        trace_block_rays<false>(a, d, J, blk, j0, min(j0 + a.ray_tile, J.Rz), lane, s_flags[wib], &s_nflags[wib]);
        __syncwarp();
        const uint32_t nf = s_nflags[wib];
        if (nf >= kWarpFlags / 2u) {
            const uint32_t n = min(nf, kWarpFlags);
            if (lane < n) retrace_ray(a, s_flags[wib][lane].x, s_flags[wib][lane].y, s_flags[wib][lane].z, sp);
            __syncwarp();
            if (lane == 0) s_nflags[wib] = 0u;
            __syncwarp();
        }
    }
    __syncwarp();
    const uint32_t n = min(s_nflags[wib], kWarpFlags);
    if (lane < n) retrace_ray(a, s_flags[wib][lane].x, s_flags[wib][lane].y, s_flags[wib][lane].z, sp);
}

// The queued rays, hybrid mode: the float-float re-trace.
// The pass's final queue state for the host (no later kernel changes it).
__device__ __forceinline__ void publish_status_all(const LaunchArgs &a)
{
    if (a.status && threadIdx.x == 0) {
        a.status->queue_count = a.ctl->queue_count;
        a.status->overflow = a.ctl->overflow;
        a.status->pad = 0u;
    }
}
__device__ __forceinline__ void publish_status(const LaunchArgs &a)
{
    if (blockIdx.x == 0) publish_status_all(a);
}

__global__ void __launch_bounds__(32) retrace_kernel(const LaunchArgs a)
{
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();  // the queue of the setup and trace kernels
    publish_status(a);
    const unsigned long long qn = a.ctl->queue_count;
    const uint64_t n = qn < a.qcap ? qn : a.qcap;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const QEntry e = a.queue[i];
        retrace_ray(a, e.design, e.k, e.j, (uint32_t)(i % kSpread));
    }
}

// The queued rays, FP64 study mode: the exact f64 trace of the reference
// (bit-identical to its CPU path). A kernel of its own, so that the hybrid re-trace
// does not carry this code.
__global__ void __launch_bounds__(32) retrace_exact_kernel(const LaunchArgs a)
{
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();  // the queue of the setup and trace kernels
    publish_status(a);
    const unsigned long long qn = a.ctl->queue_count;
    const uint64_t n = qn < a.qcap ? qn : a.qcap;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const QEntry e = a.queue[i];
        const DevDesign &D = a.designs[e.design];
        const DesignJob &J = a.jobs[e.design];
        uint32_t bin = 0;
        double t = 0.0;
        if (x::trace(D, x::wavelength(D, lam_point(a, J, e.k)), x::beam_y(D, a.z64[J.ray_off + e.j]), bin, t) ==
            0) {
            atomicAdd(a.hist + J.hist_off + (uint64_t)e.k * J.B + bin, (unsigned long long)t_fixed64(t));
            atomicAdd(&a.acc[e.design].hits[i % kSpread], 1ull);
        }
        atomicAdd(&a.acc[e.design].retraced[i % kSpread], 1ull);
    }
}

// ------------------------------------------------------------------ adaptive sampling

// The float-float exact trace of one ray as (bin or ~0u, t_fixed).
__device__ __forceinline__ uint2 trace_df_exact_packed(const DevDesign &D, const LamDF &E, float zh, float zl)
{
    uint32_t b = 0, tx = 0;
    return trace_df_exact(D, E, zh, zl, b, tx) ? make_uint2(b, tx) : make_uint2(0xffffffffu, 0u);
}

// The same, out of line: the fast kernel takes it for ~0.1% of its rays, and inlined its
// float-float code would set the register budget of the whole kernel.
__device__ __noinline__ uint2 trace_df_exact_call(const DevDesign &D, const LamDF &E, float zh, float zl)
{
    return trace_df_exact_packed(D, E, zh, zl);
}

// Per-warp scratch of the adaptive kernels (dynamic shared memory, one slot per warp,
// before the bin states). A group of KW rounds is traced by KW warps, warp w taking round
// w of the group; each warp sums its round's hits per bin into its slot, and the group's
// stop decisions are then taken by all warps at once, each from its round's exact Welford
// states (the states at the group's start plus the sums of the group's rounds up to its
// own). The first round that stops, or that the FP32 sums cannot settle, ends the row.
struct RoundSlot {
    // indexed by the leader lane of a bin the round hit: the round's sums there, in 32-bit
    // pieces (t_fixed = q 2^11 + low, q = qh 2^10 + ql, q <= 2^20): sum q, sum low,
    // sum qh^2, sum qh ql, sum ql^2, and the hits
    uint32_t p[6][32];
    uint32_t df;       // ballot of the rays traced in float-float
    uint32_t nh;       // hits of the round
    uint32_t verdict;  // 0 go on, 1 stop, 2 unsure, 3 a hit of another transmittance (ROWS_EQUAL)
    uint32_t pad;
};
static_assert(sizeof(RoundSlot) % 16 == 0, "bin states follow the slots 16-byte aligned");
// Dynamic shared memory of an adaptive block of KW warps over B-bin detectors.
constexpr size_t adapt_smem_bytes(uint32_t KW, uint32_t B) { return KW * sizeof(RoundSlot) + bin_state_bytes(B); }
static_assert(adapt_smem_bytes(kMaxAdaptWarps, CPD_MAX_BINS) <= 227u * 1024u, "shared memory per block");

// Dynamic shared memory of the one-warp form (adaptive_row1): the row's LamParams and
// FastConst, one slot, the bin states.
constexpr size_t adapt1_smem_bytes(uint32_t B)
{
    return sizeof(LamParams) + sizeof(FastConst) + adapt_smem_bytes(1, B);
}

// Byte v of a bin's group lane table (v = the round within the group).
__device__ __forceinline__ uint32_t lane_entry(const uint4 &w, uint32_t v)
{
    const uint32_t word = v < 8u ? (v < 4u ? w.x : w.y) : (v < 12u ? w.z : w.w);
    return (word >> (8u * (v & 3u))) & 0xffu;
}

// One wavelength row under adaptive sampling (the stop rule of src/spectrometer/
// kernel.rs:127-178, restated with exact integer Welford sums: cpd_model.h, sem_test)
// by one block of KW warps; the bin states live in shared memory after the KW slots.
// Tracing: lane l of warp w takes ray g0 + 32 w + l in index order; `rank` maps it to its
// place in the sorted z table, whose band / core ranges (from the setup) say how to trace
// it: lost outside the band, the FP32 fast path inside the core, the float-float trace
// (exact transmittance) otherwise or when the fast path flags it.
// Deciding: each bin a round hit is led by the lowest lane that hit it; the leader sums
// the round's hits there, and the bin's group lane table records which lane of which round
// holds those sums. A round's leaders then add the sums of the group's rounds up to theirs
// to the states at the group's start, run the SEM test, and vote: the round stops the row
// when it hit some bin and every bin it hit passes. Rounds after the first one that stops
// were traced for nothing and are dropped; the states through that round are written back
// by the leader of each bin's latest round. Everything is integer, so the result equals
// the one-round-at-a-time order bit for bit.
// kExact: every ray by the float-float trace and the exact test. Otherwise a row whose
// stop decision the FP32 transmittances cannot settle (sem_test: SEM_UNSURE) leaves
// nothing behind and returns ROW_UNSURE: the caller redoes it on the exact path. (In the
// verification mode every row is queued for adaptive_exact_kernel instead.)
// ROWS_EQUAL: a design with certified pieces (ROWS_MIXED: if it has them). Its rows have the
// arithmetic of adaptive_row1_pieces, decision for decision (one transmittance, states of samples and
// hits alone, a row with a hit of another transmittance up to its stop returned as ROW_OTHER), so
// that they come out the same here and there; kExact then concerns the transmittance and the test.
enum : int { ROW_DONE = 0, ROW_UNSURE = 1, ROW_OTHER = 2 };
enum : int { ROWS_GENERAL = 0, ROWS_EQUAL = 1, ROWS_MIXED = 2 };
template <bool kExact, int kRows = ROWS_GENERAL>
__device__ int adaptive_row(const LaunchArgs &a, uint64_t row, unsigned long long *smem, uint32_t KW,
                             uint32_t warp, uint32_t lane)
{
    const uint32_t d = find_job<F_ROW>(a.jobs, a.njobs, row);
    const DesignJob &J = a.jobs[d];
    const uint32_t k = (uint32_t)(row - J.row_off);
    const uint32_t B = J.B, R = J.R;
    const DevDesign &D = a.designs[d];
    const bool equal = kRows == ROWS_MIXED ? D.fc.pieces != 0u : kRows == ROWS_EQUAL;
    const uint32_t tid = warp * 32u + lane, nthr = KW * 32u;
    if (!kExact && a.adaptive == 2u) {
        // verification mode: every row on the exact path
        if (tid == 0) {
            const unsigned long long pos = atomicAdd(&a.ctl->queue_count, 1ull);
            if (pos < a.qcap) a.queue[pos] = QEntry{d, k, 0u, 0u};
            else atomicOr(&a.ctl->overflow, kOverflowQueue);
        }
        return ROW_DONE;
    }
    RoundSlot *slots = reinterpret_cast<RoundSlot *>(smem);
    RoundSlot &my = slots[warp];
    const FastConst C = D.fc;
    const LamParams P = a.lp[row];
    const LamDF &E = a.lx[row];
    const BinStates st(slots + KW, B);
    const uint32_t tfast = equal ? piece_tfix(P) : 0u, tfix = equal ? coated_tfix(E) : 0u;
    const uint32_t tfx = kExact ? tfix : tfast, tq = tfx >> kTqShift;
    constexpr uint32_t delta = kExact ? 0u : kTqDelta;
    if (equal && !kExact && (tfix >> kTqShift) - tq + kTqDelta > 2u * kTqDelta) return ROW_OTHER;
    for (uint32_t b = tid; b < B; b += nthr) {
        st.s1[b] = 0ull;  // equal: what the float-float hits add beside tfast
        if (!equal) st.q1[b] = st.q2[b] = 0ull;
        st.n[b] = st.h[b] = 0u;
        st.lanes[b] = make_uint4(0u, 0u, 0u, 0u);
        st.rounds[b] = 0u;
    }
    __syncthreads();
    const uint32_t *rank = a.rank + J.rank_off;
    const float2 *zt = reinterpret_cast<const float2 *>(a.z32) + J.ray_off;
    const uint32_t lt_mask = (1u << lane) - 1u;
    uint32_t count = 0, flag = 0;  // the same in every thread
    uint32_t hits = 0, ndf = 0;    // thread 0
    // no ray clears the flat faces: every round runs without a hit
    const uint32_t g_start = P.band_lo >= P.band_hi ? R : 0u;
    if (g_start == R) count = R;
    // the ray a lane traces in the next group, loaded while the current group is decided:
    // its sorted position (~0u: none, or no finite start height; outside the band either
    // way) and its start height
    uint32_t s_nx = 0xffffffffu;
    float2 z_nx = make_float2(0.f, 0.f);
    const auto fetch = [&](uint32_t g) {
        const uint32_t j = g + warp * kRoundRays + lane;
        s_nx = j < R ? rank[j] : 0xffffffffu;
        if (s_nx >= P.band_lo && s_nx < P.band_hi) z_nx = zt[s_nx];
    };
    if (g_start < R) fetch(g_start);
    for (uint32_t g0 = g_start; g0 < R; g0 += KW * kRoundRays) {
        // 1. trace round `warp` of the group; each bin's leader sums the round's hits there
        uint32_t bin = 0xffffffffu, tf = 0u;
        bool used_df = false, other = false;
        {
            const uint32_t s = s_nx;
            if (s >= P.band_lo && s < P.band_hi) {
                const float2 z = z_nx;
                int res = RAY_FLAG;
                if ((!kExact || equal) && !P.all_exact && s >= P.core_lo && s < P.core_hi) {
                    uint32_t b = 0;
                    float t = 0.f;
                    res = fast_ray(C, P, a.guards, z.x, z.y, b, t);
                    if (res == RAY_HIT) {
                        bin = b;
                        tf = t_fixed(t);
                        other = equal && tf != tfast;
                    }
                }
                if (res == RAY_FLAG) {
                    const uint2 r = trace_df_exact_call(D, E, z.x, z.y);
                    bin = r.x;
                    tf = r.y;
                    used_df = true;
                    other = equal && bin != 0xffffffffu && tf != tfix;
                }
                if (equal && kExact) used_df = true;
            }
        }
        if (g0 + KW * kRoundRays < R) fetch(g0 + KW * kRoundRays);
        const bool hit = bin != 0xffffffffu;
        const uint32_t hm = __ballot_sync(0xffffffffu, hit);
        const uint32_t dfb = __ballot_sync(0xffffffffu, used_df);
        const uint32_t grp = __match_any_sync(0xffffffffu, bin);
        const bool leader = hit && (grp & lt_mask) == 0u;
        if (lane == 0) {
            my.df = dfb;
            my.nh = (uint32_t)__popc(hm);
        }
        const bool any_other = equal && __any_sync(0xffffffffu, other);
        if (equal) {
            if (leader) my.p[0][lane] = kExact ? 0u : (uint32_t)__popc(grp & dfb);  // float-float hits
        } else {
            // the bin's sums over its lanes: shared-memory adds into the leader's slot
            my.p[0][lane] = my.p[1][lane] = my.p[2][lane] = my.p[3][lane] = my.p[4][lane] = 0u;
            __syncwarp();
            if (hit) {
                const uint32_t ld = (uint32_t)__ffs(grp) - 1u, q = tf >> kTqShift;
                const uint32_t qh = q >> 10, ql = q & 0x3ffu;
                atomicAdd(&my.p[0][ld], q);
                atomicAdd(&my.p[1][ld], tf & 0x7ffu);
                atomicAdd(&my.p[2][ld], qh * qh);
                atomicAdd(&my.p[3][ld], qh * ql);
                atomicAdd(&my.p[4][ld], ql * ql);
            }
        }
        if (leader) {
            my.p[5][lane] = (uint32_t)__popc(grp);
            atomicOr(reinterpret_cast<uint32_t *>(st.lanes + bin) + (warp >> 2), (lane + 1u) << (8u * (warp & 3u)));
            atomicOr(st.rounds + bin, 1u << warp);
        }
        __syncthreads();
        // 2. every round's decision at once, from the states through that round
        uint4 lw = make_uint4(0u, 0u, 0u, 0u);
        uint32_t rmask = 0u;  // leader: the group's rounds that hit its bin
        unsigned long long cs1 = 0, cq1 = 0, cq2 = 0;
        uint32_t cn = 0, ch = 0;
        int verdict = SEM_PASS;
        if (leader) {
            lw = st.lanes[bin];
            rmask = st.rounds[bin];
            cs1 = st.s1[bin];
            if (!equal) {
                cq1 = st.q1[bin];
                cq2 = st.q2[bin];
            }
            cn = st.n[bin];
            ch = st.h[bin];
            for (uint32_t m = rmask & ((2u << warp) - 1u); m; m &= m - 1u) {  // rounds <= warp
                const uint32_t v = (uint32_t)__ffs(m) - 1u, l = lane_entry(lw, v);
                const RoundSlot &o = slots[v];
                const uint32_t sq = o.p[0][l - 1u];
                if (equal) {
                    cs1 += sq * ((unsigned long long)tfix - tfast);
                } else {
                    cs1 += ((unsigned long long)sq << kTqShift) + o.p[1][l - 1u];
                    cq1 += sq;
                    cq2 += ((unsigned long long)o.p[2][l - 1u] << 20) + ((unsigned long long)o.p[3][l - 1u] << 11) +
                           o.p[4][l - 1u];
                }
                ch += o.p[5][l - 1u];
                cn += min(kRoundRays, R - (g0 + v * kRoundRays));
            }
            verdict = equal ? sem_quick_equal(cn, ch, sem_equal(tq, delta)) : sem_quick(cn, ch, cq1, cq2, delta);
            if (equal) {
                cq1 = (unsigned long long)ch * tq;
                cq2 = cq1 * tq;
            }
        }
        if (__any_sync(0xffffffffu, verdict < 0) && verdict < 0)
            verdict = sem_test(cn, ch, cq1, cq2, delta);
        const bool fail = __any_sync(0xffffffffu, verdict == SEM_FAIL);
        const bool unsure = __any_sync(0xffffffffu, verdict == SEM_UNSURE);
        if (lane == 0) my.verdict = any_other ? 3u : (!hm || fail) ? 0u : (!kExact && unsure) ? 2u : 1u;
        __syncthreads();
        // 3. the first round that stops ends the row; the states through it are kept
        // (lane v reads round v's verdict)
        const uint32_t vv = lane < KW ? slots[lane].verdict : 0u;
        const uint32_t vb = __ballot_sync(0xffffffffu, vv != 0u);
        const uint32_t last = vb ? (uint32_t)__ffs(vb) - 1u : KW - 1u;
        if (vb) flag = __shfl_sync(0xffffffffu, vv, last);
        for (uint32_t v = 0; v <= last && g0 + v * kRoundRays < R; v++) {
            count += min(kRoundRays, R - (g0 + v * kRoundRays));
            if (tid == 0) {  // the row's totals, published by thread 0
                hits += slots[v].nh;
                ndf += (uint32_t)__popc(slots[v].df);
            }
        }
        if (leader) {
            const uint32_t later = rmask & ((2u << last) - 1u) & ~((2u << warp) - 1u);
            const uint32_t earlier = rmask & ((1u << warp) - 1u);
            if (warp <= last && !later) {  // the bin's latest round through `last`
                st.s1[bin] = cs1;
                if (!equal) {
                    st.q1[bin] = cq1;
                    st.q2[bin] = cq2;
                }
                st.n[bin] = cn;
                st.h[bin] = ch;
            }
            if (!earlier) {  // the bin's first round of the group clears its lane table
                st.lanes[bin] = make_uint4(0u, 0u, 0u, 0u);
                st.rounds[bin] = 0u;
            }
        }
        if (!flag && g0 + KW * kRoundRays >= R) flag = 1u;  // out of rays
        __syncthreads();
        if (flag) break;
    }
    if (flag >= 2u) {
        // the caller redoes the row on the exact path at once, or queues it
        __syncthreads();
        return flag == 2u ? ROW_UNSURE : ROW_OTHER;
    } else {
        unsigned long long *hrow = a.hist + J.hist_off + (uint64_t)k * B;
        for (uint32_t b = tid; b < B; b += nthr) {
            const unsigned long long s1 = st.s1[b] + (equal ? (unsigned long long)st.h[b] * tfx : 0ull);
            if (s1) hrow[b] = rescale_cell(s1, R, count);
        }
        if (tid == 0) {
            const uint32_t sp = (uint32_t)(row % (uint64_t)kSpread);
            atomicAdd(&a.acc[d].fast[sp], (unsigned long long)count);
            if (hits) atomicAdd(&a.acc[d].hits[sp], (unsigned long long)hits);
            if (ndf) atomicAdd(&a.acc[d].retraced[sp], (unsigned long long)ndf);
        }
    }
    __syncthreads();  // the slots and bin states are reused by the block's next row
    return ROW_DONE;
}

// One wavelength row under adaptive sampling by a single warp (the form for passes with
// many rows, where the rows themselves fill the GPU): the same rounds and decisions as
// adaptive_row, one round after another. Each bin's exact integer Welford sums are kept
// cumulatively in shared memory; a round's hit lanes add their sums into the slot of their
// bin's leader (the lowest lane that hit it), the leader adds them to the bin's state and
// tests the state through the round, and the round stops the row when it hit some bin and
// every bin it hit passes. No lane tables, no barriers: one warp decides each round alone.
template <bool kExact>
__device__ bool adaptive_row1(const LaunchArgs &a, uint64_t row, unsigned long long *smem, uint32_t lane)
{
    const uint32_t d = find_job<F_ROW>(a.jobs, a.njobs, row);
    const DesignJob &J = a.jobs[d];
    const uint32_t k = (uint32_t)(row - J.row_off);
    const uint32_t B = J.B, R = J.R;
    const DevDesign &D = a.designs[d];
    if (!kExact && a.adaptive == 2u) {
        // verification mode: every row on the exact path
        if (lane == 0) {
            const unsigned long long pos = atomicAdd(&a.ctl->queue_count, 1ull);
            if (pos < a.qcap) a.queue[pos] = QEntry{d, k, 0u, 0u};
            else atomicOr(&a.ctl->overflow, kOverflowQueue);
        }
        return false;
    }
    // the row's constants are the same in every lane: they live in shared memory (read
    // where they are used), which leaves the registers to more resident warps
    LamParams &P = *reinterpret_cast<LamParams *>(smem);
    FastConst &C = *reinterpret_cast<FastConst *>(reinterpret_cast<char *>(smem) + sizeof(LamParams));
    RoundSlot &my = *reinterpret_cast<RoundSlot *>(reinterpret_cast<char *>(smem) + sizeof(LamParams) + sizeof(FastConst));
    const LamDF &E = a.lx[row];
    const BinStates st(&my + 1, B);
    static_assert(sizeof(LamParams) % 16 == 0 && sizeof(FastConst) % 16 == 0, "16-byte copies");
    if (lane < sizeof(LamParams) / 16)
        reinterpret_cast<uint4 *>(&P)[lane] = reinterpret_cast<const uint4 *>(a.lp + row)[lane];
    else if (lane < (sizeof(LamParams) + sizeof(FastConst)) / 16)
        reinterpret_cast<uint4 *>(&C)[lane - sizeof(LamParams) / 16] =
            reinterpret_cast<const uint4 *>(&D.fc)[lane - sizeof(LamParams) / 16];
    for (uint32_t b = lane; b < B; b += 32u) {
        st.s1[b] = st.q1[b] = st.q2[b] = 0ull;
        st.n[b] = st.h[b] = 0u;
    }
    __syncwarp();
    const uint32_t *rank = a.rank + J.rank_off;
    const float2 *zt = reinterpret_cast<const float2 *>(a.z32) + J.ray_off;
    const uint32_t lt_mask = (1u << lane) - 1u;
    uint32_t count = 0, flag = 0, hits = 0, ndf = 0;  // the same in every lane
    // no ray clears the flat faces: every round runs without a hit
    const uint32_t g_start = P.band_lo >= P.band_hi ? R : 0u;
    if (g_start == R) count = R;
    // the ray this lane traces in the next round, loaded while the current one is decided
    uint32_t s_nx = 0xffffffffu;
    float2 z_nx = make_float2(0.f, 0.f);
    const auto fetch = [&](uint32_t g) {
        const uint32_t j = g + lane;
        s_nx = j < R ? rank[j] : 0xffffffffu;
        if (s_nx >= P.band_lo && s_nx < P.band_hi) z_nx = zt[s_nx];
    };
    if (g_start < R) fetch(g_start);
    for (uint32_t g0 = g_start; g0 < R; g0 += kRoundRays) {
        uint32_t bin = 0xffffffffu, tf = 0u;
        bool used_df = false;
        {
            const uint32_t s = s_nx;
            if (s >= P.band_lo && s < P.band_hi) {
                const float2 z = z_nx;
                int res = RAY_FLAG;
                if (!kExact && !P.all_exact && s >= P.core_lo && s < P.core_hi) {
                    uint32_t b = 0;
                    float t = 0.f;
                    res = fast_ray(C, P, a.guards, z.x, z.y, b, t);
                    if (res == RAY_HIT) {
                        bin = b;
                        tf = t_fixed(t);
                    }
                }
                if (res == RAY_FLAG) {
                    const uint2 r = trace_df_exact_call(D, E, z.x, z.y);
                    bin = r.x;
                    tf = r.y;
                    used_df = true;
                }
            }
        }
        if (g0 + kRoundRays < R) fetch(g0 + kRoundRays);
        const bool hit = bin != 0xffffffffu;
        const uint32_t hm = __ballot_sync(0xffffffffu, hit);
        const uint32_t dfb = __ballot_sync(0xffffffffu, used_df);
        const uint32_t grp = __match_any_sync(0xffffffffu, bin);
        const bool leader = hit && (grp & lt_mask) == 0u;
        const uint32_t rn = min(kRoundRays, R - g0);  // samples of this round
        // the round's sums per bin, in 32-bit pieces (as adaptive_row): into the leader's slot
        my.p[0][lane] = my.p[1][lane] = my.p[2][lane] = my.p[3][lane] = my.p[4][lane] = 0u;
        __syncwarp();
        if (hit) {
            const uint32_t ld = (uint32_t)__ffs(grp) - 1u, q = tf >> kTqShift;
            const uint32_t qh = q >> 10, ql = q & 0x3ffu;
            atomicAdd(&my.p[0][ld], q);
            atomicAdd(&my.p[1][ld], tf & 0x7ffu);
            atomicAdd(&my.p[2][ld], qh * qh);
            atomicAdd(&my.p[3][ld], qh * ql);
            atomicAdd(&my.p[4][ld], ql * ql);
        }
        __syncwarp();
        int verdict = SEM_PASS;
        uint32_t cn = 0, ch = 0;
        unsigned long long cq1 = 0, cq2 = 0;
        if (leader) {
            const uint32_t sq = my.p[0][lane];
            st.s1[bin] += ((unsigned long long)sq << kTqShift) + my.p[1][lane];
            cq1 = st.q1[bin] + sq;
            cq2 = st.q2[bin] + ((unsigned long long)my.p[2][lane] << 20) +
                  ((unsigned long long)my.p[3][lane] << 11) + my.p[4][lane];
            cn = st.n[bin] + rn;
            ch = st.h[bin] + (uint32_t)__popc(grp);
            st.q1[bin] = cq1;
            st.q2[bin] = cq2;
            st.n[bin] = cn;
            st.h[bin] = ch;
            verdict = sem_quick(cn, ch, cq1, cq2, kExact ? 0u : kTqDelta);
        }
        if (__any_sync(0xffffffffu, verdict < 0) && verdict < 0)
            verdict = sem_test(cn, ch, cq1, cq2, kExact ? 0u : kTqDelta);
        const bool fail = __any_sync(0xffffffffu, verdict == SEM_FAIL);
        const bool unsure = __any_sync(0xffffffffu, verdict == SEM_UNSURE);
        count += rn;
        hits += (uint32_t)__popc(hm);
        ndf += (uint32_t)__popc(dfb);
        if (hm && !fail) {
            flag = (!kExact && unsure) ? 2u : 1u;
            break;
        }
        if (g0 + kRoundRays >= R) {
            flag = 1u;  // out of rays
            break;
        }
    }
    __syncwarp();
    if (flag == 2u) return true;  // the caller redoes the row on the exact path at once
    unsigned long long *hrow = a.hist + J.hist_off + (uint64_t)k * B;
    for (uint32_t b = lane; b < B; b += 32u) {
        const unsigned long long s1 = st.s1[b];
        if (s1) hrow[b] = rescale_cell(s1, R, count);
    }
    if (lane == 0) {
        const uint32_t sp = (uint32_t)(row % (uint64_t)kSpread);
        atomicAdd(&a.acc[d].fast[sp], (unsigned long long)count);
        if (hits) atomicAdd(&a.acc[d].hits[sp], (unsigned long long)hits);
        if (ndf) atomicAdd(&a.acc[d].retraced[sp], (unsigned long long)ndf);
    }
    __syncwarp();  // the slot and bin states are reused by the next row
    return false;
}

// One wavelength row under adaptive sampling by one warp, for a design with certified pieces
// (cpd_piece.h): the rounds and decisions of adaptive_row1 with the row's core range cut into up
// to 31 pieces of 2^k sorted rays once, so that a ray's bin is a quadratic of its piece (~25
// instructions against ~100 of fast_ray) and every such hit has the same transmittance. A bin's
// Welford state is then its samples n and hits h alone, the test is sem_quick_equal, and the
// shared-memory sums of q and q^2 drop out. The rays that the float-float trace decides hit with
// a transmittance of its own: for p(d|lambda) the difference is summed apart (ox), and while it is
// within kTqDelta quanta the test's error bound covers it.
// kExact: every hit with the float-float transmittance (coated_tfix), the test without an error
// bound. Returns ROW_DONE; ROW_UNSURE when the bound leaves a decision open (the caller redoes the
// row with kExact); or ROW_OTHER when a hit's transmittance is another (an exit face met at
// cos <= 0.5): the general exact path takes the row.
struct Adapt1Pieces {
    LamParams P;
    FastConst C;
    // the pieces, then the eighths of up to three pieces without a bound
    float4 rec_a[32 + 24];  // z of the left end (hi, lo), v0, v1; of a cut piece its first eighth's place
    float2 rec_b[32 + 24];  // v2, e (kCutPiece: cut)
};
constexpr float kCutPiece = 2e30f;  // an error beyond that of piece_uniform's pieces without a bound
// per bin: ox, samples and hits
constexpr size_t adapt1p_smem_bytes(uint32_t B) { return sizeof(Adapt1Pieces) + 16u * (size_t)B; }

// A row for adaptive_exact_kernel.
__device__ __forceinline__ void queue_row(const LaunchArgs &a, uint64_t row)
{
    const uint32_t d = find_job<F_ROW>(a.jobs, a.njobs, row);
    const unsigned long long pos = atomicAdd(&a.ctl->queue_count, 1ull);
    if (pos < a.qcap) a.queue[pos] = QEntry{d, (uint32_t)(row - a.jobs[d].row_off), 0u, 0u};
    else atomicOr(&a.ctl->overflow, kOverflowQueue);
}

// The records of a row's pieces, by one warp.
__device__ __forceinline__ void adapt_pieces(const Guards &g, Adapt1Pieces &w, const PieceConst &K,
                                             const float2 *__restrict__ zt, uint32_t lo, uint32_t hi, uint32_t ks,
                                             uint32_t lane)
{
    const LamParams &P = w.P;
    const FastConst &C = w.C;
    // the pieces, and then again the pieces without a bound in eighths (nine ends each): of
    // 81 rays in such pieces per row of 7591, nine in ten are decided
    uint32_t j0 = lo + (lane << ks), cut = 0u;
    for (int level = 0; level < 2; level++) {
        if (level) {
            const uint32_t pc = lane / 9u, t = lane - 9u * pc;
            uint32_t m = cut;
            for (uint32_t i = 0; i < pc; i++) m &= m - 1u;
            const uint32_t p = pc < 3u && m ? (uint32_t)__ffs(m) - 1u : 0u;
            j0 = min(lo + (p << ks) + (t << (ks - 3u)), min(lo + ((p + 1u) << ks), hi - 1u));
        }
        const float2 z = __ldg(zt + min(j0, hi - 1u));
        const PieceEnd e = piece_end(C, fast_limits(C, g), K, P, g, z.x, z.y);
        PieceEnd o = e;
        o.dz = __shfl_down_sync(0xffffffffu, e.dz, 1);
        o.v = __shfl_down_sync(0xffffffffu, e.v, 1);
        o.gv = __shfl_down_sync(0xffffffffu, e.gv, 1);
        o.ci = __shfl_down_sync(0xffffffffu, e.ci, 1);
        o.cr = __shfl_down_sync(0xffffffffu, e.cr, 1);
        o.cid = __shfl_down_sync(0xffffffffu, e.cid, 1);
        o.gn = __shfl_down_sync(0xffffffffu, e.gn, 1);
        o.px = __shfl_down_sync(0xffffffffu, e.px, 1);
        o.py = __shfl_down_sync(0xffffffffu, e.py, 1);
        o.cls = __shfl_down_sync(0xffffffffu, e.cls, 1);
        const Piece f = piece_fit(C, K, P, e, o);
        const Piece q = piece_uniform(K, f);
        if (level == 0) {
            w.rec_a[lane] = make_float4(z.x, z.y, q.v0, q.v1);
            w.rec_b[lane] = make_float2(q.v2, q.e);
            cut = ks >= 3u ? __ballot_sync(0xffffffffu, lane < 31u && j0 < hi && f.cls == PIECE_RAYS) : 0u;
            if (!cut) break;
            // their records point to their eighths
            const uint32_t place = __popc(cut & ((1u << lane) - 1u));
            __syncwarp();
            if ((cut >> lane & 1u) && place < 3u) {
                w.rec_a[lane].x = __uint_as_float(32u + 8u * place);
                w.rec_b[lane].y = kCutPiece;
            }
        } else {
            const uint32_t pc = lane / 9u, t = lane - 9u * pc;
            if (pc < 3u && t < 8u) {
                w.rec_a[32u + 8u * pc + t] = make_float4(z.x, z.y, q.v0, q.v1);
                w.rec_b[32u + 8u * pc + t] = make_float2(q.v2, q.e);
            }
        }
    }
}

// A core ray (sorted position s) on its piece: piece_ray's outcome and the bin.
__device__ __forceinline__ int adapt_ray(const Adapt1Pieces &w, const PieceConst &K, uint32_t B, uint32_t s, uint32_t lo,
                                         uint32_t ks, float2 z, uint32_t &bin)
{
    const uint32_t i = (s - lo) >> ks;
    float4 ra = w.rec_a[i];
    float2 rb = w.rec_b[i];
    if (rb.y >= kCutPiece) {
        const uint32_t c = __float_as_uint(ra.x) + ((s - lo) >> (ks - 3u) & 7u);
        ra = w.rec_a[c];
        rb = w.rec_b[c];
    }
    return piece_ray(K, B, 0.f, ra.z, ra.w, rb.x, rb.y, (ra.x - z.x) + (ra.y - z.y), bin);
}

// A ray that the pieces leave: fast_ray in the core, and the float-float trace. False when it hits
// with another transmittance than the row's (tfast by fast_ray, tfix in float-float, which is what
// a float-float hit gives); add: what its hit adds to the bin beside tfast (kExact: nothing).
template <bool kExact>
__device__ __forceinline__ bool adapt_left(const LaunchArgs &a, const DevDesign &D, const Adapt1Pieces &w, const LamDF &E,
                                           bool core, float2 z, uint32_t tfast, uint32_t tfix, uint32_t &bin,
                                           bool &used_df, long long &add)
{
    int r = RAY_FLAG;
    if (core) {
        uint32_t b = 0u;
        float t = 0.f;
        r = fast_ray(w.C, w.P, a.guards, z.x, z.y, b, t);
        if (r == RAY_HIT) {
            bin = b;
            return t_fixed(t) == tfast;
        }
    }
    if (r != RAY_FLAG) return true;
    const uint2 x = trace_df_exact_call(D, E, z.x, z.y);
    bin = x.x;
    used_df = true;
    if (bin == 0xffffffffu) return true;
    if (!kExact) add = (long long)x.y - (long long)tfast;
    return x.y == tfix;
}

template <bool kExact>
__device__ __forceinline__ int adaptive_row1_pieces(const LaunchArgs &a, uint64_t row, uint32_t d,
                                                         const DesignJob &J, unsigned long long *smem, uint32_t lane)
{
    const uint32_t k = (uint32_t)(row - J.row_off);
    const uint32_t B = J.B, R = J.R;
    const DevDesign &D = a.designs[d];
    Adapt1Pieces &w = *reinterpret_cast<Adapt1Pieces *>(smem);
    LamParams &P = w.P;
    FastConst &C = w.C;
    unsigned long long *ox = reinterpret_cast<unsigned long long *>(&w + 1);
    uint2 *st = reinterpret_cast<uint2 *>(ox + B);  // samples, hits
    const LamDF &E = a.lx[row];
    static_assert(sizeof(Adapt1Pieces) % 16 == 0, "bin arrays follow");
    if (lane < sizeof(LamParams) / 16)
        reinterpret_cast<uint4 *>(&P)[lane] = reinterpret_cast<const uint4 *>(a.lp + row)[lane];
    else if (lane < (sizeof(LamParams) + sizeof(FastConst)) / 16)
        reinterpret_cast<uint4 *>(&C)[lane - sizeof(LamParams) / 16] =
            reinterpret_cast<const uint4 *>(&D.fc)[lane - sizeof(LamParams) / 16];
    for (uint32_t b = lane; b < B; b += 32u) {
        st[b] = make_uint2(0u, 0u);
        ox[b] = 0ull;
    }
    __syncwarp();
    const uint32_t *rank = a.rank + J.rank_off;
    const float2 *__restrict__ zt = reinterpret_cast<const float2 *>(a.z32) + J.ray_off;
    const PieceConst K = piece_const(C);
    const uint32_t lo = P.core_lo, hi = P.all_exact ? P.core_lo : P.core_hi, band_lo = P.band_lo, band_hi = P.band_hi;
    const uint32_t ks = piece_shift(hi - lo);
    if (hi > lo) adapt_pieces(a.guards, w, K, zt, lo, hi, ks, lane);
    __syncwarp();
    const uint32_t lt_mask = (1u << lane) - 1u;
    const uint32_t tfast = piece_tfix(P), tfix = coated_tfix(E), tfx = kExact ? tfix : tfast, tq = tfx >> kTqShift;
    constexpr uint32_t delta = kExact ? 0u : kTqDelta;
    if (!kExact && (tfix >> kTqShift) - tq + kTqDelta > 2u * kTqDelta) return ROW_OTHER;
    const SemEqual se = sem_equal(tq, delta);
    uint32_t count = R, ndf = 0;  // the same in every lane
    // no ray clears the flat faces: every round runs without a hit
    const uint32_t g_start = band_lo >= band_hi ? R : 0u;
    // the ray this lane traces in the next round and its start height, loaded while the current
    // one is decided; its place in the table a round before that (the second load's address)
    uint32_t s_n1 = 0xffffffffu, s_n2 = 0xffffffffu;
    float2 z_n1 = make_float2(0.f, 0.f);
    const auto place = [&](uint32_t g) { return g + lane < R ? __ldg(rank + g + lane) : 0xffffffffu; };
    const auto height = [&](uint32_t s) { return s >= band_lo && s < band_hi ? __ldg(zt + s) : make_float2(0.f, 0.f); };
    if (g_start < R) {
        s_n1 = place(g_start);
        s_n2 = place(g_start + kRoundRays);
        z_n1 = height(s_n1);
    }
    for (uint32_t g0 = g_start; g0 < R; g0 += kRoundRays) {
        uint32_t bin = 0xffffffffu;
        const uint32_t s = s_n1;
        const float2 z = z_n1;
        s_n1 = s_n2;
        z_n1 = height(s_n1);
        s_n2 = place(g0 + 2u * kRoundRays);
        int res = RAY_LOST;
        const bool core = s >= lo && s < hi;
        if (core) {
            uint32_t b = 0u;
            res = adapt_ray(w, K, B, s, lo, ks, z, b);
            if (res == RAY_HIT) bin = b;
        } else if (s >= band_lo && s < band_hi) {
            res = RAY_FLAG;
        }
        bool used_df = false;
        const uint32_t left = __ballot_sync(0xffffffffu, res == RAY_FLAG);
        if (left) {
            // the rays that the pieces leave
            bool same = true;
            long long add = 0;
            if (res == RAY_FLAG) same = adapt_left<kExact>(a, D, w, E, core, z, tfast, tfix, bin, used_df, add);
            if (!__all_sync(0xffffffffu, same)) return ROW_OTHER;
            if (add) atomicAdd(ox + bin, (unsigned long long)add);
        }
        const bool hit = bin != 0xffffffffu;
        const uint32_t hm = __ballot_sync(0xffffffffu, hit);
        const uint32_t rn = min(kRoundRays, R - g0);  // samples of this round
        const uint32_t grp = __match_any_sync(0xffffffffu, bin);
        const bool leader = hit && (grp & lt_mask) == 0u;
        int verdict = SEM_PASS;
        uint32_t cn = 0u, ch = 0u;
        if (leader) {
            const uint2 v = st[bin];
            cn = v.x + rn;
            ch = v.y + (uint32_t)__popc(grp);
            st[bin] = make_uint2(cn, ch);
            verdict = sem_quick_equal(cn, ch, se);
        }
        if (kExact) ndf += (uint32_t)__popc(__ballot_sync(0xffffffffu, s >= band_lo && s < band_hi));
        else if (left) ndf += (uint32_t)__popc(__ballot_sync(0xffffffffu, used_df));
        // the row goes on when a bin fails (most rounds), or no ray hit
        if (!hm || __any_sync(0xffffffffu, verdict == SEM_FAIL)) continue;
        if (verdict < 0) verdict = sem_test(cn, ch, (uint64_t)ch * tq, (uint64_t)ch * tq * tq, delta);
        if (!__any_sync(0xffffffffu, verdict == SEM_FAIL)) {
            if (__any_sync(0xffffffffu, verdict == SEM_UNSURE)) return ROW_UNSURE;
            count = g0 + rn;
            break;
        }
    }
    __syncwarp();
    uint32_t hits = 0u;
    unsigned long long *hrow = a.hist + J.hist_off + (uint64_t)k * B;
    for (uint32_t b = lane; b < B; b += 32u) {
        const uint32_t h = st[b].y;
        hits += h;
        if (h) hrow[b] = rescale_cell((unsigned long long)h * tfx + ox[b], R, count);
    }
    hits = __reduce_add_sync(0xffffffffu, hits);
    if (lane == 0) {
        const uint32_t sp = (uint32_t)(row % (uint64_t)kSpread);
        atomicAdd(&a.acc[d].fast[sp], (unsigned long long)count);
        if (hits) atomicAdd(&a.acc[d].hits[sp], (unsigned long long)hits);
        if (ndf) atomicAdd(&a.acc[d].retraced[sp], (unsigned long long)ndf);
    }
    return ROW_DONE;
}

#ifndef CPD_ADAPT_KW_MANY
#define CPD_ADAPT_KW_MANY 1  // warps per row when at least 8 rows per SM (1: adaptive1_kernel)
#endif
#ifndef CPD_ADAPT_KW_SOME
#define CPD_ADAPT_KW_SOME 4  // warps per row at 2 to 7 rows per SM
#endif
// ------------------------------------------------------------------ adaptive sampling, few rows

constexpr uint32_t kAdaptOdd = 128;  // such hits listed per group of rounds (more: traced again once the stop is known)
struct AdaptBlock {
    Adapt1Pieces w;
    uint2 part[32 * kMaxAdaptWarps];   // samples and hits of one bin over one stretch of rounds
    uint8_t hit[kAdaptRounds], test[kAdaptRounds], df[kAdaptRounds];  // test: 1 a bin failed
    uint32_t other, ndf, nodd, pad;    // other: the row's first round with a hit for adaptive_exact_kernel
    uint32_t unsure[kAdaptRounds / 32];
    uint4 odd[kAdaptOdd];  // hits of the float-float trace: round, bin, what they add beside tfast
};
// then per bin: ox, samples and hits so far, and the counts (adapt_arrays_bytes)
constexpr size_t adapt_block_smem_bytes(uint32_t max_B, uint32_t max_rounds = kAdaptRounds)
{
    return sizeof(AdaptBlock) + adapt_arrays_bytes(max_B, max_rounds);
}

// What the float-float hits of rounds [r0, r0 + taken) add beside tfast, where there are more of them
// than the list holds: their rays traced again (out of line: a row with its rays on a bin's edge).
__device__ __noinline__ void adapt_odd_again(const LaunchArgs &a, const AdaptBlock &S, uint64_t row, const DevDesign &D,
                                             const DesignJob &J, unsigned long long *ox, uint32_t r0, uint32_t taken,
                                             uint32_t tfast, uint32_t tfix)
{
    const Adapt1Pieces &w = S.w;
    const uint32_t *rank = a.rank + J.rank_off;
    const float2 *__restrict__ zt = reinterpret_cast<const float2 *>(a.z32) + J.ray_off;
    const PieceConst K = piece_const(w.C);
    const uint32_t lo = w.P.core_lo, hi = w.P.all_exact ? w.P.core_lo : w.P.core_hi, ks = piece_shift(hi - lo);
    const uint32_t j1 = min((r0 + taken) * kRoundRays, J.R);
    for (uint32_t j = r0 * kRoundRays + threadIdx.x; j < j1; j += blockDim.x) {
        const uint32_t s = __ldg(rank + j);
        if (s < w.P.band_lo || s >= w.P.band_hi) continue;
        const float2 z = __ldg(zt + s);
        const bool core = s >= lo && s < hi;
        uint32_t bin = 0xffffffffu;
        if (core && adapt_ray(w, K, J.B, s, lo, ks, z, bin) != RAY_FLAG) continue;
        bin = 0xffffffffu;
        bool used_df = false;
        long long add = 0;
        adapt_left<false>(a, D, w, a.lx[row], core, z, tfast, tfix, bin, used_df, add);
        if (add) atomicAdd(ox + bin, (unsigned long long)add);
    }
}

// One wavelength row under adaptive sampling by one block, for a design with certified pieces
// (the form for passes with few rows: the plain call). With the pieces a round costs ~70
// instructions, so the block bins up to kAdaptRounds rounds first (a round per warp at a time)
// and decides them afterwards: counts[round][bin] holds each round's hits; a thread takes one bin
// over a stretch of rounds, adds up the stretches before its own, and tests the bin after every
// round that hit it; the row stops after the first round with a hit and no failed test. Three
// barriers for 256 rounds instead of three for 16, and no round waits for the one before.
// The rays of the float-float trace past the stop would leave their differences in ox, so those
// are listed with their round and added at the end. Returns as adaptive_row1_pieces: what lies past
// the stop decides nothing.
template <bool kExact>
__device__ __forceinline__ int adaptive_row_pieces(const LaunchArgs &a, uint64_t row, unsigned long long *smem)
{
    const uint32_t d = find_job<F_ROW>(a.jobs, a.njobs, row);
    const DesignJob &J = a.jobs[d];
    const uint32_t k = (uint32_t)(row - J.row_off), B = J.B, R = J.R;
    const DevDesign &D = a.designs[d];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, nthr = blockDim.x, nwarps = nthr >> 5;
    AdaptBlock &S = *reinterpret_cast<AdaptBlock *>(smem);
    Adapt1Pieces &w = S.w;
    unsigned long long *ox = reinterpret_cast<unsigned long long *>(&S + 1);
    uint2 *base = reinterpret_cast<uint2 *>(ox + B);
    uint8_t *counts = reinterpret_cast<uint8_t *>(base + B);
    const uint32_t stride = adapt_stride(B), C = adapt_rounds(B, adapt_arrays_bytes(a.max_B, a.max_rounds));
    const LamDF &E = a.lx[row];
    if (tid < sizeof(LamParams) / 4)
        reinterpret_cast<uint32_t *>(&w.P)[tid] = reinterpret_cast<const uint32_t *>(a.lp + row)[tid];
    if (tid < sizeof(FastConst) / 4)
        reinterpret_cast<uint32_t *>(&w.C)[tid] = reinterpret_cast<const uint32_t *>(&D.fc)[tid];
    for (uint32_t b = tid; b < B; b += nthr) {
        base[b] = make_uint2(0u, 0u);
        ox[b] = 0ull;
    }
    if (tid == 0) {
        S.other = 0xffffffffu;
        S.ndf = S.nodd = 0u;
    }
    __syncthreads();
    const uint32_t *rank = a.rank + J.rank_off;
    const float2 *__restrict__ zt = reinterpret_cast<const float2 *>(a.z32) + J.ray_off;
    const PieceConst K = piece_const(w.C);
    const uint32_t lo = w.P.core_lo, hi = w.P.all_exact ? w.P.core_lo : w.P.core_hi;
    const uint32_t band_lo = w.P.band_lo, band_hi = w.P.band_hi, ks = piece_shift(hi - lo);
    if (warp == 0u && hi > lo) adapt_pieces(a.guards, w, K, zt, lo, hi, ks, lane);
    __syncthreads();
    const uint32_t lt_mask = (1u << lane) - 1u;
    const uint32_t tfast = piece_tfix(w.P), tfix = coated_tfix(E), tfx = kExact ? tfix : tfast, tq = tfx >> kTqShift;
    constexpr uint32_t delta = kExact ? 0u : kTqDelta;
    if (!kExact && (tfix >> kTqShift) - tq + kTqDelta > 2u * kTqDelta) return ROW_OTHER;
    const SemEqual se = sem_equal(tq, delta);
    const uint32_t rounds = band_lo >= band_hi ? 0u : (R + kRoundRays - 1u) / kRoundRays;
    uint32_t stop = rounds;  // rounds taken
    const auto place = [&](uint32_t r) {
        const uint32_t j = r * kRoundRays + lane;
        return r < rounds && j < R ? __ldg(rank + j) : 0xffffffffu;
    };
    const auto height = [&](uint32_t s) { return s >= band_lo && s < band_hi ? __ldg(zt + s) : make_float2(0.f, 0.f); };
    for (uint32_t r0 = 0; r0 < rounds; r0 += C) {
        const uint32_t nr = min(C, rounds - r0);
        if (tid < kAdaptRounds / 32) S.unsure[tid] = 0u;
        // 1. every round's hits per bin
        uint32_t s_n1 = place(r0 + warp), s_n2 = place(r0 + warp + nwarps);
        float2 z_n1 = height(s_n1);
        for (uint32_t q = warp; q < nr; q += nwarps) {
            uint32_t bin = 0xffffffffu;
            const uint32_t s = s_n1;
            const float2 z = z_n1;
            s_n1 = s_n2;
            z_n1 = height(s_n1);
            s_n2 = place(r0 + q + 2u * nwarps);
            uint32_t *cw = reinterpret_cast<uint32_t *>(counts + q * stride);
            for (uint32_t i = lane; i < stride / 4u; i += 32u) cw[i] = 0u;
            __syncwarp();
            int res = RAY_LOST;
            const bool core = s >= lo && s < hi;
            if (core) {
                uint32_t b = 0u;
                res = adapt_ray(w, K, B, s, lo, ks, z, b);
                if (res == RAY_HIT) bin = b;
            } else if (s >= band_lo && s < band_hi) {
                res = RAY_FLAG;
            }
            bool used_df = false;
            long long add = 0;
            if (res == RAY_FLAG && !adapt_left<kExact>(a, D, w, E, core, z, tfast, tfix, bin, used_df, add))
                atomicMin(&S.other, r0 + q);
            if (add) {
                const uint32_t i = atomicAdd(&S.nodd, 1u);
                if (i < kAdaptOdd) S.odd[i] = make_uint4(r0 + q, bin, (uint32_t)add, (uint32_t)(add >> 32));
            }
            if (kExact) used_df = s >= band_lo && s < band_hi;
            const uint32_t grp = __match_any_sync(0xffffffffu, bin);
            const uint32_t ndf = __popc(__ballot_sync(0xffffffffu, used_df));
            const bool any = __any_sync(0xffffffffu, bin != 0xffffffffu);
            if (bin != 0xffffffffu && (grp & lt_mask) == 0u) counts[q * stride + bin] = (uint8_t)__popc(grp);
            if (lane == 0u) {
                S.hit[q] = any ? 1u : 0u;
                S.test[q] = 0u;
                S.df[q] = (uint8_t)ndf;
            }
        }
        __syncthreads();
        // 2. the tests, up to nthr bins at a time
        for (uint32_t b0 = 0; b0 < B; b0 += nthr) {
            uint32_t width = 1u;
            while (width < min(B - b0, nthr)) width <<= 1;
            const uint32_t np = nthr / width, p = tid / width, b = b0 + (tid & (width - 1u));
            const uint32_t len = (nr + np - 1u) / np, qa = min(p * len, nr), qb = min(qa + len, nr);
            const bool act = b < B;
            uint32_t n = 0u, h = 0u;
            if (np > 1u) {
                // this stretch's share, for the stretches after it (one stretch, every thread a bin of its
                // own: nothing to pass on; calls of 472 rows x 4096 rays in 200 bins 109 -> 104 us)
                for (uint32_t q = qa; q < qb && act; q++) {
                    const uint32_t c = counts[q * stride + b];
                    if (c) n += min(kRoundRays, R - (r0 + q) * kRoundRays);
                    h += c;
                }
                S.part[tid] = make_uint2(n, h);
                __syncthreads();
            }
            if (act) {
                const uint2 v = base[b];
                n = v.x;
                h = v.y;
                for (uint32_t i = 0; i < p; i++) {
                    const uint2 o = S.part[i * width + (b - b0)];
                    n += o.x;
                    h += o.y;
                }
                for (uint32_t q = qa; q < qb; q++) {
                    const uint32_t c = counts[q * stride + b];
                    if (!c) continue;
                    n += min(kRoundRays, R - (r0 + q) * kRoundRays);
                    h += c;
                    // with a thread per bin, a bin that failed has often settled the round already
                    // (the same calls: 107 -> 104 us; with stretches, no gain)
                    if (np == 1u && *(volatile uint8_t *)&S.test[q]) continue;
                    int verdict = sem_quick_equal(n, h, se);
                    if (verdict < 0) verdict = sem_test(n, h, (uint64_t)h * tq, (uint64_t)h * tq * tq, delta);
                    if (verdict == SEM_FAIL) S.test[q] = 1u;  // a failed bin settles the round
                    else if (verdict == SEM_UNSURE) atomicOr(&S.unsure[q >> 5], 1u << (q & 31u));
                }
            }
            __syncthreads();
        }
        // 3. the first round that stops the row
        uint32_t last = nr;
        for (uint32_t q0 = 0; q0 < nr; q0 += 32u) {
            const uint32_t q = q0 + lane;
            const uint32_t m = __ballot_sync(0xffffffffu, q < nr && S.hit[q] && !S.test[q]);
            if (m) {
                last = q0 + (uint32_t)__ffs(m) - 1u;
                break;
            }
        }
        const uint32_t taken = last < nr ? last + 1u : nr;
        if (S.other < r0 + taken) return ROW_OTHER;
        if (last < nr && (S.unsure[last >> 5] >> (last & 31u) & 1u)) return ROW_UNSURE;
        // the states through it, and the float-float rays
        for (uint32_t b0 = 0; b0 < B; b0 += nthr) {
            uint32_t width = 1u;
            while (width < min(B - b0, nthr)) width <<= 1;
            const uint32_t np = nthr / width, p = tid / width, b = b0 + (tid & (width - 1u));
            if (b >= B) continue;
            uint32_t n = 0u, h = 0u;
            for (uint32_t q = p; q < taken; q += np) {
                const uint32_t c = counts[q * stride + b];
                if (c) n += min(kRoundRays, R - (r0 + q) * kRoundRays);
                h += c;
            }
            if (n) atomicAdd(&base[b].x, n);
            if (h) atomicAdd(&base[b].y, h);
        }
        const uint32_t nodd = S.nodd;
        if (!kExact && nodd > kAdaptOdd) adapt_odd_again(a, S, row, D, J, ox, r0, taken, tfast, tfix);
        for (uint32_t i = tid; i < nodd && nodd <= kAdaptOdd; i += nthr) {
            const uint4 o = S.odd[i];
            if (o.x < r0 + taken) atomicAdd(ox + o.y, (unsigned long long)o.w << 32 | o.z);
        }
        if (warp == 0u) {
            uint32_t v = 0u;
            for (uint32_t q = lane; q < taken; q += 32u) v += S.df[q];
            v = __reduce_add_sync(0xffffffffu, v);
            if (lane == 0u) S.ndf += v;
        }
        __syncthreads();
        if (last < nr) {
            stop = r0 + last + 1u;
            break;
        }
        if (tid == 0) S.nodd = 0u;
        __syncthreads();
    }
    const uint32_t count = rounds ? min(R, stop * kRoundRays) : R;
    uint32_t hits = 0u;
    unsigned long long *hrow = a.hist + J.hist_off + (uint64_t)k * B;
    for (uint32_t b = tid; b < B; b += nthr) {
        const uint32_t h = base[b].y;
        hits += h;
        if (h) hrow[b] = rescale_cell((unsigned long long)h * tfx + ox[b], R, count);
    }
    hits = __reduce_add_sync(0xffffffffu, hits);
    const uint32_t sp = (uint32_t)(row % (uint64_t)kSpread);
    if (lane == 0u && hits) atomicAdd(&a.acc[d].hits[sp], (unsigned long long)hits);
    if (tid == 0u) {
        atomicAdd(&a.acc[d].fast[sp], (unsigned long long)count);
        if (S.ndf) atomicAdd(&a.acc[d].retraced[sp], (unsigned long long)S.ndf);
    }
    return ROW_DONE;
}

__device__ __noinline__ int adaptive_row_redo(const LaunchArgs &a, unsigned long long *smem)
{
    __syncthreads();
    return adaptive_row_pieces<true>(a, blockIdx.x, smem);
}

// Passes with fewer rows than adaptive1_kernel's: one row per block (rows of designs without
// pieces are adaptive_kernel's). The chain of a row bounds it: up to 256 rounds are binned at once
// by all warps and then decided, instead of 16 rounds per three barriers: a call of 128 rows x up
// to 8192 rays in 32 bins 101 -> 80 us, some of its rows redone. The tests of step 2 run for 32
// bins at a time whether one or all were hit, so wide detectors and short tables are not for it
// (adapt_by_blocks).
__global__ void __launch_bounds__(32 * kMaxAdaptWarps, 2) adaptive_block_kernel(const LaunchArgs a)
{
    extern __shared__ __align__(16) unsigned long long adapt_smem[];
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();  // the setup's LamParams and LamDF
    if (a.adapt_pieces != 1u && !a.designs[find_job<F_ROW>(a.jobs, a.njobs, blockIdx.x)].fc.pieces) return;
    int r = adaptive_row_pieces<false>(a, blockIdx.x, adapt_smem);
    if (r == ROW_UNSURE) r = adaptive_row_redo(a, adapt_smem);
    if (r == ROW_OTHER && threadIdx.x == 0) queue_row(a, blockIdx.x);
}

#ifndef CPD_ADAPT_MIN_BLOCKS
#define CPD_ADAPT_MIN_BLOCKS 2  // 64 registers at kMaxAdaptWarps warps per block
#endif
// One row per block of KW = blockDim.x / 32 warps: rows differ widely in length (a single
// round to all R / 32), and one row per block lets the block scheduler balance them.
__global__ void __launch_bounds__(32 * kMaxAdaptWarps, CPD_ADAPT_MIN_BLOCKS) adaptive_kernel(const LaunchArgs a)
{
    extern __shared__ __align__(16) unsigned long long adapt_smem[];
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();  // the setup's LamParams and LamDF
    const uint32_t kw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    if (a.adapt_pieces && a.designs[find_job<F_ROW>(a.jobs, a.njobs, blockIdx.x)].fc.pieces) return;
    // a row whose stop decision the FP32 transmittances cannot settle is redone here, on
    // the float-float path from its first round, while other blocks go on with theirs
    if (adaptive_row<false>(a, blockIdx.x, adapt_smem, kw, warp, lane))
        adaptive_row<true>(a, blockIdx.x, adapt_smem, kw, warp, lane);
}

__device__ __noinline__ int adaptive_equal_redo(const LaunchArgs &a, unsigned long long *smem)
{
    return adaptive_row<true, ROWS_EQUAL>(a, blockIdx.x, smem, blockDim.x >> 5, threadIdx.x >> 5, threadIdx.x & 31u);
}

// The same for the rows of designs with certified pieces, ray by ray: passes with few rows that
// adaptive_block_kernel is slower for (adapt_by_blocks).
__global__ void __launch_bounds__(32 * kMaxAdaptWarps, CPD_ADAPT_MIN_BLOCKS) adaptive_equal_kernel(const LaunchArgs a)
{
    extern __shared__ __align__(16) unsigned long long adapt_smem[];
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();  // the setup's LamParams and LamDF
    const uint32_t kw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    if (a.adapt_pieces != 1u && !a.designs[find_job<F_ROW>(a.jobs, a.njobs, blockIdx.x)].fc.pieces) return;
    int r = adaptive_row<false, ROWS_EQUAL>(a, blockIdx.x, adapt_smem, kw, warp, lane);
    if (r == ROW_UNSURE) r = adaptive_equal_redo(a, adapt_smem);
    if (r == ROW_OTHER && threadIdx.x == 0) queue_row(a, blockIdx.x);
}

// Out of line: rows of designs without pieces, and the rare ones that the pieces leave (exact:
// every form of a pass takes those to the exact path, so that a design's result does not depend on
// what shares its pass).
__device__ __noinline__ void adaptive_row1_rest(const LaunchArgs &a, unsigned long long *smem, bool exact)
{
    if (exact || adaptive_row1<false>(a, blockIdx.x, smem, threadIdx.x))
        adaptive_row1<true>(a, blockIdx.x, smem, threadIdx.x);
}

__device__ __noinline__ int adaptive_row1_redo(const LaunchArgs &a, uint32_t d, unsigned long long *smem)
{
    return adaptive_row1_pieces<true>(a, blockIdx.x, d, a.jobs[d], smem, threadIdx.x);
}

#ifndef CPD_ADAPT1_MIN_BLOCKS
#define CPD_ADAPT1_MIN_BLOCKS 32
#endif
// The many-rows form: one row per one-warp block (adaptive_row1).
__global__ void __launch_bounds__(32, CPD_ADAPT1_MIN_BLOCKS) adaptive1_kernel(const LaunchArgs a)
{
    extern __shared__ __align__(16) unsigned long long adapt_smem[];
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();  // the setup's LamParams and LamDF
    if (adaptive_row1<false>(a, blockIdx.x, adapt_smem, threadIdx.x))
        adaptive_row1<true>(a, blockIdx.x, adapt_smem, threadIdx.x);
}

// The same for passes of designs with certified pieces, or some of them (a kernel of its own:
// with the general form out of line, rows without pieces take 9% longer here). Issue and the rows'
// states in shared memory bound it: at 2.6 KB a row 32 rows per SM leave the L1 enough (7.7 KB:
// 2.1 ms). 256 designs x 128 rows x up to 8192 rays: 2.7 ms ray by ray, 1.15 here.
__global__ void __launch_bounds__(32, CPD_ADAPT1_MIN_BLOCKS) adaptive1_pieces_kernel(const LaunchArgs a)
{
    extern __shared__ __align__(16) unsigned long long adapt_smem[];
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();  // the setup's LamParams and LamDF
    const uint32_t d = find_job<F_ROW>(a.jobs, a.njobs, blockIdx.x);
    const bool pieces = a.designs[d].fc.pieces;
    if (pieces) {
        int r = adaptive_row1_pieces<false>(a, blockIdx.x, d, a.jobs[d], adapt_smem, threadIdx.x);
        __syncwarp();
        if (r == ROW_UNSURE) r = adaptive_row1_redo(a, d, adapt_smem);
        if (r == ROW_DONE) return;
    }
    __syncwarp();
    if (a.adapt_pieces == 1u) {
        // a pass of such designs alone has no room for the general form's states
        if (threadIdx.x == 0) queue_row(a, blockIdx.x);
        return;
    }
    adaptive_row1_rest(a, adapt_smem, pieces);
}

// The queued rows: the float-float path from the first round on, one row per block of
// blockDim.x / 32 warps (as many as the rounds kernel used: a queued row of a plain call
// is on the pass's critical path).
__global__ void __launch_bounds__(32 * kMaxAdaptWarps, 1) adaptive_exact_kernel(const LaunchArgs a)
{
    extern __shared__ __align__(16) unsigned long long adapt_smem[];
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();  // the adaptive kernel's queue
    publish_status(a);
    const unsigned long long qn = a.ctl->queue_count;
    const uint64_t n = qn < a.qcap ? qn : a.qcap;
    for (uint64_t i = blockIdx.x; i < n; i += gridDim.x) {
        const QEntry e = a.queue[i];
        const uint64_t row = a.jobs[e.design].row_off + e.k;
        if (blockDim.x == 32u) adaptive_row1<true>(a, row, adapt_smem, threadIdx.x);
        else adaptive_row<true>(a, row, adapt_smem, blockDim.x >> 5, threadIdx.x >> 5, threadIdx.x & 31u);
    }
}

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

constexpr int kEntropyThreads = 256;

// A non-negative float-float value in fixed point with `scale` units, its hi and lo
// words rounded separately: one rounding per cell, so that the sums over cells are integer
// sums whose value does not depend on how the cells are grouped.
// The conversions are 32-bit or exact bit arithmetic: 64-bit float-to-integer conversions
// issue to the FP64 unit, ~64 cycles per warp instruction on this GPU.
__device__ __forceinline__ unsigned long long df_to_fixed(ff::F2 v, float scale)
{
    const float x = v.hi * scale;  // >= 0, below 2^47
    unsigned long long q;
    if (x < 2147483648.0f) {
        q = __float2uint_rn(x);
    } else {
        // at or above 2^31 a float is an integer: its significand shifted by its exponent
        const uint32_t bits = __float_as_uint(x);
        q = (unsigned long long)((bits & 0x7fffffu) | 0x800000u) << (((bits >> 23) & 0xffu) - 150u);
    }
    // |lo| is below half an ulp of hi: |lo scale| < 2^23
    const long long r = (long long)q + __float2int_rn(v.lo * scale);
    return r > 0 ? (unsigned long long)r : 0ull;
}

// Per-design finalize: H(D) from the per-bin sums, MI, and the SEM stop of cuda_fitness
// (src/cuda_fitness.rs:392-422), by nthr threads (one warp, or the 256 threads of an entropy
// block; red: nthr / 32 scratch records in shared memory when nthr > 32). f64 costs ~64
// cycles per warp instruction here (a division or square root ~700 cycles of latency), and
// this runs on the tail of the plain call, so everything is float-float on the FP32 pipe:
// pbar = S1 / (n R 2^31), log2 pbar = log2 S1 - log2(n R) - 31 (logs of integers,
// ff::log2_u64, absolute error < 1e-12), each bin's pbar log2 pbar rounded once to 2^-50
// fixed point (so the sum over bins is the same integer for any number of threads), and
// each bin's Welford M2, S2 - S1^2 / n, against (5e-3)^2 n (n - 1). Only the conversion of
// the three results to double is f64.
struct FinalizeRed {
    long long hdet;
    float m2max;
    int conv;
};
constexpr float kHdetScale = 1125899906842624.0f;  // 2^50

__device__ void finalize_design(const LaunchArgs &a, uint32_t d, const DesignJob &J, uint32_t tid, uint32_t nthr,
                                const float *tab, FinalizeRed *red)
{
    using ff::F2;
    const uint32_t lane = tid & 31u;
    // every load first, so that their L2 round trips overlap one another and the
    // float-float prologue: the design's sums, its ray counters and this thread's first bin
    const unsigned long long rows = __ldcg(&a.acc[d].rows) + J.W;
    const unsigned long long Hsum = __ldcg(&a.acc[d].H);
    const bool cp = lane < (uint32_t)kSpread;
    const unsigned long long hits_l = cp ? __ldcg(&a.acc[d].hits[lane]) : 0ull;
    const unsigned long long retraced_l = cp ? __ldcg(&a.acc[d].retraced[lane]) : 0ull;
    const unsigned long long fast_l = cp ? __ldcg(&a.acc[d].fast[lane]) : 0ull;
    unsigned long long c1n = 0ull, c2n = 0ull;
    if (tid < J.B) {
        c1n = __ldcg(&a.S1[J.acc_off + tid]);
        c2n = __ldcg(&a.S2[J.acc_off + tid]);
    }
    const F2 n = ff::from_u64(rows);
    const F2 inv_n = df::rcp(n);
    const F2 unit{J.unit_hi, J.unit_lo};  // p per count unit, 2^-31 / R
    const F2 inv_nr = ff::mul(unit, inv_n);
    const unsigned long long nR = rows * (unsigned long long)J.R;
    const F2 lnr = ff::add_f(ff::log2_u64(nR, tab), 31.f);
    const F2 thr = df::div(ff::mul(n, ff::from_u64(rows - 1ull)), df::c(40000.f));  // (5e-3)^2 n (n - 1)
    const F2 s2unit{(float)kPScaleInv, 0.f};
    long long hdet = 0;  // sum of pbar log2 pbar (<= 0), 2^-50 units
    float m2max = 0.f;
    int conv = 1;
    for (uint32_t b = tid; b < J.B; b += nthr) {
        const unsigned long long c1 = c1n, c2 = c2n;
        if (b + nthr < J.B) {  // the next bin's sums
            c1n = __ldcg(&a.S1[J.acc_off + b + nthr]);
            c2n = __ldcg(&a.S2[J.acc_off + b + nthr]);
        }
        const F2 sc1 = ff::from_u64(c1);
        if (c1) {
            const F2 pbar = ff::mul(sc1, inv_nr);
            const F2 lg = ff::add(ff::log2_u64(c1, tab), F2{-lnr.hi, -lnr.lo});
            const F2 pl = ff::mul(pbar, lg);
            hdet -= (long long)df_to_fixed(F2{-pl.hi, -pl.lo}, kHdetScale);
        }
        // Welford M2 of the per-wavelength p(d|lambda) (welford.rs:26-57)
        const F2 s1 = ff::mul(sc1, unit);  // sum over rows of p
        const F2 s2 = ff::mul(ff::from_u64(c2), s2unit);
        F2 m2 = df::sub(s2, ff::mul(ff::mul(s1, s1), inv_n));
        if (df::neg_(m2)) m2 = F2{0.f, 0.f};
        conv &= df::lt(m2, thr) ? 1 : 0;
        m2max = fmaxf(m2max, m2.hi);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        hdet += (long long)__shfl_xor_sync(0xffffffffu, (unsigned long long)hdet, o);
        m2max = fmaxf(m2max, __shfl_xor_sync(0xffffffffu, m2max, o));
    }
    conv = __all_sync(0xffffffffu, conv);
    if (nthr > 32u) {
        if (lane == 0) red[tid >> 5] = FinalizeRed{hdet, m2max, conv};
        __syncthreads();
        if (tid >= 32u) return;
        const uint32_t nw = nthr >> 5;
        FinalizeRed r = lane < nw ? red[lane] : FinalizeRed{0, 0.f, 1};
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            r.hdet += (long long)__shfl_xor_sync(0xffffffffu, (unsigned long long)r.hdet, o);
            r.m2max = fmaxf(r.m2max, __shfl_xor_sync(0xffffffffu, r.m2max, o));
        }
        hdet = r.hdet;
        m2max = r.m2max;
        conv = __all_sync(0xffffffffu, r.conv);
    }
    const unsigned long long hits = warp_sum_u64(hits_l);
    const unsigned long long retraced = warp_sum_u64(retraced_l);
    const unsigned long long fast = warp_sum_u64(fast_l);
    if (lane == 0) {
        const F2 H = ff::mul(ff::from_u64(Hsum), F2{(float)kHScaleInv, 0.f});
        const F2 hc = ff::mul(H, inv_n);
        const double h_cond = -((double)hc.hi + (double)hc.lo);
        const double h_det = (double)hdet * (1.0 / 1125899906842624.0);
        DesignOut o;
        o.h_cond = h_cond;
        o.h_det = h_det;
        o.info = h_cond - h_det;
        const float fn = (float)rows;
        o.max_sem = rows > 1ull ? (double)sqrtf(m2max / (fn - 1.f) / fn) : (double)INFINITY;
        const DevDesign &D = a.designs[d];
        o.size = D.size;
        o.deviation = D.deviation;
        o.hits = hits;
        o.retraced = retraced;
        o.rows = rows;
        o.fast = fast;
        o.converged = conv;
        o.status = D.status;
        a.out[d] = o;
        a.acc[d].rows = rows;
        if (a.stamp != STAMP_NONE && tid == 0u) a.status->t1 = global_ns();
    }
}

// One nonzero cell of the histogram: -p log2 p (2^-40 units) and p^2 (2^-46 units) in
// fixed point, p = c 2^-31 / R in float-float on the FP32 pipe.
__device__ __forceinline__ void entropy_cell(unsigned long long cv, ff::F2 unit, ff::F2 lu, const float *tab,
                                             unsigned long long &hq, unsigned long long &pq)
{
    const ff::F2 p = ff::mul(ff::from_u64(cv), unit);
    const ff::F2 lp = ff::add(ff::log2_u64(cv, tab), lu);
    const ff::F2 plp = ff::mul(p, lp);  // p log2 p <= 0
    hq = df_to_fixed(ff::F2{-plp.hi, -plp.lo}, (float)kHScale);
    pq = df_to_fixed(ff::mul(p, p), (float)kPScale);
}

// The finalize of a single-design pass, folded into the entropy kernel: the warp that
// accounts the design's last tile runs it (after the fences that publish every tile's sums).
__device__ __forceinline__ bool last_tile_of_design(const LaunchArgs &a, const DesignJob &J, uint32_t lane)
{
    __threadfence();
    unsigned last = 0;
    if (lane == 0) last = atomicAdd(&a.ctl->tiles_done, 1u) == J.ntiles - 1u ? 1u : 0u;
    last = __shfl_sync(0xffffffffu, last, 0);
    if (last) __threadfence();
    return last != 0u;
}

// Entropy sums of the rows [r0, r1) of one design by one warp (the form for passes with
// many tiles: no block-level synchronization). Lane -> (bin, row phase): for B <= 32 the
// lanes split into 32/B row phases of one bin each; for wider detectors a lane owns bins
// lane, lane+32, ... of every row, NB of them per sweep. Each step reads 8/NB rows x NB
// bins, so eight loads per lane are in flight.
template <int NB, bool WITH_P>
__device__ __forceinline__ void entropy_tile(const LaunchArgs &a, const DesignJob &J, uint32_t r0, uint32_t r1,
                                             uint32_t lane, const float *tab, unsigned long long &hl)
{
    constexpr uint32_t RS = 8u / NB;
    const uint32_t B = J.B;
    const uint32_t groups = B <= 32u ? 32u / B : 1u;
    const uint32_t grp = B <= 32u ? lane / B : 0u;
    const uint32_t bin0 = B <= 32u ? lane % B : lane;
    const bool active = grp < groups;
    const ff::F2 unit{J.unit_hi, J.unit_lo}, lu{J.lu_hi, J.lu_lo};
    unsigned long long *base = a.hist + J.hist_off;
    const double pscale = J.pscale;  // p per count unit, for the optional p(d|lambda) output
    for (uint32_t bg = 0; bg < B; bg += 32u * NB) {
        unsigned long long c1[NB], q2[NB];
#pragma unroll
        for (int i = 0; i < NB; i++) c1[i] = q2[i] = 0ull;
        for (uint32_t row = r0 + grp; row < r1; row += RS * groups) {
            unsigned long long c[RS * NB];
#pragma unroll
            for (uint32_t rr = 0; rr < RS; rr++) {
                const uint32_t rw = row + rr * groups;
#pragma unroll
                for (int i = 0; i < NB; i++) {
                    const uint32_t b = bg + bin0 + 32u * (uint32_t)i;
                    c[rr * NB + i] = (active && rw < r1 && b < B) ? base[(uint64_t)rw * B + b] : 0ull;
                }
            }
            // one copy of the cell code, not RS x NB (instruction fetch)
#pragma unroll 1
            for (uint32_t q = 0; q < RS * NB; q++) {
                const uint32_t rw = row + (q / NB) * groups;
                const uint32_t i = q % NB;
                const uint32_t b = bg + bin0 + 32u * i;
                const unsigned long long cv = c[q];
                if (cv) {
                    base[(uint64_t)rw * B + b] = 0ull;
                    unsigned long long hq, pq;
                    entropy_cell(cv, unit, lu, tab, hq, pq);
                    hl += hq;
#pragma unroll
                    for (int ii = 0; ii < NB; ii++)
                        if (ii == (int)i) {
                            q2[ii] += pq;
                            c1[ii] += cv;
                        }
                }
                if (WITH_P && active && rw < r1 && b < B) a.p_out[(uint64_t)rw * B + b] = (double)cv * pscale;
            }
        }
#pragma unroll
        for (int i = 0; i < NB; i++) {
            const uint32_t b = bg + bin0 + 32u * (uint32_t)i;
            if (c1[i]) {
                atomicAdd(&a.S1[J.acc_off + b], c1[i]);
                atomicAdd(&a.S2[J.acc_off + b], q2[i]);
            }
        }
    }
}

// One warp per tile.
// WITH_P: the pass also writes p(d|lambda) (a.p_out); a kernel of its own, so that the
// f64 conversion of every cell is not issued when nobody reads it.
template <bool WITH_P>
__global__ void __launch_bounds__(kEntropyThreads, 4) entropy_warp_kernel(const LaunchArgs a)
{
    __shared__ float tab[4 * ff::kLogTable];
    cudaTriggerProgrammaticLaunchCompletion();
    for (uint32_t i = threadIdx.x; i < 4u * ff::kLogTable; i += blockDim.x) tab[i] = a.logtab[i];
    __syncthreads();
    cudaGridDependencySynchronize();  // the histogram of the trace and re-trace kernels
    // A pass whose re-trace queue overflowed is re-run by the host: leave every
    // accumulator untouched.
    if (a.ctl->overflow || a.ctl->queue_count > a.qcap) return;
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t tile = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; tile < a.total_tiles; tile += nw) {
        const uint32_t d = find_job<F_TILE>(a.jobs, a.njobs, tile);
        const DesignJob J = a.jobs[d];
        const uint32_t r0 = (uint32_t)(tile - J.tile_off) * J.tile_rows;
        const uint32_t r1 = min(r0 + J.tile_rows, J.W);
        const uint32_t nb = (J.B + 31u) / 32u;  // bins per lane
        unsigned long long hl = 0ull;
        if (nb >= 3u) entropy_tile<4, WITH_P>(a, J, r0, r1, lane, tab, hl);
        else if (nb == 2u) entropy_tile<2, WITH_P>(a, J, r0, r1, lane, tab, hl);
        else entropy_tile<1, WITH_P>(a, J, r0, r1, lane, tab, hl);
        hl = warp_sum_u64(hl);
        if (lane == 0 && hl) atomicAdd(&a.acc[d].H, hl);
        if (a.njobs == 1 && last_tile_of_design(a, J, lane)) finalize_design(a, d, J, lane, 32u, tab, nullptr);
    }
}

// One block per entropy tile (tile_rows rows of one design, at most kTileCells cells),
// the form for passes with few tiles (the plain call), where one warp per tile would
// leave most SMs idle: thread t takes cells t, t + 256, ... of the tile in row-major order,
// and the tile's per-bin sums meet in shared memory, then one global atomic per bin and
// sum. In both forms each cell's terms are rounded to fixed point once (entropy_cell), so
// every sum is independent of the grouping of cells into threads, tiles and launches,
// and each nonzero cell is zeroed after it is read, which leaves the histogram clear for
// the next pass.
template <bool WITH_P>
__global__ void __launch_bounds__(kEntropyThreads, 4) entropy_block_kernel(const LaunchArgs a)
{
    __shared__ float tab[4 * ff::kLogTable];
    extern __shared__ __align__(16) unsigned long long ent_smem[];  // per-bin s1, s2 (max_B each)
    __shared__ unsigned long long hsum;
    __shared__ unsigned last_tile;
    __shared__ FinalizeRed fin_red[kEntropyThreads / 32];
    cudaTriggerProgrammaticLaunchCompletion();
    for (uint32_t i = threadIdx.x; i < 4u * ff::kLogTable; i += blockDim.x) tab[i] = a.logtab[i];
    __syncthreads();
    cudaGridDependencySynchronize();  // the histogram of the trace and re-trace kernels
    // A pass whose re-trace queue overflowed is re-run by the host: leave every
    // accumulator untouched.
    if (a.ctl->overflow || a.ctl->queue_count > a.qcap) return;
    const uint32_t t = threadIdx.x, lane = t & 31u;
    for (uint64_t tile = blockIdx.x; tile < a.total_tiles; tile += gridDim.x) {
        const uint32_t d = find_job<F_TILE>(a.jobs, a.njobs, tile);
        const DesignJob J = a.jobs[d];
        const uint32_t B = J.B;
        const uint32_t r0 = (uint32_t)(tile - J.tile_off) * J.tile_rows;
        const uint32_t r1 = min(r0 + J.tile_rows, J.W);
        unsigned long long *s1 = ent_smem, *s2 = ent_smem + B;
        for (uint32_t b = t; b < B; b += kEntropyThreads) s1[b] = s2[b] = 0ull;
        if (t == 0) hsum = 0ull;
        __syncthreads();
        const ff::F2 unit{J.unit_hi, J.unit_lo}, lu{J.lu_hi, J.lu_lo};
        unsigned long long *base = a.hist + J.hist_off;
        const double pscale = J.pscale;
        const uint32_t cells = (r1 - r0) * B;
        const uint32_t db = (uint32_t)kEntropyThreads % B, dr = (uint32_t)kEntropyThreads / B;
        uint32_t b = t % B, row = r0 + t / B;
        unsigned long long hl = 0ull;
        // two cells per step, both loaded before either is processed, so that their
        // memory latencies and their float-float chains overlap
        for (uint32_t i0 = t; i0 < cells; i0 += 2u * kEntropyThreads) {
            uint64_t idx[2];
            uint32_t bc[2];
            unsigned long long cv[2];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const bool in = i0 + (uint32_t)k * kEntropyThreads < cells;
                idx[k] = (uint64_t)row * B + b;
                bc[k] = b;
                cv[k] = in ? base[idx[k]] : 0ull;
                if (WITH_P && in) a.p_out[idx[k]] = (double)cv[k] * pscale;
                b += db;
                row += dr;
                if (b >= B) {
                    b -= B;
                    row++;
                }
            }
#pragma unroll
            for (int k = 0; k < 2; k++) {
                if (cv[k]) {
                    base[idx[k]] = 0ull;
                    unsigned long long hq, pq;
                    entropy_cell(cv[k], unit, lu, tab, hq, pq);
                    hl += hq;
                    atomicAdd(s1 + bc[k], cv[k]);
                    atomicAdd(s2 + bc[k], pq);
                }
            }
        }
        hl = warp_sum_u64(hl);
        if (lane == 0 && hl) atomicAdd(&hsum, hl);
        __syncthreads();
        for (uint32_t bb = t; bb < B; bb += kEntropyThreads) {
            const unsigned long long v1 = s1[bb];
            if (v1) {
                atomicAdd(&a.S1[J.acc_off + bb], v1);
                atomicAdd(&a.S2[J.acc_off + bb], s2[bb]);
            }
        }
        if (t == 0 && hsum) atomicAdd(&a.acc[d].H, hsum);
        if (a.njobs == 1) {
            // a single design (the plain call): the block that finishes the last tile runs
            // the finalize, which saves a launch; with many designs the per-tile fences
            // would cost more than the separate finalize kernel
            __threadfence();
            __syncthreads();
            if (t == 0) last_tile = atomicAdd(&a.ctl->tiles_done, 1u) == J.ntiles - 1u ? 1u : 0u;
            __syncthreads();
            if (last_tile) {
                __threadfence();
                finalize_design(a, d, J, t, kEntropyThreads, tab, fin_red);
            }
        }
        __syncthreads();  // the shared sums are reused by the block's next tile
    }
}

// ------------------------------------------------------------------ rows by certified pieces

// 20 warps per SM without spills: 104 registers (16 warps) 5.85 ms, 96 5.45, 80 (24 warps, spills)
// 6.3, 128 6.2 on the 1024-design pass.
#ifndef CPD_ROWS_MAXNREG
#define CPD_ROWS_MAXNREG 96
#endif
constexpr uint32_t kRowsMaxTeam = 16;   // most warps of a team
constexpr uint32_t kRowsBrief = 48;     // a range of up to this many rays goes through fast_ray whole
constexpr uint32_t kRowsPieces = 15;    // pieces per half-warp (16 ends)
constexpr uint32_t kRowsSplit = 24;     // a piece without a bound is cut again from this many rays
constexpr uint32_t kRowsList = 64;      // entries of a warp's lists
constexpr uint32_t kRowsFull = 28;      // waiting ranges that make a batch: one step adds at most 34
constexpr uint32_t kRayBits = 22;       // (row of the group << kRayBits | ray) in one word
constexpr uint32_t kRayMask = (1u << kRayBits) - 1u;
static_assert(CPD_MAX_RAYS <= 1u << kRayBits && kRowsGroup <= 1u << (31 - kRayBits), "ray and row in one word");
constexpr uint32_t kDirect = 0x80000000u;  // in a range's end: rays for the re-trace, past fast_ray

// A warp's scratch.
struct RowsWarp {
    float4 rec_a[32];           // z of the left end (hi, lo), v0, v1
    float4 rec_b[32];           // v2, e, first bin, tasks | extent task << 31
    uint4 rec_c[32];            // rays [x, y), first task, row of the group
    uint2 wait[kRowsList];      // ranges of rays for fast_ray: row and first ray, one past the last
    uint32_t flag[kRowsList];   // rays for the float-float re-trace
    uint2 sub[32];              // pieces to cut again, as ranges
    uint32_t tfix[kRowsGroup];  // the rows' transmittances
};

// Shared memory of a block: the log2 table, per-bin sums (single-design passes), the warps'
// scratch, and per team the cells of its group of rows: ext (u64) and cnt (u32).
constexpr size_t rows_smem_bytes(uint32_t warps, uint32_t teams, uint32_t B)
{
    const uint32_t cells = B > kRowsCells ? B : kRowsCells;
    return 4u * 4u * ff::kLogTable + 16u * (size_t)B + warps * sizeof(RowsWarp) + teams * 12u * (size_t)((cells + 3u) & ~3u);
}

__device__ __forceinline__ void team_sync(uint32_t team, uint32_t T)
{
    // a block has at most two teams of more than one warp; constant barrier numbers, or the
    // block would reserve all sixteen
    if (T == 1u) __syncwarp();
    else if (team == 0u) asm volatile("bar.sync 1, %0;" ::"r"(T * 32u) : "memory");
    else asm volatile("bar.sync 2, %0;" ::"r"(T * 32u) : "memory");
}

// The fixed-N hybrid estimate of the designs whose coated exit face admits certified pieces
// (cpd_piece.h), from LamParams to the per-bin sums: trace, re-trace and entropy of a
// wavelength row by one team of T warps, with no histogram in memory.
//
// A team takes groups of rows of one design (J.grp_rows of them; one row when T > 1), whose
// cells live in shared memory: cnt counts the hits with the row's own transmittance (every hit
// of a certified piece), ext adds up the others. Per group:
//  1. Half a warp cuts a row's core range (T > 1: its share of it) into 15 pieces, lane i
//     evaluating the ray at the left end of piece i. A piece in one bin, or lost whole, is
//     counted at once; a mixed piece's bins come from its edges, two lanes per bin, each
//     finding one edge by bisection of the piece's rays on its quadratic, or, where the edges
//     lie too close, ray by ray. A piece without a bound is cut again into 15.
//  2. Rays within the error of an edge, and short pieces without a bound, wait in the warp's
//     list for fast_ray, 32 at a time over the rows of the group; what fast_ray flags, and the
//     setup's guard bands, wait for the float-float re-trace in the same way.
//  3. The cells' entropy terms, lane = bin, and the sums over the group's rows added to the
//     design's.
// Outcomes, flags and sums are those of trace_kernel, retrace_kernel and the entropy kernels,
// integer for integer.
//
// Issue bounds it (2.3 M rows of 1024 rays: 1680 warp instructions a row at 60% of the slots, the
// ALU pipe at 51%): 20 warps per SM, an edge's dependent bisection steps, and code the size of the
// instruction cache. 1024 designs, those rows: 10.8 ms trace and 0.97 entropy by the ray-by-ray
// kernels, 5.45 ms here; 512 designs x 128 rows x 8192 rays 2.33 -> 0.41 ms. (The steps' code
// inlined where their lists fill: 6.5 ms. One row's pieces through a histogram in memory and
// separate re-trace and entropy kernels: 6.3 ms. Edges 3.8 of 14 parts of a warp's time, rays of
// short pieces 3.6, pieces 2.8, entropy 1.5, re-trace 1.1.)
//
// HEAVY: the rows that the setup listed as having many rays for the float-float trace, each by a
// whole block, ahead of the groups. A warp takes 1.7 us per 32 such rays, and a pass waits for its
// last group: one design whose rows are re-traced whole (8 rows of 8192 rays in one warp) made a
// pass of 512 designs x 128 rows 3.5 ms instead of 0.45 (0.50 so). Without such rows the launch
// costs 2 us, so a pass of one design has it only where a group could keep its warps for 2 ms.
template <bool PARAM_FC, bool WITH_P, bool HEAVY>
__global__ void __maxnreg__(CPD_ROWS_MAXNREG) rows_kernel(const LaunchArgs a)
{
    cudaTriggerProgrammaticLaunchCompletion();
    extern __shared__ __align__(16) unsigned char rows_smem[];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, wib = tid >> 5, nwarps = blockDim.x >> 5;
    const uint32_t T = HEAVY ? nwarps : a.team, teams = HEAVY ? 1u : nwarps / T, team = HEAVY ? 0u : wib / T, tw = wib - team * T;
    const uint32_t maxc = ((a.max_B > kRowsCells ? a.max_B : kRowsCells) + 3u) & ~3u;
    float *tab = reinterpret_cast<float *>(rows_smem);
    unsigned long long *bs1 = reinterpret_cast<unsigned long long *>(tab + 4 * ff::kLogTable), *bs2 = bs1 + a.max_B;
    RowsWarp *wsm = reinterpret_cast<RowsWarp *>(bs2 + a.max_B);
    RowsWarp &w = wsm[wib];
    unsigned long long *ext = reinterpret_cast<unsigned long long *>(wsm + nwarps) + (size_t)team * maxc;
    uint32_t *cnt = reinterpret_cast<uint32_t *>(reinterpret_cast<unsigned long long *>(wsm + nwarps) + (size_t)teams * maxc) +
                    (size_t)team * maxc;
    const uint32_t tt = tw * 32u + lane, tn = T * 32u;  // thread of the team
    const uint32_t lt_mask = (1u << lane) - 1u;
    for (uint32_t i = tid; i < 4u * ff::kLogTable; i += blockDim.x) tab[i] = a.logtab[i];
    for (uint32_t b = tid; b < 2u * a.max_B; b += blockDim.x) bs1[b] = 0ull;
    for (uint32_t c = tt; c < maxc; c += tn) {
        cnt[c] = 0u;
        ext[c] = 0ull;
    }
    __syncthreads();
    cudaGridDependencySynchronize();  // the setup's LamParams and LamDF
    const uint32_t gteam = blockIdx.x * teams + team, nteams = gridDim.x * teams;
    const uint32_t sp = (blockIdx.x * nwarps + wib) % (uint32_t)kSpread;
    // a pass whose table could not be made is re-run by the host: nothing is added
    const bool bad = a.ctl->overflow != 0u;
    const uint64_t total = HEAVY ? (uint64_t)a.ctl->heavy_count : a.total_groups;
    for (uint64_t grp = gteam; grp < total && !bad;) {
        const uint64_t at = HEAVY ? a.heavy[grp].row : grp;
        const uint32_t d = PARAM_FC ? 0u : find_job<HEAVY ? F_ROW : F_GROUP>(a.jobs, a.njobs, at);
        const DesignJob &J = PARAM_FC ? a.one : a.jobs[d];
        const uint32_t B = J.B;
        const uint32_t k0 = HEAVY ? (uint32_t)(at - J.row_off) : (uint32_t)(at - J.grp_off) * J.grp_rows;
        const uint32_t g = HEAVY ? 1u : min(J.grp_rows, J.W - k0);
        const uint64_t row0 = J.row_off + k0;
        const float2 *__restrict__ zt = reinterpret_cast<const float2 *>(a.z32) + J.ray_off;
        const LamParams *lp = a.lp + row0;
        uint32_t nhit = 0u, nret = 0u, nfast = 0u;
        PieceConst K;
        {
            const FastConst Cd = PARAM_FC ? FastConst{} : a.designs[d].fc;
            K = piece_const(PARAM_FC ? a.fc : Cd);
        }
        // the same in every lane: entries of the lists, the next row, and what is left of the
        // last rows' mixed pieces: tasks [t0, ntask), records [ir, nrec) from ray js on
        uint32_t nwait = 0u, nflag = 0u, nsub = 0u, next = 0u;
        uint32_t t0 = 0u, ntask = 0u, ir = 0u, nrec = 0u, js = 0u;
        // of the lane's piece: its tasks
        uint32_t incl = 0u, excl = 0u;
        bool by_edge = false;
        const uint32_t half = lane >> 4, hl = lane & 15u;
        // One step per turn, each kind in one place (the code of every step once: inlined where
        // their lists fill, the float-float steps alone would exceed the instruction cache).
        for (;;) {
            const bool rows_left = next < g || nsub != 0u;
            const bool work_left = t0 < ntask || ir < nrec || rows_left;
            if (nflag >= 32u || (nflag && !work_left && !nwait)) {
                // ---- 32 flagged rays re-traced, one per lane
                __syncwarp();
                const uint32_t n = min(nflag, 32u);
                if (lane < n) {
                    const uint32_t r = w.flag[lane], rl = r >> kRayBits;
                    const float2 z = __ldg(zt + (r & kRayMask));
                    uint32_t bin = 0u;
                    float t = 0.f;
                    if (trace_df(a.designs[d], a.lx[row0 + rl], z.x, z.y, bin, t)) {
                        atomicAdd(ext + rl * B + bin, (unsigned long long)t_fixed(t));
                        nhit++;
                    }
                    nret++;
                }
                __syncwarp();
                nflag -= n;
                const uint32_t v = w.flag[32u + lane];
                __syncwarp();
                if (lane < nflag) w.flag[lane] = v;
                continue;
            }
            if (nwait >= kRowsFull || (nwait && !work_left)) {
                // ---- the first 32 rays of the waiting ranges through fast_ray
                __syncwarp();
                uint2 e0 = lane < nwait ? w.wait[lane] : make_uint2(0u, 0u);
                const uint2 e1 = w.wait[32u + lane];
                const uint32_t j0 = e0.x & kRayMask, len = (e0.y & ~kDirect) - j0;
                uint32_t ic = lane < nwait ? len : 0u;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t v = __shfl_up_sync(0xffffffffu, ic, o);
                    if (lane >= (uint32_t)o) ic = min(ic + v, 64u);  // only the first 32 matter
                }
                const uint32_t sum = __shfl_sync(0xffffffffu, ic, 31), m = min(sum, 32u);
                uint32_t ec = __shfl_up_sync(0xffffffffu, ic, 1);
                if (lane == 0u) ec = 0u;
                // the range of ray `lane` of the batch: ranges marked at their first ray
                const uint32_t starts = __reduce_or_sync(0xffffffffu, lane < nwait && ec < 32u ? 1u << ec : 0u);
                const int i = __popc(starts & (lt_mask | 1u << lane)) - 1;
                const uint32_t ent = __shfl_sync(0xffffffffu, e0.x, i) + lane - __shfl_sync(0xffffffffu, ec, i);
                const bool direct = (__shfl_sync(0xffffffffu, e0.y, i) & kDirect) != 0u;
                // ranges used up leave the list
                const uint32_t gone = __popc(__ballot_sync(0xffffffffu, lane < nwait && ic <= m && ec < m));
                if (lane < nwait && ec < m && ic > m) e0.x += m - ec;
                __syncwarp();
                if (lane >= gone && lane < nwait) w.wait[lane - gone] = e0;
                if (32u + lane < nwait) w.wait[32u + lane - gone] = e1;
                nwait -= gone;
                int r = RAY_LOST;
                if (lane < m) {
                    r = RAY_FLAG;
                    if (!direct) {
                        const uint32_t rl = ent >> kRayBits;
                        const FastConst Cd = PARAM_FC ? FastConst{} : a.designs[d].fc;
                        const FastConst &C = PARAM_FC ? a.fc : Cd;
                        const FastLimits Ld = PARAM_FC ? FastLimits{} : fast_limits(Cd, a.guards);
                        const FastLimits &Lm = PARAM_FC ? a.fl : Ld;
                        const LamParams P = lp[rl];
                        const float2 z = __ldg(zt + (ent & kRayMask));
                        uint32_t bin = 0u;
                        float t = 0.f;
                        r = fast_ray(C, Lm, P, a.guards, z.x, z.y, bin, t);
                        if (r == RAY_HIT) {
                            const uint32_t tf = t_fixed(t);
                            if (tf == piece_tfix(P)) {
                                atomicAdd(cnt + rl * B + bin, 1u);
                            } else {
                                atomicAdd(ext + rl * B + bin, (unsigned long long)tf);
                                nhit++;
                            }
                        }
                    }
                }
                const uint32_t f = __ballot_sync(0xffffffffu, r == RAY_FLAG);
                if (r == RAY_FLAG) w.flag[nflag + __popc(f & lt_mask)] = ent;
                nflag += __popc(f);
                continue;
            }
            if (t0 < ntask) {
                // ---- 16 tasks of the mixed pieces: two lanes per bin, one edge each
                // the record of task t: those that start after t0 are marked at their first task
                const uint32_t tau = lane >> 1, t = t0 + tau;
                const uint32_t first_rec = __popc(__ballot_sync(0xffffffffu, by_edge && incl <= t0));
                const uint32_t starts =
                    __reduce_or_sync(0xffffffffu, by_edge && excl > t0 && excl < t0 + 16u ? 1u << (excl - t0) : 0u);
                const bool act = t < ntask;
                const uint32_t i = act ? first_rec + __popc(starts & ((2u << tau) - 1u)) : 0u;
                const float4 ra = w.rec_a[i], rb = w.rec_b[i];
                const uint4 rc = w.rec_c[i];
                const uint32_t cw = __float_as_uint(rb.w), kt = t - rc.z;
                const bool xt = (cw >> 31) && kt + 1u == (cw & 0x7fffffffu);
                const int bq = __float_as_int(rb.z) + (int)kt;
                const bool up = lane & 1u;
                const Edge ed = piece_edge(K, bq, xt, up);
                const float sg = ra.w > 0.f ? -1.f : 1.f;  // the rays' dz fall with their index
                uint32_t jb = 0u, je = 0u;
                if (act) {
                    const float a0 = sg * (ra.z - ed.v), a1 = sg * ra.w, a2 = sg * rb.x;
                    const EdgeRays er = edge_rays(rc.x, rc.y, rb.y, [&](uint32_t j) {
                        const float2 z = __ldg(zt + j);
                        const float dd = (ra.x - z.x) + (ra.y - z.y);
                        return a0 + dd * (a1 + dd * a2);
                    });
                    jb = er.jb;
                    je = er.je;
                }
                // the bin's rays lie between its two edges' windows
                const uint32_t ob = __shfl_xor_sync(0xffffffffu, jb, 1), oe = __shfl_xor_sync(0xffffffffu, je, 1);
                const uint32_t first = sg > 0.f ? je : oe, last = sg > 0.f ? ob : jb;
                const uint32_t bin = bq > 0 ? (uint32_t)bq : 0u;
                if (act && !up && !xt && last > first && bin < B) atomicAdd(cnt + rc.w * B + bin, last - first);
                const bool put = ed.emit && jb < je;
                const uint32_t f = __ballot_sync(0xffffffffu, put);
                if (put) w.wait[nwait + __popc(f & lt_mask)] = make_uint2(rc.w << kRayBits | jb, je);
                nwait += __popc(f);
                t0 += 16u;
                continue;
            }
            if (ir < nrec) {
                // ---- 32 rays of a mixed piece on its quadratic
                const float4 ra = w.rec_a[ir], rb = w.rec_b[ir];
                const uint4 rc = w.rec_c[ir];
                const uint32_t j = rc.x + js + lane;
                uint32_t bin = 0u;
                int r = RAY_LOST;
                if (j < rc.y) {
                    const float2 z = __ldg(zt + j);
                    r = piece_ray(K, B, 0.f, ra.z, ra.w, rb.x, rb.y, (ra.x - z.x) + (ra.y - z.y), bin);
                }
                // runs of consecutive rays in one bin: the first lane of each counts it
                const uint32_t key = r == RAY_HIT ? bin : 0xffffffffu;
                const uint32_t prev = __shfl_up_sync(0xffffffffu, key, 1);
                const uint32_t heads = __ballot_sync(0xffffffffu, lane == 0u || key != prev);
                if (r == RAY_HIT && (heads >> lane & 1u)) {
                    const uint32_t after = heads & ~(lt_mask | 1u << lane);
                    atomicAdd(cnt + rc.w * B + bin, (after ? (uint32_t)__ffs(after) - 1u : 32u) - lane);
                }
                const uint32_t f = __ballot_sync(0xffffffffu, r == RAY_FLAG);
                if (r == RAY_FLAG) w.wait[nwait + __popc(f & lt_mask)] = make_uint2(rc.w << kRayBits | j, j + 1u);
                nwait += __popc(f);
                js += 32u;
                if (rc.x + js >= rc.y) {
                    ir++;
                    js = 0u;
                }
                continue;
            }
            if (!rows_left) break;
            // ---- the next two rows (T > 1: two shares of the row), pieces to cut again first
            __syncwarp();
            uint32_t rl = 0u, lo = 0u, hi = 0u;
            const bool again = nsub != 0u;
            if (again) {
                if (nsub > half) {
                    const uint2 v = w.sub[nsub - 1u - half];
                    rl = v.x >> kRayBits;
                    lo = v.x & kRayMask;
                    hi = v.y;
                }
                nsub -= min(nsub, 2u);
            } else {
                // the half's row, its core range, and the guard bands around it
                rl = T == 1u ? min(next + half, g - 1u) : 0u;
                const bool has = T > 1u || next + half < g;
                const uint4 rg = HEAVY ? a.heavy[grp].ranges : *reinterpret_cast<const uint4 *>(&lp[rl].core_lo);  // core, band
                lo = rg.x;
                hi = rg.y;
                uint32_t blo = rg.z, b1 = lo, b2 = hi, bhi = rg.w;
                if (!has) hi = lo = blo = b1 = b2 = bhi = 0u;
                if (hl == 0u && tw == 0u && (T == 1u || half == 0u)) nfast += hi - lo;
                if (T > 1u) {
                    const uint32_t sh = 31u - __clz(2u * T), s = 2u * tw + half;  // share s of 2 T
                    const auto share = [&](uint32_t &p, uint32_t &q) {
                        const uint32_t n = q - p;
                        q = p + (n * (s + 1u) >> sh);
                        p = p + (n * s >> sh);
                    };
                    share(lo, hi);
                    share(blo, b1);
                    share(b2, bhi);
                }
                const bool ba = hl == 0u && b1 > blo, bb = hl == 1u && bhi > b2;
                const uint32_t f = __ballot_sync(0xffffffffu, ba || bb);
                if (f) {
                    if (ba || bb)
                        w.wait[nwait + __popc(f & lt_mask)] =
                            make_uint2(rl << kRayBits | (ba ? blo : b2), (ba ? b1 : bhi) | kDirect);
                    nwait += __popc(f);
                }
                next += 2u;
            }
            const uint32_t n = hi - lo;
            // a short range goes to fast_ray whole: one "piece", of lane 0
            const bool brief = n <= kRowsBrief;
            const uint32_t L = brief ? n : (n + kRowsPieces - 1u) / kRowsPieces;
            const uint32_t j0 = lo + hl * L, j1 = min(j0 + L, hi);
            const bool mine = hl < kRowsPieces && j0 < hi;
            Piece q;
            PieceEdges pe;
            float2 z = make_float2(0.f, 0.f);
            {
                const FastConst Cd = PARAM_FC ? FastConst{} : a.designs[d].fc;
                const FastConst &C = PARAM_FC ? a.fc : Cd;
                const FastLimits Ld = PARAM_FC ? FastLimits{} : fast_limits(Cd, a.guards);
                const FastLimits &Lm = PARAM_FC ? a.fl : Ld;
                const LamParams P = lp[rl];
                if (!again && hl == 0u) w.tfix[rl] = WITH_P && !HEAVY && P.core_lo == kNotHere ? kNotHere : piece_tfix(P);
                if (n) z = __ldg(zt + min(j0, hi - 1u));
                const PieceEnd e = piece_end(C, Lm, K, P, a.guards, z.x, z.y);
                PieceEnd o = e;
                o.dz = __shfl_down_sync(0xffffffffu, e.dz, 1);
                o.v = __shfl_down_sync(0xffffffffu, e.v, 1);
                o.gv = __shfl_down_sync(0xffffffffu, e.gv, 1);
                o.ci = __shfl_down_sync(0xffffffffu, e.ci, 1);
                o.cr = __shfl_down_sync(0xffffffffu, e.cr, 1);
                o.cid = __shfl_down_sync(0xffffffffu, e.cid, 1);
                o.gn = __shfl_down_sync(0xffffffffu, e.gn, 1);
                o.px = __shfl_down_sync(0xffffffffu, e.px, 1);
                o.py = __shfl_down_sync(0xffffffffu, e.py, 1);
                o.cls = __shfl_down_sync(0xffffffffu, e.cls, 1);
                q = piece_fit(C, K, P, e, o);
                if (!C.pieces || brief) q.cls = PIECE_RAYS;
                pe = piece_edges(K, q, o.dz - e.dz, j1 - j0);
            }
            if (mine && q.cls == PIECE_BIN) atomicAdd(cnt + rl * B + q.bin, j1 - j0);
            // pieces without a bound: cut again, or their rays wait for fast_ray
            const bool rays = mine && q.cls == PIECE_RAYS;
            const bool cut = rays && !again && !brief && j1 - j0 >= kRowsSplit, wait = rays && !cut;
            const uint32_t mc = __ballot_sync(0xffffffffu, cut), mw = __ballot_sync(0xffffffffu, wait);
            const uint2 range = make_uint2(rl << kRayBits | j0, j1);
            if (cut) w.sub[nsub + __popc(mc & lt_mask)] = range;
            if (wait) w.wait[nwait + __popc(mw & lt_mask)] = range;
            nsub += __popc(mc);
            nwait += __popc(mw);
            // mixed pieces: records of those binned by edges, then of those binned ray by ray
            const bool mixed = mine && q.cls == PIECE_MIXED;
            by_edge = mixed && pe.count != 0u;
            const uint32_t me = __ballot_sync(0xffffffffu, by_edge), mr = __ballot_sync(0xffffffffu, mixed && !by_edge);
            incl = by_edge ? pe.count : 0u;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= (uint32_t)o) incl += v;
            }
            excl = by_edge ? incl - pe.count : 0u;
            t0 = js = 0u;
            ntask = __shfl_sync(0xffffffffu, incl, 31);
            ir = __popc(me);
            nrec = ir + __popc(mr);
            if (mixed) {
                const uint32_t at = by_edge ? __popc(me & lt_mask) : ir + __popc(mr & lt_mask);
                w.rec_a[at] = make_float4(z.x, z.y, q.v0, q.v1);
                w.rec_b[at] = make_float4(q.v2, q.e, __int_as_float(pe.qa),
                                          __uint_as_float(pe.count | (pe.ext ? 0x80000000u : 0u)));
                w.rec_c[at] = make_uint4(j0, j1, excl, rl);
            }
            __syncwarp();
        }
        team_sync(team, T);
        // 3. the cells' entropy terms
        {
            const ff::F2 unit{J.unit_hi, J.unit_lo}, lu{J.lu_hi, J.lu_lo};
            const uint32_t *tfix = (wsm + team * T)->tfix;
            const uint32_t phases = tn > B && T == 1u ? 32u / B : 1u;  // rows side by side when B < 32
            const uint32_t ph = phases > 1u ? tt / B : 0u;
            unsigned long long hl_sum = 0ull;
            for (uint32_t b = phases > 1u ? tt - ph * B : tt; b < B; b += phases > 1u ? B : tn) {
                unsigned long long c1 = 0ull, q2 = 0ull;
                for (uint32_t r = ph; r < g; r += phases) {
                    if (ph >= phases) break;
                    const uint32_t c = r * B + b;
                    const uint32_t v = cnt[c];
                    const unsigned long long cv = ext[c] + (unsigned long long)v * tfix[r];
                    if (v) {
                        cnt[c] = 0u;
                        nhit += v;
                    }
                    if (cv) {
                        ext[c] = 0ull;
                        unsigned long long hq, pq;
                        entropy_cell(cv, unit, lu, tab, hq, pq);
                        hl_sum += hq;
                        q2 += pq;
                        c1 += cv;
                    }
                    if (WITH_P && (HEAVY || tfix[r] != kNotHere)) a.p_out[(uint64_t)(k0 + r) * B + b] = (double)cv * J.pscale;
                }
                if (c1) {
                    if (PARAM_FC) {
                        atomicAdd(bs1 + b, c1);
                        atomicAdd(bs2 + b, q2);
                    } else {
                        atomicAdd(&a.S1[J.acc_off + b], c1);
                        atomicAdd(&a.S2[J.acc_off + b], q2);
                    }
                }
            }
            hl_sum = warp_sum_u64(hl_sum);
            nhit = __reduce_add_sync(0xffffffffu, nhit);
            nret = __reduce_add_sync(0xffffffffu, nret);
            nfast = __reduce_add_sync(0xffffffffu, nfast);
            if (lane == 0u) {
                if (hl_sum) atomicAdd(&a.acc[d].H, hl_sum);
                if (nhit) atomicAdd(&a.acc[d].hits[sp], (unsigned long long)nhit);
                if (nret) atomicAdd(&a.acc[d].retraced[sp], (unsigned long long)nret);
                if (nfast) atomicAdd(&a.acc[d].fast[sp], (unsigned long long)nfast);
            }
        }
        team_sync(team, T);  // the cells are clear for the next group
        if (nteams >= total) break;
        if (!HEAVY && T == 1u) {
            unsigned long long c = 0;
            if (lane == 0) c = atomicAdd(&a.ctl->group_counter, 1ull);
            grp = nteams + __shfl_sync(0xffffffffu, c, 0);
        } else {
            grp += nteams;
        }
    }
    if (PARAM_FC) {
        // a single design: the block's per-bin sums, then the finalize by the last block
        __shared__ unsigned last_block;
        __shared__ FinalizeRed fin_red[kRowsMaxTeam];
        __syncthreads();
        const uint32_t B = a.one.B;
        for (uint32_t b = tid; b < B; b += blockDim.x)
            if (bs1[b]) {
                atomicAdd(&a.S1[b], bs1[b]);
                atomicAdd(&a.S2[b], bs2[b]);
            }
        __threadfence();
        __syncthreads();
        if (tid == 0) last_block = atomicAdd(&a.ctl->tiles_done, 1u) == gridDim.x - 1u ? 1u : 0u;
        __syncthreads();
        if (last_block) {
            __threadfence();
            publish_status_all(a);
            if (!bad) finalize_design(a, 0u, a.jobs[0], tid, blockDim.x, tab, fin_red);
        }
    }
}

// One warp per design after the entropy kernel.
__global__ void __launch_bounds__(128) finalize_kernel(const LaunchArgs a)
{
    __shared__ float tab[4 * ff::kLogTable];
    for (uint32_t i = threadIdx.x; i < 4u * ff::kLogTable; i += blockDim.x) tab[i] = a.logtab[i];
    __syncthreads();
    cudaGridDependencySynchronize();  // the entropy kernel's sums
    if (!a.total_items && !a.adaptive) publish_status(a);  // no re-trace kernel in this pass
    // A pass whose re-trace queue overflowed is re-run by the host: write nothing.
    if (a.ctl->overflow || a.ctl->queue_count > a.qcap) return;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t d = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; d < a.njobs; d += nw) {
        const DesignJob J = a.jobs[d];
        finalize_design(a, d, J, lane, 32u, tab, nullptr);
    }
}

__global__ void __launch_bounds__(128) trace_pairs_kernel(const DevDesign *__restrict__ dd,
                                                          const double *__restrict__ lam_u,
                                                          const double *__restrict__ z64, uint32_t n,
                                                          uint32_t mode, uint32_t *bins, double *ts,
                                                          uint8_t *flags)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const DevDesign &D = *dd;
    const double z = z64[i];
    uint32_t bin = D.B;
    double t = 0.0;
    uint8_t fl = 0;
    if (isfinite(z)) {
        if (mode == CPD_TRACE_FP64) {
            uint32_t b = 0;
            double te = 0.0;
            if (x::trace(D, x::wavelength(D, lam_u[i]), x::beam_y(D, z), b, te) == 0) {
                bin = b;
                t = te;
            }
        } else {
            float zz[2];
            split_f32(z, zz[0], zz[1]);
            LamParams P;
            LamDF E;
            const double yg = mode == CPD_TRACE_FP32 ? 0.0 : kYGuardRel;
            lambda_setup_df(D, lam_u[i], zz, 1u, P, yg, &E);
            bool retrace = false;
            if (P.core_lo == 0 && P.core_hi == 1 && !P.all_exact) {
                const Guards g = mode == CPD_TRACE_FP32 ? no_guards() : default_guards();
                uint32_t b = 0;
                float tf = 0.f;
                const int r = fast_ray(D.fc, P, g, zz[0], zz[1], b, tf);
                if (r == RAY_HIT) {
                    bin = b;
                    t = tf;
                } else if (r == RAY_FLAG) {
                    retrace = true;
                }
            } else if (P.band_lo == 0 && P.band_hi == 1) {
                // in a y-interval guard band, or its own reference ray without a usable
                // exit/detector geometry
                retrace = mode == CPD_TRACE_HYBRID;
            }
            if (retrace) {
                fl = 1;
                uint32_t b = 0;
                float tf = 0.f;
                if (trace_df(D, E, zz[0], zz[1], b, tf)) {
                    bin = b;
                    t = tf;
                }
            }
        }
    }
    bins[i] = bin;
    ts[i] = t;
    if (flags) flags[i] = fl;
}

// ------------------------------------------------------------------ p_dets_l_wavelength
//
// The reference CPU estimator of p(d|lambda) for one wavelength
// (vector_quasi_monte_carlo_integration + p_dets_l_wavelength, src/fitness.rs:5-34,48-69),
// the one Spectrometer.transmission_probability returns (src/pylib.rs:1028-1058): rays in
// order; a ray that hits bin b pads b's Welford state with zeros up to the ray count
// (Welford::skip), adds its t (next_sample), and the integration stops at the first hit
// after which its bin's SEM^2 <= (5e-3)^2 (sem_le_error_threshold, welford.rs:5-57); every
// bin is then padded to the final count and p = its mean. The bin that fired the stop keeps
// a count one ahead of the rays (skip then next_sample), as the reference does.
//
// One block per wavelength, kTpRays threads. A round traces kTpRays rays in exact f64
// (x::trace, bit-identical to the reference's f64 trace), sorts the round's hits by (bin,
// ray), and the first thread of each bin's run replays the run's Welford updates in the
// reference's f64 operation order, keeping the state after each update and stopping at the
// run's first passing hit. The round's stop is the earliest passing hit over all bins;
// each bin then keeps its state after its last hit before or at that ray. The result is
// the one-ray-at-a-time order of the reference bit for bit: the bins' states are
// independent, and every hit up to the stop is applied in ray order within its bin.
constexpr uint32_t kTpRays = 256;

struct TpWelford {
    double c, m, m2;
};

// Welford::skip (welford.rs:34-42).
__device__ __forceinline__ void tp_skip(TpWelford &w, double n)
{
    if (w.c < n) {
        const double z = x::sub(n, w.c);
        w.m = x::div(x::mul(w.c, w.m), n);
        w.m2 = x::add(w.m2, x::div(x::mul(x::mul(x::sqr(w.m), w.c), z), n));
        w.c = n;
    }
}

// Welford::next_sample (welford.rs:26-32).
__device__ __forceinline__ void tp_next(TpWelford &w, double v)
{
    w.c = x::add(w.c, 1.0);
    const double d = x::sub(v, w.m);
    w.m = x::add(w.m, x::div(d, w.c));
    w.m2 = x::add(w.m2, x::mul(d, x::sub(v, w.m)));
}

__global__ void __launch_bounds__(kTpRays) tp_adaptive_kernel(const DevDesign *__restrict__ dd,
                                                              const double *__restrict__ lambdas,
                                                              const double *__restrict__ z64, uint32_t max_m,
                                                              double *out, uint32_t *rays_out, bool left_only)
{
    if (left_only && rays_out[blockIdx.x]) return;  // tp_pieces_kernel has done it
    __shared__ __align__(16) DevDesign sD;
    __shared__ uint32_t key[kTpRays];   // (bin << 8) | ray within the round; ~0u: no hit
    __shared__ double tv[kTpRays];      // t of the round's ray i
    __shared__ double sc[kTpRays], sm[kTpRays], sm2[kTpRays];  // state after sorted hit k
    __shared__ uint32_t stop_i;
    extern __shared__ __align__(16) double wst[];  // c[B] | m[B] | m2[B]
    const uint32_t tid = threadIdx.x;
    for (uint32_t i = tid; i < sizeof(DevDesign) / 4; i += blockDim.x)
        reinterpret_cast<uint32_t *>(&sD)[i] = reinterpret_cast<const uint32_t *>(dd)[i];
    const uint32_t B = dd->B;
    double *wc = wst, *wm = wst + B, *wm2 = wst + 2 * B;
    for (uint32_t b = tid; b < B; b += blockDim.x) wc[b] = wm[b] = wm2[b] = 0.0;
    __syncthreads();
    const double lambda = lambdas[blockIdx.x];
    const double e2 = x::mul(5e-3, 5e-3);
    uint32_t count = max_m;
    for (uint32_t j0 = 0; j0 < max_m; j0 += kTpRays) {
        const uint32_t j = j0 + tid;
        uint32_t k = ~0u;
        if (j < max_m) {
            uint32_t bin = 0;
            double t = 0.0;
            if (x::trace(sD, lambda, x::beam_y(sD, z64[j]), bin, t) == 0) {
                k = (bin << 8) | tid;
                tv[tid] = t;
            }
        }
        key[tid] = k;
        if (tid == 0) stop_i = ~0u;
        if (!__syncthreads_or(k != ~0u)) continue;  // no hit this round
        // bitonic sort of the keys: hits grouped by bin, in ray order within a bin
        for (uint32_t w = 2; w <= kTpRays; w <<= 1)
            for (uint32_t h = w >> 1; h > 0; h >>= 1) {
                const uint32_t o = tid ^ h;
                if (o > tid) {
                    const uint32_t a = key[tid], b = key[o];
                    if ((a > b) == ((tid & w) == 0)) {
                        key[tid] = b;
                        key[o] = a;
                    }
                }
                __syncthreads();
            }
        const uint32_t kk = key[tid];
        const bool head = kk != ~0u && (tid == 0 || (key[tid - 1] >> 8) != (kk >> 8));
        uint32_t last = tid;  // sorted position of the run's last hit
        if (head) {
            const uint32_t b = kk >> 8;
            TpWelford st{wc[b], wm[b], wm2[b]};
            while (last + 1 < kTpRays && key[last + 1] != ~0u && (key[last + 1] >> 8) == b) last++;
            for (uint32_t q = tid; q <= last; q++) {
                const uint32_t i = key[q] & 0xffu;
                tp_skip(st, (double)(j0 + i + 1u));
                tp_next(st, tv[i]);
                sc[q] = st.c;
                sm[q] = st.m;
                sm2[q] = st.m2;
                if (st.m2 < x::mul(e2, x::mul(st.c, x::sub(st.c, 1.0)))) {
                    atomicMin(&stop_i, i);
                    break;
                }
            }
        }
        __syncthreads();
        const uint32_t si = stop_i;
        if (head) {
            // the bin's state after its last hit at or before the stop
            int q_keep = -1;
            for (uint32_t q = tid; q <= last && (key[q] & 0xffu) <= si; q++) q_keep = (int)q;
            if (q_keep >= 0) {
                const uint32_t b = kk >> 8;
                wc[b] = sc[q_keep];
                wm[b] = sm[q_keep];
                wm2[b] = sm2[q_keep];
            }
        }
        __syncthreads();
        if (si != ~0u) {
            count = j0 + si + 1u;
            break;
        }
    }
    // every bin padded to the final ray count (the reference's closing skip)
    for (uint32_t b = tid; b < B; b += blockDim.x) {
        TpWelford st{wc[b], wm[b], wm2[b]};
        tp_skip(st, (double)count);
        out[(uint64_t)blockIdx.x * B + b] = st.m;
    }
    if (tid == 0 && rays_out) rays_out[blockIdx.x] = count;
}

// The same estimator for a design with certified pieces (cpd_piece.h), bit for bit. What bounds
// the kernel above is FP64: a warp instruction takes its scheduler ~64 cycles, a trace of 256 rays
// ~28k cycles, and a hit's Welford update three divisions. Here
//  * the bins come from the wavelength's pieces, fast_ray and, for the few rays in its guard
//    bands, the exact f64 trace; every ray's transmittance is the same f64 value, formed once per
//    wavelength by the trace's own operations (tp_setup_kernel). So FP32 decides most bins, and that
//    they are the f64 trace's rests on the guards' measured widths (default_guards): over 1500
//    designs of wider ranges than the optimizer's, 48 wavelengths x up to 8192 rays each, every bit
//    and count equals the kernel above's with these guards and with a tenth of them, and not with
//    0.03 (4 designs);
//  * a chunk's hits are bits of a mask per bin, so one thread per bin replays its hits in ray order
//    with all bins of 32 packed in one warp, and runs ahead of the other bins up to the earliest
//    stop known;
//  * the divisors are ray counts, whose reciprocals are a table: a division is three FP64
//    instructions (x::div_by);
//  * of an update only the mean is replayed in f64 (9 instructions; the result is its bits). The
//    squared deviations are read by the SEM test alone and have a closed form for hits of one t:
//    after hit k + 1 at ray n, with c the count before it, they grow by
//    (k t / n)^2 c (n - c) / n + t^2 (n - k)^2 / (n (n + 1)). All terms are positive, a term's
//    roundings are at most 22 2^-24 (a reciprocal counts 4), the limit's 3, and the sum is kept in
//    two floats: within 2e-6 of the f64 recurrence. A test within kTpMargin leaves the wavelength
//    to a replay in full (21 instructions) from the start.
// A bin that ran past the stop is replayed from the chunk's start. The longest bin's replay bounds
// it now. 100 wavelengths x up to 16384 rays, device: 119 -> 56 us where they stop early, 1223 -> 425
// and 2312 -> 761 where some run all rays (every update in full: 641 and 1166).
constexpr uint32_t kTpList = 1024;

// Per wavelength, by two warps of a block: the setup in float-float, and the transmittance of its
// hits in the f64 trace's operations (the flat faces and a coated exit face).
__global__ void __launch_bounds__(64) tp_setup_kernel(const TpArgs a)
{
    cudaTriggerProgrammaticLaunchCompletion();
    const uint32_t i = blockIdx.x * 32u + (threadIdx.x & 31u);
    if (i >= a.n) return;
    const DevDesign &D = *a.d;
    const double lambda = a.lambdas[i];
    if (threadIdx.x < 32u) {
        LamParams P;
        LamDF E;
        lambda_setup_df(D, lambda, reinterpret_cast<const float *>(a.z32), a.Rz, P, kYGuardRel, &E);
        a.lp[i] = P;
    } else {
        x::Ray r{0.0, 0.0, 1.0, 0.0, 1.0, 1.0};
        double n1 = 1.0;
        bool ok = true;
        for (int k = 0; k < D.G && ok; k++) {
            const double n2 = x::calc_n(D.glass[k], lambda);
            ok = x::refract(r, D.pnx[k], D.pny[k], n1, n2, D.ar != 0);
            n1 = n2;
        }
        a.t64[i] = x::mul(x::add(x::mul(r.ts, 0.99), x::mul(r.tp, 0.99)), 0.5);
    }
}

constexpr float kTpMargin = 1e-5f;
// One bin: its mean, squared deviations (fast: an FP32 sum and its error; full: f64), the count
// and the hits.
struct TpBin {
    double m;
    union {
        double m2;
        float2 f2;
    };
    uint32_t c, k;
};

__host__ __device__ constexpr uint32_t tp_chunk(uint32_t B) { return B <= 256u ? 1024u : 256u; }
constexpr size_t tp_pieces_smem_bytes(uint32_t B)
{
    // per bin: the state, its copy at the chunk's start, the mask
    return sizeof(Adapt1Pieces) + (size_t)B * (2u * sizeof(TpBin) + tp_chunk(B) / 8u) + 8u * kTpList;
}

__global__ void __launch_bounds__(256) tp_pieces_kernel(const TpArgs a)
{
    extern __shared__ __align__(16) unsigned char tp_smem[];
    __shared__ uint32_t s_stop, s_n1, s_n2, s_open;
    Adapt1Pieces &w = *reinterpret_cast<Adapt1Pieces *>(tp_smem);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, nthr = blockDim.x;
    const DevDesign &D = *a.d;
    const uint32_t B = D.B, C = tp_chunk(B), words = C / 32u;
    TpBin *st = reinterpret_cast<TpBin *>(&w + 1), *st0 = st + B;
    uint32_t *list1 = reinterpret_cast<uint32_t *>(st0 + B), *list2 = list1 + kTpList;
    uint32_t *mask = list2 + kTpList;  // [bin][word]
    TpBin zero;
    zero.m = zero.m2 = 0.0;
    zero.c = zero.k = 0u;
    for (uint32_t b = tid; b < B; b += nthr) st[b] = zero;
    if (tid == 0) s_open = 0u;
    if (tid < sizeof(FastConst) / 4)
        reinterpret_cast<uint32_t *>(&w.C)[tid] = reinterpret_cast<const uint32_t *>(&D.fc)[tid];
    const uint32_t il = blockIdx.x;
    const double lambda = a.lambdas[il];
    cudaGridDependencySynchronize();  // tp_setup_kernel
    if (tid < sizeof(LamParams) / 4)
        reinterpret_cast<uint32_t *>(&w.P)[tid] = reinterpret_cast<const uint32_t *>(a.lp + il)[tid];
    __syncthreads();
    const PieceConst K = piece_const(w.C);
    const uint32_t lo = w.P.core_lo, hi = w.P.all_exact ? w.P.core_lo : w.P.core_hi;
    const uint32_t band_lo = w.P.band_lo, band_hi = w.P.band_hi, ks = piece_shift(hi - lo);
    const uint32_t tfast = piece_tfix(w.P);
    const double t64 = a.t64[il];
    if (tid < 32u && hi > lo) adapt_pieces(a.guards, w, K, a.z32, lo, hi, ks, lane);
    uint32_t count = a.max_m;
    bool full = false;
    const float tf = (float)t64, tf2 = tf * tf;
    // no ray clears the flat faces: no hit
    for (uint32_t j0 = band_lo >= band_hi ? a.max_m : 0u; j0 < a.max_m; j0 += C) {
        const uint32_t nj = min(C, a.max_m - j0);
        for (uint32_t i = tid; i < B * words; i += nthr) mask[i] = 0u;
        for (uint32_t b = tid; b < B; b += nthr) st0[b] = st[b];
        if (tid == 0) {
            s_stop = ~0u;
            s_n1 = s_n2 = 0u;
        }
        __syncthreads();
        // the rays' bins: their pieces, then fast_ray for what those leave
        for (uint32_t i = tid; i < nj; i += nthr) {
            const uint32_t s = __ldg(a.rank + j0 + i);
            if (s < band_lo || s >= band_hi) continue;
            uint32_t bin = 0u;
            int r = RAY_FLAG;
            if (s >= lo && s < hi) r = adapt_ray(w, K, B, s, lo, ks, __ldg(a.z32 + s), bin);
            if (r == RAY_HIT) atomicOr(mask + bin * words + (i >> 5), 1u << (i & 31u));
            else if (r == RAY_FLAG) list1[atomicAdd(&s_n1, 1u)] = i;
        }
        __syncthreads();
        for (uint32_t q = tid; q < s_n1; q += nthr) {
            const uint32_t i = list1[q], s = __ldg(a.rank + j0 + i);
            const float2 z = __ldg(a.z32 + s);
            uint32_t bin = 0u;
            float t = 0.f;
            int r = RAY_FLAG;
            if (s >= lo && s < hi) r = fast_ray(w.C, w.P, a.guards, z.x, z.y, bin, t);
            if (r == RAY_HIT && t_fixed(t) != tfast) r = RAY_FLAG;  // not the wavelength's transmittance
            if (r == RAY_HIT) atomicOr(mask + bin * words + (i >> 5), 1u << (i & 31u));
            else if (r == RAY_FLAG) list2[atomicAdd(&s_n2, 1u)] = i;
        }
        __syncthreads();
        // what fast_ray leaves, in exact f64; a hit with another transmittance would break the
        // replay's one value, and the wavelength is then left to tp_adaptive_kernel
        bool other = false;
        for (uint32_t q = tid; q < s_n2; q += nthr) {
            const uint32_t i = list2[q];
            uint32_t bin = 0u;
            double t = 0.0;
            if (x::trace(D, lambda, x::beam_y(D, a.z64[j0 + i]), bin, t) == 0) {
                if (t == t64) atomicOr(mask + bin * words + (i >> 5), 1u << (i & 31u));
                else other = true;
            }
        }
        if (__syncthreads_or(other)) {
            if (tid == 0) a.rays_out[il] = 0u;  // no wavelength takes 0 rays: the mark
            return;
        }
        // the bins' updates in ray order, up to the earliest stop
        const auto replay = [&](uint32_t b, bool last) {
            TpBin v = last ? st0[b] : st[b];
            // the hits in ray order; the next one's counts are loaded before the current update
            // (their latency is as long as its chain)
            uint32_t q = 0, m = mask[b * words];
            const auto next = [&]() {
                while (!m && ++q < words) m = mask[b * words + q];
                if (!m) return ~0u;
                const uint32_t i = 32u * q + (uint32_t)__ffs(m) - 1u;
                m &= m - 1u;
                return i;
            };
            uint32_t ni = next();
            double2 tn = make_double2(0.0, 0.0), tc = tn;
            if (ni != ~0u) {
                tn = __ldg(a.cnt + j0 + ni + 1u);
                tc = __ldg(a.cnt + j0 + ni + 2u);
            }
            double c = (double)v.c;
            while (ni != ~0u && ni <= *(volatile uint32_t *)&s_stop) {
                const uint32_t i = ni, n = j0 + i + 1u;  // the ray's number
                const double rn = tn.x, nd = tn.y, rc = tc.x, cd = tc.y;
                ni = next();
                if (ni != ~0u) {
                    tn = __ldg(a.cnt + j0 + ni + 1u);
                    tc = __ldg(a.cnt + j0 + ni + 2u);
                }
                int pass;
                if (full) {
                    if (v.c < n) {  // Welford::skip
                        v.m = x::div_by(x::mul(c, v.m), nd, rn);
                        v.m2 = x::add(v.m2, x::div_by(x::mul(x::mul(x::sqr(v.m), c), x::sub(nd, c)), nd, rn));
                    }
                    // Welford::next_sample: the count becomes the ray's number plus one
                    const double dl = x::sub(t64, v.m);
                    v.m = x::add(v.m, x::div_by(dl, cd, rc));
                    v.m2 = x::add(v.m2, x::mul(dl, x::sub(t64, v.m)));
                    pass = v.m2 < x::mul(x::mul(5e-3, 5e-3), x::mul(cd, nd));  // c (c - 1), c = n + 1
                } else {
                    if (v.c < n) v.m = x::div_by(x::mul(c, v.m), nd, rn);
                    v.m = x::add(v.m, x::div_by(x::sub(t64, v.m), cd, rc));
                    const float nf = (float)n, ir = __fdividef(1.f, nf), kt = (float)v.k * tf * ir, cf = (float)v.c;
                    const float sk = kt * kt * cf * (float)(n - v.c) * ir;
                    const float rest = (float)(n - v.k);
                    const float nx = tf2 * (rest * ir) * __fdividef(rest, nf + 1.f);
                    const ff::F2 e = ff::two_sum(v.f2.x, sk), f = ff::two_sum(e.hi, nx);
                    v.f2.x = f.hi;
                    v.f2.y += e.lo + f.lo;
                    const float m2 = v.f2.x + v.f2.y, lim = 2.5e-5f * ((nf + 1.f) * nf);
                    pass = m2 < lim * (1.f - kTpMargin) ? 1 : m2 > lim * (1.f + kTpMargin) ? 0 : 2;
                }
                c = cd;
                v.c = n + 1u;
                v.k++;
                if (!last && pass) {
                    if (pass == 2) s_open = 1u;
                    atomicMin(&s_stop, i);
                    break;
                }
            }
            st[b] = v;
        };
        for (uint32_t b = tid; b < B; b += nthr) replay(b, false);
        __syncthreads();
        const uint32_t stop = s_stop;
        if (s_open) {
            // a test too close to call: the wavelength again from its first ray, in full
            __syncthreads();
            for (uint32_t b = tid; b < B; b += nthr) st[b] = zero;
            if (tid == 0) s_open = 0u;
            full = true;
            j0 = 0u - C;
            __syncthreads();
            continue;
        }
        if (stop != ~0u) {
            // bins that took a ray past the stop: again from the chunk's start
            for (uint32_t b = tid; b < B; b += nthr)
                if (st[b].c > j0 + stop + 2u) replay(b, true);
            __syncthreads();
            count = j0 + stop + 1u;
            break;
        }
        __syncthreads();
    }
    // every bin padded to the final ray count (the reference's closing skip)
    const double2 fin = a.cnt[count];
    for (uint32_t b = tid; b < B; b += nthr) {
        const TpBin v = st[b];
        a.out[(uint64_t)il * B + b] = v.c < count ? x::div_by(x::mul((double)v.c, v.m), fin.y, fin.x) : v.m;
    }
    if (tid == 0) a.rays_out[il] = count;
}

__global__ void fma_peak_kernel(float *out, uint32_t iters)
{
    float a0 = threadIdx.x * 1e-7f, a1 = a0 + 1e-7f, a2 = a0 + 2e-7f, a3 = a0 + 3e-7f;
    float a4 = a0 + 4e-7f, a5 = a0 + 5e-7f, a6 = a0 + 6e-7f, a7 = a0 + 7e-7f;
    const float b = 0.999999f, c = 1e-7f;
    for (uint32_t i = 0; i < iters; i++) {
#pragma unroll
        for (int u = 0; u < 16; u++) {
            a0 = fmaf(a0, b, c);
            a1 = fmaf(a1, b, c);
            a2 = fmaf(a2, b, c);
            a3 = fmaf(a3, b, c);
            a4 = fmaf(a4, b, c);
            a5 = fmaf(a5, b, c);
            a6 = fmaf(a6, b, c);
            a7 = fmaf(a7, b, c);
        }
    }
    const float s = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
    if (s == 12345.0f) out[blockIdx.x] = s;  // keeps the chains live
}

// SFU throughput probe: eight independent chains of the reciprocal-square-root estimate
// (MUFU.RSQ) per thread; the values stay near 1.
__global__ void mufu_peak_kernel(float *out, uint32_t iters)
{
    float a[8];
#pragma unroll
    for (int k = 0; k < 8; k++) a[k] = 1.0f + 1e-3f * (float)k + 1e-7f * (float)threadIdx.x;
    for (uint32_t i = 0; i < iters; i++) {
#pragma unroll
        for (int u = 0; u < 16; u++)
#pragma unroll
            for (int k = 0; k < 8; k++) asm volatile("rsqrt.approx.ftz.f32 %0, %0;" : "+f"(a[k]));
    }
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 8; k++) s += a[k];
    if (s == 12345.0f) out[blockIdx.x] = s;  // keeps the chains live
}

// ------------------------------------------------------------------ device-resident loop
//
// One CTA evaluates one design at a time, start to finish, with the pass's device code:
// lambda_setup_df per wavelength row, fast_ray over the core rays (lane = wavelength, items
// of 32 rows x a ray chunk claimed from a shared counter), trace_df for the guard-band rays
// of every row and the rays fast_ray flagged, entropy_cell over the W x B cells, then
// finalize_design. Every sum is the same integer as in the pass, so a design's result is
// bitwise its batched result. The CTA then claims the next published ring entry.

constexpr uint32_t kLoopThreads = 256;
#ifndef CPD_LOOP_MIN_BLOCKS
#define CPD_LOOP_MIN_BLOCKS 3
#endif

struct SlabLayout {
    size_t hist, lp, lx, queue, s1, s2, acc, band, bytes;
};

__host__ __device__ inline SlabLayout slab_layout(uint32_t rows, uint32_t cells, uint32_t maxB, uint32_t qcap)
{
    SlabLayout L;
    size_t o = 0;
    L.hist = o;
    o += (8 * (size_t)cells + 255) & ~size_t(255);
    L.lp = o;
    o += (sizeof(LamParams) * (size_t)rows + 255) & ~size_t(255);
    L.lx = o;
    o += (sizeof(LamDF) * (size_t)rows + 255) & ~size_t(255);
    L.queue = o;
    o += (sizeof(QEntry) * (size_t)qcap + 255) & ~size_t(255);
    L.s1 = o;
    o += (8 * (size_t)maxB + 255) & ~size_t(255);
    L.s2 = o;
    o += (8 * (size_t)maxB + 255) & ~size_t(255);
    L.acc = o;
    o += (sizeof(DesignAcc) + 255) & ~size_t(255);
    L.band = o;
    o += (4 * ((size_t)rows + 1) + 255) & ~size_t(255);
    L.bytes = o;
    return L;
}

__device__ __forceinline__ unsigned long long load_acquire_sys(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void store_release_sys(unsigned long long *p, unsigned long long v)
{
    asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// The float-float re-trace of one ray into the CTA's histogram; returns 1 on a hit.
__device__ __noinline__ uint32_t loop_retrace(const DevDesign &D, const LamDF &E, const float *z32, uint32_t j,
                                              unsigned long long *hrow)
{
    uint32_t bin = 0;
    float t = 0.f;
    if (trace_df(D, E, z32[2 * j], z32[2 * j + 1], bin, t)) {
        atomicAdd(hrow + bin, (unsigned long long)t_fixed(t));
        return 1u;
    }
    return 0u;
}

// The loop's per-wavelength setup: rows t, t + nthr, ... (out of line, so that its
// float-float program does not set the register budget of the trace loop).
__device__ __noinline__ void loop_setup(const DevDesign &D, const double *lam, const float *z32, uint32_t Rz, uint32_t W,
                                        LamParams *lp, LamDF *lx, uint32_t t, uint32_t nthr)
{
    for (uint32_t k = t; k < W; k += nthr) {
        LamParams P;
        lambda_setup_df(D, lam[k], z32, Rz, P, kYGuardRel, lx + k, false);
        if (P.all_exact) {
            // no reference ray: every ray of the band is re-traced
            P.core_lo = P.core_hi = 0;
        }
        lp[k] = P;
    }
}

// Counters of one design in the loop (shared memory).
struct LoopTally {
    unsigned long long hits, retraced, fast, H, inl;
    uint32_t item, qn;
};

// The loop's FP32 trace of the core rays by one warp: items of 32 rows x a ray chunk,
// claimed from the shared counter; hits as run-length fixed-point sums into the slab's
// histogram; flagged rays to the slab's queue, or re-traced here when it is full.
__device__ __noinline__ void loop_trace(const DevDesign &D, const LamParams *lp, const LamDF *lx, const float *z32,
                                        uint32_t W, uint32_t B, uint32_t Rz, uint32_t ray_tile,
                                        unsigned long long *hist, QEntry *queue, uint32_t qcap, LoopTally *tally,
                                        uint32_t lane)
{
    const uint32_t nblk = (W + 31u) / 32u;
    const uint32_t nchunk = Rz ? (Rz + ray_tile - 1u) / ray_tile : 1u;
    const uint32_t total = nblk * nchunk;
    // the design's constants in registers (read from shared memory at every use, they cost
    // more than the registers: loop alone 171 -> 172 k designs/s)
    const FastConst C = D.fc;
    const Guards guards = default_guards();
    const FastLimits Lm = fast_limits(C, guards);
    for (;;) {
        uint32_t item = 0;
        if (lane == 0) item = atomicAdd(&tally->item, 1u);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= total) break;
        const uint32_t blk = item / nchunk, chunk = item - blk * nchunk;
        const uint32_t k = blk * 32u + lane;
        LamParams P;
        uint32_t lo = 0, hi = 0;
        if (k < W) {
            P = lp[k];
            const uint32_t j0 = chunk * ray_tile;
            const uint32_t j1 = min(j0 + ray_tile, Rz);
            lo = max(j0, P.core_lo);
            hi = min(j1, P.core_hi);
        }
        const float2 *__restrict__ zt = reinterpret_cast<const float2 *>(z32);
        unsigned long long *hrow = hist + (uint64_t)k * B;
        uint32_t cur = 0xffffffffu;
        unsigned long long sum = 0ull;
        uint32_t nhit = 0, ninl = 0;
        for (uint32_t j = lo; j < hi; ++j) {
            const float2 z = __ldg(zt + j);
            uint32_t bin = 0;
            float tt = 0.f;
            const int r = fast_ray(C, Lm, P, guards, z.x, z.y, bin, tt);
            if (r == RAY_HIT) {
                if (bin != cur) {
                    if (sum) atomicAdd(hrow + cur, sum);
                    cur = bin;
                    sum = 0ull;
                }
                sum += t_fixed(tt);
                nhit++;
            } else if (r == RAY_FLAG) {
                const uint32_t pos = atomicAdd(&tally->qn, 1u);
                if (pos < qcap) {
                    queue[pos] = QEntry{0u, k, j, 0u};
                } else {
                    // the queue is full: re-trace here (counted as re-traced, as queued)
                    nhit += loop_retrace(D, lx[k], z32, j, hrow);
                    ninl++;
                }
            }
        }
        if (sum) atomicAdd(hrow + cur, sum);
        nhit = __reduce_add_sync(0xffffffffu, nhit);
        ninl = __reduce_add_sync(0xffffffffu, ninl);
        const uint32_t nfast = __reduce_add_sync(0xffffffffu, hi > lo ? hi - lo : 0u);
        if (lane == 0) {
            if (nhit) atomicAdd(&tally->hits, (unsigned long long)nhit);
            if (nfast) atomicAdd(&tally->fast, (unsigned long long)nfast);
            if (ninl) {
                atomicAdd(&tally->retraced, (unsigned long long)ninl);
                atomicAdd(&tally->inl, (unsigned long long)ninl);
            }
        }
    }
}

__global__ void __launch_bounds__(kLoopThreads, CPD_LOOP_MIN_BLOCKS) loop_kernel(const LoopArgs L)
{
    __shared__ __align__(16) LoopWork sW;
    DevDesign &sD = sW.d;
    DesignJob &sJ = sW.j;
    __shared__ float tab[4 * ff::kLogTable];
    __shared__ FinalizeRed fin_red[kLoopThreads / 32];
    __shared__ unsigned long long s_idx;
    __shared__ LoopTally tally;
    extern __shared__ __align__(16) unsigned long long loop_smem[];  // per-bin s1, s2 (max_B each)
    const uint32_t t = threadIdx.x, lane = t & 31u;
    for (uint32_t i = t; i < 4u * ff::kLogTable; i += blockDim.x) tab[i] = L.logtab[i];
    const SlabLayout SL = slab_layout(L.max_rows, L.max_cells, L.max_B, L.qcap);
    unsigned char *slab = L.slabs + (size_t)blockIdx.x * L.slab_bytes;
    unsigned long long *hist = reinterpret_cast<unsigned long long *>(slab + SL.hist);
    LamParams *lp = reinterpret_cast<LamParams *>(slab + SL.lp);
    LamDF *lx = reinterpret_cast<LamDF *>(slab + SL.lx);
    QEntry *queue = reinterpret_cast<QEntry *>(slab + SL.queue);
    unsigned long long *S1 = reinterpret_cast<unsigned long long *>(slab + SL.s1);
    unsigned long long *S2 = reinterpret_cast<unsigned long long *>(slab + SL.s2);
    DesignAcc *acc = reinterpret_cast<DesignAcc *>(slab + SL.acc);
    uint32_t *band = reinterpret_cast<uint32_t *>(slab + SL.band);  // exclusive prefix of band rays per row
    unsigned long long *s1 = loop_smem, *s2 = loop_smem + L.max_B;
    __shared__ uint32_t s_part[kLoopThreads];
    // the idle wait: bounded in time and in polls (a poll sleeps about a microsecond)
    const unsigned long long max_polls = L.idle_ns / 500ull + 1000ull;
    unsigned long long idle_start = global_ns();
    for (;;) {
        // ---- claim the next published ring entry, or leave after the idle limit
        if (t == 0) {
            unsigned long long got = ~0ull;
            for (unsigned long long polls = 0;; polls++) {
                const unsigned long long pub = load_acquire_sys(&L.ctl->published);
                const unsigned long long n = *reinterpret_cast<volatile unsigned long long *>(&L.cnt->claimed);
                if (n < pub) {
                    if (atomicCAS(&L.cnt->claimed, n, n + 1ull) == n) {
                        got = n;
                        break;
                    }
                    continue;
                }
                if (*reinterpret_cast<volatile unsigned int *>(&L.ctl->stop)) {
                    atomicAdd(&L.cnt->stop_exits, 1u);
                    break;
                }
                if (polls >= max_polls || global_ns() - idle_start > L.idle_ns) {
                    atomicAdd(&L.cnt->idle_exits, 1u);
                    break;
                }
                __nanosleep(1000);
            }
            s_idx = got;
            tally = LoopTally{0ull, 0ull, 0ull, 0ull, 0ull, 0u, 0u};
        }
        __syncthreads();
        const unsigned long long idx = s_idx;
        if (idx == ~0ull) break;
        const uint32_t slot = (uint32_t)(idx % L.capacity);
        {
            // the record (after thread 0's acquire of `published` and the barrier), in 16-byte
            // words from mapped host memory
            const uint4 *src = reinterpret_cast<const uint4 *>(&L.ring[slot]);
            uint4 *dst = reinterpret_cast<uint4 *>(&sW);
            for (uint32_t i = t; i < sizeof(LoopWork) / 16; i += blockDim.x) dst[i] = __ldcv(src + i);
        }
        unsigned long long *accw = reinterpret_cast<unsigned long long *>(acc);
        for (uint32_t i = t; i < sizeof(DesignAcc) / 8; i += blockDim.x) accw[i] = 0ull;
        __syncthreads();
        const uint32_t W = sJ.W, B = sJ.B, Rz = sJ.Rz, ray_tile = sW.ray_tile;
        const float *z32 = L.z32 + 2 * sJ.ray_off;
        for (uint32_t b = t; b < B; b += blockDim.x) s1[b] = s2[b] = 0ull;

        // ---- per-wavelength setup
        loop_setup(sD, L.lam + sJ.lam_off, z32, Rz, W, lp, lx, t, blockDim.x);
        __syncthreads();

        // ---- FP32 trace of the core rays
        loop_trace(sD, lp, lx, z32, W, B, Rz, ray_tile, hist, queue, L.qcap, &tally, lane);
        __syncthreads();

        // ---- float-float re-trace of every row's guard bands, spread over all threads (an
        // exclusive prefix sum of the rows' band rays: rows differ widely), then the queue
        {
            // per thread: a contiguous run of rows; its band rays, then a scan over threads
            const uint32_t per = (W + blockDim.x - 1u) / blockDim.x;
            const uint32_t k0 = min(t * per, W), k1 = min(k0 + per, W);
            uint32_t run = 0;
            for (uint32_t k = k0; k < k1; k++) {
                const LamParams &P = lp[k];
                band[k] = run;
                run += P.all_exact ? P.band_hi - P.band_lo : (P.core_lo - P.band_lo) + (P.band_hi - P.core_hi);
            }
            s_part[t] = run;
            __syncthreads();
            if (t == 0) {
                uint32_t acc_n = 0;
                for (uint32_t i = 0; i < blockDim.x; i++) {
                    const uint32_t v = s_part[i];
                    s_part[i] = acc_n;
                    acc_n += v;
                }
                band[W] = acc_n;
            }
            __syncthreads();
            for (uint32_t k = k0; k < k1; k++) band[k] += s_part[t];
            __syncthreads();
        }
        {
            unsigned long long hits = 0ull, ret = 0ull;
            const uint32_t nband = band[W];
            for (uint32_t i = t; i < nband; i += blockDim.x) {
                // the row holding band ray i: the last k with band[k] <= i
                uint32_t lo = 0, hi = W;
                while (hi - lo > 1u) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (band[mid] <= i) lo = mid;
                    else hi = mid;
                }
                const uint32_t k = lo, r = i - band[k];
                const LamParams &P = lp[k];
                const uint32_t na = P.all_exact ? P.band_hi - P.band_lo : P.core_lo - P.band_lo;
                const uint32_t j = r < na ? P.band_lo + r : P.core_hi + (r - na);
                hits += loop_retrace(sD, lx[k], z32, j, hist + (uint64_t)k * B);
                ret++;
            }
            const uint32_t qn = min(tally.qn, L.qcap);
            for (uint32_t i = t; i < qn; i += blockDim.x) {
                const QEntry e = queue[i];
                hits += loop_retrace(sD, lx[e.k], z32, e.j, hist + (uint64_t)e.k * B);
                ret++;
            }
            hits = warp_sum_u64(hits);
            ret = warp_sum_u64(ret);
            if (lane == 0) {
                if (hits) atomicAdd(&tally.hits, hits);
                if (ret) atomicAdd(&tally.retraced, ret);
            }
        }
        __syncthreads();

        // ---- entropy over the W x B cells; each nonzero cell is cleared for the next design
        {
            const ff::F2 unit{sJ.unit_hi, sJ.unit_lo}, lu{sJ.lu_hi, sJ.lu_lo};
            const uint32_t cells = W * B;
            unsigned long long hl = 0ull;
            for (uint32_t i = t; i < cells; i += blockDim.x) {
                const unsigned long long cv = hist[i];
                if (cv) {
                    hist[i] = 0ull;
                    unsigned long long hq, pq;
                    entropy_cell(cv, unit, lu, tab, hq, pq);
                    hl += hq;
                    const uint32_t b = i % B;
                    atomicAdd(s1 + b, cv);
                    atomicAdd(s2 + b, pq);
                }
            }
            hl = warp_sum_u64(hl);
            if (lane == 0 && hl) atomicAdd(&tally.H, hl);
        }
        __syncthreads();
        for (uint32_t b = t; b < B; b += blockDim.x) {
            S1[b] = s1[b];
            S2[b] = s2[b];
        }
        if (t == 0) {
            acc->H = tally.H;
            acc->rows = 0ull;
            acc->hits[0] = tally.hits;
            acc->retraced[0] = tally.retraced;
            acc->fast[0] = tally.fast;
            if (tally.inl) atomicAdd(&L.cnt->inline_retraced, tally.inl);
        }
        __syncthreads();

        // ---- finalize into the ring entry's result slot (mapped host memory)
        {
            LaunchArgs a;
            memset(&a, 0, sizeof(a));
            a.designs = &sD;
            a.acc = acc;
            a.S1 = S1;
            a.S2 = S2;
            a.out = &L.done[slot].o;
            DesignJob J = sJ;
            J.acc_off = 0;
            finalize_design(a, 0u, J, t, blockDim.x, tab, fin_red);
        }
        __syncthreads();
        if (t == 0) {
            L.done[slot].status = 0u;
            __threadfence_system();
            store_release_sys(&L.done[slot].seq, idx + 1ull);
            atomicAdd(&L.cnt->designs, 1ull);
        }
        idle_start = global_ns();
    }
}

}  // namespace

// A launch that, with `pdl`, may start before the previous kernel on the stream has
// finished (programmatic dependent launch): the kernel waits for its predecessor's
// results in cudaGridDependencySynchronize.
template <class Args>
void launch_k(void (*k)(const Args), dim3 grid, unsigned block, size_t smem, cudaStream_t st, bool pdl, const Args &a)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = pdl ? attr : nullptr;
    cfg.numAttrs = pdl ? 1 : 0;
    cudaLaunchKernelEx(&cfg, k, a);
}

// Resident blocks of rows_kernel per SM for blocks of `warps` warps and detectors of up to B
// bins (asked once each: the answer depends on the block and its shared memory alone).
static uint32_t rows_blocks_per_sm(uint32_t warps, uint32_t B)
{
    static std::atomic<uint8_t> known[3][CPD_MAX_BINS + 1];
    std::atomic<uint8_t> &k = known[warps <= kRowsWarps ? 0 : warps <= 8u ? 1 : 2][B];
    uint32_t n = k.load(std::memory_order_relaxed);
    if (!n) {
        // one-warp teams need the most shared memory of a kRowsWarps block
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, rows_kernel<false, false, false>, 32 * warps,
                                                      rows_smem_bytes(warps, warps <= kRowsWarps ? warps : 1u, B));
        n = per_sm < 1 ? 1u : (uint32_t)per_sm;
        k.store((uint8_t)n, std::memory_order_relaxed);
    }
    return n;
}

RowsPlan plan_rows(uint64_t rows, uint32_t R, uint32_t max_B, int num_sms)
{
    RowsPlan p;
    // Several warps per row while all teams are resident at once (4096 rows of 1024 rays by teams of
    // two, in three waves: 69 us a call instead of 52), and each half-warp's share of the row is up
    // to 64 rays (mostly fast_ray's, whole) or 256 and more: between, its 15 pieces are so short
    // that a bin's edges cost more than its rays. 512 rows of 1024 rays (a call, four designs): 128
    // rays 45.6 us, 256 rays 42.0; 128 rows of 4096: 128 rays 44.3, 256 rays 41.8; but 256 rows of
    // 1024: 64 rays 40.6, 256 rays 41.7; 128 rows of 2048: 40.3, 41.1.
    p.team = 1u;
    for (uint32_t T = 2u; T <= kRowsMaxTeam && R >= 64u * T; T *= 2u) {
        if (R > 2u * T * 64u && R < 2u * T * 256u) continue;
        const uint32_t warps = std::max(kRowsWarps, T);
        if (rows <= (uint64_t)num_sms * rows_blocks_per_sm(warps, max_B) * (warps / T)) p.team = T;
    }
    // two rows or more per warp once every warp has one
    const uint64_t resident = (uint64_t)num_sms * rows_blocks_per_sm(kRowsWarps, max_B) * kRowsWarps;
    p.group = rows <= resident ? 1u : (uint32_t)std::min<uint64_t>(kRowsGroup, std::max<uint64_t>(2u, rows / resident));
    return p;
}

// Both kinds of rows in one launch, for passes of few rows that have some of each: a kernel for each
// kind stands one behind the other in the pass's chain, and the second waits for the slowest row of the
// first. A coated and an uncoated design of 128 rows x 4096 rays 125 -> 106 us, four of each 218 -> 176
// (both forms inlined: 108 and 181, the kernel spills).
__device__ __noinline__ int adaptive_mixed_redo(const LaunchArgs &a, unsigned long long *smem)
{
    return adaptive_row<true, ROWS_MIXED>(a, blockIdx.x, smem, blockDim.x >> 5, threadIdx.x >> 5, threadIdx.x & 31u);
}
__global__ void __launch_bounds__(32 * kMaxAdaptWarps, CPD_ADAPT_MIN_BLOCKS) adaptive_mixed_kernel(const LaunchArgs a)
{
    extern __shared__ __align__(16) unsigned long long adapt_smem[];
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();  // the setup's LamParams and LamDF
    const uint32_t kw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    int r = adaptive_row<false, ROWS_MIXED>(a, blockIdx.x, adapt_smem, kw, warp, lane);
    if (r == ROW_UNSURE) r = adaptive_mixed_redo(a, adapt_smem);
    if (r == ROW_OTHER && threadIdx.x == 0) queue_row(a, blockIdx.x);
}

// Whether the rows of designs with pieces go through adaptive_block_kernel (true) or
// adaptive_equal_kernel, in adaptive passes of fewer than 8 rows per SM. The first bins by pieces, but
// tests every bin of every round; the second traces ray by ray, 16 (4) rounds at a time, and tests
// the bins that a round hit. So the first is for long tables and narrow detectors. Calls in us, first /
// second (three designs each; over 4032 sizes of up to 1024 bins and 1200 rows the lines below are within
// 0.3 % of the faster of the two on average):
//   up to 2 rows per SM, 100 rows: 64 bins x 300 rays 47 / 46, x 1024 49 / 50, x 4096 59 / 75; 256 bins
//     x 2048 61 / 61, x 4096 78 / 80; 800 bins x 1024 64 / 53, x 16384 264 / 163: a round costs the first
//     more with more bins, and a group of 16 rounds the second hardly more than one;
//   up to 4, 472 rows: as long as all blocks are resident, 200 bins x 4096 112 / 130, x 8192 (4 rows on
//     some SM, room for 3) 222 / 206; 512 bins x 8192 314 / 243;
//   beyond, 900 rows: 64 bins x 300 55 / 53, x 8192 158 / 214; 128 x 16384 315 / 321; 160 x 16384 366 / 259;
//     512 x 8192 463 / 292: rows wait for a place, and of blocks of the second twice as many fit.
static bool adapt_by_blocks(uint32_t max_B, uint64_t rows, uint32_t max_rounds, int num_sms)
{
    const uint64_t per_sm = rows / (uint64_t)num_sms, setup = (rows + 31u) / 32u;  // setup: its blocks
    const size_t bytes = adapt_block_smem_bytes(max_B, max_rounds);
    // Beside a setup block an SM has no room for arrays of 50 KB: from 148 rows on two rows share an SM,
    // though there is one for each. 236 bins x 16384, 147 rows 156 / 165, 148 rows 193 / 165
    if (rows <= (uint64_t)num_sms && rows + setup > (uint64_t)num_sms && bytes > 50u * 1024u) return false;
    if (per_sm < 2) return max_B <= 256u && max_rounds > 20u + max_B / 4u;
    if (per_sm >= 4) return max_B <= 128u && max_rounds >= 24u && max_rounds * max_B <= 65536u;
    // (blocks of 8 warps at 64 registers: four)
    const uint64_t room = std::min<uint64_t>(4u, (227u * 1024u) / (bytes + 1024u));
    return max_B <= 400u && max_rounds >= 16u && rows <= room * (uint64_t)num_sms;
}

int launch_pass(const LaunchArgs &a, int num_sms, uint32_t warps_per_cta, cudaStream_t stream, cudaEvent_t *ev,
                bool pdl)
{
    // per-kernel events would stand between the kernels
    pdl = pdl && ev == nullptr;
    int launches = 0;
    if (ev) cudaEventRecord(ev[0], stream);
    if (a.ntables) {
        uint32_t M = 1024u;
        while (M < a.table_max) M <<= 1;
        if (a.nsort) {
            launch_k(table_sort_kernel, a.nsort, kTableThreads, table_smem_bytes(M, a.table_max), stream, false, a);
            launches++;
        }
        launch_k(table_z_kernel, dim3(a.ntables, (a.table_max + 63u) / 64u), 64, 0, stream, pdl && a.nsort, a);
        launches++;
    }
    if (a.params) {
        launch_k(build_kernel, (a.njobs + kBuildPerWarp - 1u) / kBuildPerWarp, 32, 0, stream, false, a);
        launches++;
    }
    if (a.total_rows) {
        // 16 warps or more per SM: larger blocks; fewer: each row is one thread's latency-bound
        // float-float chain, so spreading the rows over every SM matters. A single-design pass
        // (spans) splits each row's chain over two warps.
        const uint32_t rows = !a.spans && a.total_rows >= (uint64_t)num_sms * 32u * 16u ? kSetupThreads : 32u;
        const uint32_t blocks = (uint32_t)((a.total_rows + rows - 1u) / rows);
        const uint32_t cap = a.stage_cap < kStageRays ? a.stage_cap : kStageRays;
        launch_k(a.spans ? setup_pair_kernel : a.stamp == STAMP_SETUP ? setup_kernel<true> : setup_kernel<false>, blocks, a.spans ? 64 : rows,
                 2 * ((cap + 1u) & ~1u) * sizeof(float), stream, pdl && a.ntables && !a.params, a);
        launches++;
    }
    if (a.adaptive) {
        const uint32_t maxB = a.max_B ? a.max_B : (uint32_t)CPD_MAX_BINS;
        if (ev) cudaEventRecord(ev[1], stream);
        if (a.total_rows) {
            // enough rows to fill the GPU: few warps per row (rounds traced past a row's
            // stop are wasted); fewer rows: up to kMaxAdaptWarps warps per row trace and
            // decide that many rounds at once
            const uint64_t per_sm = a.total_rows / (uint64_t)num_sms;
            const uint32_t kw = per_sm >= 8 ? CPD_ADAPT_KW_MANY : per_sm >= 2 ? CPD_ADAPT_KW_SOME : kMaxAdaptWarps;
            if (kw == 1u) {
                const size_t smem = adapt1p_smem_bytes(maxB);
                launch_k(a.adapt_pieces ? adaptive1_pieces_kernel : adaptive1_kernel, (unsigned)a.total_rows, 32,
                         a.adapt_pieces == 1u ? smem : std::max(smem, adapt1_smem_bytes(maxB)), stream, pdl, a);
                launches++;
            } else {
                if (a.adapt_pieces == 3u) {
                    launch_k(adaptive_mixed_kernel, (unsigned)a.total_rows, 32 * kw, adapt_smem_bytes(kw, maxB), stream, pdl, a);
                    launches++;
                } else if (a.adapt_pieces && !adapt_by_blocks(maxB, a.total_rows, a.max_rounds, num_sms)) {
                    launch_k(adaptive_equal_kernel, (unsigned)a.total_rows, 32 * kw, adapt_smem_bytes(kw, maxB), stream, pdl, a);
                    launches++;
                } else if (a.adapt_pieces) {
                    // 2 to 7 rows per SM: 8 warps, four such blocks per SM; 4 warps where more rows
                    // than that have few rounds. Calls, 16 / 8 / 4 warps: 472 x 602 rays in 100 bins 57 /
                    // 52 / 55 us, 472 x 4096 in 200 119 / 103 / 135, 1000 x 8192 in 64 174 / 161 / 181,
                    // 700 x 1024 in 64 66 / 61 / 57, 1200 x 1024 in 100 92 / 75 / 67
                    const uint32_t kb = kw == kMaxAdaptWarps ? kw : per_sm >= 4 && a.max_rounds <= 32u ? 4u : 8u;
                    launch_k(adaptive_block_kernel, (unsigned)a.total_rows, 32 * kb,
                             adapt_block_smem_bytes(maxB, a.max_rounds), stream, pdl, a);
                    launches++;
                }
                if (a.adapt_pieces == 0u || a.adapt_pieces == 2u) {
                    launch_k(adaptive_kernel, (unsigned)a.total_rows, 32 * kw, adapt_smem_bytes(kw, maxB), stream, pdl, a);
                    launches++;
                }
            }
        }
        if (ev) cudaEventRecord(ev[2], stream);
        const uint32_t kwe = a.total_rows / (uint64_t)num_sms >= 8 ? 1u : kMaxAdaptWarps;
        launch_k(adaptive_exact_kernel, (unsigned)(num_sms * (kwe == 1u ? 8 : 1)), 32 * kwe,
                 kwe == 1u ? adapt1_smem_bytes(maxB) : adapt_smem_bytes(kwe, maxB), stream, pdl, a);
        launches++;
    } else {
    if (ev) cudaEventRecord(ev[1], stream);
    if (a.total_groups) {
        const uint32_t warps = std::max(kRowsWarps, a.team), teams = warps / a.team;
        const uint64_t need = (a.total_groups + teams - 1u) / teams;
        const uint64_t resident = (uint64_t)num_sms * rows_blocks_per_sm(warps, a.max_B);
        if (a.heavy) {
            launch_k(a.p_out ? rows_kernel<false, true, true> : rows_kernel<false, false, true>, (unsigned)num_sms,
                     32 * kRowsMaxTeam, rows_smem_bytes(kRowsMaxTeam, 1u, a.max_B), stream, pdl, a);
            launches++;
        }
        auto k = a.spans ? (a.p_out ? rows_kernel<true, true, false> : rows_kernel<true, false, false>)
                         : (a.p_out ? rows_kernel<false, true, false> : rows_kernel<false, false, false>);
        launch_k(k, (unsigned)std::min(need, resident), 32 * warps, rows_smem_bytes(warps, teams, a.max_B), stream, pdl, a);
        launches++;
    }
    if (a.mode != CPD_TRACE_FP64 && a.total_items) {
        int per_sm = 0;
        const int threads = (int)warps_per_cta * 32;
        auto k = a.spans ? trace_spans_kernel : trace_kernel;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, threads, 0);
        if (per_sm < 1) per_sm = 1;
        uint64_t grid = (uint64_t)num_sms * per_sm;
        // equal shares: every resident warp; work items: no more warps than items
        const uint64_t need = (a.total_items + warps_per_cta - 1) / warps_per_cta;
        if (!a.spans && grid > need) grid = need;
        launch_k(k, (unsigned)grid, threads, 0, stream, pdl, a);
        launches++;
    }
    if (ev) cudaEventRecord(ev[2], stream);
    // the single-design trace re-traces its own flagged rays; what reaches the queue there
    // (the setup's guard bands, a warp's flags past kWarpFlags) is usually little, and a
    // grid of one block per SM is resident beside the trace, ready when it completes
    if (a.total_items) {
        launch_k(a.mode == CPD_TRACE_FP64 ? retrace_exact_kernel : retrace_kernel,
                 (unsigned)(num_sms * (a.spans ? 1 : 8)), 32, 0, stream, pdl, a);
        launches++;
    }
    }
    if (ev) cudaEventRecord(ev[3], stream);
    if (a.total_tiles) {
        const uint64_t wpb = (uint64_t)kEntropyThreads / 32u;
        if (a.total_tiles <= (uint64_t)num_sms * wpb) {
            // few tiles: one block per tile
            const size_t smem = 2u * sizeof(unsigned long long) * (a.max_B ? a.max_B : (uint32_t)CPD_MAX_BINS);
            int per_sm = 0;
            auto k = a.p_out ? entropy_block_kernel<true> : entropy_block_kernel<false>;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kEntropyThreads, smem);
            if (per_sm < 1) per_sm = 1;
            uint64_t grid = a.total_tiles;
            if (grid > (uint64_t)num_sms * per_sm) grid = (uint64_t)num_sms * per_sm;
            launch_k(k, (unsigned)grid, kEntropyThreads, smem, stream, pdl, a);
        } else {
            // one warp per tile, as many blocks as are resident at once
            int per_sm = 0;
            auto k = a.p_out ? entropy_warp_kernel<true> : entropy_warp_kernel<false>;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kEntropyThreads, 0);
            if (per_sm < 1) per_sm = 1;
            uint64_t grid = (a.total_tiles + wpb - 1) / wpb;
            if (grid > (uint64_t)num_sms * per_sm) grid = (uint64_t)num_sms * per_sm;
            launch_k(k, (unsigned)grid, kEntropyThreads, 0, stream, pdl, a);
        }
        launches++;
    }
    if (a.njobs > 1 || (!a.total_tiles && !(a.spans && a.total_groups))) {
        launch_k(finalize_kernel, (a.njobs + 3u) / 4u, 128, 0, stream, pdl, a);
        launches++;
    }
    if (ev) cudaEventRecord(ev[4], stream);
    return launches;
}

cudaError_t configure_kernels()
{
    const int bytes = (int)adapt_smem_bytes(kMaxAdaptWarps, CPD_MAX_BINS);
    cudaError_t e = cudaFuncSetAttribute(adaptive_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(adaptive_equal_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(adaptive_mixed_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(adaptive1_pieces_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)std::max(adapt1_smem_bytes(CPD_MAX_BINS), adapt1p_smem_bytes(CPD_MAX_BINS)));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(adaptive1_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)std::max(adapt1_smem_bytes(CPD_MAX_BINS), adapt1p_smem_bytes(CPD_MAX_BINS)));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(adaptive_exact_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    size_t block_bytes = 0;
    for (uint32_t B = 1; B <= CPD_MAX_BINS; B++) block_bytes = std::max(block_bytes, adapt_block_smem_bytes(B));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(adaptive_block_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)block_bytes);
    size_t tp_bytes = 0;
    for (uint32_t B = 1; B <= CPD_MAX_BINS; B++) tp_bytes = std::max(tp_bytes, tp_pieces_smem_bytes(B));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(tp_pieces_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tp_bytes);
    const int rows_bytes = (int)std::max(rows_smem_bytes(kRowsWarps, kRowsWarps, CPD_MAX_BINS),
                                         rows_smem_bytes(kRowsMaxTeam, 1u, CPD_MAX_BINS));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(table_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)table_smem_bytes(kTableRays, kTableRays));
    const auto rows = {rows_kernel<false, false, false>, rows_kernel<false, true, false>, rows_kernel<true, false, false>,
                       rows_kernel<true, true, false>, rows_kernel<false, false, true>, rows_kernel<false, true, true>};
    for (auto k : rows)
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, rows_bytes);
    return e;
}

const void *single_trace_kernel_fn(const LaunchArgs &a)
{
    if (!a.total_groups) return reinterpret_cast<const void *>(trace_spans_kernel);
    return a.p_out ? reinterpret_cast<const void *>(rows_kernel<true, true, false>)
                   : reinterpret_cast<const void *>(rows_kernel<true, false, false>);
}

uint64_t trace_resident_warps(int num_sms, uint32_t warps_per_cta)
{
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, trace_kernel, (int)warps_per_cta * 32, 0);
    if (per_sm < 1) per_sm = 1;
    return (uint64_t)num_sms * (uint64_t)per_sm * warps_per_cta;
}

void launch_build_records(const cpd_spectrometer_params *p, uint32_t n, double acceptance, cpd_design *out,
                          int32_t *status, cudaStream_t stream)
{
    if (!n) return;
    build_records_kernel<<<(n + kBuildPerWarp - 1u) / kBuildPerWarp, 32, 0, stream>>>(p, n, acceptance, out, status);
}

void launch_trace_pairs(const DevDesign *d, const double *lam_u, const double *z64, uint32_t n, uint32_t mode,
                        uint32_t *bins, double *ts, uint8_t *flags, cudaStream_t stream)
{
    if (!n) return;
    trace_pairs_kernel<<<(n + 127) / 128, 128, 0, stream>>>(d, lam_u, z64, n, mode, bins, ts, flags);
}

void launch_tp_adaptive(const DevDesign *d, uint32_t B, const double *lambdas, uint32_t n, const double *z64,
                        uint32_t max_m, double *out, uint32_t *rays_out, bool left_only, cudaStream_t stream)
{
    if (!n) return;
    tp_adaptive_kernel<<<n, kTpRays, 3 * sizeof(double) * B, stream>>>(d, lambdas, z64, max_m, out, rays_out, left_only);
}

void launch_tp_pieces(const TpArgs &a, uint32_t B, cudaStream_t stream)
{
    if (!a.n) return;
    tp_setup_kernel<<<(a.n + 31) / 32, 64, 0, stream>>>(a);
    launch_k(tp_pieces_kernel, a.n, 256, tp_pieces_smem_bytes(B), stream, true, a);
}

void launch_mufu_peak(float *out, uint32_t iters, int blocks, int threads, cudaStream_t stream)
{
    mufu_peak_kernel<<<blocks, threads, 0, stream>>>(out, iters);
}

size_t loop_slab_bytes(uint32_t max_rows, uint32_t max_cells, uint32_t max_B, uint32_t qcap)
{
    return slab_layout(max_rows, max_cells, max_B, qcap).bytes;
}

void launch_loop(const LoopArgs &a, uint32_t grid, cudaStream_t stream)
{
    loop_kernel<<<grid, kLoopThreads, 2 * sizeof(unsigned long long) * a.max_B, stream>>>(a);
}

int loop_ctas_per_sm()
{
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, loop_kernel, kLoopThreads,
                                                  2 * sizeof(unsigned long long) * CPD_MAX_BINS);
    return per_sm < 1 ? 1 : per_sm;
}

void launch_fma_peak(float *out, uint32_t iters, int blocks, int threads, cudaStream_t stream)
{
    fma_peak_kernel<<<blocks, threads, 0, stream>>>(out, iters);
}

}  // namespace cpd
