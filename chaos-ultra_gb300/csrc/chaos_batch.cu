// chaos_batch.cu -- many viewports of uneven size and iteration limit in one
// CUDA-graph launch.
//
// Each viewport is rendered at a precision tier chosen from its pixel size
// (binary32, float-float or binary64).  Per tier one persistent kernel serves
// all of that tier's viewports from a single job space (job = one pixel with
// its samples; a lane maps its job to a viewport by binary search over the
// viewports' job offsets held in shared memory).  The three kernels sit in one
// fork-join CUDA graph, so the tail of one tier's kernel overlaps the next.
// The escape loop is the frame path's: blocks of K untested steps, and a lane
// whose block overshot an escape halves its search window inside the warp's
// regular blocks.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/chaos_gb300.h"
#include "chaos_frame.cuh"
#include "chaos_trace.h"

namespace chaos {

int api_fail(int code, const char *fmt, ...);  // chaos_api.cu
bool api_budget(double seconds, unsigned long long *ns);
int api_orbit_create_d(double center_x, double center_y, uint32_t bits, uint32_t max_iterations,
                       chaos_orbit **out);  // chaos_perturb.cu
int api_perturb_enqueue(const chaos_frame_desc *desc, const chaos_orbit *orbit, const chaos_frame_out *out,
                        cudaStream_t stream, uint32_t *counter);  // chaos_perturb.cu

struct BatchViewport {
    uint32_t w, h, spp, mode, max_iter;
    uint32_t job_base;  // first job of this viewport in its tier's job space
    uint32_t w_magic;   // div_magic(w)
    uint64_t seed;
    double center_x, center_y, ps;
    uint32_t *counts;
    float *smooth;
    uint32_t *rgba;
};

struct BatchArgs {
    const BatchViewport *vps;
    uint32_t n_vp, n_jobs;
    uint32_t chunk;  // consecutive jobs a lane claims per work-counter update
    uint32_t *counter;
    unsigned long long *total;  // [0] pixel-iterations, [1] iterations proven interior (by c or a repeated state), not run
    const uint32_t *palette;
    uint32_t palette_len;
    uint32_t interior_rgba;
    unsigned long long budget_ns;  // 0, or the run time after which warps stop (RUN_STATUS_TIMEOUT into *status)
    uint32_t *status;
};

// Number policies: binary32, binary64 (fused multiply-adds) and float-float.
template <class N> struct Num;
template <> struct Num<float> {
    using T = float;
    static __device__ __forceinline__ T from(double d) { return (float)d; }
    static __device__ __forceinline__ T zero() { return 0.f; }
    static __device__ __forceinline__ void step(T &x, T &y, T cx, T cy) { chaos::step<float, ARITH_FMA>(x, y, cx, cy); }
    static __device__ __forceinline__ float r2(T x, T y) { return radius2<float, ARITH_FMA>(x, y); }
    static __device__ __forceinline__ bool below(T x, T y) { return below_four<ARITH_FMA>(x, y); }
    static __device__ __forceinline__ bool blockable(T cx, T cy) { return blockable_c(cx, cy); }
    static __device__ __forceinline__ bool interior(T cx, T cy) { return interior_c(cx, cy); }
};
template <> struct Num<double> {
    using T = double;
    static __device__ __forceinline__ T from(double d) { return d; }
    static __device__ __forceinline__ T zero() { return 0.0; }
    static __device__ __forceinline__ void step(T &x, T &y, T cx, T cy) { chaos::step<double, ARITH_FMA>(x, y, cx, cy); }
    static __device__ __forceinline__ double r2(T x, T y) { return radius2<double, ARITH_FMA>(x, y); }
    static __device__ __forceinline__ bool below(T x, T y) { return below_four<ARITH_FMA>(x, y); }
    static __device__ __forceinline__ bool blockable(T cx, T cy) { return blockable_c(cx, cy); }
    static __device__ __forceinline__ bool interior(T cx, T cy) { return interior_c(cx, cy); }
};
template <> struct Num<FF> {
    using T = FF;
    static __device__ __forceinline__ T from(double d) { return ff_from_double(d); }
    static __device__ __forceinline__ T zero() { return FF{0.f, 0.f}; }
    static __device__ __forceinline__ void step(T &x, T &y, T cx, T cy) { ff_step(x, y, cx, cy); }
    static __device__ __forceinline__ float r2(T x, T y) { return ff_radius2(x, y); }
    static __device__ __forceinline__ bool blockable(T cx, T cy) { return blockable_c(cx.hi, cy.hi); }
    static __device__ __forceinline__ bool interior(T cx, T cy) { return interior_c(cx.hi, cy.hi); }
};

// Binary64 with the reference's rounding (tier CHAOS_TIER_F64_ROUNDED): the
// rounded step of the frame path, five binary64 operations with x*x - y*y on
// the integer units, redone with the literal step when its checks ask for it.
struct R64 {};
template <> struct Num<R64> {
    using T = double;
    static __device__ __forceinline__ T from(double d) { return d; }
    static __device__ __forceinline__ T zero() { return 0.0; }
    static __device__ __forceinline__ void step(T &x, T &y, T cx, T cy)
    {
        chaos::step<double, ARITH_PARITY>(x, y, cx, cy);
    }
    static __device__ __forceinline__ double r2(T x, T y) { return radius2<double, ARITH_PARITY>(x, y); }
    static __device__ __forceinline__ bool below(T x, T y) { return below_four<ARITH_PARITY>(x, y); }
    static __device__ __forceinline__ bool blockable(T cx, T cy) { return blockable_c(cx, cy); }
    static __device__ __forceinline__ bool interior(T cx, T cy) { return interior_c(cx, cy); }
};
template <class N> constexpr bool is_binary64() { return std::is_same<N, double>::value || std::is_same<N, R64>::value; }

constexpr uint32_t BATCH_MAX_VIEWPORTS = 1024;

template <class N, int K> __global__ void __launch_bounds__(512) k_batch(BatchArgs a)
{
    using P = Num<N>;
    using T = typename P::T;
    constexpr uint32_t FULLM = 0xffffffffu;
    __shared__ uint32_t s_pal[4096];
    __shared__ uint32_t s_base[BATCH_MAX_VIEWPORTS + 1];
    const uint32_t *pal = a.palette;
    if (a.palette && a.palette_len <= 4096u) {
        for (uint32_t k = threadIdx.x; k < a.palette_len; k += blockDim.x) s_pal[k] = a.palette[k];
        pal = s_pal;
    }
    for (uint32_t k = threadIdx.x; k < a.n_vp; k += blockDim.x) s_base[k] = a.vps[k].job_base;
    if (threadIdx.x == 0) s_base[a.n_vp] = a.n_jobs;
    __syncthreads();
    // a kernel launched after this one with programmatic serialization (the next
    // tier sharing the SMs) may start now: it reads nothing this kernel writes
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lt_mask = (1u << lane) - 1u;
    uint32_t job = 0xffffffffu, job_end = 0, vp = 0, pix = 0, s = 0, i = 0, window = 0, max_iter = 0, spp = 1;
    T x = P::zero(), y = P::zero(), cx = P::zero(), cy = P::zero();
    bool blk = false, need = true, begin = false;
    float acc_v = 0.f, acc[4] = {0.f, 0.f, 0.f, 0.f};
    unsigned long long iters = 0, skipped = 0;
    CycleWatch<T> cw;  // exact cycle detection at the end of every full block (see CycleWatch)

    // a job's viewport: the last one whose job_base <= job
    auto start_job = [&]() {
        uint32_t lo = 0, hi = a.n_vp;
        while (hi - lo > 1) {
            uint32_t mid = (lo + hi) >> 1;
            if (s_base[mid] <= job)
                lo = mid;
            else
                hi = mid;
        }
        vp = lo;
        pix = job - s_base[lo];
        max_iter = a.vps[lo].max_iter;
        spp = a.vps[lo].spp;
        begin = true;
        s = 0;
        acc_v = 0.f;
        acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
    };

    const unsigned long long t_start = a.budget_ns ? global_ns() : 0ull;
    for (;;) {
        // a time limit: the warp stops where it is (its samples in flight stay unwritten)
        if (out_of_time(a.budget_ns, t_start, a.status, lane)) break;
        uint32_t need_mask = __ballot_sync(FULLM, need);
        if (need_mask) {
            uint32_t leader = __ffs(need_mask) - 1u;
            uint32_t base = 0;
            if (lane == leader) base = atomicAdd(a.counter, (uint32_t)__popc(need_mask) * a.chunk);
            base = __shfl_sync(FULLM, base, leader);
            if (need) {
                job = base + (uint32_t)__popc(need_mask & lt_mask) * a.chunk;
                job_end = job + a.chunk;
                need = false;
                if (job < a.n_jobs) start_job();
            }
        }
        const bool active = job < a.n_jobs;
        if (!__any_sync(FULLM, active)) break;

        bool done = false;
        float r2 = 0.f;
        uint32_t lim = 0;
        if (active) {
            if (begin) {
                begin = false;
                const BatchViewport &v = a.vps[vp];
                uint32_t px, py;
                divmod_magic(pix, v.w, v.w_magic, py, px);
                double ox = 0.5, oy = 0.5;
                if (v.mode == SAMPLES_JITTER) {
                    ox = unit_interval_t<double>(sample_hash(v.seed, pix, s, 0));
                    oy = unit_interval_t<double>(sample_hash(v.seed, pix, s, 1));
                }
                double dxp = __dsub_rn(__dadd_rn((double)px, ox), 0.5 * v.w);
                double dyp = __dsub_rn(__dadd_rn((double)py, oy), 0.5 * v.h);
                cx = P::from(__fma_rn(dxp, v.ps, v.center_x));
                cy = P::from(__fma_rn(-dyp, v.ps, v.center_y));
                x = P::zero();
                y = P::zero();
                blk = P::blockable(cx, cy);
                i = 0;
                window = 0;
                cw.reset(x, y);
                if (max_iter == 0) done = true;
                if constexpr (is_binary64<N>()) {
                    // start at z = c, the first step's result (+0 for -0), so that no
                    // block begins with x = 0 (which the integer doubling redoes)
                    if (max_iter > 0) {
                        x = __dadd_rn(cx, 0.0);
                        y = __dadd_rn(cy, 0.0);
                        cw.reset(x, y);
                        i = 1;
                        const double rr = P::r2(x, y);
                        r2 = (float)rr;
                        if (i == max_iter || !(rr < 4.0)) done = true;
                    }
                }
                if (!done && P::interior(cx, cy)) {
                    skipped += max_iter - i;
                    i = max_iter;
                    done = true;
                }
            }
            if (!done && !std::is_same<N, FF>::value) {
                if (!blk) {
                    lim = 1;
                } else if (window) {
                    lim = window > 1u ? window >> 1 : 1u;
                } else {
                    uint32_t rest = max_iter - i;
                    lim = rest >= (uint32_t)K ? (uint32_t)K : 1u << (31 - __clz(rest));
                }
            }
        }
        const bool stepping = active && !done;
        const bool partial = stepping && lim < (uint32_t)K;
        const bool any_partial = !std::is_same<N, FF>::value && __any_sync(FULLM, partial);
        // K steps of `stepper`, keeping the state after lim steps on partial lanes
        auto run_block = [&](auto stepper) {
            if (any_partial) {
                T kx = x, ky = y;
#pragma unroll
                for (int k = 0; k < K; k++) {
                    stepper(x, y);
                    if (((k + 1) & k) == 0 && k + 1 < K && (uint32_t)(k + 1) == lim) {
                        kx = x;
                        ky = y;
                    }
                }
                if (partial) {
                    x = kx;
                    y = ky;
                }
            } else {
#pragma unroll
                for (int k = 0; k < K; k++) stepper(x, y);
            }
        };
        if constexpr (std::is_same<N, FF>::value) {
            // float-float: every step carries its own test (two binary32
            // operations on the leading words beside the step's 43), so a lane
            // that escapes stops at its exact state: no roll-back, no search
            if (stepping) {
                const uint32_t rest = max_iter - i;
                const uint32_t lim_t = rest >= (uint32_t)K ? (uint32_t)K : rest;
                uint32_t k = 0;
                bool esc = false;
#pragma unroll
                for (int u = 0; u < K; u++) {
                    if ((uint32_t)u == lim_t) break;
                    const float rr = P::r2(x, y);
                    if (!(rr < 4.f)) {
                        esc = true;
                        r2 = rr;
                        break;
                    }
                    P::step(x, y, cx, cy);
                    k++;
                }
                i += k;
                if (!esc && lim_t == (uint32_t)K && cw.check(x, y)) {  // a repeated state: interior
                    skipped += max_iter - i;
                    i = max_iter;
                }
                if (!esc && i == max_iter) r2 = P::r2(x, y);
                if (esc || i == max_iter) done = true;
            }
        } else if (stepping) {
            const T sx = x, sy = y;
            if constexpr (std::is_same<N, double>::value) {
                // 2x on the integer pipe; blocks it cannot double exactly are redone
                uint32_t emin = 0xffffffffu;
                run_block([&](T &u, T &v) { step_fma3(u, v, cx, cy, emin); });
                if (emin == 0u) {
                    x = sx;
                    y = sy;
                    run_block([&](T &u, T &v) { P::step(u, v, cx, cy); });
                }
            } else if constexpr (std::is_same<N, R64>::value) {
                // x*x - y*y on the integer units, fma(2, x*y, cy); a block with a
                // product or difference near the subnormal range is redone literally
                uint32_t emin = 0xffffffffu;
                run_block([&](T &u, T &v) { step_rounded6<double>(u, v, cx, cy, emin); });
                if (emin < exponent_bits_two<double>()) {
                    x = sx;
                    y = sy;
                    run_block([&](T &u, T &v) { P::step(u, v, cx, cy); });
                }
            } else {
                run_block([&](T &u, T &v) { P::step(u, v, cx, cy); });
            }
            if (P::below(x, y)) {
                const bool full = window == 0u && lim == (uint32_t)K;  // a checkpoint every K steps
                i += lim;
                window = window > 1u ? window - lim : 0u;
                if (full && cw.template check_every<cycle_blocks<T>()>(x, y)) {  // a repeated state: interior
                    skipped += max_iter - i;
                    i = max_iter;
                }
                if (i == max_iter) done = true;
            } else if (lim == 1u) {
                i += 1u;
                r2 = (float)P::r2(x, y);
                done = true;
            } else {
                x = sx;
                y = sy;
                window = lim;
            }
        }
        if (done) {
            const BatchViewport &v = a.vps[vp];
            const bool escaped = i < max_iter;
            const float nu = frame_smooth(i, r2, max_iter);
            const size_t sidx = (size_t)pix * spp + s;
            if (v.counts) v.counts[sidx] = i;
            if (v.smooth) v.smooth[sidx] = nu;
            iters += i;
            acc_v = __fadd_rn(acc_v, escaped ? nu : 0.f);
            if (v.rgba) {
                float ch[4];
                if (escaped) {
                    frame_palette_lerp(pal, a.palette_len, nu, ch);
                } else {
#pragma unroll
                    for (int k = 0; k < 4; k++) ch[k] = (float)((a.interior_rgba >> (8 * k)) & 255u);
                }
#pragma unroll
                for (int k = 0; k < 4; k++) acc[k] = __fadd_rn(acc[k], ch[k]);
            }
            ++s;
            if (s == spp) {
                if (v.rgba) v.rgba[pix] = frame_pack_rgba(acc, spp);
                if (job + 1u < job_end && job + 1u < a.n_jobs) {
                    ++job;  // the next job of this lane's chunk
                    start_job();
                } else {
                    need = true;
                }
            } else {
                begin = true;
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) iters += __shfl_down_sync(FULLM, iters, o);
    if (lane == 0 && iters && a.total) atomicAdd(a.total, iters);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) skipped += __shfl_down_sync(FULLM, skipped, o);
    if (lane == 0 && skipped && a.total) atomicAdd(a.total + 1, skipped);
    // when launched after a kernel that is still running (programmatic dependent
    // launch), the kernel ends only after that one has completed, so that the
    // stream's later work sees both.  Block 0 alone waits: the other blocks
    // leave at once and free their SM for what is queued behind them.  Without
    // such a predecessor this returns at once; the predecessor never waits on
    // this kernel, so the wait always ends.
    if (blockIdx.x == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
}

// blocks_per_sm > 0 caps the persistent grid at that many blocks per SM (the
// share of each SM a co-resident tier leaves this kernel); 0 = as many as fit.
template <class N, int K>
static cudaError_t launch_batch_k(const BatchArgs &a, int threads, int sms, int blocks_per_sm, bool after_started,
                                  cudaStream_t s)
{
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_batch<N, K>, threads, 0) != cudaSuccess || occ < 1)
        occ = 1;
    if (blocks_per_sm > 0 && blocks_per_sm < occ) occ = blocks_per_sm;
    const unsigned long long per_warp = 32ull * a.chunk;
    unsigned long long warps = ((unsigned long long)a.n_jobs + per_warp - 1ull) / per_warp;
    unsigned long long per_block = (unsigned long long)threads / 32ull;
    unsigned long long blocks = (warps + per_block - 1) / per_block;
    unsigned long long cap = (unsigned long long)occ * (unsigned long long)sms;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    cudaLaunchConfig_t lc{};
    lc.gridDim = dim3((unsigned)blocks);
    lc.blockDim = dim3((unsigned)threads);
    lc.stream = s;
    // after_started: start as soon as every block of the previous kernel in the
    // stream has started (programmatic dependent launch), not when it ends
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = after_started ? 1 : 0;
    lc.attrs = attr;
    lc.numAttrs = after_started ? 1 : 0;
    return cudaLaunchKernelEx(&lc, k_batch<N, K>, a);
}

template <class N>
static cudaError_t launch_batch(const BatchArgs &a, int threads, int k, int sms, int blocks_per_sm, bool after_started,
                                cudaStream_t s)
{
    if (k == 8) return launch_batch_k<N, 8>(a, threads, sms, blocks_per_sm, after_started, s);
    if (k == 32) return launch_batch_k<N, 32>(a, threads, sms, blocks_per_sm, after_started, s);
    return launch_batch_k<N, 16>(a, threads, sms, blocks_per_sm, after_started, s);
}

// Every tier kernel asks for the same shared-memory carveout (all of it): blocks
// of two kernels can share an SM only when the SM's L1/shared split suits
// both, and a split picked per kernel would keep them apart.
template <class N, int K> static void set_carveout()
{
    cudaFuncSetAttribute(k_batch<N, K>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         (int)cudaSharedmemCarveoutMaxShared);
}
static void prepare_batch_kernels()
{
    static const bool done = [] {
        set_carveout<float, 8>(), set_carveout<float, 16>(), set_carveout<float, 32>();
        set_carveout<FF, 8>(), set_carveout<FF, 16>(), set_carveout<FF, 32>();
        set_carveout<double, 8>(), set_carveout<double, 16>(), set_carveout<double, 32>();
        set_carveout<R64, 8>(), set_carveout<R64, 16>(), set_carveout<R64, 32>();
        return true;
    }();
    (void)done;
}

// Per-SM footprint of one block of a tier kernel.
struct Footprint {
    int regs = 0, smem = 0, warps = 0, alone = 1;  // alone: blocks per SM with the SM to itself
};
template <class N, int K> static Footprint footprint_k(int threads)
{
    Footprint f;
    cudaFuncAttributes fa{};
    if (cudaFuncGetAttributes(&fa, k_batch<N, K>) != cudaSuccess) return f;
    f.warps = threads / 32;
    f.regs = ((fa.numRegs * 32 + 255) / 256) * 256 * f.warps;  // registers are allocated per warp, 256 at a time
    f.smem = (int)fa.sharedSizeBytes + 1024;                     // plus the per-block reservation
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&f.alone, k_batch<N, K>, threads, 0) != cudaSuccess ||
        f.alone < 1)
        f.alone = 1;
    return f;
}
template <class N> static Footprint footprint(int threads, int k)
{
    if (k == 8) return footprint_k<N, 8>(threads);
    if (k == 32) return footprint_k<N, 32>(threads);
    return footprint_k<N, 16>(threads);
}

// Binary64 tier warps per SM when it shares the SMs with a binary32-pipe tier
// (chaos_batch_config.fp64_warps_per_sm, default 8): the binary64 pipe is
// saturated by a few warps (a warp-wide DFMA occupies it for ~19 cycles), so
// the binary64 kernel takes that many warps per SM and the float-float /
// binary32 kernels the rest, and the two pipes work at once.

}  // namespace chaos

using namespace chaos;

namespace {
constexpr int kTiers = 3;  // 0 binary32, 1 float-float, 2 binary64
int tier_slot(uint32_t tier) { return tier == CHAOS_TIER_F32 ? 0 : tier == CHAOS_TIER_FLOATFLOAT ? 1 : 2; }  // F64 or F64_ROUNDED: 2
}  // namespace

// A viewport of the batch rendered by perturbation (its own reference orbit).
struct PerturbJob {
    chaos_frame_desc desc{};
    chaos_frame_out out{};
    chaos_orbit *orbit = nullptr;
};

struct chaos_batch {
    int device = -1;
    std::vector<uint32_t> tiers;  // chosen tier per viewport
    std::vector<PerturbJob> perturb;
    BatchViewport *d_vps[kTiers] = {nullptr, nullptr, nullptr};
    uint32_t n_vp[kTiers] = {0, 0, 0}, n_jobs[kTiers] = {0, 0, 0};
    uint32_t *d_counters = nullptr;
    // [0] pixel-iterations, [1] iterations proven interior and not run,
    // [2] low word: the RUN_STATUS_* bits of the last launch
    unsigned long long *d_total = nullptr;
    unsigned long long budget_ns = 0;  // each launch's time limit (0: none)
    const uint32_t *palette = nullptr;
    uint32_t palette_len = 0, interior = 0;
    int threads[kTiers] = {256, 256, 256}, k[kTiers] = {16, 16, 16}, chunk[kTiers] = {1, 1, 1};
    int fp64_warps = 8;  // binary64 warps per SM when it shares the SMs
    bool rounded64 = false;  // the binary64 slot runs CHAOS_TIER_F64_ROUNDED
    int sms = 0;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    unsigned long long pixel_iterations_hint = 0;
};

uint32_t chaos_batch_auto_tier(double center_x, double center_y, double pixel_size)
{
    double m = std::max(std::max(std::fabs(center_x), std::fabs(center_y)), 1.0 / 256);
    if (pixel_size >= m * 0x1p-18) return CHAOS_TIER_F32;
    if (pixel_size >= m * 0x1p-42) return CHAOS_TIER_FLOATFLOAT;
    return CHAOS_TIER_F64;
}

static uint32_t auto_deep_tier(double center_x, double center_y, double pixel_size)
{
    uint32_t t = chaos_batch_auto_tier(center_x, center_y, pixel_size);
    return t == CHAOS_TIER_F64 ? CHAOS_TIER_PERTURB_F32 : t;
}

static void batch_free(chaos_batch *b)
{
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    for (int t = 0; t < kTiers; t++)
        if (b->d_vps[t]) cudaFree(b->d_vps[t]);
    for (PerturbJob &j : b->perturb)
        if (j.orbit) chaos_orbit_destroy(j.orbit);
    if (b->d_counters) cudaFree(b->d_counters);
    if (b->d_total) cudaFree(b->d_total);
    delete b;
}

// *rc: the status of a perturbation enqueue that failed (its message is the last error)
static cudaError_t batch_enqueue(chaos_batch *b, cudaStream_t s0, cudaStream_t s1, cudaStream_t s2, cudaStream_t s3,
                                 cudaEvent_t fork, cudaEvent_t j1, cudaEvent_t j2, cudaEvent_t j3, int *rc)
{
    // work counters: one per tier kernel, then one per perturbation viewport
    cudaError_t e = cudaMemsetAsync(b->d_counters, 0, (kTiers + b->perturb.size()) * sizeof(uint32_t), s0);
    if (e == cudaSuccess) e = cudaMemsetAsync(b->d_total, 0, 3 * sizeof(unsigned long long), s0);
    if (e == cudaSuccess) e = cudaEventRecord(fork, s0);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s1, fork, 0);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s2, fork, 0);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s3, fork, 0);
    // perturbation viewports, one after another on the fourth branch
    for (size_t k = 0; k < b->perturb.size() && e == cudaSuccess; k++) {
        PerturbJob &j = b->perturb[k];
        *rc = api_perturb_enqueue(&j.desc, j.orbit, &j.out, s3, b->d_counters + kTiers + k);
        if (*rc != CHAOS_OK) e = cudaErrorInvalidValue;
    }
    cudaStream_t st[kTiers] = {s0, s1, s2};
    // binary64 first: its kernels are the longest, the cheaper tiers fill in behind
    const int order[kTiers] = {2, 1, 0};
    // co-residency: with a binary64 tier and a binary32-pipe tier present, the
    // binary64 grid is capped at fp64_warps warps per SM and launched first; the
    // binary32-pipe kernels follow in the same stream as programmatic dependent
    // launches, so they start once every binary64 block is resident, with their
    // grids capped at what fits beside it.  A binary64 tail grid follows (see
    // below) to widen the binary64 tier when the others finish first.
    int per_sm[kTiers] = {0, 0, 0};
    bool shared = false;
    if (b->n_jobs[2] && (b->n_jobs[0] || b->n_jobs[1])) {
        Footprint f64 = b->rounded64 ? footprint<R64>(b->threads[2], b->k[2]) : footprint<double>(b->threads[2], b->k[2]);
        int b64 = std::max(1, std::min(f64.alone, b->fp64_warps / std::max(1, f64.warps)));
        int dev = 0, smem_sm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
        const int regs_left = 65536 - b64 * f64.regs, smem_left = smem_sm - b64 * f64.smem;
        const int warps_left = 64 - b64 * f64.warps, blocks_left = 32 - b64;
        bool fits = true;
        for (int t = 0; t < 2; t++) {
            if (!b->n_jobs[t]) continue;
            Footprint f = t == 0 ? footprint<float>(b->threads[t], b->k[t]) : footprint<FF>(b->threads[t], b->k[t]);
            int n = f.alone;
            if (f.regs > 0) n = std::min(n, regs_left / f.regs);
            if (f.smem > 0) n = std::min(n, smem_left / f.smem);
            if (f.warps > 0) n = std::min(n, warps_left / f.warps);
            n = std::min(n, blocks_left);
            if (n < 1) fits = false;
            per_sm[t] = n;
        }
        if (fits) {
            per_sm[2] = b64;
            shared = true;
        } else {
            per_sm[0] = per_sm[1] = 0;
        }
    }
    for (int oi = 0; oi < kTiers && e == cudaSuccess; oi++) {
        int t = order[oi];
        if (!b->n_jobs[t]) continue;
        BatchArgs a{};
        a.vps = b->d_vps[t];
        a.n_vp = b->n_vp[t];
        a.n_jobs = b->n_jobs[t];
        a.counter = b->d_counters + t;
        a.chunk = (uint32_t)b->chunk[t];
        a.total = b->d_total;
        a.palette = b->palette;
        a.palette_len = b->palette_len;
        a.interior_rgba = b->interior;
        a.budget_ns = b->budget_ns;
        a.status = reinterpret_cast<uint32_t *>(b->d_total + 2);
        cudaStream_t s = shared ? s0 : st[oi];
        const bool after = shared && t != 2;
        if (t == 0) e = launch_batch<float>(a, b->threads[t], b->k[t], b->sms, per_sm[t], after, s);
        if (t == 1) e = launch_batch<FF>(a, b->threads[t], b->k[t], b->sms, per_sm[t], after, s);
        if (t == 2)
            e = b->rounded64 ? launch_batch<R64>(a, b->threads[t], b->k[t], b->sms, per_sm[t], after, s)
                             : launch_batch<double>(a, b->threads[t], b->k[t], b->sms, per_sm[t], after, s);
    }
    if (shared && e == cudaSuccess) {
        // the binary64 tail: a second, full-size grid on the same job counter.
        // It starts once every binary32-pipe block has started, and its blocks
        // take the room those blocks leave when their tier runs out of work, so
        // a binary64 tier that outlasts the others widens to whole SMs.
        BatchArgs a{};
        a.vps = b->d_vps[2];
        a.n_vp = b->n_vp[2];
        a.n_jobs = b->n_jobs[2];
        a.counter = b->d_counters + 2;
        a.chunk = (uint32_t)b->chunk[2];
        a.total = b->d_total;
        a.palette = b->palette;
        a.palette_len = b->palette_len;
        a.interior_rgba = b->interior;
        a.budget_ns = b->budget_ns;
        a.status = reinterpret_cast<uint32_t *>(b->d_total + 2);
        e = b->rounded64 ? launch_batch<R64>(a, b->threads[2], b->k[2], b->sms, 0, true, s0)
                         : launch_batch<double>(a, b->threads[2], b->k[2], b->sms, 0, true, s0);
    }
    if (e == cudaSuccess) e = cudaEventRecord(j1, s1);
    if (e == cudaSuccess) e = cudaEventRecord(j2, s2);
    if (e == cudaSuccess) e = cudaEventRecord(j3, s3);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s0, j1, 0);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s0, j2, 0);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s0, j3, 0);
    return e;
}

int chaos_batch_create(const chaos_viewport *vps, uint32_t n, const uint32_t *palette, uint32_t palette_len,
                       uint32_t interior_rgba, const chaos_batch_config *cfg, chaos_batch **out)
{
    if (!vps || !out || n == 0) return api_fail(CHAOS_ERR_INVALID_ARGUMENT, "viewports required");
    if (n > BATCH_MAX_VIEWPORTS) return api_fail(CHAOS_ERR_INVALID_ARGUMENT, "at most %u viewports", BATCH_MAX_VIEWPORTS);
    std::vector<BatchViewport> per[kTiers];
    std::vector<uint32_t> tiers(n);
    uint64_t jobs[kTiers] = {0, 0, 0};
    bool any_rgba = false, any_f64 = false, any_rounded = false;
    for (uint32_t k = 0; k < n; k++) {
        const chaos_viewport &v = vps[k];
        if (v.width == 0 || v.height == 0 || (uint64_t)v.width * v.height > (1ull << 31))
            return api_fail(CHAOS_ERR_INVALID_ARGUMENT, "viewport %u: bad size", k);
        if (v.samples_per_pixel < 1 || v.samples_per_pixel > 64)
            return api_fail(CHAOS_ERR_INVALID_ARGUMENT, "viewport %u: samples_per_pixel must be 1..64", k);
        if (v.sample_mode > CHAOS_SAMPLES_JITTER ||
            (v.sample_mode == CHAOS_SAMPLES_CENTER && v.samples_per_pixel != 1))
            return api_fail(CHAOS_ERR_INVALID_ARGUMENT, "viewport %u: bad sample mode", k);
        if (!std::isfinite(v.center_x) || !std::isfinite(v.center_y) || !(v.pixel_size > 0) ||
            !std::isfinite(v.pixel_size))
            return api_fail(CHAOS_ERR_INVALID_ARGUMENT, "viewport %u: centre/pixel size", k);
        uint32_t tier = v.tier == CHAOS_TIER_AUTO        ? chaos_batch_auto_tier(v.center_x, v.center_y, v.pixel_size)
                        : v.tier == CHAOS_TIER_AUTO_DEEP ? auto_deep_tier(v.center_x, v.center_y, v.pixel_size)
                                                         : v.tier;
        if (tier != CHAOS_TIER_F32 && tier != CHAOS_TIER_FLOATFLOAT && tier != CHAOS_TIER_F64 &&
            tier != CHAOS_TIER_F64_ROUNDED && tier != CHAOS_TIER_PERTURB_F32 && tier != CHAOS_TIER_PERTURB_F64)
            return api_fail(CHAOS_ERR_UNSUPPORTED, "viewport %u: tier %u not batchable", k, tier);
        tiers[k] = tier;
        any_f64 |= tier == CHAOS_TIER_F64;
        any_rounded |= tier == CHAOS_TIER_F64_ROUNDED;
        if (any_f64 && any_rounded)
            return api_fail(CHAOS_ERR_INVALID_ARGUMENT,
                            "viewport %u: binary64 viewports of one batch must all be fused or all rounded", k);
        if (tier == CHAOS_TIER_PERTURB_F32 || tier == CHAOS_TIER_PERTURB_F64) {
            if (!(v.pixel_size >= 1e-290))
                return api_fail(CHAOS_ERR_INVALID_ARGUMENT, "viewport %u: perturbation needs pixel >= 1e-290", k);
            any_rgba |= v.rgba != nullptr;
            continue;  // its orbit is computed below
        }
        int t = tier_slot(tier);
        BatchViewport bv{};
        bv.w = v.width;
        bv.w_magic = div_magic(v.width);
        bv.h = v.height;
        bv.spp = v.samples_per_pixel;
        bv.mode = v.sample_mode;
        bv.max_iter = v.max_iterations;
        bv.job_base = (uint32_t)jobs[t];
        bv.seed = v.seed;
        bv.center_x = v.center_x;
        bv.center_y = v.center_y;
        bv.ps = v.pixel_size;
        bv.counts = v.counts;
        bv.smooth = v.smooth;
        bv.rgba = v.rgba;
        any_rgba |= v.rgba != nullptr;
        jobs[t] += (uint64_t)v.width * v.height;
        if (jobs[t] > (1ull << 31)) return api_fail(CHAOS_ERR_INVALID_ARGUMENT, "batch too large");
        per[t].push_back(bv);
    }
    if (any_rgba && (!palette || palette_len == 0 || palette_len > 4096))
        return api_fail(CHAOS_ERR_INVALID_ARGUMENT, "rgba outputs need a device palette of 1..4096 entries");
    // Costly viewports first: lanes claim a tier's job space in order, so the
    // pixels with the highest maxIter x samples start first and the end of the
    // launch, where lanes run out of work, is made of short ones.
    for (int t = 0; t < kTiers; t++) {
        std::stable_sort(per[t].begin(), per[t].end(), [](const BatchViewport &p, const BatchViewport &q) {
            return (uint64_t)p.max_iter * p.spp > (uint64_t)q.max_iter * q.spp;
        });
        uint32_t base = 0;
        for (BatchViewport &bv : per[t]) {
            bv.job_base = base;
            base += bv.w * bv.h;
        }
    }

    chaos_batch *b = new (std::nothrow) chaos_batch();
    if (!b) return api_fail(CHAOS_ERR_OUT_OF_MEMORY, "out of host memory");
    cudaGetDevice(&b->device);
    cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, b->device);
    b->tiers = tiers;
    b->rounded64 = any_rounded;
    b->palette = palette;
    b->palette_len = palette_len;
    b->interior = interior_rgba;
    if (cfg) {
        for (int t = 0; t < kTiers; t++) {
            if (cfg->block_threads[t]) b->threads[t] = (int)cfg->block_threads[t];
            if (cfg->escape_block[t]) b->k[t] = (int)cfg->escape_block[t];
            if (cfg->chunk[t]) b->chunk[t] = (int)cfg->chunk[t];
            if (b->threads[t] % 32 || b->threads[t] < 32 || b->threads[t] > 512 ||
                (b->k[t] != 8 && b->k[t] != 16 && b->k[t] != 32) || b->chunk[t] < 1 || b->chunk[t] > 64) {
                batch_free(b);
                return api_fail(CHAOS_ERR_INVALID_ARGUMENT,
                                "tier %d: threads 32..512 (multiple of 32), block 8/16/32, chunk 1..64", t);
            }
        }
        if (cfg->fp64_warps_per_sm) b->fp64_warps = (int)cfg->fp64_warps_per_sm;
        if (!api_budget(cfg->time_limit_s, &b->budget_ns)) {
            batch_free(b);
            return api_fail(CHAOS_ERR_INVALID_ARGUMENT, "time_limit_s must be >= 0");
        }
        if (b->fp64_warps < 1 || b->fp64_warps > 32) {
            batch_free(b);
            return api_fail(CHAOS_ERR_INVALID_ARGUMENT, "fp64_warps_per_sm must be 1..32");
        }
    }
    size_t n_perturb = 0;
    for (uint32_t k = 0; k < n; k++) n_perturb += tiers[k] == CHAOS_TIER_PERTURB_F32 || tiers[k] == CHAOS_TIER_PERTURB_F64;
    cudaError_t e = cudaMalloc(&b->d_counters, (kTiers + n_perturb) * sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMalloc(&b->d_total, 3 * sizeof(unsigned long long));
    // reference orbits of the perturbation viewports (host, multi-word)
    for (uint32_t k = 0; k < n && e == cudaSuccess; k++) {
        if (tiers[k] != CHAOS_TIER_PERTURB_F32 && tiers[k] != CHAOS_TIER_PERTURB_F64) continue;
        const chaos_viewport &v = vps[k];
        PerturbJob j;
        double bits = -std::log2(v.pixel_size) + 96.0;
        uint32_t want = (uint32_t)std::min(1536.0, std::max(128.0, std::ceil(bits / 64.0) * 64.0));
        int rc = api_orbit_create_d(v.center_x, v.center_y, want, v.max_iterations, &j.orbit);
        if (rc != CHAOS_OK) {
            batch_free(b);
            return rc;
        }
        j.desc.width = v.width;
        j.desc.height = v.height;
        j.desc.max_iterations = v.max_iterations;
        j.desc.samples_per_pixel = v.samples_per_pixel;
        j.desc.sample_mode = v.sample_mode;
        j.desc.tier = tiers[k];
        j.desc.fractal = 0;
        j.desc.seed = v.seed;
        j.desc.pixel_size = v.pixel_size;
        j.desc.time_limit_s = cfg ? cfg->time_limit_s : 0.0;
        j.out.counts = v.counts;
        j.out.smooth = v.smooth;
        j.out.rgba = v.rgba;
        j.out.palette = palette;
        j.out.palette_len = palette_len;
        j.out.interior_rgba = interior_rgba;
        j.out.total_iterations = b->d_total;
        j.out.status = reinterpret_cast<uint32_t *>(b->d_total + 2);
        b->perturb.push_back(j);
    }
    for (int t = 0; t < kTiers && e == cudaSuccess; t++) {
        b->n_vp[t] = (uint32_t)per[t].size();
        b->n_jobs[t] = (uint32_t)jobs[t];
        if (per[t].empty()) continue;
        e = cudaMalloc(&b->d_vps[t], per[t].size() * sizeof(BatchViewport));
        if (e == cudaSuccess)
            e = cudaMemcpy(b->d_vps[t], per[t].data(), per[t].size() * sizeof(BatchViewport), cudaMemcpyHostToDevice);
    }
    prepare_batch_kernels();
    // capture the fork-join launch into a graph
    cudaStream_t s0 = nullptr, s1 = nullptr, s2 = nullptr, s3 = nullptr;
    cudaEvent_t fork = nullptr, j1 = nullptr, j2 = nullptr, j3 = nullptr;
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&s0, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&s1, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&s2, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&s3, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&fork, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&j1, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&j2, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&j3, cudaEventDisableTiming);
    int enqueue_rc = CHAOS_OK;
    if (e == cudaSuccess) e = cudaStreamBeginCapture(s0, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
        cudaError_t ee = batch_enqueue(b, s0, s1, s2, s3, fork, j1, j2, j3, &enqueue_rc);
        e = cudaStreamEndCapture(s0, &b->graph);
        if (ee != cudaSuccess) e = ee;
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&b->exec, b->graph, 0);
    if (fork) cudaEventDestroy(fork);
    if (j1) cudaEventDestroy(j1);
    if (j2) cudaEventDestroy(j2);
    if (j3) cudaEventDestroy(j3);
    if (s3) cudaStreamDestroy(s3);
    if (s0) cudaStreamDestroy(s0);
    if (s1) cudaStreamDestroy(s1);
    if (s2) cudaStreamDestroy(s2);
    if (e != cudaSuccess) {
        batch_free(b);
        if (enqueue_rc != CHAOS_OK) return enqueue_rc;
        return api_fail(CHAOS_ERR_CUDA, "batch set-up: %s", cudaGetErrorString(e));
    }
    *out = b;
    return CHAOS_OK;
}

int chaos_batch_launch(chaos_batch *b, void *stream)
{
    TraceRange trace_("chaos_batch_launch");
    if (!b) return api_fail(CHAOS_ERR_INVALID_ARGUMENT, "NULL batch");
    cudaError_t e = cudaGraphLaunch(b->exec, (cudaStream_t)stream);
    if (e != cudaSuccess) return api_fail(CHAOS_ERR_CUDA, "cudaGraphLaunch: %s", cudaGetErrorString(e));
    return CHAOS_OK;
}

int chaos_batch_tiers(const chaos_batch *b, uint32_t *tiers, uint32_t n)
{
    if (!b || !tiers || n < b->tiers.size()) return api_fail(CHAOS_ERR_INVALID_ARGUMENT, "bad argument");
    std::copy(b->tiers.begin(), b->tiers.end(), tiers);
    return CHAOS_OK;
}

int chaos_batch_total(const chaos_batch *b, unsigned long long **device_total)
{
    if (!b || !device_total) return api_fail(CHAOS_ERR_INVALID_ARGUMENT, "bad argument");
    *device_total = b->d_total;
    return CHAOS_OK;
}

int chaos_batch_read_total(const chaos_batch *b, unsigned long long *total)
{
    if (!b || !total) return api_fail(CHAOS_ERR_INVALID_ARGUMENT, "bad argument");
    cudaError_t e = cudaMemcpy(total, b->d_total, sizeof *total, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return api_fail(CHAOS_ERR_CUDA, "read total: %s", cudaGetErrorString(e));
    return CHAOS_OK;
}

int chaos_batch_read_cycle_skipped(const chaos_batch *b, unsigned long long *skipped)
{
    if (!b || !skipped) return api_fail(CHAOS_ERR_INVALID_ARGUMENT, "bad argument");
    cudaError_t e = cudaMemcpy(skipped, b->d_total + 1, sizeof *skipped, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return api_fail(CHAOS_ERR_CUDA, "read skipped: %s", cudaGetErrorString(e));
    return CHAOS_OK;
}

int chaos_batch_read_status(const chaos_batch *b, uint32_t *status)
{
    if (!b || !status) return api_fail(CHAOS_ERR_INVALID_ARGUMENT, "bad argument");
    cudaError_t e = cudaMemcpy(status, b->d_total + 2, sizeof *status, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return api_fail(CHAOS_ERR_CUDA, "read status: %s", cudaGetErrorString(e));
    return CHAOS_OK;
}

int chaos_batch_destroy(chaos_batch *b)
{
    if (b) batch_free(b);
    return CHAOS_OK;
}

// ---- autotuner ------------------------------------------------------------------
//
// Per tier slot present in the viewport list, time every launch shape of the
// search space on a sample of that tier's viewports (each cut to its central
// window of 1/8 of its width and height, at least 32 pixels, same pixel size,
// samples and iteration limit) and keep the fastest; then, when binary64
// shares the batch with a binary32-pipe tier, tune the shared launch on the
// joint sample.  Results are cached in a text file, one line
// per key: "<key> <threads> <escape block> <chunk> <ms>", the key being the
// device name, its SM count, the tier slot and a hash of that tier's viewport
// parameters.

namespace {

uint64_t fnv1a(uint64_t h, const void *p, size_t n)
{
    const unsigned char *c = static_cast<const unsigned char *>(p);
    for (size_t k = 0; k < n; k++) {
        h ^= c[k];
        h *= 1099511628211ull;
    }
    return h;
}

struct TuneEntry {
    int threads, k, chunk;
    double ms;
};

std::vector<std::pair<std::string, TuneEntry>> read_tune_cache(const char *path)
{
    std::vector<std::pair<std::string, TuneEntry>> out;
    if (!path) return out;
    FILE *f = std::fopen(path, "r");
    if (!f) return out;
    char key[512];
    TuneEntry e{};
    while (std::fscanf(f, "%511s %d %d %d %lf", key, &e.threads, &e.k, &e.chunk, &e.ms) == 5) out.push_back({key, e});
    std::fclose(f);
    return out;
}

// Launch time of a batch of `vps` under `cfg`: the faster of two launches
// after a warm-up.  Negative on failure.
double time_config(const std::vector<chaos_viewport> &vps, const chaos_batch_config &cfg, cudaStream_t s)
{
    chaos_batch *b = nullptr;
    if (chaos_batch_create(vps.data(), (uint32_t)vps.size(), nullptr, 0, 0, &cfg, &b) != CHAOS_OK) return -1.0;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    double best = -1.0;
    if (cudaEventCreate(&e0) == cudaSuccess && cudaEventCreate(&e1) == cudaSuccess &&
        chaos_batch_launch(b, s) == CHAOS_OK) {
        for (int rep = 0; rep < 2; rep++) {
            float ms = 0.f;
            if (cudaEventRecord(e0, s) != cudaSuccess || chaos_batch_launch(b, s) != CHAOS_OK ||
                cudaEventRecord(e1, s) != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess ||
                cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess) {
                best = -1.0;
                break;
            }
            if (best < 0 || ms < best) best = ms;
        }
    }
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    chaos_batch_destroy(b);
    return best;
}

// One tier's viewports (forced) under one shape.
double time_shape(const std::vector<chaos_viewport> &vps, int slot, int threads, int k, int chunk, cudaStream_t s)
{
    chaos_batch_config cfg{};
    cfg.block_threads[slot] = (uint32_t)threads;
    cfg.escape_block[slot] = (uint32_t)k;
    cfg.chunk[slot] = (uint32_t)chunk;
    return time_config(vps, cfg, s);
}

}  // namespace

int chaos_batch_autotune(const chaos_viewport *vps, uint32_t n, const char *cache_path, chaos_batch_config *config,
                         uint32_t *from_cache)
{
    if (!vps || !config || n == 0) return api_fail(CHAOS_ERR_INVALID_ARGUMENT, "viewports and config required");
    if (n > BATCH_MAX_VIEWPORTS) return api_fail(CHAOS_ERR_INVALID_ARGUMENT, "at most %u viewports", BATCH_MAX_VIEWPORTS);
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceProp prop{};
    if (cudaGetDeviceProperties(&prop, dev) != cudaSuccess) return api_fail(CHAOS_ERR_CUDA, "device properties");
    sms = prop.multiProcessorCount;
    std::string devname = prop.name;
    for (char &c : devname)
        if (c == ' ' || c == '\t') c = '_';

    // the tuning sample per tier slot
    std::vector<chaos_viewport> sample[kTiers];
    uint64_t sig[kTiers] = {1469598103934665603ull, 1469598103934665603ull, 1469598103934665603ull};
    size_t pixels[kTiers] = {0, 0, 0};
    for (uint32_t k = 0; k < n; k++) {
        const chaos_viewport &v = vps[k];
        uint32_t tier = v.tier == CHAOS_TIER_AUTO        ? chaos_batch_auto_tier(v.center_x, v.center_y, v.pixel_size)
                        : v.tier == CHAOS_TIER_AUTO_DEEP ? auto_deep_tier(v.center_x, v.center_y, v.pixel_size)
                                                         : v.tier;
        if (tier != CHAOS_TIER_F32 && tier != CHAOS_TIER_FLOATFLOAT && tier != CHAOS_TIER_F64 &&
            tier != CHAOS_TIER_F64_ROUNDED)
            continue;
        const int t = tier_slot(tier);
        chaos_viewport c = v;
        c.tier = tier;
        // the central window of 1/8 of the width and height (at least 32 pixels), so
        // that the sample keeps the viewports' proportions of work
        c.width = std::min<uint32_t>(v.width, std::max<uint32_t>(32, v.width / 8));
        c.height = std::min<uint32_t>(v.height, std::max<uint32_t>(32, v.height / 8));
        c.counts = nullptr;
        c.smooth = nullptr;
        c.rgba = nullptr;
        const uint32_t fields[6] = {c.width, c.height, c.samples_per_pixel, c.sample_mode, c.max_iterations, c.tier};
        sig[t] = fnv1a(sig[t], fields, sizeof(fields));
        const double geo[3] = {c.center_x, c.center_y, c.pixel_size};
        sig[t] = fnv1a(sig[t], geo, sizeof(geo));
        pixels[t] += (size_t)c.width * c.height * c.samples_per_pixel;
        sample[t].push_back(c);
    }
    auto cache = read_tune_cache(cache_path);
    std::vector<std::string> new_lines;
    *config = chaos_batch_config{};
    bool all_cached = true;
    cudaStream_t s = nullptr;
    if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess)
        return api_fail(CHAOS_ERR_CUDA, "stream create");
    // the counts go to one scratch buffer, tier after tier, viewport after viewport
    uint32_t *scratch = nullptr;
    size_t all = pixels[0] + pixels[1] + pixels[2];
    if (all && cudaMalloc(&scratch, all * sizeof(uint32_t)) != cudaSuccess) {
        cudaStreamDestroy(s);
        return api_fail(CHAOS_ERR_OUT_OF_MEMORY, "autotune scratch");
    }
    {
        size_t off = 0;
        for (int t = 0; t < kTiers; t++)
            for (chaos_viewport &c : sample[t]) {
                c.counts = scratch + off;
                off += (size_t)c.width * c.height * c.samples_per_pixel;
            }
    }
    static const int kThreads[] = {128, 256, 512}, kBlocks[] = {8, 16, 32}, kChunks[] = {1, 2, 4};
    int rc = CHAOS_OK;
    for (int t = 0; t < kTiers && rc == CHAOS_OK; t++) {
        if (sample[t].empty()) continue;
        char key[512];
        std::snprintf(key, sizeof(key), "%s|sm%d|slot%d|%016llx", devname.c_str(), sms, t, (unsigned long long)sig[t]);
        bool hit = false;
        for (auto &kv : cache)
            if (kv.first == key) {
                config->block_threads[t] = (uint32_t)kv.second.threads;
                config->escape_block[t] = (uint32_t)kv.second.k;
                config->chunk[t] = (uint32_t)kv.second.chunk;
                hit = true;
            }
        if (hit) continue;
        all_cached = false;
        TuneEntry best{0, 0, 0, -1.0};
        for (int th : kThreads)
            for (int kb : kBlocks)
                for (int ch : kChunks) {
                    double ms = time_shape(sample[t], t, th, kb, ch, s);
                    if (ms >= 0 && (best.ms < 0 || ms < best.ms)) best = {th, kb, ch, ms};
                }
        if (best.ms < 0) {
            rc = api_fail(CHAOS_ERR_CUDA, "autotune: no launch shape ran for tier slot %d", t);
            break;
        }
        config->block_threads[t] = (uint32_t)best.threads;
        config->escape_block[t] = (uint32_t)best.k;
        config->chunk[t] = (uint32_t)best.chunk;
        char line[640];
        std::snprintf(line, sizeof(line), "%s %d %d %d %.6f\n", key, best.threads, best.k, best.chunk, best.ms);
        new_lines.push_back(line);
    }
    // the shared launch: binary64 next to a binary32-pipe tier.  Cache line
    // "<key> <binary32-pipe threads> <binary64 threads> <binary64 warps per SM
    // + 65536 x binary64 escape block> <ms>".
    if (rc == CHAOS_OK && !sample[2].empty() && (!sample[0].empty() || !sample[1].empty())) {
        char key[512];
        std::snprintf(key, sizeof(key), "%s|sm%d|shared|%016llx", devname.c_str(), sms,
                      (unsigned long long)(sig[0] ^ (sig[1] * 31ull) ^ (sig[2] * 1009ull)));
        bool hit = false;
        for (auto &kv : cache)
            if (kv.first == key) {
                for (int t = 0; t < 2; t++)
                    if (!sample[t].empty()) config->block_threads[t] = (uint32_t)kv.second.threads;
                config->block_threads[2] = (uint32_t)kv.second.k;
                config->fp64_warps_per_sm = (uint32_t)(kv.second.chunk & 0xffff);
                if (kv.second.chunk >> 16) config->escape_block[2] = (uint32_t)(kv.second.chunk >> 16);
                hit = true;
            }
        if (!hit) {
            all_cached = false;
            // a larger sample than the per-tier one (1/4 of each side, at least 64
            // pixels): the shared launch's balance depends on the tail of each tier
            std::vector<chaos_viewport> joint;
            size_t jpix = 0;
            for (uint32_t k = 0; k < n; k++) {
                const chaos_viewport &v = vps[k];
                uint32_t tier = v.tier == CHAOS_TIER_AUTO ? chaos_batch_auto_tier(v.center_x, v.center_y, v.pixel_size)
                                : v.tier == CHAOS_TIER_AUTO_DEEP
                                    ? auto_deep_tier(v.center_x, v.center_y, v.pixel_size)
                                    : v.tier;
                if (tier != CHAOS_TIER_F32 && tier != CHAOS_TIER_FLOATFLOAT && tier != CHAOS_TIER_F64 &&
            tier != CHAOS_TIER_F64_ROUNDED)
            continue;
                chaos_viewport c = v;
                c.tier = tier;
                c.width = std::min<uint32_t>(v.width, std::max<uint32_t>(64, v.width / 4));
                c.height = std::min<uint32_t>(v.height, std::max<uint32_t>(64, v.height / 4));
                c.counts = nullptr;
                c.smooth = nullptr;
                c.rgba = nullptr;
                jpix += (size_t)c.width * c.height * c.samples_per_pixel;
                joint.push_back(c);
            }
            uint32_t *jscratch = nullptr;
            if (cudaMalloc(&jscratch, jpix * sizeof(uint32_t)) != cudaSuccess) joint.clear();
            size_t joff = 0;
            for (chaos_viewport &c : joint) {
                c.counts = jscratch + joff;
                joff += (size_t)c.width * c.height * c.samples_per_pixel;
            }
            // 512-thread blocks of the binary32-pipe kernels are left out: beside the
            // binary64 blocks only one fits (16 warps, against 24 for 256-thread
            // blocks), and on the full C4 batch they lost every pairing (586 ms vs
            // 544 ms); 32-step binary64 blocks likewise (596 vs 544).
            static const int kSideThreads[] = {128, 256}, kF64Threads[] = {128, 256}, kF64Block[] = {16},
                             kF64Warps[] = {8, 12, 16};
            TuneEntry best{0, 0, 0, -1.0};
            int best_k64 = config->escape_block[2];
            for (int ts : kSideThreads)
                for (int t64 : kF64Threads)
                    for (int k64 : kF64Block)
                        for (int w64 : kF64Warps) {
                            chaos_batch_config c = *config;
                            for (int t = 0; t < 2; t++)
                                if (!sample[t].empty()) c.block_threads[t] = (uint32_t)ts;
                            c.block_threads[2] = (uint32_t)t64;
                            c.escape_block[2] = (uint32_t)k64;
                            c.fp64_warps_per_sm = (uint32_t)w64;
                            double ms = joint.empty() ? -1.0 : time_config(joint, c, s);
                            if (ms >= 0 && (best.ms < 0 || ms < best.ms)) {
                                best = {ts, t64, w64, ms};
                                best_k64 = k64;
                            }
                        }
            if (jscratch) cudaFree(jscratch);
            if (best.ms >= 0) {
                for (int t = 0; t < 2; t++)
                    if (!sample[t].empty()) config->block_threads[t] = (uint32_t)best.threads;
                config->block_threads[2] = (uint32_t)best.k;
                config->escape_block[2] = (uint32_t)best_k64;
                config->fp64_warps_per_sm = (uint32_t)best.chunk;
                char line[640];
                // the binary64 escape block rides in the warps field's upper half
                std::snprintf(line, sizeof(line), "%s %d %d %d %.6f\n", key, best.threads, best.k,
                              best.chunk | (best_k64 << 16), best.ms);
                new_lines.push_back(line);
            }
        }
    }
    if (scratch) cudaFree(scratch);
    cudaStreamDestroy(s);
    if (rc != CHAOS_OK) return rc;
    if (cache_path && !new_lines.empty()) {
        FILE *f = std::fopen(cache_path, "a");
        if (f) {
            for (const std::string &l : new_lines) std::fputs(l.c_str(), f);
            std::fclose(f);
        }
    }
    if (from_cache) *from_cache = all_cached ? 1u : 0u;
    return CHAOS_OK;
}
