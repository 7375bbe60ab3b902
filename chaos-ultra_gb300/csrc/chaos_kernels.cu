// chaos_kernels.cu -- library kernels of the escape-time path (sm_103a).
//
//   k_main / k_advanced   reference-mode frames (fractalRenderMain/Advanced,
//                         gen.cu:168-181, 307-368): persistent warps take 8x4
//                         tiles from a work counter, one tile = one vote group
//   k_frame               independent binary64 samples (pixel centres or
//                         jittered): persistent warps with per-lane refill, so a
//                         lane whose sample escaped takes the next one without
//                         waiting for the slowest lane of its warp; untested
//                         blocks with an in-warp search of an overshot block
//   k_frame32             independent binary32 samples: short orbits as they
//                         come, long ones queued and packed into full warps
//   k_compose             palette compose (gen.cu:455-475), HBM-bound
//   k_under_sampled       fractalRenderUnderSampled (gen.cu:478-503)
#include <algorithm>
#include <cstdio>

#include "chaos_frame.cuh"
#include "chaos_kernels.cuh"
#include "chaos_refmode.cuh"

namespace chaos {

constexpr uint32_t PALETTE_SMEM = 4096;

// ---------------------------------------------------------------------------
// Packing a block's working lanes into as few warps as hold them
// ---------------------------------------------------------------------------

template <class S> constexpr uint32_t LANE_WORDS = (uint32_t)(sizeof(S) / 4);

// All threads of the block take part.  `left` is the number of lanes at work
// that the caller packed for last (the block's threads at first) and becomes
// their number now; the states move only where that saves a warp.  `keep`:
// this lane is at work; on return `on` says so of the lane's new state.
// buf holds LANE_WORDS<S> words a thread, count one a warp.
template <class S>
__device__ __forceinline__ void pack_lanes(S &st, bool keep, bool &on, uint32_t &left, uint32_t *buf, uint32_t *count)
{
    const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const uint32_t mask = __ballot_sync(FULL, keep);
    __syncthreads();  // the last packing's words and counts have been read
    if (lane == 0) count[wib] = (uint32_t)__popc(mask);
    __syncthreads();
    uint32_t at = (uint32_t)__popc(mask & ((1u << lane) - 1u)), now = 0;
    for (uint32_t k = 0; k < warps; k++) {
        const uint32_t c = count[k];
        at += k < wib ? c : 0u;
        now += c;
    }
    const bool pack = (now + 31u) / 32u < (left + 31u) / 32u;
    left = now;
    on = keep;
    if (!pack) return;
    constexpr uint32_t W = LANE_WORDS<S>;
    uint32_t words[W];
    if (keep) {
        memcpy(words, &st, sizeof(S));
#pragma unroll
        for (uint32_t k = 0; k < W; k++) buf[k * blockDim.x + at] = words[k];
    }
    __syncthreads();
    on = threadIdx.x < now;
    if (on) {
#pragma unroll
        for (uint32_t k = 0; k < W; k++) words[k] = buf[k * blockDim.x + threadIdx.x];
        memcpy(&st, words, sizeof(S));
    }
}

// ---------------------------------------------------------------------------
// Independent-sample frames with per-lane refill
// ---------------------------------------------------------------------------

template <class R>
__device__ __forceinline__ void frame_point(const FrameArgs<R> &a, uint32_t w_magic, uint32_t pix, uint32_t s, R &cx,
                                            R &cy)
{
    using O = Op<R>;
    uint32_t px, py;
    divmod_magic(pix, a.w, w_magic, py, px);
    R ox = R(0.5), oy = R(0.5);
    if (a.mode == SAMPLES_JITTER) {
        ox = unit_interval_t<R>(sample_hash(a.seed, pix, s, 0));
        oy = unit_interval_t<R>(sample_hash(a.seed, pix, s, 1));
    }
    R dxp = O::sub(O::add((R)px, ox), a.half_w);
    R dyp = O::sub(O::add((R)py, oy), a.half_h);
    cx = O::fma(dxp, a.ps, a.center_x);
    cy = O::fma(-dyp, a.ps, a.center_y);
}

// Binary64 frames.  Bound: the binary64 pipe (a warp's operation takes its
// scheduler's pipe 76 cycles; five operations a step rounded, three fused).
// Once the pixels are claimed the remaining lanes are packed: 640x360 pixels of
// 4 samples at span 1.7e-8, maxIter 20000, are 1.5 pixels a lane and took 222 ms
// with the lanes left where they were, 175 packed and 172 with the clear escape
// tests in binary32 (480x270: 115 -> 99 ms); 512-step epochs, 128 and 2048 steps
// gave 175 and 180, three or four blocks an SM (80 and 64 registers) 176 and 185.
constexpr int DRAIN_ROUNDS = 32;  // rounds between packings
struct FrameLane {
    double x, y, cx, cy;
    CycleWatch<double> cw;
    uint32_t pix, s, i, window;
    float acc_v, acc[4];
    bool blk, begin;
};

template <int A, int F> __global__ void __launch_bounds__(PERSIST_THREADS) k_frame(FrameArgs<double> a)
{
    using R = double;
    constexpr int K = ESCAPE_BLOCK;
    __shared__ uint32_t s_pal[PALETTE_SMEM];
    __shared__ uint32_t s_state[LANE_WORDS<FrameLane> * PERSIST_THREADS], s_count[PERSIST_THREADS / 32], s_drain, s_retired;
    if (threadIdx.x == 0) s_drain = s_retired = 0;
    const uint32_t *pal = a.palette;
    if (a.rgba && a.palette_len <= PALETTE_SMEM) {
        for (uint32_t k = threadIdx.x; k < a.palette_len; k += blockDim.x) s_pal[k] = a.palette[k];
        pal = s_pal;
    }
    __syncthreads();

    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lt_mask = (1u << lane) - 1u;
    const uint32_t w_magic = div_magic(a.w);
    FrameLane st{};
    R &x = st.x, &y = st.y, &cx = st.cx, &cy = st.cy;
    CycleWatch<R> &cw = st.cw;  // exact cycle detection (see CycleWatch)
    uint32_t &pix = st.pix, &s = st.s, &i = st.i;
    uint32_t &window = st.window;  // > 0: the escape lies within the next `window` steps
    float &acc_v = st.acc_v, (&acc)[4] = st.acc;
    pix = 0xffffffffu;
    bool need = true;
    unsigned long long iters = 0, skipped = 0;
    const unsigned long long t_start = a.budget_ns ? global_ns() : 0ull;

    // the grid's first pixels go out without a claim (32 to a warp, neighbouring
    // ones to different blocks), so the launch does not start with every warp's
    // atomic on one counter; claims then count from there
    const uint32_t n_warps = gridDim.x * (blockDim.x >> 5);
    bool first = true;

    // Two phases, one loop.  First every lane whose pixel is complete takes the
    // next one.  Once the pixels are gone for one of the block's warps (s_drain)
    // the lanes still at work are packed into as few warps as hold them, again
    // and again as they end: a warp's step takes the binary64 pipe the same time
    // with one lane as with 32, and a pixel runs for up to samples x maxIterations
    // steps.
    bool drain = false, on = true;
    uint32_t left = blockDim.x, rounds = 0;
    for (;;) {
        // a time limit: the warp stops where it is (its samples in flight stay unwritten)
        const bool late = out_of_time(a.budget_ns, t_start, a.status, lane);
        if (!drain) {
            const uint32_t need_mask = __ballot_sync(FULL, need);
            if (need_mask && !late) {
                uint32_t base = 0;
                if (first) {
                    base = 32u * ((threadIdx.x >> 5) * gridDim.x + blockIdx.x);
                    first = false;
                } else {
                    const uint32_t leader = __ffs(need_mask) - 1u;
                    if (lane == leader) base = 32u * n_warps + atomicAdd(a.work.next, (uint32_t)__popc(need_mask));
                    base = __shfl_sync(FULL, base, leader);
                }
                if (need) {
                    pix = base + (uint32_t)__popc(need_mask & lt_mask);
                    need = false;
                    st.begin = true;
                    s = 0;
                    acc_v = 0.f;
                    acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
                }
            }
            if (late || __any_sync(FULL, pix >= a.n_pix)) {
                if (lane == 0) *(volatile uint32_t *)&s_drain = 1;
                drain = true;
            } else {
                // (the lanes' reads may straddle the store; the warp decides as one)
                drain = __any_sync(FULL, *(volatile uint32_t *)&s_drain != 0);
            }
            on = !need && pix < a.n_pix;
            rounds = 0;
        }
        if (drain) {
            on = on && !need && !late;
            if (rounds == 0) {
                pack_lanes(st, on, on, left, s_state, s_count);
                if (left == 0) break;
                need = false;
                rounds = DRAIN_ROUNDS;
            }
            --rounds;
            if (!__any_sync(FULL, on)) {
                rounds = 0;  // to the next packing
                continue;
            }
        }
        const bool active = on;

        bool done = false;
        R r2 = R(0);
        uint32_t lim = 0;  // steps this lane takes this round: a power of two <= K
        if (active) {
            if (st.begin) {
                st.begin = false;
                R px, py;
                frame_point(a, w_magic, pix, s, px, py);
                i = 0;
                if (F == FRACTAL_MANDELBROT) {
                    cx = px;
                    cy = py;
                    // the first step from z = 0 gives z = c (+0 in place of -0, as the
                    // step's own additions do); starting there spares every sample a
                    // step whose products are 0
                    x = R(0);
                    y = R(0);
                    if (a.max_iter > 0) {
                        x = Op<R>::add(cx, R(0));
                        y = Op<R>::add(cy, R(0));
                        i = 1;
                    }
                } else {
                    x = px;
                    y = py;
                    cx = a.jcx;
                    cy = a.jcy;
                }
                st.blk = blockable_c(cx, cy);
                window = 0;
                cw.reset(x, y);
                r2 = radius2<R, A>(x, y);
                if (i == a.max_iter || !(r2 < R(4))) {
                    done = true;
                } else if (F == FRACTAL_MANDELBROT && interior_c(cx, cy)) {
                    skipped += a.max_iter - i;
                    i = a.max_iter;
                    done = true;
                }
            }
            if (!done) {
                if (!st.blk) {
                    lim = 1;
                } else if (window) {
                    lim = window > 1u ? window >> 1 : 1u;
                } else {
                    uint32_t rest = a.max_iter - i;
                    lim = rest >= (uint32_t)K ? (uint32_t)K : 1u << (31 - __clz(rest));
                }
            }
        }
        // Every stepping lane runs the same K unrolled steps.  A lane with
        // lim < K keeps the state it had after lim steps (captured after steps
        // 1, 2, 4, ...): that is how a lane whose block overshot an escape
        // halves its search window each round without holding up the others.
        const bool stepping = active && !done;
        const bool partial = stepping && lim < (uint32_t)K;
        const bool any_partial = __any_sync(FULL, partial);
        // K steps of `stepper`, keeping the state after lim steps on partial lanes
        auto run_block = [&](auto stepper) {
            if (any_partial) {
                R kx = x, ky = y;
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
        if (stepping) {
            const R sx = x, sy = y;
            if constexpr (A == ARITH_PARITY) {
                // one binary64 operation fewer per step for two integer ones
                uint32_t emin = 0xffffffffu;
                run_block([&](R &u, R &v) { step_rounded6<R>(u, v, cx, cy, emin); });
                if (emin < exponent_bits_two<R>()) {
                    // a product below twice the smallest normal: redo the block literally
                    x = sx;
                    y = sy;
                    run_block([&](R &u, R &v) { step<R, A>(u, v, cx, cy); });
                }
            } else {
                uint32_t emin = 0xffffffffu;
                run_block([&](R &u, R &v) { step_fma3(u, v, cx, cy, emin); });
                if (emin == 0u) {
                    // x = 0 or subnormal: redo the block with x + x
                    x = sx;
                    y = sy;
                    run_block([&](R &u, R &v) { step<R, A>(u, v, cx, cy); });
                }
            }
            if (below_four<A>(x, y)) {
                const bool full = window == 0u && lim == (uint32_t)K;  // a checkpoint every K steps
                i += lim;
                window = window > 1u ? window - lim : 0u;
                if (full && cw.template check_every<cycle_blocks<R>()>(x, y)) {  // a repeated state: interior
                    skipped += a.max_iter - i;
                    i = a.max_iter;
                }
                if (i == a.max_iter) done = true;
            } else if (lim == 1u) {
                i += 1u;  // the escape step
                r2 = radius2<R, A>(x, y);
                done = true;
            } else {
                // the escape lies within these lim steps: search them
                x = sx;
                y = sy;
                window = lim;
            }
        }
        if (done) {
            const bool escaped = i < a.max_iter;
            const float nu = (a.smooth || a.pixels || a.rgba) ? frame_smooth(i, (float)r2, a.max_iter) : 0.f;
            const size_t sidx = (size_t)pix * a.spp + s;
            if (a.counts) a.counts[sidx] = i;
            if (a.smooth) a.smooth[sidx] = nu;
            iters += i;
            float v = escaped ? nu : (F == FRACTAL_MANDELBROT ? 0.f : (float)a.max_iter);
            acc_v = __fadd_rn(acc_v, v);
            if (a.rgba) {
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
            if (s == a.spp) {
                uint32_t px, py;
                divmod_magic(pix, a.w, w_magic, py, px);
                if (a.pixels)
                    store_pixel(pixel_ptr(a.pixels, a.pixels_pitch, px, py),
                                make_pixel(__fdiv_rn(acc_v, (float)a.spp), (float)a.spp));
                if (a.rgba) a.rgba[pix] = frame_pack_rgba(acc, a.spp);
                need = true;
            } else {
                st.begin = true;
            }
        }
    }
    if (a.total) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) iters += __shfl_down_sync(FULL, iters, o);
        if (lane == 0 && iters) atomicAdd(a.total, iters);
    }
    if (a.skipped) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) skipped += __shfl_down_sync(FULL, skipped, o);
        if (lane == 0 && skipped) atomicAdd(a.skipped, skipped);
    }
    if (lane == 0) leave_counter(a.work, &s_retired);
}

// ---------------------------------------------------------------------------
// Binary32 frames: fresh pixels and long orbits apart
// ---------------------------------------------------------------------------
//
// After interior_c most samples of a view end within a few steps, and the few
// that go on (samples close to the boundary, interiors of the smaller
// components) go on for hundreds.  Mixed in one warp, each long orbit held its
// 31 neighbours to a round of 64 steps.  So a warp takes fresh pixels 32 at a
// time and gives every sample up to `fresh_steps` steps; samples still running
// then wait in the warp's queue in shared memory, and when the queue holds a
// warp's worth they run by themselves in rounds of 64 steps, lanes that end
// refilled from the queue, until fewer than REQUEUE lanes are left.  When the
// fresh pixels are gone the block's waiting orbits are packed into as few
// warps as hold them, again and again as they end: a warp alone would run its
// few leftovers, often up to maxIterations, with most lanes idle.
//
// Fresh pixels: a fixed share first (batch k of warp w is batch k n_warps + w),
// the rest claimed 32 at a time from the work counter.  One claim per 32
// pixels from the start made the counter's address the bottleneck of cheap
// frames (32768 atomics on one word for 1024x1024 pixels).
//
// The bound is issue: 1024x1024 pixels of the whole set, maxIter 1000, take
// 20 us for the fresh part (360 instructions a batch) and 25 us for the long
// orbits, whose end is the block with the most of them.  Measured there with
// the memset of the counter: 85 us with per-lane refill in tested 64-step
// rounds, 81 with interior_c, 72 with queues alone, 55 with untested blocks for
// the long orbits, 51 with ended samples written several at a time, 46 with
// packing and the skew (FRESH_STEPS 16: 49; REQUEUE 12: 49).  256x144 pixels,
// maxIter 500: 20.6 -> 15.
//
// Samples that the iteration limit ends soon are not worth a queue: up to
// FRESH_ALL steps a batch runs to the limit as it is, and up to FRESH_ALL_SMALL
// where no warp has a second batch.  us with per-lane refill / 32 fresh steps /
// all: Julia set, 260x240 of 4 samples, maxIter 50 23 / 38 / 22, 134 46 / 50 / 28;
// 1500x1000 of 1 at 50 47 / 57 / 41, 200 71 / 72 / 69, 256 73 / 74 / 79; -1.25, span
// 0.2, 370x280 at 500 41 / 40 / 34, 2400x1700 at 200 374 / 190 / 205.
constexpr uint32_t FRESH_STEPS = 32, FRESH_ALL = 200, FRESH_ALL_SMALL = 512;
constexpr int LONG_STEPS = 64;
constexpr uint32_t REQUEUE = 24;
constexpr int MAX_EPOCH = 16;         // rounds between packings, at most
constexpr uint32_t FINISH_LANES = 12;  // samples of a warp that end before any of them is written
constexpr uint32_t QUEUE = 64;  // entries per warp: at most 31 waiting and 32 fresh

template <bool MULTI> constexpr int frame32_threads() { return MULTI ? 256 : 512; }

template <int A, int F, bool MULTI>
__global__ void __launch_bounds__(frame32_threads<MULTI>())
k_frame32(FrameArgs<float> a, uint32_t fixed_rounds, uint32_t fresh_steps)
{
    constexpr int WORDS = MULTI ? 12 : 6, WARPS = frame32_threads<MULTI>() / 32;
    __shared__ uint32_t s_pal[PALETTE_SMEM];
    __shared__ uint32_t s_queue[WARPS][WORDS][QUEUE];
    __shared__ uint32_t s_count[WARPS], s_retired;
    if (threadIdx.x == 0) s_retired = 0;
    const uint32_t *pal = a.palette;
    if (a.rgba && a.palette_len <= PALETTE_SMEM) {
        for (uint32_t k = threadIdx.x; k < a.palette_len; k += blockDim.x) s_pal[k] = a.palette[k];
        pal = s_pal;
    }
    __syncthreads();

    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lt_mask = (1u << lane) - 1u;
    const uint32_t w_magic = div_magic(a.w);
    const uint32_t wib = threadIdx.x >> 5;
    uint32_t(*q)[QUEUE] = s_queue[wib];
    uint32_t qn = 0;  // entries waiting
    const uint32_t n_warps = gridDim.x * (blockDim.x >> 5);
    // neighbouring batches go to different blocks, and a block's batches are spread
    // over the columns of frames of any width (the skew)
    const uint32_t warp = wib * gridDim.x + (blockIdx.x + 37u * wib) % gridDim.x;
    const uint32_t claim_base = 32u * n_warps * fixed_rounds;
    uint32_t round = 0;
    bool more = true;

    uint32_t pix = 0, s = 0, i = 0;
    float x = 0.f, y = 0.f, cx = 0.f, cy = 0.f, r2 = 0.f;
    float acc_v = 0.f, acc[4] = {0.f, 0.f, 0.f, 0.f};
    unsigned long long iters = 0, skipped = 0;
    const unsigned long long t_start = a.budget_ns ? global_ns() : 0ull;

    // start sample s of pixel pix; true when it ends before its first step
    auto start = [&]() -> bool {
        float px, py;
        frame_point(a, w_magic, pix, s, px, py);
        i = 0;
        if (F == FRACTAL_MANDELBROT) {
            cx = px;
            cy = py;
            x = y = 0.f;
            if (a.max_iter > 0) {  // from z = c, as k_frame
                x = __fadd_rn(cx, 0.f);
                y = __fadd_rn(cy, 0.f);
                i = 1;
            }
        } else {
            x = px;
            y = py;
            cx = a.jcx;
            cy = a.jcy;
        }
        r2 = radius2<float, A>(x, y);
        if (i == a.max_iter || !(r2 < 4.f)) return true;
        if (F == FRACTAL_MANDELBROT && interior_c(cx, cy)) {
            skipped += a.max_iter - i;
            i = a.max_iter;
            return true;
        }
        return false;
    };
    // write the sample that ended; true when its pixel is complete
    auto finish = [&]() -> bool {
        const bool escaped = i < a.max_iter;
        const float nu = (a.smooth || a.pixels || a.rgba) ? frame_smooth(i, r2, a.max_iter) : 0.f;
        const size_t sidx = (size_t)pix * a.spp + s;
        if (a.counts) a.counts[sidx] = i;
        if (a.smooth) a.smooth[sidx] = nu;
        iters += i;
        const float v = escaped ? nu : (F == FRACTAL_MANDELBROT ? 0.f : (float)a.max_iter);
        acc_v = __fadd_rn(MULTI ? acc_v : 0.f, v);
        if (a.rgba) {
            float ch[4];
            if (escaped) {
                frame_palette_lerp(pal, a.palette_len, nu, ch);
            } else {
#pragma unroll
                for (int k = 0; k < 4; k++) ch[k] = (float)((a.interior_rgba >> (8 * k)) & 255u);
            }
#pragma unroll
            for (int k = 0; k < 4; k++) acc[k] = __fadd_rn(MULTI ? acc[k] : 0.f, ch[k]);
        }
        if (MULTI && ++s < a.spp) return false;
        if (a.pixels) {
            uint32_t px, py;
            divmod_magic(pix, a.w, w_magic, py, px);
            store_pixel(pixel_ptr(a.pixels, a.pixels_pitch, px, py),
                        make_pixel(__fdiv_rn(acc_v, (float)a.spp), (float)a.spp));
        }
        if (a.rgba) a.rgba[pix] = frame_pack_rgba(acc, a.spp);
        return true;
    };
    // lanes with `put` append their samples to the queue
    auto push = [&](bool put) {
        const uint32_t mask = __ballot_sync(FULL, put);
        if (put) {
            const uint32_t at = qn + (uint32_t)__popc(mask & lt_mask);
            q[0][at] = __float_as_uint(x);
            q[1][at] = __float_as_uint(y);
            q[2][at] = __float_as_uint(cx);
            q[3][at] = __float_as_uint(cy);
            q[4][at] = i;
            q[5][at] = pix;
            if constexpr (MULTI) {
                q[6][at] = s;
                q[7][at] = __float_as_uint(acc_v);
#pragma unroll
                for (int k = 0; k < 4; k++) q[8 + k][at] = __float_as_uint(acc[k]);
            }
        }
        qn += (uint32_t)__popc(mask);
        __syncwarp();
    };
    auto pop = [&](uint32_t(*q)[QUEUE], uint32_t at) {
        x = __uint_as_float(q[0][at]);
        y = __uint_as_float(q[1][at]);
        cx = __uint_as_float(q[2][at]);
        cy = __uint_as_float(q[3][at]);
        i = q[4][at];
        pix = q[5][at];
        if constexpr (MULTI) {
            s = q[6][at];
            acc_v = __uint_as_float(q[7][at]);
#pragma unroll
            for (int k = 0; k < 4; k++) acc[k] = __uint_as_float(q[8 + k][at]);
        }
    };

    // a round of a long orbit; true when the sample ended.  While |c| allows,
    // blocks of 16 untested steps as in escape(), with no branch between them: the
    // state after the last block that ended below 4 is kept, and a block that
    // overshot is gone over again with tests, by all the lanes that overshot in
    // the round together.
    CycleWatch<float> cw;
    auto long_round = [&]() -> bool {
        const uint32_t rest = a.max_iter - i;
        bool tested = true;
        if (rest >= (uint32_t)ESCAPE_BLOCK && blockable_c(cx, cy)) {
            float kx = x, ky = y;
            uint32_t n = 0;
            bool ok = true, cyc = false;
#pragma unroll 1
            for (uint32_t end = ESCAPE_BLOCK; end <= (uint32_t)LONG_STEPS; end += ESCAPE_BLOCK) {
#pragma unroll
                for (int k = 0; k < ESCAPE_BLOCK; k++) step<float, A>(x, y, cx, cy);
                ok = ok && radius2<float, A>(x, y) < 4.f && end <= rest;
                cyc = cyc || (ok && same_state(x, cw.sx) && same_state(y, cw.sy));  // a repeated state: interior
                cw.ck += ok ? 1u : 0u;
                const bool save = ok && cw.ck == cw.save_at;
                cw.sx = save ? x : cw.sx;
                cw.sy = save ? y : cw.sy;
                cw.save_at <<= save ? 1 : 0;
                kx = ok ? x : kx;
                ky = ok ? y : ky;
                n = ok ? end : n;
            }
            x = kx;
            y = ky;
            i += n;
            if (cyc) {
                skipped += a.max_iter - i;
                i = a.max_iter;
            }
            if (i == a.max_iter) return true;
            tested = n < (uint32_t)LONG_STEPS && n + (uint32_t)ESCAPE_BLOCK <= rest;
        }
        if (tested) {
            tested_steps<float, A>(x, y, cx, cy, i, a.max_iter - i > (uint32_t)LONG_STEPS ? i + LONG_STEPS : a.max_iter, r2);
            if (!(r2 < 4.f) || i == a.max_iter) return true;
            if (cw.check(x, y)) {
                skipped += a.max_iter - i;
                i = a.max_iter;
                return true;
            }
        }
        return false;
    };
    // the samples that ended: written, the pixel's next sample started; true
    // when the pixel is complete
    auto finish_ended = [&]() -> bool {
        do {
            if (finish()) return true;
        } while (start());
        cw.reset(x, y);
        return false;
    };

    bool late = false;
    while (!late) {
        // ---- fresh pixels
        while (more && qn < 32u) {
            // a time limit: the warp stops where it is (its samples in flight stay unwritten)
            if ((late = out_of_time(a.budget_ns, t_start, a.status, lane))) break;
            uint32_t base = 0;
            if (round < fixed_rounds) {
                base = 32u * (round++ * n_warps + warp);
            } else {
                if (lane == 0) base = claim_base + atomicAdd(a.work.next, 32u);
                base = __shfl_sync(FULL, base, 0);
            }
            if (base >= a.n_pix) {
                more = false;
                break;
            }
            pix = base + lane;
            bool live = pix < a.n_pix, running = false, put = false;
            s = 0;
            acc_v = 0.f;
            acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
            do {
                if (live) {
                    bool ended = start();
                    if (!ended) {
                        const uint32_t end = a.max_iter - i > fresh_steps ? i + fresh_steps : a.max_iter;
                        tested_steps<float, A>(x, y, cx, cy, i, end, r2);
                        ended = !(r2 < 4.f) || i == a.max_iter;
                    }
                    if (ended) {
                        live = !finish();
                    } else {
                        put = true;
                        live = false;
                    }
                }
                running = MULTI && __any_sync(FULL, live);
            } while (running);
            push(put);
        }
        if (late || !more) break;
        // ---- long orbits: a warp's worth of them
        qn -= 32u;
        pop(q, qn + lane);
        __syncwarp();
        bool on = true, ended = false;
        cw.reset(x, y);
        for (;;) {
            if ((late = out_of_time(a.budget_ns, t_start, a.status, lane))) break;
            if (on && !ended) ended = long_round();
            const uint32_t end_mask = __ballot_sync(FULL, ended);
            const uint32_t running = (uint32_t)__popc(__ballot_sync(FULL, on && !ended));
            if ((uint32_t)__popc(end_mask) < FINISH_LANES && running >= REQUEUE) continue;
            if (ended) {
                on = !finish_ended();
                ended = false;
            }
            const uint32_t free_mask = __ballot_sync(FULL, !on);
            if (free_mask && qn) {
                const uint32_t k = (uint32_t)__popc(free_mask & lt_mask);
                const uint32_t take = min((uint32_t)__popc(free_mask), qn);
                if (!on && k < take) {
                    pop(q, qn - 1u - k);
                    cw.reset(x, y);
                    on = true;
                }
                qn -= take;
                __syncwarp();
            }
            if ((uint32_t)__popc(__ballot_sync(FULL, on)) < REQUEUE) {
                push(on);
                break;
            }
        }
    }
    // ---- the block's remaining orbits, one per thread (at most 31 a warp), packed
    // into as few warps as hold them every `epoch` rounds
    if (lane == 0) s_count[wib] = late ? 0u : qn;
    __syncthreads();
    uint32_t left = 0;
#pragma unroll
    for (int k = 0; k < WARPS; k++) left += s_count[k];
    bool on = threadIdx.x < left, ended = false;
    if (on) {
        uint32_t w = 0, at = threadIdx.x;
        while (at >= s_count[w]) at -= s_count[w++];
        pop(s_queue[w], at);
        cw.reset(x, y);
    }
    int epoch = 2;
    while (left) {
        late = out_of_time(a.budget_ns, t_start, a.status, lane);
        for (int k = 0; k < epoch && __any_sync(FULL, on && !ended); k++)
            if (on && !ended) ended = long_round();
        epoch = min(2 * epoch, MAX_EPOCH);  // orbits end at a falling rate
        if (ended) {
            on = !finish_ended();
            ended = false;
        }
        const uint32_t mask = __ballot_sync(FULL, on && !late);
        __syncthreads();  // the last epoch's queue and counts have been read
        if (lane == 0) s_count[wib] = (uint32_t)__popc(mask);
        __syncthreads();
        uint32_t at = (uint32_t)__popc(mask & lt_mask), now = 0;
#pragma unroll
        for (int k = 0; k < WARPS; k++) {
            at += (uint32_t)k < wib ? s_count[k] : 0u;
            now += s_count[k];
        }
        const bool pack = (now + 31u) / 32u < (left + 31u) / 32u;
        left = now;
        if (!pack) {
            on = on && !late;
            continue;
        }
        // words 0.. of every waiting orbit at [word][at], then its cycle watch
        uint32_t *flat = &s_queue[0][0][0];
        constexpr uint32_t T = frame32_threads<MULTI>();
        static_assert((WORDS + 4) * T <= WARPS * WORDS * QUEUE, "a packed orbit per thread fits the queues");
        auto swap_words = [&](bool put, uint32_t e) {
            auto word = [&](uint32_t k, auto &v) {
                if (put)
                    memcpy(&flat[k * T + e], &v, 4);
                else
                    memcpy(&v, &flat[k * T + e], 4);
            };
            word(0, x), word(1, y), word(2, cx), word(3, cy), word(4, i), word(5, pix);
            if constexpr (MULTI) {
                word(6, s), word(7, acc_v);
#pragma unroll
                for (int k = 0; k < 4; k++) word(8 + k, acc[k]);
            }
            word(WORDS, cw.sx), word(WORDS + 1, cw.sy), word(WORDS + 2, cw.ck), word(WORDS + 3, cw.save_at);
        };
        if ((mask >> lane) & 1u) swap_words(true, at);
        __syncthreads();
        on = threadIdx.x < left;
        if (on) swap_words(false, threadIdx.x);
    }
    if (a.total) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) iters += __shfl_down_sync(FULL, iters, o);
        if (lane == 0 && iters) atomicAdd(a.total, iters);
    }
    if (a.skipped) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) skipped += __shfl_down_sync(FULL, skipped, o);
        if (lane == 0 && skipped) atomicAdd(a.skipped, skipped);
    }
    if (lane == 0) leave_counter(a.work, &s_retired);
}

// ---------------------------------------------------------------------------
// Compose, under-sampled preview, debug
// ---------------------------------------------------------------------------

__global__ void __launch_bounds__(256) k_compose(ComposeArgs a)
{
    __shared__ uint32_t s_pal[PALETTE_SMEM];
    const uint32_t *pal = a.palette;
    if (!a.visualize && a.palette && a.palette_len <= PALETTE_SMEM) {
        for (uint32_t k = threadIdx.x; k < a.palette_len; k += blockDim.x) s_pal[k] = a.palette[k];
        pal = s_pal;
    }
    __syncthreads();
    // A warp takes a run of 128 pixels of one row; lane l handles pixels
    // x0 + 32k + l (k = 0..3), so every load instruction reads 32 consecutive
    // 16-byte records (512 B) and every store writes 32 consecutive words.  The
    // four records are loaded before any is composed, four loads in flight
    // (eight measured the same and cost 57 registers instead of 32).
    constexpr int R = 4;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t runs = (a.w + 32u * R - 1u) / (32u * R);
    const size_t n = (size_t)runs * a.h;
    const size_t warps = (size_t)gridDim.x * (blockDim.x / 32u);
    for (size_t c = (size_t)blockIdx.x * (blockDim.x / 32u) + (threadIdx.x >> 5); c < n; c += warps) {
        const uint32_t y = (uint32_t)(c / runs), x0 = 32u * R * (uint32_t)(c % runs);
        PixelInfo p[R];
#pragma unroll
        for (int k = 0; k < R; k++) {
            const uint32_t x = x0 + 32u * k + lane;
            if (x < a.w) p[k] = load_pixel(pixel_ptr(a.in, a.pitch, x, y));
        }
        uint32_t *row = reinterpret_cast<uint32_t *>(reinterpret_cast<char *>(a.out) + (size_t)y * (size_t)a.out_pitch);
#pragma unroll
        for (int k = 0; k < R; k++) {
            const uint32_t x = x0 + 32u * k + lane;
            if (x < a.w)
                row[x] = compose_pixel(p[k], pal, a.palette_len, a.max_ss, a.visualize, a.color_mode, a.magnifier);
        }
    }
}

template <int F>
__global__ void k_under_sampled(void *out, long pitch, uint32_t w, uint32_t h, Rect<float> r, uint32_t max_iter,
                                uint32_t level, float jcx, float jcy)
{
    const uint32_t ix = (blockDim.x * blockIdx.x + threadIdx.x) * level;
    const uint32_t iy = (blockDim.y * blockIdx.y + threadIdx.y) * level;
    if (ix >= w - level || iy >= h - level) return;
    float pw = __fdiv_rn(__fsub_rn(r.rtx, r.lbx), (float)w);
    float ph = __fdiv_rn(__fsub_rn(r.rty, r.lby), (float)h);
    float cx = __fadd_rn(r.lbx, __fmul_rn((float)ix, pw));
    float cy = __fsub_rn(r.rty, __fmul_rn((float)iy, ph));
    uint32_t e = compute_fractal<float, ARITH_PARITY, F>(max_iter, cx, cy, jcx, jcy);
    store_pixel(pixel_ptr(out, pitch, ix, iy), make_pixel((float)e, __fdiv_rn(1.f, (float)level)));
}

template <int F> __global__ void k_debug()
{
    if (blockIdx.x == 0 && threadIdx.x == 0) printf("hello from %s\n", F == FRACTAL_MANDELBROT ? "mandelbrot" : "julia");
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------


template <class R>
cudaError_t launch_main(const MainArgs<R> &a, int arith, int fractal, int sms, cudaStream_t s)
{
    if (fractal >= FRACTAL_NEWTON_WIRED) return launch_main_newton<R>(a, fractal, sms, s);
    if (arith == ARITH_PARITY)
        return fractal == FRACTAL_JULIA ? launch_main_t<R, ARITH_PARITY, FRACTAL_JULIA>(a, sms, s)
                                        : launch_main_t<R, ARITH_PARITY, FRACTAL_MANDELBROT>(a, sms, s);
    if (arith == ARITH_CONTRACTED)
        return fractal == FRACTAL_JULIA ? launch_main_t<R, ARITH_CONTRACTED, FRACTAL_JULIA>(a, sms, s)
                                        : launch_main_t<R, ARITH_CONTRACTED, FRACTAL_MANDELBROT>(a, sms, s);
    return fractal == FRACTAL_JULIA ? launch_main_t<R, ARITH_FMA, FRACTAL_JULIA>(a, sms, s)
                                    : launch_main_t<R, ARITH_FMA, FRACTAL_MANDELBROT>(a, sms, s);
}


template <class R>
cudaError_t launch_advanced(const AdvancedArgs<R> &a, int arith, int fractal, int sms, cudaStream_t s)
{
    if (fractal >= FRACTAL_NEWTON_WIRED) return launch_advanced_newton<R>(a, fractal, sms, s);
    if (arith == ARITH_PARITY)
        return fractal == FRACTAL_JULIA ? launch_advanced_t<R, ARITH_PARITY, FRACTAL_JULIA>(a, sms, s)
                                        : launch_advanced_t<R, ARITH_PARITY, FRACTAL_MANDELBROT>(a, sms, s);
    if (arith == ARITH_CONTRACTED)
        return fractal == FRACTAL_JULIA ? launch_advanced_t<R, ARITH_CONTRACTED, FRACTAL_JULIA>(a, sms, s)
                                        : launch_advanced_t<R, ARITH_CONTRACTED, FRACTAL_MANDELBROT>(a, sms, s);
    return fractal == FRACTAL_JULIA ? launch_advanced_t<R, ARITH_FMA, FRACTAL_JULIA>(a, sms, s)
                                    : launch_advanced_t<R, ARITH_FMA, FRACTAL_MANDELBROT>(a, sms, s);
}

template <int A, int F> static cudaError_t launch_frame64(const FrameArgs<double> &a, int sms, cudaStream_t s)
{
    static const int occ = occupancy(k_frame<A, F>, PERSIST_THREADS);
    unsigned long long warps = ((unsigned long long)a.n_pix + 31ull) / 32ull;
    const LaunchShape l = shape_for(warps, occ, sms);
    k_frame<A, F><<<l.blocks, l.threads, 0, s>>>(a);
    return cudaGetLastError();
}

template <int A, int F, bool MULTI> static cudaError_t launch_frame32_t(const FrameArgs<float> &a, int sms, cudaStream_t s)
{
    constexpr int threads = frame32_threads<MULTI>();
    static const int occ = occupancy(k_frame32<A, F, MULTI>, threads);
    const unsigned long long batches = ((unsigned long long)a.n_pix + 31ull) / 32ull, warps = threads / 32;
    const unsigned long long fill = (unsigned long long)occ * (unsigned long long)sms;
    const unsigned grid = (unsigned)std::min(fill, batches);
    const unsigned long long n_warps = (unsigned long long)grid * warps;
    uint32_t fixed = (uint32_t)(batches * 5ull / 8ull / n_warps);  // rounds of fixed batches
    if (fixed < 1) fixed = 1;
    const uint32_t all = batches <= n_warps ? FRESH_ALL_SMALL : FRESH_ALL;
    k_frame32<A, F, MULTI><<<grid, threads, 0, s>>>(a, fixed, a.max_iter <= all ? all : FRESH_STEPS);
    return cudaGetLastError();
}
template <int A, int F> static cudaError_t launch_frame32(const FrameArgs<float> &a, int sms, cudaStream_t s)
{
    return a.spp > 1 ? launch_frame32_t<A, F, true>(a, sms, s) : launch_frame32_t<A, F, false>(a, sms, s);
}

template <class R>
cudaError_t launch_frame(const FrameArgs<R> &a, int arith, int fractal, int sms, cudaStream_t s)
{
    const bool julia = fractal == FRACTAL_JULIA;
    if constexpr (sizeof(R) == 4) {
        if (arith == ARITH_PARITY)
            return julia ? launch_frame32<ARITH_PARITY, FRACTAL_JULIA>(a, sms, s)
                         : launch_frame32<ARITH_PARITY, FRACTAL_MANDELBROT>(a, sms, s);
        return julia ? launch_frame32<ARITH_FMA, FRACTAL_JULIA>(a, sms, s)
                     : launch_frame32<ARITH_FMA, FRACTAL_MANDELBROT>(a, sms, s);
    } else {
        if (arith == ARITH_PARITY)
            return julia ? launch_frame64<ARITH_PARITY, FRACTAL_JULIA>(a, sms, s)
                         : launch_frame64<ARITH_PARITY, FRACTAL_MANDELBROT>(a, sms, s);
        return julia ? launch_frame64<ARITH_FMA, FRACTAL_JULIA>(a, sms, s)
                     : launch_frame64<ARITH_FMA, FRACTAL_MANDELBROT>(a, sms, s);
    }
}

cudaError_t launch_compose(const ComposeArgs &a, cudaStream_t s)
{
    unsigned long long runs = (unsigned long long)((a.w + 127u) / 128u) * a.h;  // one warp each
    unsigned long long blocks = (runs + 7ull) / 8ull;
    if (blocks > 152ull * 16ull) blocks = 152ull * 16ull;
    if (blocks < 1) blocks = 1;
    k_compose<<<(unsigned)blocks, 256, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_under_sampled(void *out, long pitch, uint32_t w, uint32_t h, Rect<float> rect, uint32_t max_iter,
                                 uint32_t level, int fractal, double jcx, double jcy, cudaStream_t s)
{
    dim3 block(32, 32);
    dim3 grid((w + 31u) / 32u, (h + 31u) / 32u);
    if (fractal == FRACTAL_JULIA)
        k_under_sampled<FRACTAL_JULIA><<<grid, block, 0, s>>>(out, pitch, w, h, rect, max_iter, level, (float)jcx,
                                                              (float)jcy);
    else
        k_under_sampled<FRACTAL_MANDELBROT><<<grid, block, 0, s>>>(out, pitch, w, h, rect, max_iter, level, 0.f, 0.f);
    return cudaGetLastError();
}

cudaError_t launch_debug(int fractal, cudaStream_t s)
{
    if (fractal >= FRACTAL_NEWTON_WIRED) return cudaSuccess;  // the Newton modules' debugFractal is empty
    if (fractal == FRACTAL_JULIA)
        k_debug<FRACTAL_JULIA><<<1, 1, 0, s>>>();
    else
        k_debug<FRACTAL_MANDELBROT><<<1, 1, 0, s>>>();
    return cudaGetLastError();
}

template <class R> __global__ void __launch_bounds__(256) k_fma_peak(uint32_t iters, double *sink)
{
    R a[8];
#pragma unroll
    for (int k = 0; k < 8; k++) a[k] = R(threadIdx.x + k) * R(1e-3);
    const R m = R(0.999999), c = R(1e-7);
    for (uint32_t i = 0; i < iters; i++) {
#pragma unroll
        for (int k = 0; k < 8; k++) a[k] = Op<R>::fma(a[k], m, c);
    }
    R t = R(0);
#pragma unroll
    for (int k = 0; k < 8; k++) t += a[k];
    if (t == R(-1)) sink[0] = (double)t;  // never true; keeps the chains live
}

cudaError_t launch_fma_peak(bool dbl, int blocks, uint32_t iters, double *sink, cudaStream_t s)
{
    if (dbl)
        k_fma_peak<double><<<blocks, 256, 0, s>>>(iters, sink);
    else
        k_fma_peak<float><<<blocks, 256, 0, s>>>(iters, sink);
    return cudaGetLastError();
}

template cudaError_t launch_main<float>(const MainArgs<float> &, int, int, int, cudaStream_t);
template cudaError_t launch_main<double>(const MainArgs<double> &, int, int, int, cudaStream_t);
template cudaError_t launch_advanced<float>(const AdvancedArgs<float> &, int, int, int, cudaStream_t);
template cudaError_t launch_advanced<double>(const AdvancedArgs<double> &, int, int, int, cudaStream_t);
template cudaError_t launch_frame<float>(const FrameArgs<float> &, int, int, int, cudaStream_t);
template cudaError_t launch_frame<double>(const FrameArgs<double> &, int, int, int, cudaStream_t);

}  // namespace chaos
