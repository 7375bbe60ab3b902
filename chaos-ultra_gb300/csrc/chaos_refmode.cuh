// chaos_refmode.cuh -- the reference-mode persistent kernels (fractalRenderMain
// and fractalRenderAdvanced semantics, gen.cu:168-181, 307-368): persistent
// warps take 8x4 pixel tiles from a work counter; one tile is one vote group
// of the adaptive super-sampling.  Included by chaos_kernels.cu (escape-time
// modules) and chaos_newton.cu (Newton modules, built without contraction).
#pragma once

#include <algorithm>

#include "chaos_claim.cuh"
#include "chaos_kernels.cuh"

namespace chaos {

constexpr uint32_t FULL = 0xffffffffu;
constexpr int PERSIST_THREADS = 256;


__device__ __forceinline__ void add_total(unsigned long long *total, unsigned long long iters, uint32_t lane)
{
    if (!total) return;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) iters += __shfl_down_sync(FULL, iters, o);
    if (lane == 0 && iters) atomicAdd(total, iters);
}

// Tiles are claimed in strips of consecutive tiles.  With one counter for the
// whole frame, a claim per tile made the counter the bottleneck of large
// reuse-dominated frames, whose tiles take a few loads each.  Claims are
// guided: a quarter of an even share of the tiles left after the warp's
// previous strip, between 1 and `max_chunk`, so long strips early keep the
// counter quiet and short ones late keep the end of the frame balanced.
// AHEAD (short, even tiles): a strip of several tiles is claimed before the one
// before it is rendered.  Where a tile may run for long, the strip that its warp
// holds already would wait as long, so strips are claimed when needed
// (1801x1769, maxIter 1600, 5 samples, strips of two: 413 us ahead, 348).
// SPREAD: the warps' first strips go out without a claim, neighbouring ones to
// different SMs.  Claimed, a block's warps take neighbouring tiles: the sampled
// border at the top of a binary64 zoom-out was on a third of the SMs, eight warps
// to a binary64 pipe (966x515, maxIter 300, 2 samples 385 -> 306 us; in binary32,
// where the rows' reads come from the L2 together, 5199x4054 382 -> 403).
template <bool AHEAD, bool SPREAD, class Body>
__device__ __forceinline__ void for_each_strip(uint32_t *counter, uint32_t n_tiles, uint32_t max_chunk, uint32_t lane,
                                               Body body)
{
    const uint32_t warps = gridDim.x * (blockDim.x >> 5), share = 4u * warps;
    auto size_after = [&](uint32_t at) -> uint32_t {
        const uint32_t c = (at < n_tiles ? n_tiles - at : 0u) / share;
        return c < 1u ? 1u : c > max_chunk ? max_chunk : c;
    };
    uint32_t size = size_after(0u), claim = 0;
    const uint32_t base = SPREAD ? warps * size : 0u;  // claims count from here
    if (SPREAD)
        claim = ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * size;
    else if (lane == 0)
        claim = atomicAdd(counter, size);
    uint32_t t0 = __shfl_sync(FULL, claim, 0);
    while (t0 < n_tiles) {
        const uint32_t t1 = min(t0 + size, n_tiles);
        const bool ahead = AHEAD && size > 1u;
        if (ahead) {
            size = size_after(t1);
            if (lane == 0) claim = base + atomicAdd(counter, size);
        }
        body(t0, t1);
        if (!ahead) {
            size = size_after(t1);
            if (lane == 0) claim = base + atomicAdd(counter, size);
        }
        t0 = __shfl_sync(FULL, claim, 0);
    }
}

// The same with strips of up to `strip` tiles from the block's pieces, each
// taken when it is needed.
template <class Body> __device__ __forceinline__ void for_each_claim(Claims &claims, uint32_t strip, Body body)
{
    for (;;) {
        uint32_t got;
        const uint32_t t0 = claims.take(strip, got);
        if (got == 0u) break;
        body(t0, t0 + got);
    }
}

// A tile's column and row in a frame `tiles_x` tiles wide, stepped tile by
// tile: one division per strip instead of two per tile (a reuse tile is ~90
// instructions; the divisions were another ~100).
struct TileCursor {
    uint32_t tx, ty;
    __device__ __forceinline__ TileCursor(uint32_t t, uint32_t tiles_x) : tx(t % tiles_x), ty(t / tiles_x) {}
    __device__ __forceinline__ void next(uint32_t tiles_x)
    {
        if (++tx == tiles_x) {
            tx = 0;
            ++ty;
        }
    }
    // the cursor k tiles further on
    __device__ __forceinline__ TileCursor plus(uint32_t k, uint32_t tiles_x) const
    {
        TileCursor c = *this;
        c.tx += k;
        while (c.tx >= tiles_x) {
            c.tx -= tiles_x;
            ++c.ty;
        }
        return c;
    }
    __device__ __forceinline__ uint32_t x0() const { return 8u * tx; }
    __device__ __forceinline__ uint32_t y0() const { return 4u * ty; }
};

// body(x0, y0) for every tile claimed, (x0, y0) its top-left pixel
template <bool AHEAD, class Body>
__device__ __forceinline__ void for_each_tile(uint32_t *counter, uint32_t n_tiles, uint32_t tiles_x, uint32_t chunk,
                                              uint32_t lane, Body body)
{
    for_each_strip<AHEAD, false>(counter, n_tiles, chunk, lane, [&](uint32_t t0, uint32_t t1) {
        TileCursor c(t0, tiles_x);
        for (uint32_t t = t0; t < t1; t++, c.next(tiles_x)) body(c.x0(), c.y0());
    });
}

// The longest strip a warp claims: up to `cap` tiles, while every resident
// warp still gets 8 claims.  (An 8K reuse frame is a million tiles: at 4 per
// claim its single work counter took a quarter of a million atomics in
// ~0.3 ms.)
static inline uint32_t tile_chunk_for(uint32_t n_tiles, int occ, int sms, uint32_t cap = 16)
{
    const unsigned long long warps = (unsigned long long)occ * sms * (PERSIST_THREADS / 32);
    unsigned long long c = n_tiles / (warps * 8ull);
    return (uint32_t)(c < 1 ? 1 : c > cap ? cap : c);
}

template <class R, int A, int F> __global__ void __launch_bounds__(PERSIST_THREADS) k_main(MainArgs<R> a)
{
    __shared__ uint32_t s_retired;
    if (threadIdx.x == 0) s_retired = 0;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u;
    SampleGeometry<R> g = make_geometry(a.image, a.size, a.max_iter, a.jcx, a.jcy);
    g.newton = a.newton;
    unsigned long long iters = 0;
    constexpr bool even = F >= FRACTAL_NEWTON_WIRED;  // Newton tiles
    for_each_tile<even>(a.work.next, a.n_tiles, a.tiles_x, a.tile_chunk, lane, [&](uint32_t x0, uint32_t y0) {
        render_main_tile<R, A, F>(g, a.out, a.pitch, a.size, x0, y0, lane, a.max_ss, a.flags, iters);
    });
    add_total(a.total, iters, lane);
    if (lane == 0) leave_counter(a.work, &s_retired);
}

constexpr uint32_t PIECE_TILES = 4 * PERSIST_THREADS / 32;  // a group of four for each warp

// Tiles whose previous-frame reads are in flight together.  A reuse-dominated
// frame is a stream of small dependent steps per tile (origin -> four loads
// -> filter -> store); with one tile's loads in flight per warp and the
// origin's four divisions computed per pixel it ran at about half the copy
// rate, bound by the loads' latency and the issue of the divisions.  Two
// tiles (eight 8-byte loads per lane) measured best: four need registers
// that cost a fifth of the warps.
// The strip [t0, t1) of a fractalRenderAdvanced frame, in groups of four
// tiles (32x4 pixels).  The reuse reads of a group run in row order: lane l
// takes column l & 7 of the group's tile l >> 3 and walks its four rows, so
// that a warp's read of one row covers 32 consecutive pixels (contiguous
// records under a near-identity warp), and the reads of all four rows are in
// flight before the first is filtered.  The origin's column term is the
// lane's own; its row terms are computed once per row (lane l: row l & 3 of
// tile (l >> 2) & 3) and taken by shuffles.  The filtered (value, weight)
// pairs (the weight -1 where the origin is out of range) go to the warp's
// `stage` (4 x 32 pairs of shared memory), from which each tile is finished
// in its own 8x4 lane layout (votes, samples, record): the group's tiles that
// only reuse first, then the others, in a loop of their own with one copy of
// the sampling code.  Sampled within the loop of all four, which is unrolled,
// it was 200 KB of code (790 KB in binary64; 74 and 229 so), and the warps of a
// frame that samples its borders waited for instructions (1.7 of every 13 cycles
// a warp is resident for an instruction; 0.8 with less code): zooming out at
// 7000x4000, span 3, maxIter 133, 2 samples 252 -> 209 us, 4681x4384 184 -> 164,
// 5199x4054 of the antenna, maxIter 274, 435 -> 382.
template <class R, int A, int F, bool AL8>
__device__ __forceinline__ void advanced_strip(const AdvancedArgs<R> &a, const SampleGeometry<R> &g, uint32_t lane,
                                               float2 *stage, uint32_t t0, uint32_t t1, unsigned long long &iters)
{
    // (frames smaller than 5x5 pixels reuse nothing, see reuse_axis)
    const bool reuse = (a.m.flags & FLAG_SAMPLE_REUSE) != 0 && a.m.size.x >= 5u && a.m.size.y >= 5u;
    // zooming in with foveation, a reusing pixel in the foveal region takes new samples
    const bool fov =
        (a.m.flags & FLAG_FOVEATION) && (a.m.flags & FLAG_IS_ZOOMING) && (a.m.flags & FLAG_ZOOMING_IN);
    const uint32_t col = 4u * (lane >> 4) + (lane & 3u), row = (lane >> 2) & 3u;  // the 8x4 tile layout
    const uint32_t tiles_x = a.m.tiles_x;
    TileCursor cur(t0, tiles_x);  // the next tile to finish
    for (uint32_t tg = t0; tg < t1; tg += 4u) {
        const uint32_t ng = min(4u, t1 - tg);
        if (reuse) {
            // this lane's column (of its tile k; lanes past the group's end repeat its last tile)
            const uint32_t k = min(lane >> 3, ng - 1u);
            const TileCursor tc = cur.plus(k, tiles_x);
            const TileCursor tr = cur.plus(min((lane >> 2) & 3u, ng - 1u), tiles_x);
            const uint32_t x = tc.x0() + (lane & 7u);
            const ReuseAxis mx = reuse_axis(warping_origin_x<R, A>(x, a.m.size, a.m.image, a.image_reused), a.m.size.x);
            const ReuseAxis my = reuse_axis(
                warping_origin_y<R, A>(tr.y0() + (lane & 3u), a.m.size, a.m.image, a.image_reused), a.m.size.y);
            ReuseFetch f[4];
#pragma unroll
            for (uint32_t r = 0; r < 4u; r++) {
                ReuseAxis ay;
                ay.at = __shfl_sync(FULL, my.at, 4u * k + r);
                ay.frac = __shfl_sync(FULL, my.frac, 4u * k + r);
                f[r] = reuse_fetch<AL8>(mx, ay, a.in, a.in_pitch);
            }
#pragma unroll
            for (uint32_t r = 0; r < 4u; r++) {
                float vv, ww;
                reuse_filter<A>(f[r], vv, ww);
                stage[32u * r + lane] = make_float2(vv, f[r].in_range ? ww : -1.f);
            }
            __syncwarp();
        }
        // the tiles whose pixels all reuse and take no new samples: the record is
        // (value, weight, isReused = 1, 0), as the full path stores it
        TileCursor at = cur;
        uint32_t rest = 0;  // the others
        for (uint32_t k = 0; k < ng; k++, at.next(tiles_x)) {
            const uint32_t x0 = at.x0(), y0 = at.y0();
            const UInt2 p = tile_pixel(x0, y0, lane);
            const bool valid = p.x < a.m.size.x && p.y < a.m.size.y;
            const float2 vw = reuse ? stage[32u * row + 8u * k + col] : make_float2(0.f, 0.f);
            const bool reusing = valid && reuse && !(vw.y < 0.1f);
            if ((!fov || clear_of_fovea(a.focus, x0, y0)) && __all_sync(FULL, reusing || !valid)) {
                if (valid) {
                    PixelInfo rec = make_pixel(vw.x, vw.y);
                    rec.is_reused = 1;
                    store_pixel_streaming(pixel_ptr(a.m.out, a.m.pitch, p.x, p.y), rec);
                }
            } else {
                rest |= 1u << k;
            }
        }
        while (rest) {
            const uint32_t k = __ffs(rest) - 1u;
            rest &= rest - 1u;
            const TileCursor c = cur.plus(k, tiles_x);
            const UInt2 p = tile_pixel(c.x0(), c.y0(), lane);
            const bool valid = p.x < a.m.size.x && p.y < a.m.size.y;
            const float2 vw = reuse ? stage[32u * row + 8u * k + col] : make_float2(0.f, 0.f);
            finish_advanced_tile<R, A, F>(g, a.m.out, a.m.pitch, a.m.size, a.focus, c.x0(), c.y0(), lane, a.m.max_ss,
                                          a.m.flags, valid && reuse && !(vw.y < 0.1f), vw.x, vw.y, iters);
        }
        cur = at;
        __syncwarp();
    }
}

// PIECES: strips of one group from 32-tile pieces that a block claims, for large
// frames with a foveal region, whose tiles take samples: guided strips of up to
// 16 tiles gave one warp that many of them, and single groups from the one
// counter are 65,000 claims of 2 ns.  3840x2160, zooming in: 142 -> 112 us.  A
// resting 7680x4320 frame takes 209 us with guided strips and 240 with pieces
// (64- and 128-tile pieces 268 and 276, guided strips of up to 32 tiles 235: the
// longer a warp's strip, the wider the band of rows that is read at a time).
template <class R, int A, int F, bool PIECES>
__global__ void __launch_bounds__(PERSIST_THREADS) k_advanced(AdvancedArgs<R> a)
{
    const uint32_t lane = threadIdx.x & 31u;
    SampleGeometry<R> g = make_geometry(a.m.image, a.m.size, a.m.max_iter, a.m.jcx, a.m.jcy);
    g.newton = a.m.newton;
    unsigned long long iters = 0;
    __shared__ float2 s_stage[PERSIST_THREADS / 32][4 * 32];
    __shared__ uint32_t s_retired;
    if (threadIdx.x == 0) s_retired = 0;
    __syncthreads();
    float2 *stage = s_stage[threadIdx.x >> 5];
    const bool al8 = ((reinterpret_cast<uintptr_t>(a.in) | (uintptr_t)a.in_pitch) & 7u) == 0;
    auto each = [&](auto strip) {
        if constexpr (PIECES) {
            __shared__ ClaimShared s_claims;
            Claims claims(s_claims, a.m.work.next, ClaimPlan{a.m.n_tiles, PIECE_TILES});
            __syncthreads();
            for_each_claim(claims, 4u, strip);
        } else {
            for_each_strip<true, sizeof(R) == 8>(a.m.work.next, a.m.n_tiles, a.m.tile_chunk, lane, strip);
        }
    };
    if (PIECES || al8)
        each([&](uint32_t t0, uint32_t t1) { advanced_strip<R, A, F, true>(a, g, lane, stage, t0, t1, iters); });
    else
        each([&](uint32_t t0, uint32_t t1) { advanced_strip<R, A, F, false>(a, g, lane, stage, t0, t1, iters); });
    add_total(a.m.total, iters, lane);
    if (lane == 0) leave_counter(a.m.work, &s_retired);
}

template <class KernelPtr> static int occupancy(KernelPtr k, int threads)
{
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, threads, 0) != cudaSuccess || n < 1) n = 1;
    return n;
}

struct LaunchShape {
    unsigned blocks, threads;
};

// The launch for work that `work_warps` warps share, up to `occ` blocks an SM.
// Work that fits goes out in blocks sized for the busiest SM: it gets no more than
// an even share, rounded up to whole warps of each of its blocks (just above a
// multiple of the SMs others get fewer: 153 tiles are 77 blocks of two warps).
// Full blocks put the 437 tiles of a 150x90
// frame on 55 of the 152 SMs and a 300x200 frame's 1900 on 86 SMs twice and on
// 66 once.  Seahorse valley, maxIter 3500, 2 samples in binary64, whose warps
// queue for their SM's pipe: 2823 / 1767 us and 5543 /
// 4970, 400x250 8265 / 7855; 160x100 of 4 samples in binary32: 82 / 78 us.
static inline LaunchShape shape_for(unsigned long long work_warps, int occ, int sms)
{
    constexpr unsigned FULL_WARPS = PERSIST_THREADS / 32;
    const unsigned long long per_sm = std::max(1ull, (work_warps + (unsigned)sms - 1ull) / (unsigned)sms);
    const unsigned long long n = std::min((per_sm + FULL_WARPS - 1ull) / FULL_WARPS, (unsigned long long)occ);
    const unsigned warps = (unsigned)std::min((per_sm + n - 1ull) / n, (unsigned long long)FULL_WARPS);
    const unsigned long long blocks = std::min((work_warps + warps - 1ull) / warps, n * (unsigned)sms);
    return {(unsigned)std::max(1ull, blocks), 32u * warps};
}

// k_main's residency for escape-time tiles.  A tile across the boundary runs up
// to maxIterations sample after sample, and the last such tiles are the launch's
// end: with 64 warps an SM each had a sixteenth of its scheduler, with 32 an
// eighth, and 32 still fill the issue slots before that (three blocks are slower
// for shallow frames: 219 against 200 us at 3840x2160, maxIter 64).  Newton tiles
// are short and even: they keep all warps (136 against 139 us at 1920x1080).
// Binary64 tiles queue for one pipe, which four warps a scheduler fill: two
// blocks (with 1 / 2 / 4: 500x300 of 2 samples 7.71 / 7.42 / 7.93 ms, 853x479 of 1
// 14.29 / 13.91 / 14.00, 640x400 of 4 24.07 / 23.08 / 23.11).  Float-float ones are
// binary32 work.
template <class R, int A> constexpr int main_blocks() { return sizeof(R) == 8 && A != ARITH_FLOATFLOAT ? 2 : 4; }

// And their longest strip of tiles.  Single tiles make the counter the bound of
// shallow frames (0.7 ns a claim), strips lengthen the frame's end: one warp
// renders a strip, and its worst case, every step of every sample, is about 8 ns
// a step.  So the tiles past a strip's first may cost a thirtieth of the least
// such a frame takes, about 0.45 ns (1 + worst / 600) a tile; frames with 32 tiles
// a warp and more, which a claim a tile could hold up by a quarter of a
// millisecond, have strips of two at least.  Binary64 tiles take longer than a claim.
// us with strips of up to 1 / 2 / 4 / 8, default view: 1801x1769 of 1 sample at
// maxIter 64 83 / 68 / 69 / 69, 250 81 / 71 / 71 / 71, of 5 at 250 124 / 137 / 137 / 137, 1600
// 282 / 348 / 356 / 356; 3840x2160 of 1 at 64 189 / 143 / 137 / 135, 250 188 / 154 / 154 /
// 157, 1600 229 / 231 / 252 / 269; 7680x4320 at 64 719 / 501 / 475 / 465, 250 713 / 544 /
// 521 / 519, 1600 776 / 720 / 728 / 769 (all points outside 717 / 386 / 357 / 344).
// Longer strips after short tiles: lost wherever the boundary came next (3840x2160 at
// 1600: 274 us; 1801x1769 in binary64 at 250: 885 -> 1035).
template <class R>
static inline uint32_t main_strip(uint32_t n_tiles, int occ, int sms, uint32_t max_iter, float max_ss)
{
    if (sizeof(R) == 8) return 1;
    const double worst = std::max(1.0, (double)max_iter * std::max(1.0, (double)max_ss));
    const double least = 0.45 * n_tiles * (1.0 + worst / 600.0);  // ns
    const double floor = n_tiles / 32u >= (uint32_t)(occ * sms * (PERSIST_THREADS / 32)) ? 2.0 : 1.0;
    return (uint32_t)std::min(8.0, std::max(floor, 1.0 + least / 30.0 / (8.0 * worst)));
}

template <class R, int A, int F> static cudaError_t launch_main_t(const MainArgs<R> &args, int sms, cudaStream_t s)
{
    constexpr bool newton = F >= FRACTAL_NEWTON_WIRED;
    static const int fit = occupancy(k_main<R, A, F>, PERSIST_THREADS);
    const int occ = newton ? fit : std::min(main_blocks<R, A>(), fit);
    MainArgs<R> a = args;
    a.tile_chunk = newton ? tile_chunk_for(a.n_tiles, occ, sms)
                          : tile_chunk_for(a.n_tiles, occ, sms, main_strip<R>(a.n_tiles, occ, sms, a.max_iter, a.max_ss));
    const LaunchShape l = shape_for((a.n_tiles + a.tile_chunk - 1) / a.tile_chunk, occ, sms);
    k_main<R, A, F><<<l.blocks, l.threads, 0, s>>>(a);
    return cudaGetLastError();
}

template <class R, int A, int F>
static cudaError_t launch_advanced_t(const AdvancedArgs<R> &args, int sms, cudaStream_t s)
{
    static const int occ = occupancy(k_advanced<R, A, F, false>, PERSIST_THREADS);
    AdvancedArgs<R> a = args;
    a.m.tile_chunk = tile_chunk_for(a.m.n_tiles, occ, sms);
    if constexpr (sizeof(R) == 4 && F <= FRACTAL_JULIA) {
        // where guided strips would hold whole groups (smaller frames go tile by
        // tile), and the previous frame's pairs can be read 8 bytes at a time
        const bool fov =
            (a.m.flags & FLAG_FOVEATION) && (a.m.flags & FLAG_IS_ZOOMING) && (a.m.flags & FLAG_ZOOMING_IN);
        const bool al8 = ((reinterpret_cast<uintptr_t>(a.in) | (uintptr_t)a.in_pitch) & 7u) == 0;
        if (fov && al8 && a.m.tile_chunk >= 4u) {
            static const int occ_p = occupancy(k_advanced<R, A, F, true>, PERSIST_THREADS);
            const LaunchShape l = shape_for((a.m.n_tiles + 3u) / 4u, occ_p, sms);
            k_advanced<R, A, F, true><<<l.blocks, l.threads, 0, s>>>(a);
            return cudaGetLastError();
        }
    }
    const LaunchShape l = shape_for((a.m.n_tiles + a.m.tile_chunk - 1) / a.m.tile_chunk, occ, sms);
    k_advanced<R, A, F, false><<<l.blocks, l.threads, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace chaos
