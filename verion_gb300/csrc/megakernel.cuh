// Whole paths in one launch: the megakernel (shaders/pathtrace.slang), and the streaming wavefront's tail.
#pragma once
#include "kernels.cuh"

namespace vgk {

// ---------------------------------------------------------------------------------------------
// Block wavefront. A thread that runs its path alone (trace, shade, trace, ...) shares its SM with paths
// at other places of a large kernel: 8 of 32 lanes active, and 25 cycles per issue with no instruction
// fetched yet. Here a block keeps up to BLOCK_SLOTS paths, each a pixel that runs its samples one after the
// other, and moves them together through the stages of the streaming wavefront (trace with dynamic
// fetch, resolve, shade by class), its queues in shared memory, its paths in the wave planes. A slot whose
// pixel is done takes the next one. Stages are a block barrier apart instead of a launch: nothing waits
// for the chip's slowest ray, and there is no host in the loop. Same functions, same order per pixel, same
// sums.
//
// One block per SM, so that all its warps run the same code (the shade code alone is larger than the
// instruction cache): 8 samples of a 641x359 frame of the 110k-triangle scene and of a 1920x1080 frame
// of the 1M-triangle one took 11.9 and 97 ms with a path per thread; with blocks of 128 threads, four to an SM,
// 5.1 and 47.5 ms; 256, two to an SM, 3.9 and 41.1; 512, one, 3.6 and 38.7; 768, one, 3.85 and 34.3; 1024,
// one (64 registers), 4.0 and 33.6.
constexpr uint32_t BLOCK_SLOTS = 3072;
// Threads of a block: the megakernel's, over whole frames, and the tail's, over at most some hundred
// thousand slots (640x360, 8 samples: 7.12 ms with 512, 7.27 with 768, 7.41 with 1024).
constexpr uint32_t MK_THREADS = 768, FINISH_THREADS = 512;

// Appends the `pred` lanes of a converged warp to a queue in shared memory, from its front (step 1) or from
// its back (step -1, `queue` at its last word).
static __device__ __forceinline__ void shared_append(uint32_t* count, uint16_t* queue, int step, bool pred, uint32_t value)
{
    uint32_t b = __ballot_sync(FULL, pred);
    if (b == 0)
        return;
    uint32_t base = 0;
    if (lane_id() == 0)
        base = atomicAdd(count, __popc(b));
    base = __shfl_sync(FULL, base, 0);
    if (pred)
        queue[step * (int)(base + __popc(b & ((1u << lane_id()) - 1u)))] = (uint16_t)value;
}

static __device__ __forceinline__ bool pixel_active(const Ctx& c, bool f64, uint32_t pixel)
{
    return f64 ? pixelActive<double>(c, pixel) : pixelActive<float>(c, pixel);
}

// Where a block's slots get their pixels: the megakernel's come from a counter over the frame, slot k of
// block b in plane entry b x slots + k; the tail's are the entries left in a wave's queue, which stay where
// they are. take(k, want): lanes with `want` get the next pixel for local slot k (one atomic per warp and
// round; every lane of the warp calls it), and say whether it has a shadow ray in flight.
template <bool LIGHT>
struct FrameSource {
    uint32_t* pixels;
    uint32_t* next;
    uint32_t first;
    bool f64;
    __device__ __forceinline__ uint32_t slot(const uint32_t*, uint32_t k) const { return first + k; }
    __device__ __forceinline__ uint32_t pixel(uint32_t p) const { return pixels[p]; }
    // Work items run through 16 x 8 tiles; those outside the frame and converged pixels are skipped.
    __device__ __forceinline__ bool take(const Ctx& c, const Wave& w, uint32_t*, uint32_t k, bool want, bool& shadow) const
    {
        uint32_t width = c.p[P_WIDTH], height = c.p[P_HEIGHT];
        uint32_t tiles_x = (width + 15) / 16;
        uint32_t nitems = tiles_x * ((height + 7) / 8) * 128u;
        bool got = false;
        shadow = false;
        for (;;) {
            uint32_t need = __ballot_sync(FULL, want);
            if (need == 0)
                return got;
            uint32_t base = 0;
            if (lane_id() == 0)
                base = atomicAdd(next, __popc(need));
            base = __shfl_sync(FULL, base, 0);
            if (base >= nitems)
                return got;
            if (want) {
                uint32_t idx = base + __popc(need & ((1u << lane_id()) - 1u));
                uint32_t t = idx >> 7, r = idx & 127u;
                uint32_t x = (t % tiles_x) * 16 + (r & 15u), y = (t / tiles_x) * 8 + (r >> 4);
                if (idx >= nitems) {
                    want = false;
                } else if (x < width && y < height && (c.p[P_ADAPTIVE] == 0 || pixel_active(c, f64, y * width + x))) {
                    uint32_t p = first + k;
                    storePath<LIGHT>(w, generatePathFor<LIGHT>(c, x, y, c.p[P_SAMPLE]), p);
                    w.meta[p] = 0;
                    w.flags[p] = SLOT_RAY;
                    pixels[p] = y * width + x;
                    got = true;
                    want = false;
                }
            }
        }
    }
};

struct QueueSource {
    const uint32_t* queue;
    uint32_t count;
    uint32_t* next;
    __device__ __forceinline__ uint32_t slot(const uint32_t* slot_of, uint32_t k) const { return slot_of[k]; }
    __device__ __forceinline__ uint32_t pixel(uint32_t p) const { return p; }
    __device__ __forceinline__ bool take(const Ctx&, const Wave& w, uint32_t* slot_of, uint32_t k, bool want, bool& shadow) const
    {
        shadow = false;
        uint32_t need = __ballot_sync(FULL, want);
        if (need == 0)
            return false;
        uint32_t base = 0;
        if (lane_id() == 0)
            base = atomicAdd(next, __popc(need));
        base = __shfl_sync(FULL, base, 0);
        uint32_t i = base + __popc(need & ((1u << lane_id()) - 1u));
        if (!want || i >= count)
            return false;
        uint32_t p = queue[i];
        slot_of[k] = p;
        shadow = (w.flags[p] & SLOT_SHADOW) != 0;
        return true;
    }
};

// The block's paths, from its source's first pixels until it has none left and all are done. `slots`: at most
// BLOCK_SLOTS. slot_of: shared memory for QueueSource.
template <uint32_t THREADS, bool LIGHT, bool RESTIR, bool CACHE, typename Source>
__device__ __forceinline__ void block_wavefront(const Ctx& c, const Wave& w, const Source& src, uint32_t slots, bool f64,
                                                const CacheWave& q, uint32_t* slot_of)
{
    // by_class[j]: class 2 j from the front, 2 j + 1 from the back.
    __shared__ uint16_t live[2][BLOCK_SLOTS], by_class[2][BLOCK_SLOTS], shadow[BLOCK_SLOTS];
    __shared__ uint32_t n_live[2], n_class[SHADE_CLASSES], n_shadow[2], fetch;
    uint32_t tid = threadIdx.x, in = 0;
    if (tid < 2)
        n_live[tid] = n_shadow[tid] = 0;
    if (tid == 0)
        fetch = 0;
    __syncthreads();
    for (uint32_t k = tid; k < (slots + 31u) / 32u * 32u; k += THREADS) {
        bool sh;
        bool got = src.take(c, w, slot_of, k, k < slots, sh);
        shared_append(&n_live[0], live[0], 1, got, k);
        shared_append(&n_shadow[0], shadow, 1, sh, k);
    }
    __syncthreads();
    for (;;) {
        uint32_t out = in ^ 1u, rays = n_live[in], count = rays + n_shadow[in];
        if (rays == 0)
            break;
        // Path rays, then shadow rays. Meanwhile nobody reads the counters that the next stages fill.
        if (tid == 0)
            n_live[out] = n_shadow[out] = 0;
        if (tid < SHADE_CLASSES)
            n_class[tid] = 0;
        vgt::trace_queue<vgt::HITS_EITHER>(
            c.s.nodes, c.s.tris, &fetch, count, c.err, w.refill, w.steps,
            [&](uint32_t i, V3& o, V3& d, float& tmax, bool& any) {
                any = i >= rays;
                if (!any)
                    return slot_ray(w, src.slot(slot_of, live[in][i]), o, d, tmax);
                slot_shadow_ray(w, src.slot(slot_of, shadow[i - rays]), o, d, tmax);
                return c.s.shadow_any != 0;
            },
            [&](uint32_t i, const vgt::TraceHit& h) {
                if (i < rays)
                    put_slot_hit(w, src.slot(slot_of, live[in][i]), h);
                else if (h.hit)
                    atomicOr(&w.flags[src.slot(slot_of, shadow[i - rays])], SLOT_BLOCKED);
            });
        __syncthreads();
        if (tid == 0)
            fetch = 0;
        for (uint32_t i = tid; i < (rays + 31u) / 32u * 32u; i += THREADS) {
            uint32_t k = 0, cls = SHADE_CLASSES;
            bool going = false;
            if (i < rays) {
                k = live[in][i];
                uint32_t p = src.slot(slot_of, k), pixel = src.pixel(p), fl = w.flags[p];
                bool blocked = (fl & SLOT_BLOCKED) != 0;
                if ((fl & SLOT_SHADOW) && !c.s.shadow_any) {
                    V3 o, d;
                    float tmax;
                    slot_shadow_ray(w, p, o, d, tmax);
                    blocked = occluded(c, o, d, tmax);
                }
                going = f64 ? resolveSlot<double, RESTIR, LIGHT>(c, w, p, pixel, fl, blocked)
                            : resolveSlot<float, RESTIR, LIGHT>(c, w, p, pixel, fl, blocked);
                if (going)
                    cls = shadeClass(c, w.hits[p]);
            }
            __syncwarp();
#pragma unroll
            for (uint32_t j = 0; j < SHADE_CLASSES; j++)
                shared_append(&n_class[j], by_class[j >> 1] + ((j & 1u) ? BLOCK_SLOTS - 1 : 0), (j & 1u) ? -1 : 1, cls == j, k);
            bool sh;
            bool started = src.take(c, w, slot_of, k, i < rays && !going, sh);
            __syncwarp();
            shared_append(&n_live[out], live[out], 1, going || started, k);
            shared_append(&n_shadow[out], shadow, 1, sh, k);
        }
        __syncthreads();
        uint32_t seg[SHADE_CLASSES + 1] = {0, 0, 0, 0, 0};
        for (uint32_t j = 0; j < SHADE_CLASSES; j++)
            seg[j + 1] = seg[j] + n_class[j];
        for (uint32_t i = tid; i < (seg[SHADE_CLASSES] + 31u) / 32u * 32u; i += THREADS) {
            bool sh = false, query = false;
            uint32_t k = 0, p = 0, kq = 0;
            CacheHook hk;
            if (i < seg[SHADE_CLASSES]) {
                uint32_t j = i >= seg[1] ? (i >= seg[2] ? (i >= seg[3] ? 3u : 2u) : 1u) : 0u;
                uint32_t at = i - seg[j];
                k = by_class[j >> 1][(j & 1u) ? BLOCK_SLOTS - 1 - at : at];
                p = src.slot(slot_of, k);
                sh = shadeSlot<CACHE, RESTIR, LIGHT>(c, w, p, src.pixel(p), q, hk, kq, query);
            }
            __syncwarp();
            shared_append(&n_shadow[out], shadow, 1, sh, k);
            if (CACHE)
                append_queries(q, query, kq, hk, p);
        }
        __syncthreads();
        in = out;
    }
}

// pathtrace.slang:9-26: params[35] samples from params[6] for every pixel.
template <bool LIGHT, bool RESTIR>
__global__ void __launch_bounds__(MK_THREADS, 1) mk_pathtrace(const __grid_constant__ Ctx c, const __grid_constant__ Wave w,
                                                                 uint32_t slots, uint32_t f64, uint32_t* pixels,
                                                                 uint32_t* next)
{
    FrameSource<LIGHT> src{pixels, next, blockIdx.x * slots, f64 != 0};
    block_wavefront<MK_THREADS, LIGHT, RESTIR, false>(c, w, src, slots, f64 != 0, CacheWave{}, nullptr);
}

// The tail of a streaming batch with deferred shadows: the slots left in a wave's queue, with the shadow rays
// that their last shade stage asked for still to be traced, run to the end.
template <bool LIGHT, bool RESTIR, bool CACHE>
__global__ void __launch_bounds__(FINISH_THREADS, 1) wf_stream_finish(const __grid_constant__ Ctx c,
                                                                     const __grid_constant__ Wave w, uint32_t wave,
                                                                     uint32_t slots, uint32_t f64,
                                                                     const __grid_constant__ CacheWave q)
{
    __shared__ uint32_t slot_of[BLOCK_SLOTS];
    uint32_t in = wave & 1u;
    QueueSource src{w.queue[in], w.counts[in], &w.fetch[FINISH_FETCH]};
    block_wavefront<FINISH_THREADS, LIGHT, RESTIR, CACHE>(c, w, src, slots, f64 != 0, q, slot_of);
}

// One path per thread over 16 x 8 tiles, for what the block wavefront's deferred light samples cannot
// follow: ReSTIR GI (the second vertex's direct light is recorded while it is shaded) and ReSTIR with the
// lighting split. One sample per launch (the host's, under ReSTIR). At 16 blocks per SM (32 registers):
// occupancy pays more than registers.
template <bool LIGHT, typename A>
__global__ void __launch_bounds__(128, 16) mk_pathtrace_restir(const __grid_constant__ Ctx c)
{
    uint32_t width = c.p[P_WIDTH], n = c.p[P_SAMPLES_PER_DISPATCH];
    bool adaptive = c.p[P_ADAPTIVE] != 0;
    uint32_t x = blockIdx.x * 16 + (threadIdx.x & 15u);
    uint32_t y = blockIdx.y * 8 + (threadIdx.x >> 4);
    if (x >= width || y >= c.p[P_HEIGHT])
        return;
    uint32_t pixel = y * width + x;
    if (n == 0 || (adaptive && !pixelActive<A>(c, pixel)))
        return;
    uint32_t k = 0, depth = 0;
    PathState<LIGHT> st = generatePathFor<LIGHT>(c, x, y, c.p[P_SAMPLE]);
    for (;;) {
        if (shadePathCall<LIGHT, true>(c, st, traceClosest(c, st.org, st.dir), depth, pixel) &&
            depth + 1 < c.p[P_MAX_DEPTH]) {
            depth++;
            continue;
        }
        finishPath<LIGHT, A, true>(c, st, pixel);
        if (++k >= n || (adaptive && !pixelActive<A>(c, pixel)))
            break;
        depth = 0;
        st = generatePathFor<LIGHT>(c, x, y, c.p[P_SAMPLE] + k);
    }
}

} // namespace vgk
