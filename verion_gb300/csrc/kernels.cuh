// Kernels of the CUDA backend (sm_103a): the megakernel and the wavefront stages.
//
// Reference entry points: shaders/pathtrace.slang (megakernel), shaders/wf_select.slang,
// shaders/wf_args.slang, shaders/wf_extend.slang, shaders/wf_shade.slang, with the path state of
// shaders/include/wf_state.slang.
//
// GB300 design:
// * Extend and shade are persistent kernels: a grid sized to fill the 152 SMs once, each warp
//   fetching 32 consecutive queue entries with one atomic until the depth's queue is drained.
//   The queue length is read on the device, so no indirect dispatch (wf_args) and no host wait
//   sit between depths.
// * Compaction (live paths into the next depth's queue, pixels into the depth-0 queue) is warp
//   aggregated: one ballot, one atomic per warp, each lane writes at its rank.
// * Path state is structure-of-arrays in 16-byte planes: a path's 16 words are four 128-bit
//   loads, each plane contiguous over paths.
#pragma once
#include "pt_device.cuh"

namespace vgk {

using namespace vgd;

constexpr uint32_t FULL = 0xffffffffu;

// Minimum resident 128-thread blocks per SM requested for the shade kernels (a register cap): 5, 6, 8 or 16
// blocks are slower than 4 (the inlined shadePath spills heavily below 128 registers), and so is calling the
// out-of-line shadePathCall (8.99 ms of shading per benchmark step inline at 4 blocks; out of line 9.67 at 4
// blocks, 10.5 at 8, 10.9 at 12, 11.4 at 16).
#ifndef VG_SHADE_MIN_BLOCKS
#define VG_SHADE_MIN_BLOCKS 4
#endif
// The deferred shade stage's ReSTIR instantiations wait on the candidate loop's memory and, with many small
// blocks, on instructions: their warps run a loop and a shade each of which fills the instruction cache.
// One block per SM takes its slots together (one fetch and two barriers a round), so that its warps run the
// same part: the many-light 1080p frame takes 5.15 ms with 128 threads at 12 blocks per SM, each warp
// fetching for itself (10 blocks 5.33, 8 5.59, 6 5.79); together 4.93, with 256 threads at 6 blocks 4.77, 512 at
// 3 4.63, 768 at 2 4.58, 1024 at 1 (64 registers) 4.49. The plain stage is 1-3% slower that way.
constexpr uint32_t SHADE_THREADS = 128, RESTIR_SHADE_THREADS = 1024;
// The same for the kernels that run whole paths per thread through the out-of-line shadePathCall
// (the streaming tail, the batch wavefront's tail).
#ifndef VG_TAIL_MIN_BLOCKS
#define VG_TAIL_MIN_BLOCKS VG_SHADE_MIN_BLOCKS
#endif

// State planes (16 bytes each, plane k of path p at state[k * N + p]):
//   0 (org.xyz, rng)  1 (dir.xyz, flags)  2 (thr.xyz, pathLen)  3 (total.xyz, qPrev)
//   with the lighting split: 4 (directDiffuse.xyz, visLit) 5 (indirectDiffuse.xyz, visTotal)
//   6 (specular.xyz, 0) 7 (transmission.xyz, 0) 8 (emission.xyz, 0)
// flags as in wf_state.slang:42: cls bits 0-1, chan + 1 bits 2-3, misPrev bit 4, restir bit 5,
// gi bit 6, prevInst bits 8 and up.

static __device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }

// Appends `pred` lanes of a converged warp to `queue` (counter `count`); returns the slot.
static __device__ __forceinline__ void warp_append(uint32_t* count, uint32_t* queue, bool pred, uint32_t value)
{
    uint32_t b = __ballot_sync(FULL, pred);
    if (b == 0)
        return;
    uint32_t base = 0;
    if (lane_id() == 0)
        base = atomicAdd(count, __popc(b));
    base = __shfl_sync(FULL, base, 0);
    if (pred)
        queue[base + __popc(b & ((1u << lane_id()) - 1u))] = value;
}

// Warp-wide work fetch: 32 consecutive items per atomic.
static __device__ __forceinline__ uint32_t warp_fetch(uint32_t* counter)
{
    uint32_t base = 0;
    if (lane_id() == 0)
        base = atomicAdd(counter, 32u);
    return __shfl_sync(FULL, base, 0);
}

// Block-level compaction: appends the `pred` threads of a block of WARPS warps to `queue` with one
// atomic per block. Every thread of the block calls it. A block-wide exclusive scan over the warps'
// ballot counts (warp 0 scans them with shuffles) gives each warp its offset in the block's range;
// each lane writes at its warp's offset plus its rank in the ballot. `slot` is WARPS words of
// shared memory. Each warp writes and reads only its own word outside the scan, so calls in a loop
// need no barrier after the writes.
template <uint32_t WARPS>
__device__ __forceinline__ void block_append(uint32_t* count, uint32_t* queue, bool pred, uint32_t value, uint32_t* slot)
{
    uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    uint32_t b = __ballot_sync(FULL, pred);
    if (lane == 0)
        slot[warp] = __popc(b);
    __syncthreads();
    if (warp == 0) {
        uint32_t v = lane < WARPS ? slot[lane] : 0u;
        uint32_t incl = v;
#pragma unroll
        for (uint32_t o = 1; o < WARPS; o <<= 1) {
            uint32_t t = __shfl_up_sync(FULL, incl, o);
            if (lane >= o)
                incl += t;
        }
        uint32_t total = __shfl_sync(FULL, incl, WARPS - 1);
        uint32_t base = 0;
        if (lane == 0 && total)
            base = atomicAdd(count, total);
        base = __shfl_sync(FULL, base, 0);
        if (lane < WARPS)
            slot[lane] = base + incl - v;
    }
    __syncthreads();
    if (pred)
        queue[slot[warp] + __popc(b & ((1u << lane) - 1u))] = value;
}

// block_append to a queue (the `live` threads) and, in the same pass, to one of CLASSES more (threads with
// cls < CLASSES): queue k at squeue + k n, counter counts[k]. One atomic per queue and block; warp q
// scans the warps' counts of queues q, q + WARPS, .... `slot` is WARPS (1 + CLASSES) words of shared
// memory; it may be used again at once after the call.
template <uint32_t WARPS, uint32_t CLASSES>
__device__ __forceinline__ void block_append_classes(uint32_t* count, uint32_t* queue, bool live, uint32_t* counts,
                                                     uint32_t* squeue, uint32_t n, uint32_t cls, uint32_t value,
                                                     uint32_t* slot)
{
    uint32_t lane = lane_id(), warp = threadIdx.x >> 5, lt = (1u << lane) - 1u;
    uint32_t mine = __ballot_sync(FULL, live), own = 0;
    if (lane == 0)
        slot[warp] = __popc(mine);
#pragma unroll
    for (uint32_t k = 0; k < CLASSES; k++) {
        uint32_t b = __ballot_sync(FULL, cls == k);
        if (lane == 0)
            slot[(1 + k) * WARPS + warp] = __popc(b);
        own = cls == k ? b : own;
    }
    __syncthreads();
    for (uint32_t q = warp; q < 1 + CLASSES; q += WARPS) {
        uint32_t v = lane < WARPS ? slot[q * WARPS + lane] : 0u;
        uint32_t incl = v;
#pragma unroll
        for (uint32_t o = 1; o < WARPS; o <<= 1) {
            uint32_t t = __shfl_up_sync(FULL, incl, o);
            if (lane >= o)
                incl += t;
        }
        uint32_t total = __shfl_sync(FULL, incl, WARPS - 1);
        uint32_t first = 0;
        if (lane == 0 && total)
            first = atomicAdd(q == 0 ? count : counts + q - 1, total);
        first = __shfl_sync(FULL, first, 0);
        if (lane < WARPS)
            slot[q * WARPS + lane] = first + incl - v;
    }
    __syncthreads();
    if (live)
        queue[slot[warp] + __popc(mine & lt)] = value;
    if (CLASSES > 0 && cls < CLASSES)
        squeue[(size_t)cls * n + slot[(1 + cls) * WARPS + warp] + __popc(own & lt)] = value;
    __syncthreads();
}

// The split's five planes of slot p.
template <bool LIGHT>
__device__ __forceinline__ void store_split(float4* planes, size_t n, const PathState<LIGHT>& s, uint32_t p)
{
    const Parts<LIGHT>& q = s.parts;
    planes[p] = make_float4(q.directDiffuse.x, q.directDiffuse.y, q.directDiffuse.z, s.visLit);
    planes[n + p] = make_float4(q.indirectDiffuse.x, q.indirectDiffuse.y, q.indirectDiffuse.z, s.visTotal);
    planes[2 * n + p] = make_float4(q.specular.x, q.specular.y, q.specular.z, 0.0f);
    planes[3 * n + p] = make_float4(q.transmission.x, q.transmission.y, q.transmission.z, 0.0f);
    planes[4 * n + p] = make_float4(q.emission.x, q.emission.y, q.emission.z, 0.0f);
}

template <bool LIGHT>
__device__ __forceinline__ void storePath(const Wave& w, const PathState<LIGHT>& s, uint32_t p)
{
    uint32_t n = w.n;
    uint32_t flags = s.cls | ((uint32_t)(s.chan + 1) << 2) | (s.misPrev ? 16u : 0u) | (s.restir ? 32u : 0u) |
                     (s.gi ? 64u : 0u) | (s.prevInst << 8);
    w.state[p] = make_float4(s.org.x, s.org.y, s.org.z, __uint_as_float(s.rng));
    w.state[n + p] = make_float4(s.dir.x, s.dir.y, s.dir.z, __uint_as_float(flags));
    w.state[2 * n + p] = make_float4(s.thr.x, s.thr.y, s.thr.z, s.pathLen);
    w.state[3 * n + p] = make_float4(s.parts.total.x, s.parts.total.y, s.parts.total.z, s.qPrev);
    if (LIGHT)
        store_split(w.state + 4 * (size_t)n, n, s, p);
}

// wf_state.slang:60-92. Depth 0 keeps no state: the camera path is generated again.
template <bool LIGHT>
__device__ __forceinline__ PathState<LIGHT> loadPath(const Ctx& c, const Wave& w, uint32_t p, uint32_t depth)
{
    if (depth == 0)
        return generatePathFor<LIGHT>(c, p % c.p[P_WIDTH], p / c.p[P_WIDTH], c.p[P_SAMPLE]);
    uint32_t n = w.n;
    PathState<LIGHT> s;
    float4 a = w.state[p];
    float4 b = w.state[n + p];
    float4 t = w.state[2 * n + p];
    float4 r = w.state[3 * n + p];
    s.org = v3(a.x, a.y, a.z);
    s.rng = __float_as_uint(a.w);
    s.dir = v3(b.x, b.y, b.z);
    uint32_t flags = __float_as_uint(b.w);
    s.thr = v3(t.x, t.y, t.z);
    s.pathLen = t.w;
    s.cls = flags & 3u;
    s.chan = (int)((flags >> 2) & 3u) - 1;
    s.misPrev = (flags & 16u) != 0;
    s.restir = (flags & 32u) != 0;
    s.gi = (flags & 64u) != 0;
    s.prevInst = flags >> 8;
    s.qPrev = r.w;
    s.parts.zero();
    s.parts.total = v3(r.x, r.y, r.z);
    s.visLit = 0.0f;
    s.visTotal = 0.0f;
    if (LIGHT) {
        float4 q4 = w.state[4 * n + p], q5 = w.state[5 * n + p], q6 = w.state[6 * n + p], q7 = w.state[7 * n + p],
               q8 = w.state[8 * n + p];
        s.parts.directDiffuse = v3(q4.x, q4.y, q4.z);
        s.visLit = q4.w;
        s.parts.indirectDiffuse = v3(q5.x, q5.y, q5.z);
        s.visTotal = q5.w;
        s.parts.specular = v3(q6.x, q6.y, q6.z);
        s.parts.transmission = v3(q7.x, q7.y, q7.z);
        s.parts.emission = v3(q8.x, q8.y, q8.z);
    }
    return s;
}

// wf_args.slang:9-24 at depth 0: starts a sample. Every pixel's path is live unless adaptive
// sampling fills the depth-0 queue (wf_select); the later queues and all work counters restart.
static __global__ void wf_begin(const __grid_constant__ Ctx c, const __grid_constant__ Wave w)
{
    uint32_t i = threadIdx.x;
    for (uint32_t k = i; k <= w.depth; k += blockDim.x) {
        w.counts[k] = (k == 0 && c.p[P_ADAPTIVE] == 0) ? w.n : 0u;
        w.fetch[k] = 0;
        w.fetch[w.depth + 1 + k] = 0;
    }
}

// wf_select.slang:7-18: queues the pixels that still take samples; one atomic per block of 256
// (the reference takes one per pixel).
template <typename A>
__global__ void __launch_bounds__(256) wf_select(const __grid_constant__ Ctx c, const __grid_constant__ Wave w)
{
    __shared__ uint32_t slot[8];
    uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    bool active = p < w.n && pixelActive<A>(c, p);
    block_append<8>(&w.counts[0], w.queue[0], active, p, slot);
}

// Sums a per-lane counter over the warp and adds it to a global 64-bit counter (lane 0).
static __device__ __forceinline__ void warp_count(unsigned long long* dst, uint32_t v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_xor_sync(FULL, v, o);
    if (lane_id() == 0 && v)
        atomicAdd(dst, (unsigned long long)v);
}

// wf_extend.slang:6-30: closest hit for every live path of depth d. STATS also counts rays,
// BVH nodes visited and triangles tested into w.tstats[0..2] (rays at depth > 0 into [3]).
template <bool STATS>
__global__ void __launch_bounds__(128, 8) wf_extend(const __grid_constant__ Ctx c, const __grid_constant__ Wave w, uint32_t d)
{
    uint32_t count = w.counts[d];
    const uint32_t* qin = w.queue[d & 1u];
    bool direct = d == 0 && c.p[P_ADAPTIVE] == 0;
    uint32_t n_rays = 0, n_nodes = 0, n_tests = 0;
    for (;;) {
        uint32_t base = warp_fetch(&w.fetch[d]);
        if (base >= count)
            break;
        uint32_t i = base + lane_id();
        if (i < count) {
            uint32_t p = direct ? i : qin[i];
            V3 org, dir;
            if (d == 0) {
                PathState<false> s = generatePathFor<false>(c, p % c.p[P_WIDTH], p / c.p[P_WIDTH], c.p[P_SAMPLE]);
                org = s.org;
                dir = s.dir;
            } else {
                float4 a = w.state[p];
                float4 b = w.state[w.n + p];
                org = v3(a.x, a.y, a.z);
                dir = v3(b.x, b.y, b.z);
            }
            vgt::TraceHit q = vgt::trace_bvh<false>(c.s.nodes, c.s.tris, org, dir, 1.0e30f, c.err);
            w.hits[p] = make_uint4(q.hit ? 1u : 0u, q.hit ? q.inst : 0u, q.hit ? q.prim : 0u,
                                   __float_as_uint(q.hit ? q.t : 0.0f));
            if (STATS) {
                n_rays++;
                n_nodes += q.nodes;
                n_tests += q.tests;
            }
        }
        __syncwarp();
    }
    if (STATS) {
        warp_count(&w.tstats[0], n_rays);
        warp_count(&w.tstats[1], n_nodes);
        warp_count(&w.tstats[2], n_tests);
        warp_count(&w.tstats[3], d > 0 ? n_rays : 0u);
    }
}

// wf_shade.slang:7-29: shade each live path of depth d, then queue it for d + 1 or finish it.
template <bool LIGHT, bool RESTIR, typename A>
__global__ void __launch_bounds__(128, VG_SHADE_MIN_BLOCKS) wf_shade(const __grid_constant__ Ctx c, const __grid_constant__ Wave w, uint32_t d)
{
    uint32_t count = w.counts[d];
    const uint32_t* qin = w.queue[d & 1u];
    uint32_t* qout = w.queue[(d + 1) & 1u];
    bool direct = d == 0 && c.p[P_ADAPTIVE] == 0;
    for (;;) {
        uint32_t base = warp_fetch(&w.fetch[w.depth + 1 + d]);
        if (base >= count)
            break;
        uint32_t i = base + lane_id();
        bool live = false;
        uint32_t p = 0;
        if (i < count) {
            p = direct ? i : qin[i];
            PathState<LIGHT> st = loadPath<LIGHT>(c, w, p, d);
            uint4 hr = w.hits[p];
            Hit h;
            h.hit = hr.x != 0;
            h.inst = hr.y;
            h.prim = hr.z;
            h.t = __uint_as_float(hr.w);
            if (shadePath<LIGHT, RESTIR>(c, st, h, d, p) && d + 1 < w.depth) {
                storePath<LIGHT>(w, st, p);
                live = true;
            } else {
                finishPath<LIGHT, A, RESTIR>(c, st, p);
            }
        }
        __syncwarp();
        warp_append(&w.counts[d + 1], qout, live, p);
    }
}

// ---------------------------------------------------------------------------------------------
// Streaming wavefront (path regeneration). The reference's wavefront runs one sample at a time,
// depth by depth (renderer/wavefront.rs:93-177): 2 x depth launches per sample, most of them on a
// small tail of long paths. Here each pixel's slot runs the batch's params[35] samples back to
// back: when its path ends, the same thread adds it to the pixel's sums and starts the pixel's next
// sample in the same slot. A wave covers every live slot, whatever the depth of its path: with
// deferred shadows it is trace (the slots' path rays and the shadow rays that the last wave's shade
// asked for, one kernel), resolve (shadow results and ended paths into the sums, the next queue and the
// class queues) and shade; without, extend and a shade that traces its own light samples. Per pixel the
// samples are still added in order, one at a time, and adaptive sampling still decides before each
// sample from the statistics of the samples before it, so the sums are those of the sample-by-sample
// loop, bit for bit.
// Counters: queue lengths counts[wave & 1] (in) / counts[~wave & 1] (out), trace work counters
// fetch[0..1], shade work counters fetch[2..3], the separate shadow stage's fetch[4..5]; the kernel that
// calls clear_wave_counters resets the ones that the stages after it use.

// Path state as stored, for any depth (depth 0 included: it was stored when the sample started).
template <bool LIGHT>
__device__ __forceinline__ PathState<LIGHT> loadState(const Wave& w, uint32_t p)
{
    uint32_t n = w.n;
    PathState<LIGHT> s;
    float4 a = w.state[p], b = w.state[n + p], t = w.state[2 * n + p], r = w.state[3 * n + p];
    s.org = v3(a.x, a.y, a.z);
    s.rng = __float_as_uint(a.w);
    s.dir = v3(b.x, b.y, b.z);
    uint32_t flags = __float_as_uint(b.w);
    s.thr = v3(t.x, t.y, t.z);
    s.pathLen = t.w;
    s.cls = flags & 3u;
    s.chan = (int)((flags >> 2) & 3u) - 1;
    s.misPrev = (flags & 16u) != 0;
    s.restir = (flags & 32u) != 0;
    s.gi = (flags & 64u) != 0;
    s.prevInst = flags >> 8;
    s.qPrev = r.w;
    s.parts.zero();
    s.parts.total = v3(r.x, r.y, r.z);
    s.visLit = 0.0f;
    s.visTotal = 0.0f;
    if (LIGHT) {
        float4 q4 = w.state[4 * n + p], q5 = w.state[5 * n + p], q6 = w.state[6 * n + p], q7 = w.state[7 * n + p],
               q8 = w.state[8 * n + p];
        s.parts.directDiffuse = v3(q4.x, q4.y, q4.z);
        s.visLit = q4.w;
        s.parts.indirectDiffuse = v3(q5.x, q5.y, q5.z);
        s.visTotal = q5.w;
        s.parts.specular = v3(q6.x, q6.y, q6.z);
        s.parts.transmission = v3(q7.x, q7.y, q7.z);
        s.parts.emission = v3(q8.x, q8.y, q8.z);
    }
    return s;
}

// Starts the batch: every pixel that takes a sample (wf_select's test) begins sample params[6].
// With CACHE the training pixels of the frame are left out (a kernel of their own traces them).
template <bool LIGHT, typename A, bool CACHE = false>
__global__ void __launch_bounds__(256) wf_stream_start(const __grid_constant__ Ctx c, const __grid_constant__ Wave w, CacheWave q)
{
    __shared__ uint32_t slot[8];
    uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    bool live = false;
    if (p == 0)
        w.fetch[FINISH_FETCH] = 0;
    if (p < w.n && c.p[P_SAMPLES_PER_DISPATCH] > 0 && (c.p[P_ADAPTIVE] == 0 || pixelActive<A>(c, p)) &&
        !(CACHE && (p + q.train_offset) % q.train_stride == 0)) {
        PathState<LIGHT> st = generatePathFor<LIGHT>(c, p % c.p[P_WIDTH], p / c.p[P_WIDTH], c.p[P_SAMPLE]);
        storePath<LIGHT>(w, st, p);
        w.meta[p] = 0;
        if (w.flags)
            w.flags[p] = SLOT_RAY;
        live = true;
    }
    block_append<8>(&w.counts[0], w.queue[0], live, p, slot);
}

// The counters that the stages of wave parity `in` use after its first kernel, which calls this: the
// next queue's length, the work counters of the stages that follow, and the shading class counts.
static __device__ __forceinline__ void clear_wave_counters(const Wave& w, uint32_t in)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        w.counts[in ^ 1u] = 0;
        w.fetch[2 + in] = 0;
        w.fetch[4 + in] = 0;
    }
    if (w.flags && blockIdx.x == 0 && threadIdx.x < SHADE_CLASSES)
        w.scount[in * SHADE_CLASSES + threadIdx.x] = 0;
}

template <bool STATS>
__global__ void __launch_bounds__(128, 8) wf_stream_extend(const __grid_constant__ Ctx c, const __grid_constant__ Wave w, uint32_t wave)
{
    uint32_t in = wave & 1u;
    clear_wave_counters(w, in);
    uint32_t count = w.counts[in];
    const uint32_t* qin = w.queue[in];
    uint32_t n_rays = 0, n_nodes = 0, n_tests = 0, n_later = 0;
    for (;;) {
        uint32_t base = warp_fetch(&w.fetch[in]);
        if (base >= count)
            break;
        uint32_t i = base + lane_id();
        uint32_t p = i < count ? qin[i] : 0u;
        if (i < count && (!w.flags || (w.flags[p] & SLOT_RAY))) {
            float4 a = w.state[p];
            float4 b = w.state[w.n + p];
            vgt::TraceHit q = vgt::trace_bvh<false>(c.s.nodes, c.s.tris, v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), 1.0e30f,
                                                    c.err);
            w.hits[p] = make_uint4(q.hit ? 1u : 0u, q.hit ? q.inst : 0u, q.hit ? q.prim : 0u,
                                   __float_as_uint(q.hit ? q.t : 0.0f));
            if (STATS) {
                n_rays++;
                n_nodes += q.nodes;
                n_tests += q.tests;
                n_later += (w.meta[p] & 0xffu) != 0 ? 1u : 0u;
            }
        }
        __syncwarp();
    }
    if (STATS) {
        warp_count(&w.tstats[0], n_rays);
        warp_count(&w.tstats[1], n_nodes);
        warp_count(&w.tstats[2], n_tests);
        warp_count(&w.tstats[3], n_later);
    }
}

template <bool LIGHT, typename A, bool RESTIR = false>
__global__ void __launch_bounds__(128, VG_SHADE_MIN_BLOCKS) wf_stream_shade(const __grid_constant__ Ctx c, const __grid_constant__ Wave w, uint32_t wave)
{
    uint32_t in = wave & 1u, out = in ^ 1u;
    if (blockIdx.x == 0 && threadIdx.x == 0)
        w.fetch[out] = 0;
    uint32_t count = w.counts[in];
    const uint32_t* qin = w.queue[in];
    uint32_t* qout = w.queue[out];
    uint32_t batch = c.p[P_SAMPLES_PER_DISPATCH];
    for (;;) {
        uint32_t base = warp_fetch(&w.fetch[2 + in]);
        if (base >= count)
            break;
        uint32_t i = base + lane_id();
        bool live = false;
        uint32_t p = 0;
        if (i < count) {
            p = qin[i];
            uint32_t meta = w.meta[p];
            uint32_t depth = meta & 0xffu, k = meta >> 8;
            PathState<LIGHT> st = loadState<LIGHT>(w, p);
            uint4 hr = w.hits[p];
            Hit h;
            h.hit = hr.x != 0;
            h.inst = hr.y;
            h.prim = hr.z;
            h.t = __uint_as_float(hr.w);
            if (shadePath<LIGHT, RESTIR>(c, st, h, depth, p) && depth + 1 < w.depth) {
                storePath<LIGHT>(w, st, p);
                w.meta[p] = (depth + 1) | (k << 8);
                live = true;
            } else {
                finishPath<LIGHT, A, RESTIR>(c, st, p);
                if (k + 1 < batch && (c.p[P_ADAPTIVE] == 0 || pixelActive<A>(c, p))) {
                    PathState<LIGHT> nx =
                        generatePathFor<LIGHT>(c, p % c.p[P_WIDTH], p / c.p[P_WIDTH], c.p[P_SAMPLE] + k + 1);
                    storePath<LIGHT>(w, nx, p);
                    w.meta[p] = (k + 1) << 8;
                    live = true;
                }
            }
        }
        __syncwarp();
        warp_append(&w.counts[out], qout, live, p);
    }
}

// What the shadow ray (SLOT_SHADOW) of slot p, of pixel `pixel`, decides once it is traced, in the order of the pixel's samples:
// its contribution is the last add of the vertex that asked for it. Returns whether the slot still has
// a path to go on with.
template <typename A, bool RESTIR, bool LIGHT = false>
__device__ __forceinline__ bool resolveSlot(const Ctx& c, const Wave& w, uint32_t p, uint32_t pixel, uint32_t fl, bool blocked)
{
    uint32_t n = w.n;
    if constexpr (LIGHT) {
        if (!(fl & (SLOT_ENDED | SLOT_SHADOW)))
            return (fl & SLOT_RAY) != 0;
        // The path's parts, in the order of the state planes 3 to 8.
        float4* P = (fl & SLOT_ENDED) ? w.pend : w.state + 3 * (size_t)n;
        float4 q[6];
#pragma unroll
        for (uint32_t k = 0; k < 6; k++)
            q[k] = P[k * (size_t)n + p];
        PathState<true> st;
        st.parts.total = v3(q[0].x, q[0].y, q[0].z);
        st.parts.directDiffuse = v3(q[1].x, q[1].y, q[1].z);
        st.visLit = q[1].w;
        st.parts.indirectDiffuse = v3(q[2].x, q[2].y, q[2].z);
        st.visTotal = q[2].w;
        st.parts.specular = v3(q[3].x, q[3].y, q[3].z);
        st.parts.transmission = v3(q[4].x, q[4].y, q[4].z);
        st.parts.emission = v3(q[5].x, q[5].y, q[5].z);
        if (fl & SLOT_SHADOW) {
            float4 r1 = w.sreq[n + p], r2 = w.sreq[2 * n + p], r3 = w.sreq[3 * (size_t)n + p],
                   r4 = w.sreq[4 * (size_t)n + p];
            V3 cd = v3(r3.x, r3.y, r3.z), cs = v3(r4.x, r4.y, r4.z);
            float cosi = r3.w;
            uint32_t bits = __float_as_uint(r4.w);
            bool first = (bits & 1u) != 0;
            if (!blocked)
                st.parts.addLight(first ? 0u : 1u, (bits >> 1) & 3u, v3(r2.x, r2.y, r2.z), cd, cs);
            if (first) {
                float vv = lum(cd + cs);
                st.visTotal += vv;
                st.visLit += blocked ? 0.0f : vv;
                if (bits & 8u)
                    addSlot(c, pixel, 3u, cd / cosi, cs / cosi, v3(r1.x, r1.y, r1.z), blocked ? 0.0f : 1.0f, blocked ? 0.0f : cosi);
            }
        }
        if (fl & SLOT_ENDED) {
            st.gi = false;
            st.chan = -1;
            finishPath<true, A, RESTIR>(c, st, pixel);
            return (fl & SLOT_RAY) && (c.p[P_ADAPTIVE] == 0 || pixelActive<A>(c, pixel));
        }
        const Parts<true>& t = st.parts;
        P[p] = make_float4(t.total.x, t.total.y, t.total.z, q[0].w);
        P[n + p] = make_float4(t.directDiffuse.x, t.directDiffuse.y, t.directDiffuse.z, st.visLit);
        P[2 * (size_t)n + p] = make_float4(t.indirectDiffuse.x, t.indirectDiffuse.y, t.indirectDiffuse.z, st.visTotal);
        P[3 * (size_t)n + p] = make_float4(t.specular.x, t.specular.y, t.specular.z, 0.0f);
        P[4 * (size_t)n + p] = make_float4(t.transmission.x, t.transmission.y, t.transmission.z, 0.0f);
        return (fl & SLOT_RAY) != 0;
    }
    bool lit = (fl & SLOT_SHADOW) && !blocked;
    if (fl & SLOT_ENDED) {
        float4 t = w.pend[p];
        V3 total = v3(t.x, t.y, t.z);
        if (lit) {
            float4 r = w.sreq[2 * n + p];
            total += v3(r.x, r.y, r.z);
        }
        PathState<false> st;
        st.parts.zero();
        st.parts.total = total;
        st.visLit = st.visTotal = 0.0f;
        // The deferred stages never carry ReSTIR GI (the host traces the light sample inside shade
        // when GI is on), so the path's GI flag is false here.
        st.gi = false;
        st.chan = -1;
        finishPath<false, A, RESTIR>(c, st, pixel);
        // The next sample was started before this one's radiance was known: it is dropped untouched when
        // the pixel takes no more.
        return (fl & SLOT_RAY) && (c.p[P_ADAPTIVE] == 0 || pixelActive<A>(c, pixel));
    }
    if (lit) {
        float4 t = w.state[3 * n + p], r = w.sreq[2 * n + p];
        V3 total = v3(t.x, t.y, t.z) + v3(r.x, r.y, r.z);
        w.state[3 * n + p] = make_float4(total.x, total.y, total.z, t.w);
    }
    return (fl & SLOT_RAY) != 0;
}

// Shading classes of material-sorted shading (SHADE_CLASSES, ctx.h): a missed ray (environment or
// sky), a diffuse surface, a conductor, a dielectric. Only the order in which slots are shaded
// changes (each slot adds to its own pixel), so the sums stay bit-identical.

static __device__ __forceinline__ uint32_t shadeClass(const Ctx& c, uint4 hr)
{
    if (hr.x == 0)
        return 0;
    uint32_t mi = uget(c.s.instances, hr.y * 16 + 2) * 24;
    if (fget(c.s.materials, mi + 8) > 0.0f)
        return 3;
    return fget(c.s.materials, mi + 6) >= 0.5f ? 2u : 1u;
}

// Between trace and shade (deferred shadows): what the wave's rays brought each slot
// of its queue. A shadow ray that got through adds its contribution, to the slot's path or, when that
// path ended at the vertex, to its radiance in w.pend, which then goes to the pixel's sums; adaptive
// sampling decides from them whether the slot's next sample, whose camera ray was traced meanwhile, is
// kept. Every slot that has a ray goes to the next wave's queue, in the order of this one, and (SORT)
// to the queue of its hit's shading class, so that the shade stage's warps mostly run one BSDF's code.
// One pass and one atomic per queue and 256 slots: as two kernels (classify with up to four atomics a
// warp, 61 us per wave of about a million slots, and finish, 69 us) it was a seventh of the wave.
template <typename A, bool RESTIR = false, bool SORT = false, bool LIGHT = false>
__global__ void __launch_bounds__(256) wf_stream_resolve(const __grid_constant__ Ctx c, const __grid_constant__ Wave w,
                                                         uint32_t wave)
{
    __shared__ uint32_t slot[8 * (1 + (SORT ? SHADE_CLASSES : 0))];
    uint32_t in = wave & 1u, out = in ^ 1u;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        w.fetch[out] = 0;
        w.shcount[out] = 0;
    }
    uint32_t count = w.counts[in];
    const uint32_t* qin = w.queue[in];
    uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t base = blockIdx.x * blockDim.x; base < count; base += stride) {
        uint32_t i = base + threadIdx.x;
        uint32_t p = 0, cls = SHADE_CLASSES;
        bool live = false;
        if (i < count) {
            p = qin[i];
            uint32_t fl = w.flags[p];
            live = resolveSlot<A, RESTIR, LIGHT>(c, w, p, p, fl, (fl & SLOT_BLOCKED) != 0);
            if (SORT && live)
                cls = shadeClass(c, w.hits[p]);
        }
        block_append_classes<8, SORT ? SHADE_CLASSES : 0>(&w.counts[out], w.queue[out], live,
                                                          w.scount + in * SHADE_CLASSES, w.squeue, w.n, cls, p, slot);
    }
}

// Shades the hit of slot p, of pixel `pixel`, without any traversal: its path goes on, or ends and the
// pixel's next sample starts in its place (a path that ends leaves its radiance in w.pend). Returns
// whether the vertex's light sample needs a shadow ray, left in w.sreq. With CACHE: the hook, the path's sample within the batch and whether it ended at the cache.
template <bool CACHE, bool RESTIR, bool LIGHT>
__device__ __forceinline__ bool shadeSlot(const Ctx& c, const Wave& w, uint32_t p, uint32_t pixel, const CacheWave& q,
                                          CacheHook& hk, uint32_t& kq, bool& query)
{
    uint32_t n = w.n, meta = w.meta[p], depth = meta & 0xffu;
    kq = meta >> 8;
    PathState<LIGHT> st = loadState<LIGHT>(w, p);
    uint4 hr = w.hits[p];
    Hit h;
    h.hit = hr.x != 0;
    h.inst = hr.y;
    h.prim = hr.z;
    h.t = __uint_as_float(hr.w);
    ShadowReq req;
    if (CACHE) {
        // The spread starts at zero with each sample (a path may pass a cut-out surface at
        // depth 0 without meeting the hook).
        float2 sp = depth > 0 ? q.st[p] : make_float2(0.0f, 0.0f);
        hk.c = q.spread;
        hk.train = false;
        hk.a0 = sp.x;
        hk.a = sp.y;
    }
    bool alive = shadePath<LIGHT, RESTIR, true, CACHE>(c, st, h, depth, pixel, &req, &hk) && depth + 1 < w.depth;
    if (CACHE) {
        query = hk.query && !bad3(st.parts.total);
        if (alive)
            q.st[p] = make_float2(hk.a0, hk.a);
    }
    uint32_t fl = SLOT_RAY;
    if (alive) {
        w.meta[p] = (depth + 1) | (kq << 8);
    } else {
        w.pend[p] = make_float4(st.parts.total.x, st.parts.total.y, st.parts.total.z, 0.0f);
        if (LIGHT)
            store_split(w.pend + n, n, st, p);
        fl = SLOT_ENDED;
        if (kq + 1 < c.p[P_SAMPLES_PER_DISPATCH]) {
            fl |= SLOT_RAY;
            st = generatePathFor<LIGHT>(c, pixel % c.p[P_WIDTH], pixel / c.p[P_WIDTH], c.p[P_SAMPLE] + kq + 1);
            w.meta[p] = (kq + 1) << 8;
        }
    }
    if (fl & SLOT_RAY)
        storePath<LIGHT>(w, st, p);
    if (req.valid) {
        fl |= SLOT_SHADOW;
        w.sreq[p] = make_float4(req.o.x, req.o.y, req.o.z, req.tmax);
        w.sreq[n + p] = make_float4(req.d.x, req.d.y, req.d.z, 0.0f);
        w.sreq[2 * (size_t)n + p] = make_float4(req.c.x, req.c.y, req.c.z, 0.0f);
        if (LIGHT) {
            w.sreq[3 * (size_t)n + p] = make_float4(req.cd.x, req.cd.y, req.cd.z, req.cosi);
            w.sreq[4 * (size_t)n + p] = make_float4(req.cs.x, req.cs.y, req.cs.z, __uint_as_float(req.bits));
        }
    }
    w.flags[p] = fl;
    return req.valid;
}

// The `query` lanes of a converged warp leave their paths' query records: those of sample kq go to range kq
// (one atomic per sample present in the warp).
static __device__ __forceinline__ void append_queries(const CacheWave& q, bool query, uint32_t kq, const CacheHook& hk,
                                                      uint32_t pixel)
{
    if (!__ballot_sync(FULL, query))
        return;
    uint32_t grp = __match_any_sync(FULL, query ? kq : 0xffffffffu);
    uint32_t leader = __ffs(grp) - 1u;
    uint32_t first = 0;
    if (query && lane_id() == leader)
        first = atomicAdd(q.qcount + kq, __popc(grp));
    first = __shfl_sync(FULL, first, leader);
    uint32_t slot = first + __popc(grp & ((1u << lane_id()) - 1u));
    if (query && slot < q.qcap)
        cacheQueryRecord(q.qrec + ((size_t)kq * q.qcap + slot) * CACHE_REC_WORDS, hk, pixel);
}

// Streaming wave in three stages: trace, resolve, then shade without any traversal.
// Shade leaves its emitter / environment light sample as a request of the slot (w.sreq planes: origin +
// tmax, direction, contribution) in the shadow queue; the next wave traces it along with the slot's next
// ray, and the resolve stage adds the contribution when it is unoccluded. A path that ends leaves its
// radiance in w.pend and the slot starts the pixel's next sample at once.
// With CACHE a path also ends where its spread passes the cache threshold (shadePath's cache
// hook); it then leaves a query record (one atomic per warp) and finishes like any other.
// With SORTED the wave's slots are taken class by class from the resolve stage's queues.
template <bool CACHE = false, bool RESTIR = false, bool SORTED = false, bool LIGHT = false>
__global__ void __launch_bounds__(RESTIR ? RESTIR_SHADE_THREADS : SHADE_THREADS, RESTIR ? 1 : VG_SHADE_MIN_BLOCKS) wf_stream_shade_deferred(const __grid_constant__ Ctx c,
                                                                                    const __grid_constant__ Wave w, uint32_t wave,
                                                                                    CacheWave q)
{
    uint32_t in = wave & 1u, out = in ^ 1u;
    uint32_t count = w.counts[out];
    const uint32_t* qin = w.queue[out];
    uint32_t n = w.n;
    uint32_t seg[SHADE_CLASSES + 1] = {0, 0, 0, 0, 0};
    if (SORTED)
        for (uint32_t k = 0; k < SHADE_CLASSES; k++)
            seg[k + 1] = seg[k] + w.scount[in * SHADE_CLASSES + k];
    __shared__ uint32_t fetched;
    for (;;) {
        uint32_t base;
        if (RESTIR) {
            __syncthreads();
            if (threadIdx.x == 0)
                fetched = atomicAdd(&w.fetch[2 + in], blockDim.x);
            __syncthreads();
            base = fetched;
            if (base >= count)
                break;
            base += threadIdx.x & ~31u;
        } else {
            base = warp_fetch(&w.fetch[2 + in]);
            if (base >= count)
                break;
        }
        uint32_t i = base + lane_id();
        bool query = false, shadow = false;
        uint32_t p = 0, kq = 0;
        CacheHook hk;
        if (i < count) {
            if (SORTED) {
                uint32_t k = i >= seg[1] ? (i >= seg[2] ? (i >= seg[3] ? 3u : 2u) : 1u) : 0u;
                p = w.squeue[(size_t)k * n + (i - seg[k])];
            } else {
                p = qin[i];
            }
            shadow = shadeSlot<CACHE, RESTIR, LIGHT>(c, w, p, p, q, hk, kq, query);
        }
        __syncwarp();
        warp_append(&w.shcount[out], w.shqueue, shadow, p);
        if (CACHE)
            append_queries(q, query, kq, hk, p);
        __syncwarp();
    }
}

// Shadow rays of scenes with translucent surfaces (layers, opacity rolls), and of the static-fetch form:
// one ray per lane, 32 queue entries per fetch.
static __global__ void __launch_bounds__(128, 8) wf_stream_shadow_layers(const __grid_constant__ Ctx c,
                                                                         const __grid_constant__ Wave w, uint32_t wave)
{
    uint32_t in = wave & 1u, n = w.n;
    uint32_t count = w.shcount[in];
    for (;;) {
        uint32_t base = warp_fetch(&w.fetch[4 + in]);
        if (base >= count)
            break;
        uint32_t i = base + lane_id();
        if (i < count) {
            uint32_t p = w.shqueue[i];
            float4 r0 = w.sreq[p], r1 = w.sreq[n + p];
            if (occluded(c, v3(r0.x, r0.y, r0.z), v3(r1.x, r1.y, r1.z), r0.w))
                w.flags[p] |= SLOT_BLOCKED;
        }
        __syncwarp();
    }
}

// Dynamic-fetch forms of the streaming extend and shadow stages (vgt::trace_queue). A warp refills
// when at least w.refill of its lanes are idle and runs at most w.steps node visits between refills
// (w.shadow_refill, w.shadow_steps for the shadow stage; vg_set_traversal_fetch). Measured on the
// 1M-triangle workload (BVH8 with SAH node cost 0.5, each lane testing its own triangles): refills
// of 4 to 10 lanes are within 0.5% of one another and 2% faster than 16; 24 is 3% slower; 2 or 8
// steps are slower than 4.

// The defaults of the dynamic fetch, for the ray queries.
constexpr uint32_t TRACE_REFILL = 8, TRACE_STEPS = 4;

// Runs trace_queue, or with COOP trace_queue_coop (warp-cooperative leaf testing; blocks of 128
// threads, the launchers' size): the same hits either way.
template <vgt::Hits H, bool COOP, typename GetRay, typename PutHit>
__device__ __forceinline__ void trace_queue_any(const Ctx& c, uint32_t* fetch, uint32_t count, uint32_t refill,
                                                uint32_t steps, GetRay get, PutHit put)
{
    if (COOP) {
        __shared__ vgt::CoopWarp coop[vgt::COOP_WARPS];
        vgt::trace_queue_coop<H == vgt::HITS_ANY>(c.s.nodes, c.s.tris, fetch, count, c.err, refill, steps,
                                                  coop[threadIdx.x >> 5], get, put);
    } else {
        vgt::trace_queue<H>(c.s.nodes, c.s.tris, fetch, count, c.err, refill, steps, get, put);
    }
}

// The path ray of slot p, if it has one (a slot whose last path has ended keeps its place in the queue
// until its shadow ray is resolved).
static __device__ __forceinline__ bool slot_ray(const Wave& w, uint32_t p, V3& o, V3& d, float& tmax)
{
    tmax = 1.0e30f;
    if (w.flags && !(w.flags[p] & SLOT_RAY))
        return false;
    float4 a = w.state[p];
    float4 b = w.state[w.n + p];
    o = v3(a.x, a.y, a.z);
    d = v3(b.x, b.y, b.z);
    return true;
}

static __device__ __forceinline__ void slot_shadow_ray(const Wave& w, uint32_t p, V3& o, V3& d, float& tmax)
{
    float4 r0 = w.sreq[p], r1 = w.sreq[w.n + p];
    o = v3(r0.x, r0.y, r0.z);
    d = v3(r1.x, r1.y, r1.z);
    tmax = r0.w;
}

static __device__ __forceinline__ void put_slot_hit(const Wave& w, uint32_t p, const vgt::TraceHit& q)
{
    w.hits[p] = make_uint4(q.hit ? 1u : 0u, q.hit ? q.inst : 0u, q.hit ? q.prim : 0u, __float_as_uint(q.hit ? q.t : 0.0f));
}

// Minimum resident 128-thread blocks per SM requested for the dynamic-fetch traversal stages (a
// register cap: 9 blocks leave 56 registers per thread; the 1080p frame of the 1M-triangle scene, 32 samples,
// takes 131.2 ms with 8, 129.9 with 9; before the merged launch 10 made it 3% slower and 7 2%).
#ifndef VG_TRACE_MIN_BLOCKS
#define VG_TRACE_MIN_BLOCKS 9
#endif

// A wave's rays in one launch: the path ray of every queued slot (closest hit) and the shadow rays that
// the last shade stage left (any hit), one after the other in one work counter. As two launches each
// waits for its longest ray with most of the chip idle: at 960x540 a fifth of both stages' time.
static __global__ void __launch_bounds__(128, VG_TRACE_MIN_BLOCKS) wf_stream_trace(const __grid_constant__ Ctx c,
                                                                                  const __grid_constant__ Wave w,
                                                                                  uint32_t wave)
{
    uint32_t in = wave & 1u;
    clear_wave_counters(w, in);
    uint32_t rays = w.counts[in], count = rays + w.shcount[in];
    const uint32_t* qin = w.queue[in];
    trace_queue_any<vgt::HITS_EITHER, false>(
        c, &w.fetch[in], count, w.refill, w.steps,
        [&](uint32_t i, V3& o, V3& d, float& tmax, bool& any) {
            any = i >= rays;
            if (!any)
                return slot_ray(w, qin[i], o, d, tmax);
            slot_shadow_ray(w, w.shqueue[i - rays], o, d, tmax);
            return true;
        },
        [&](uint32_t i, const vgt::TraceHit& q) {
            if (i < rays)
                put_slot_hit(w, qin[i], q);
            else if (q.hit)
                atomicOr(&w.flags[w.shqueue[i - rays]], SLOT_BLOCKED);
        });
}

// The path rays alone. STATS counts rays, nodes and triangle tests (tstats[0..2], rays past depth 0 in [3]).
template <bool STATS, bool COOP>
__global__ void __launch_bounds__(128, VG_TRACE_MIN_BLOCKS) wf_stream_extend_dyn(const __grid_constant__ Ctx c, const __grid_constant__ Wave w, uint32_t wave)
{
    uint32_t in = wave & 1u;
    clear_wave_counters(w, in);
    uint32_t count = w.counts[in];
    const uint32_t* qin = w.queue[in];
    uint32_t n_rays = 0, n_nodes = 0, n_tests = 0, n_later = 0;
    trace_queue_any<vgt::HITS_CLOSEST, COOP>(
        c, &w.fetch[in], count, w.refill, w.steps,
        [&](uint32_t i, V3& o, V3& d, float& tmax, bool&) {
            bool ray = slot_ray(w, qin[i], o, d, tmax);
            if (STATS && ray)
                n_rays++;
            return ray;
        },
        [&](uint32_t i, const vgt::TraceHit& q) {
            uint32_t p = qin[i];
            put_slot_hit(w, p, q);
            if (STATS) {
                n_nodes += q.nodes;
                n_tests += q.tests;
                n_later += q.nodes != 0 && (w.meta[p] & 0xffu) != 0 ? 1u : 0u;
            }
        });
    if (STATS) {
        warp_count(&w.tstats[0], n_rays);
        warp_count(&w.tstats[1], n_nodes);
        warp_count(&w.tstats[2], n_tests);
        warp_count(&w.tstats[3], n_later);
    }
}

// The shadow rays of the deferred light samples alone, any hit (opaque scenes: one layer, no opacity
// roll). STATS: the rays traced are counted into tstats[4]. (10 or 12 blocks per SM, 48 or 40
// registers, make the stage 4% and 9% slower than 8.)
template <bool STATS, bool COOP>
__global__ void __launch_bounds__(128, VG_TRACE_MIN_BLOCKS) wf_stream_shadow_trace(const __grid_constant__ Ctx c, const __grid_constant__ Wave w, uint32_t wave)
{
    uint32_t in = wave & 1u;
    uint32_t count = w.shcount[in];
    uint32_t n_rays = 0;
    trace_queue_any<vgt::HITS_ANY, COOP>(
        c, &w.fetch[4 + in], count, w.shadow_refill, w.shadow_steps,
        [&](uint32_t i, V3& o, V3& d, float& tmax, bool&) {
            slot_shadow_ray(w, w.shqueue[i], o, d, tmax);
            if (STATS)
                n_rays++;
            return true;
        },
        [&](uint32_t i, const vgt::TraceHit& q) {
            if (q.hit)
                w.flags[w.shqueue[i]] |= SLOT_BLOCKED;
        });
    if (STATS)
        warp_count(&w.tstats[4], n_rays);
}

// The tail of a streaming batch whose shade stage traces the light samples itself: once few slots are live,
// one thread per remaining slot runs its path and the rest of its samples to the end, trace and shade in a
// loop, instead of one half-empty wave per bounce. Same functions, same order per pixel, same sums.
// (With deferred shadows: wf_stream_finish.)
template <bool LIGHT, typename A, bool RESTIR = false>
__global__ void __launch_bounds__(128, VG_TAIL_MIN_BLOCKS) wf_stream_tail(const __grid_constant__ Ctx c, const __grid_constant__ Wave w,
                                                                          uint32_t wave)
{
    uint32_t in = wave & 1u;
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= w.counts[in])
        return;
    uint32_t p = w.queue[in][i];
    uint32_t meta = w.meta[p];
    uint32_t depth = meta & 0xffu, k = meta >> 8;
    uint32_t batch = c.p[P_SAMPLES_PER_DISPATCH];
    PathState<LIGHT> st = loadState<LIGHT>(w, p);
    for (;;) {
        if (shadePathCall<LIGHT, RESTIR>(c, st, traceClosest(c, st.org, st.dir), depth, p) && depth + 1 < w.depth) {
            depth++;
            continue;
        }
        finishPath<LIGHT, A, RESTIR>(c, st, p);
        if (k + 1 < batch && (c.p[P_ADAPTIVE] == 0 || pixelActive<A>(c, p))) {
            k++;
            depth = 0;
            st = generatePathFor<LIGHT>(c, p % c.p[P_WIDTH], p / c.p[P_WIDTH], c.p[P_SAMPLE] + k);
            continue;
        }
        break;
    }
}

// Closest hits of caller-given rays (6 floats each: origin, direction): the traversal alone, for tools, for
// checking it against an independent implementation and for timing it. Dynamic fetch, as the wavefront's: a
// million random rays over the 12k-triangle scene took 344 us with 32 rays to a warp at a time.
static __global__ void __launch_bounds__(128, VG_TRACE_MIN_BLOCKS) trace_rays(const __grid_constant__ Ctx c, const float* rays,
                                                                             uint4* out, uint32_t n, uint32_t* fetch)
{
    trace_queue_any<vgt::HITS_CLOSEST, false>(
        c, fetch, n, TRACE_REFILL, TRACE_STEPS,
        [&](uint32_t i, V3& o, V3& d, float& tmax, bool&) {
            const float* r = rays + 6 * (size_t)i; // (a caller's device pointer need be no more than float-aligned)
            o = v3(r[0], r[1], r[2]);
            d = v3(r[3], r[4], r[5]);
            tmax = 1.0e30f;
            return true;
        },
        [&](uint32_t i, const vgt::TraceHit& q) {
            out[i] = make_uint4(q.hit ? 1u : 0u, q.hit ? q.inst : 0u, q.hit ? q.prim : 0u, __float_as_uint(q.hit ? q.t : 0.0f));
        });
}

// Any-hit queries of caller-given rays (7 floats each: origin, direction, tmax) through the
// shadow-ray path (`occluded`, including translucent layers).
static __global__ void __launch_bounds__(128) occlusion_rays(const __grid_constant__ Ctx c, const float* rays, uint32_t* out,
                                                       uint32_t n)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const float* r = rays + 7 * (size_t)i;
    out[i] = occluded(c, v3(r[0], r[1], r[2]), v3(r[3], r[4], r[5]), r[6]) ? 1u : 0u;
}

// The same where every surface is solid: any hit, with dynamic fetch (262 us a million rays with one to a thread).
static __global__ void __launch_bounds__(128, VG_TRACE_MIN_BLOCKS) occlusion_rays_any(const __grid_constant__ Ctx c,
                                                                                     const float* rays, uint32_t* out,
                                                                                     uint32_t n, uint32_t* fetch)
{
    trace_queue_any<vgt::HITS_ANY, false>(
        c, fetch, n, TRACE_REFILL, TRACE_STEPS,
        [&](uint32_t i, V3& o, V3& d, float& tmax, bool&) {
            const float* r = rays + 7 * (size_t)i;
            o = v3(r[0], r[1], r[2]);
            d = v3(r[3], r[4], r[5]);
            tmax = r[6];
            return true;
        },
        [&](uint32_t i, const vgt::TraceHit& q) { out[i] = q.hit ? 1u : 0u; });
}

} // namespace vgk
