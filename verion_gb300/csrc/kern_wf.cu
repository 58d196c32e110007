// Wavefront kernel variants (shaders/wf_*.slang) and the traversal-only kernels.
#include <algorithm>

#include "kernels.cuh"
#include "launch.h"
#include "ray_chunks.h"

namespace vgx {

template <bool L, bool R, typename A>
static cudaError_t shade(int blocks, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w, uint32_t d)
{
    vgk::wf_shade<L, R, A><<<blocks, 128, 0, s>>>(c, w, d);
    return cudaGetLastError();
}

template <bool L, bool R, typename A>
static int shade_occ()
{
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, vgk::wf_shade<L, R, A>, 128, 0);
    return n > 0 ? n : 1;
}

cudaError_t launch_wf_shade(Variant v, int blocks, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w, uint32_t d)
{
    switch (v.index()) {
    case 0: return shade<false, false, float>(blocks, s, c, w, d);
    case 1: return shade<true, false, float>(blocks, s, c, w, d);
    case 2: return shade<false, true, float>(blocks, s, c, w, d);
    case 3: return shade<true, true, float>(blocks, s, c, w, d);
    case 4: return shade<false, false, double>(blocks, s, c, w, d);
    case 5: return shade<true, false, double>(blocks, s, c, w, d);
    case 6: return shade<false, true, double>(blocks, s, c, w, d);
    default: return shade<true, true, double>(blocks, s, c, w, d);
    }
}

int wf_shade_blocks_per_sm(Variant v)
{
    switch (v.index()) {
    case 0: return shade_occ<false, false, float>();
    case 1: return shade_occ<true, false, float>();
    case 2: return shade_occ<false, true, float>();
    case 3: return shade_occ<true, true, float>();
    case 4: return shade_occ<false, false, double>();
    case 5: return shade_occ<true, false, double>();
    case 6: return shade_occ<false, true, double>();
    default: return shade_occ<true, true, double>();
    }
}

cudaError_t launch_wf_begin(cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w)
{
    vgk::wf_begin<<<1, 64, 0, s>>>(c, w);
    return cudaGetLastError();
}

cudaError_t launch_wf_select(bool f64, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w)
{
    unsigned blocks = (w.n + 255) / 256;
    if (f64)
        vgk::wf_select<double><<<blocks, 256, 0, s>>>(c, w);
    else
        vgk::wf_select<float><<<blocks, 256, 0, s>>>(c, w);
    return cudaGetLastError();
}

cudaError_t launch_wf_extend(bool stats, int blocks, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w,
                             uint32_t d)
{
    if (stats)
        vgk::wf_extend<true><<<blocks, 128, 0, s>>>(c, w, d);
    else
        vgk::wf_extend<false><<<blocks, 128, 0, s>>>(c, w, d);
    return cudaGetLastError();
}

int wf_extend_blocks_per_sm()
{
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, vgk::wf_extend<false>, 128, 0);
    return n > 0 ? n : 1;
}

static int query_blocks(int sms, uint64_t n, const void* kernel)
{
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 128, 0) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    return (int)std::min<uint64_t>({(uint64_t)per_sm * sms, (n + 31) / 32, RAY_QUERY_WARPS / 4});
}

cudaError_t launch_trace_rays(int sms, cudaStream_t s, const vgd::Ctx& c, const float* rays, uint4* out, uint32_t n,
                              uint32_t* fetch)
{
    for (uint32_t k = 0; k < ray_chunks(n); k++) {
        RayChunk q = ray_chunk(n, k);
        cudaError_t e = k ? cudaMemsetAsync(fetch, 0, 4, s) : cudaSuccess;
        if (e != cudaSuccess)
            return e;
        vgk::trace_rays<<<query_blocks(sms, q.n, (const void*)vgk::trace_rays), 128, 0, s>>>(
            c, rays + 6 * (size_t)q.at, out + q.at, q.n, fetch);
        if ((e = cudaGetLastError()) != cudaSuccess)
            return e;
    }
    return cudaSuccess;
}

static __global__ void emitter_aux(const float* emitters, uint32_t n, float4* out)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        out[i] = vgd::emitterAux(emitters + 16 * (size_t)i);
}

cudaError_t launch_emitter_aux(cudaStream_t s, const float* emitters, uint32_t n, float4* out)
{
    emitter_aux<<<(n + 255) / 256, 256, 0, s>>>(emitters, n, out);
    return cudaGetLastError();
}

cudaError_t launch_occlusion_rays(int sms, cudaStream_t s, const vgd::Ctx& c, const float* rays, uint32_t* out, uint32_t n,
                                  uint32_t* fetch)
{
    for (uint32_t k = 0; k < ray_chunks(n); k++) {
        RayChunk q = ray_chunk(n, k);
        const float* r = rays + 7 * (size_t)q.at;
        cudaError_t e = k ? cudaMemsetAsync(fetch, 0, 4, s) : cudaSuccess;
        if (e != cudaSuccess)
            return e;
        if (c.s.solid)
            vgk::occlusion_rays_any<<<query_blocks(sms, q.n, (const void*)vgk::occlusion_rays_any), 128, 0, s>>>(c, r, out + q.at, q.n, fetch);
        else
            vgk::occlusion_rays<<<(q.n + 127) / 128, 128, 0, s>>>(c, r, out + q.at, q.n);
        if ((e = cudaGetLastError()) != cudaSuccess)
            return e;
    }
    return cudaSuccess;
}

} // namespace vgx

namespace vgx {

template <bool L, typename A>
static cudaError_t sshade(int blocks, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w, uint32_t wave)
{
    vgk::wf_stream_shade<L, A><<<blocks, 128, 0, s>>>(c, w, wave);
    return cudaGetLastError();
}

template <bool L, typename A>
static int sshade_occ()
{
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, vgk::wf_stream_shade<L, A>, 128, 0);
    return n > 0 ? n : 1;
}

cudaError_t launch_stream_start(Variant v, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w)
{
    unsigned blocks = (w.n + 255) / 256;
    if (v.light && v.f64)
        vgk::wf_stream_start<true, double><<<blocks, 256, 0, s>>>(c, w, vgk::CacheWave{});
    else if (v.light)
        vgk::wf_stream_start<true, float><<<blocks, 256, 0, s>>>(c, w, vgk::CacheWave{});
    else if (v.f64)
        vgk::wf_stream_start<false, double><<<blocks, 256, 0, s>>>(c, w, vgk::CacheWave{});
    else
        vgk::wf_stream_start<false, float><<<blocks, 256, 0, s>>>(c, w, vgk::CacheWave{});
    return cudaGetLastError();
}

cudaError_t launch_stream_extend(bool stats, int blocks, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w,
                                 uint32_t wave)
{
    if (stats)
        vgk::wf_stream_extend<true><<<blocks, 128, 0, s>>>(c, w, wave);
    else
        vgk::wf_stream_extend<false><<<blocks, 128, 0, s>>>(c, w, wave);
    return cudaGetLastError();
}

cudaError_t launch_stream_shade(Variant v, int blocks, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w,
                                uint32_t wave)
{
    if (v.restir)
        return launch_stream_shade_restir(v, blocks, s, c, w, wave);
    if (v.light && v.f64)
        return sshade<true, double>(blocks, s, c, w, wave);
    if (v.light)
        return sshade<true, float>(blocks, s, c, w, wave);
    if (v.f64)
        return sshade<false, double>(blocks, s, c, w, wave);
    return sshade<false, float>(blocks, s, c, w, wave);
}

int stream_shade_blocks_per_sm(Variant v)
{
    if (v.restir)
        return stream_shade_restir_blocks_per_sm(v);
    if (v.light && v.f64)
        return sshade_occ<true, double>();
    if (v.light)
        return sshade_occ<true, float>();
    if (v.f64)
        return sshade_occ<false, double>();
    return sshade_occ<false, float>();
}

} // namespace vgx

namespace vgx {

cudaError_t launch_stream_tail(Variant v, uint32_t max_slots, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w,
                               uint32_t wave)
{
    if (v.restir)
        return launch_stream_tail_restir(v, max_slots, s, c, w, wave);
    unsigned blocks = (max_slots + 127) / 128;
    if (blocks == 0)
        return cudaSuccess;
    if (v.light && v.f64)
        vgk::wf_stream_tail<true, double><<<blocks, 128, 0, s>>>(c, w, wave);
    else if (v.light)
        vgk::wf_stream_tail<true, float><<<blocks, 128, 0, s>>>(c, w, wave);
    else if (v.f64)
        vgk::wf_stream_tail<false, double><<<blocks, 128, 0, s>>>(c, w, wave);
    else
        vgk::wf_stream_tail<false, float><<<blocks, 128, 0, s>>>(c, w, wave);
    return cudaGetLastError();
}

} // namespace vgx

namespace vgx {

cudaError_t launch_stream_shade_deferred(bool sorted, int blocks, cudaStream_t s, const vgd::Ctx& c,
                                         const vgk::Wave& w, uint32_t wave)
{
    if (sorted)
        vgk::wf_stream_shade_deferred<false, false, true><<<blocks, vgk::SHADE_THREADS, 0, s>>>(c, w, wave, vgk::CacheWave{});
    else
        vgk::wf_stream_shade_deferred<><<<blocks, vgk::SHADE_THREADS, 0, s>>>(c, w, wave, vgk::CacheWave{});
    return cudaGetLastError();
}

cudaError_t launch_stream_resolve(bool f64, bool sorted, int blocks, cudaStream_t s, const vgd::Ctx& c,
                                  const vgk::Wave& w, uint32_t wave)
{
    if (f64 && sorted)
        vgk::wf_stream_resolve<double, false, true><<<blocks, 256, 0, s>>>(c, w, wave);
    else if (f64)
        vgk::wf_stream_resolve<double><<<blocks, 256, 0, s>>>(c, w, wave);
    else if (sorted)
        vgk::wf_stream_resolve<float, false, true><<<blocks, 256, 0, s>>>(c, w, wave);
    else
        vgk::wf_stream_resolve<float><<<blocks, 256, 0, s>>>(c, w, wave);
    return cudaGetLastError();
}

int stream_resolve_blocks_per_sm(bool f64)
{
    static int n[2] = {0, 0};
    int& k = n[f64 ? 1 : 0];
    if (k == 0) {
        if (f64)
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, vgk::wf_stream_resolve<double, false, true>, 256, 0);
        else
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, vgk::wf_stream_resolve<float, false, true>, 256, 0);
        k = k > 0 ? k : 1;
    }
    return k;
}

// Radiance-cache frames (lighting split off): start without the training pixels, shade with the
// cache hook, and the tail with it.
cudaError_t launch_stream_cache_start(bool f64, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w,
                                      const vgk::CacheWave& q)
{
    unsigned blocks = (w.n + 255) / 256;
    if (f64)
        vgk::wf_stream_start<false, double, true><<<blocks, 256, 0, s>>>(c, w, q);
    else
        vgk::wf_stream_start<false, float, true><<<blocks, 256, 0, s>>>(c, w, q);
    return cudaGetLastError();
}

cudaError_t launch_stream_cache_shade(bool sorted, int blocks, cudaStream_t s, const vgd::Ctx& c,
                                      const vgk::Wave& w, uint32_t wave, const vgk::CacheWave& q)
{
    if (sorted)
        vgk::wf_stream_shade_deferred<true, false, true><<<blocks, vgk::SHADE_THREADS, 0, s>>>(c, w, wave, q);
    else
        vgk::wf_stream_shade_deferred<true><<<blocks, vgk::SHADE_THREADS, 0, s>>>(c, w, wave, q);
    return cudaGetLastError();
}

int stream_cache_shade_blocks_per_sm()
{
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, vgk::wf_stream_shade_deferred<true>, vgk::SHADE_THREADS, 0);
    return n > 0 ? n : 1;
}

cudaError_t launch_stream_shadow_layers(int blocks, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w,
                                        uint32_t wave)
{
    vgk::wf_stream_shadow_layers<<<blocks, 128, 0, s>>>(c, w, wave);
    return cudaGetLastError();
}

int stream_shadow_layers_blocks_per_sm()
{
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, vgk::wf_stream_shadow_layers, 128, 0);
    return n > 0 ? n : 1;
}

int stream_deferred_blocks_per_sm()
{
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, vgk::wf_stream_shade_deferred<>, vgk::SHADE_THREADS, 0);
    return n > 0 ? n : 1;
}

} // namespace vgx

namespace vgx {

cudaError_t launch_stream_extend_dyn(bool stats, bool coop, int blocks, cudaStream_t s, const vgd::Ctx& c,
                                     const vgk::Wave& w, uint32_t wave)
{
    if (stats && coop)
        vgk::wf_stream_extend_dyn<true, true><<<blocks, 128, 0, s>>>(c, w, wave);
    else if (stats)
        vgk::wf_stream_extend_dyn<true, false><<<blocks, 128, 0, s>>>(c, w, wave);
    else if (coop)
        vgk::wf_stream_extend_dyn<false, true><<<blocks, 128, 0, s>>>(c, w, wave);
    else
        vgk::wf_stream_extend_dyn<false, false><<<blocks, 128, 0, s>>>(c, w, wave);
    return cudaGetLastError();
}

cudaError_t launch_stream_trace(int blocks, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w, uint32_t wave)
{
    vgk::wf_stream_trace<<<blocks, 128, 0, s>>>(c, w, wave);
    return cudaGetLastError();
}

cudaError_t launch_stream_shadow_trace(bool stats, bool coop, int blocks, cudaStream_t s, const vgd::Ctx& c,
                                       const vgk::Wave& w, uint32_t wave)
{
    if (stats && coop)
        vgk::wf_stream_shadow_trace<true, true><<<blocks, 128, 0, s>>>(c, w, wave);
    else if (stats)
        vgk::wf_stream_shadow_trace<true, false><<<blocks, 128, 0, s>>>(c, w, wave);
    else if (coop)
        vgk::wf_stream_shadow_trace<false, true><<<blocks, 128, 0, s>>>(c, w, wave);
    else
        vgk::wf_stream_shadow_trace<false, false><<<blocks, 128, 0, s>>>(c, w, wave);
    return cudaGetLastError();
}

int stream_shadow_trace_blocks_per_sm()
{
    static int n = 0;
    if (n == 0) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, vgk::wf_stream_shadow_trace<false, false>, 128, 0);
        n = n > 0 ? n : 1;
    }
    return n;
}

int stream_trace_blocks_per_sm()
{
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, vgk::wf_stream_trace, 128, 0);
    return n > 0 ? n : 1;
}

} // namespace vgx
