// The deferred stages of the streaming wavefront with the lighting split (kernels.cuh, LIGHT = true): a
// translation unit of their own so the build compiles them beside the plain variants (kern_wf.cu).
// With the shadow rays traced inside shade, that stage was 55% of a 481x270 split call (1.91 of 3.45 ms).
#include "kernels.cuh"
#include "launch.h"

namespace vgx {

cudaError_t launch_stream_shade_deferred_light(bool sorted, int blocks, cudaStream_t s, const vgd::Ctx& c,
                                               const vgk::Wave& w, uint32_t wave)
{
    if (sorted)
        vgk::wf_stream_shade_deferred<false, false, true, true><<<blocks, vgk::SHADE_THREADS, 0, s>>>(c, w, wave, vgk::CacheWave{});
    else
        vgk::wf_stream_shade_deferred<false, false, false, true><<<blocks, vgk::SHADE_THREADS, 0, s>>>(c, w, wave, vgk::CacheWave{});
    return cudaGetLastError();
}

int stream_deferred_light_blocks_per_sm()
{
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, vgk::wf_stream_shade_deferred<false, false, true, true>, vgk::SHADE_THREADS, 0);
    return n > 0 ? n : 1;
}

cudaError_t launch_stream_resolve_light(bool f64, bool sorted, int blocks, cudaStream_t s, const vgd::Ctx& c,
                                        const vgk::Wave& w, uint32_t wave)
{
    if (f64 && sorted)
        vgk::wf_stream_resolve<double, false, true, true><<<blocks, 256, 0, s>>>(c, w, wave);
    else if (f64)
        vgk::wf_stream_resolve<double, false, false, true><<<blocks, 256, 0, s>>>(c, w, wave);
    else if (sorted)
        vgk::wf_stream_resolve<float, false, true, true><<<blocks, 256, 0, s>>>(c, w, wave);
    else
        vgk::wf_stream_resolve<float, false, false, true><<<blocks, 256, 0, s>>>(c, w, wave);
    return cudaGetLastError();
}

} // namespace vgx
