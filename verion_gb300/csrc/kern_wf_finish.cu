// The block wavefront's kernels but for the plain megakernel (megakernel.cuh): a translation unit of their own
// so the build compiles them beside the others.
#include "launch.h"
#include "megakernel.cuh"

namespace vgx {

cudaError_t launch_stream_finish(Variant v, const BlockGrid& g, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w,
                                 uint32_t wave, const vgk::CacheWave* q)
{
    if (g.blocks == 0)
        return cudaSuccess;
    uint32_t f64 = v.f64 ? 1u : 0u;
    if (q)
        vgk::wf_stream_finish<false, false, true><<<g.blocks, vgk::FINISH_THREADS, 0, s>>>(c, w, wave, g.slots, f64, *q);
    else if (v.light)
        vgk::wf_stream_finish<true, false, false><<<g.blocks, vgk::FINISH_THREADS, 0, s>>>(c, w, wave, g.slots, f64, vgk::CacheWave{});
    else if (v.restir)
        vgk::wf_stream_finish<false, true, false><<<g.blocks, vgk::FINISH_THREADS, 0, s>>>(c, w, wave, g.slots, f64, vgk::CacheWave{});
    else
        vgk::wf_stream_finish<false, false, false><<<g.blocks, vgk::FINISH_THREADS, 0, s>>>(c, w, wave, g.slots, f64, vgk::CacheWave{});
    return cudaGetLastError();
}

} // namespace vgx
