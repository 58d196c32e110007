// Megakernel variants (shaders/pathtrace.slang).
#include <algorithm>

#include "launch.h"
#include "megakernel.cuh"

namespace vgx {

template <bool L, typename A>
static cudaError_t mk_tiles(uint32_t w, uint32_t h, cudaStream_t s, const vgd::Ctx& c)
{
    vgk::mk_pathtrace_restir<L, A><<<dim3((w + 15) / 16, (h + 7) / 8), 128, 0, s>>>(c);
    return cudaGetLastError();
}

// A small frame is spread over all SMs, eight paths to a block at least.
BlockGrid block_grid(int sms, uint64_t items)
{
    uint64_t per = (items + (uint64_t)sms - 1) / (uint64_t)sms;
    BlockGrid g;
    g.slots = (uint32_t)std::min<uint64_t>((per + 7) / 8 * 8, vgk::BLOCK_SLOTS);
    g.blocks = g.slots == 0 ? 0 : (uint32_t)std::min<uint64_t>((uint64_t)sms, (items + g.slots - 1) / g.slots);
    return g;
}

bool megakernel_blocks(Variant v, bool gi) { return !v.restir || !(v.light || gi); }

uint64_t megakernel_items(uint32_t w, uint32_t h) { return (uint64_t)((w + 15) / 16) * ((h + 7) / 8) * 128; }

cudaError_t launch_megakernel(Variant v, const BlockGrid& g, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w,
                              uint32_t* pixels, uint32_t* next)
{
    cudaError_t e = cudaMemsetAsync(next, 0, 4, s);
    if (e != cudaSuccess)
        return e;
    uint32_t f64 = v.f64 ? 1u : 0u;
    if (v.restir)
        vgk::mk_pathtrace<false, true><<<g.blocks, vgk::MK_THREADS, 0, s>>>(c, w, g.slots, f64, pixels, next);
    else if (v.light)
        vgk::mk_pathtrace<true, false><<<g.blocks, vgk::MK_THREADS, 0, s>>>(c, w, g.slots, f64, pixels, next);
    else
        vgk::mk_pathtrace<false, false><<<g.blocks, vgk::MK_THREADS, 0, s>>>(c, w, g.slots, f64, pixels, next);
    return cudaGetLastError();
}

cudaError_t launch_megakernel_restir(Variant v, uint32_t w, uint32_t h, cudaStream_t s, const vgd::Ctx& c)
{
    if (v.light)
        return v.f64 ? mk_tiles<true, double>(w, h, s, c) : mk_tiles<true, float>(w, h, s, c);
    return v.f64 ? mk_tiles<false, double>(w, h, s, c) : mk_tiles<false, float>(w, h, s, c);
}

} // namespace vgx

#include "aov.cuh"

namespace vgx {

cudaError_t launch_aov_normals(cudaStream_t s, const vgd::Ctx& c, const float* camera18, float* out)
{
    vga::CameraRecord cam;
    for (int i = 0; i < 18; i++)
        cam.v[i] = camera18[i];
    uint32_t w = (uint32_t)cam.v[0], h = (uint32_t)cam.v[1];
    dim3 grid((w + 15) / 16, (h + 7) / 8);
    vga::aov_normals<<<grid, 128, 0, s>>>(c, cam, out);
    return cudaGetLastError();
}

// The launches that cover the frame's tiles, and the bytes of their scratch (two counters, then the pixels left).
size_t aov_scratch_bytes(uint32_t w, uint32_t h)
{
    uint64_t tiles = (uint64_t)((w + 15) / 16) * ((h + 7) / 8);
    return 256 + std::min<uint64_t>(tiles, vga::COVER_TILES) * 128 * sizeof(uint2);
}

cudaError_t launch_aov_main(int sms, cudaStream_t s, const vgd::Ctx& c, const float* camera18, float* albedo,
                            uint32_t albedo_stride, float* depth, uint32_t depth_stride, uint32_t* object_ids,
                            uint32_t* material_ids, float* coverage, void* scratch)
{
    vga::CameraRecord cam;
    for (int i = 0; i < 18; i++)
        cam.v[i] = camera18[i];
    uint32_t w = (uint32_t)cam.v[0], h = (uint32_t)cam.v[1];
    dim3 grid((w + 15) / 16, (h + 7) / 8);
    uint32_t* counters = (uint32_t*)scratch;
    vga::aov_main<<<grid, 128, 0, s>>>(c, cam, albedo, albedo_stride, depth, depth_stride, object_ids, material_ids, counters);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return e;
    if (!c.s.solid) {
        vga::aov_coverage_layers<<<grid, 128, 0, s>>>(c, cam, coverage);
        return cudaGetLastError();
    }
    vga::CoverRest rest{(uint2*)(counters + 64), counters, counters + 1};
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, vga::aov_coverage_rest, 128, 0) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    uint64_t tiles = (uint64_t)grid.x * grid.y;
    for (uint64_t at = 0; at < tiles; at += vga::COVER_TILES) {
        uint32_t n = (uint32_t)std::min<uint64_t>(tiles - at, vga::COVER_TILES);
        if (at && (e = cudaMemsetAsync(counters, 0, 8, s)) != cudaSuccess)
            return e;
        vga::aov_coverage_solid<<<n, 128, 0, s>>>(c, cam, coverage, (uint32_t)at, rest);
        // (A tile's pixels are at most 64 warps of rays: 16 blocks.)
        vga::aov_coverage_rest<<<(unsigned)std::min<uint64_t>((uint64_t)per_sm * sms, 16ull * n), 128, 0, s>>>(c, cam, coverage, (uint32_t)at, rest);
        if ((e = cudaGetLastError()) != cudaSuccess)
            return e;
    }
    return cudaSuccess;
}

} // namespace vgx
