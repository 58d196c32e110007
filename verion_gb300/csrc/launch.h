// Host-side launchers of the kernel variants. The variants are compiled in separate translation
// units (kern_mk.cu, kern_wf.cu) so the build runs them in parallel.
#pragma once
#include <cuda_runtime.h>

#include "ctx.h"

namespace vgx {

// Compile-time variant of the path core: lighting split on, ReSTIR compiled in (the reference's
// `restirCompiled` specialisation constant, pt_core.slang:51-53), double-precision sums.
struct Variant {
    bool light;
    bool restir;
    bool f64;
    int index() const { return (light ? 1 : 0) | (restir ? 2 : 0) | (f64 ? 4 : 0); }
};

// The block wavefront (megakernel.cuh) over `items` pixels or slots: one block per SM, `slots` paths to a block.
struct BlockGrid {
    uint32_t blocks, slots;
};
BlockGrid block_grid(int sms, uint64_t items);
// The megakernel over a frame. w's planes hold blocks x slots paths, as many words are at `pixels`; `next` is a
// device word, its pixel counter. Without megakernel_blocks: one path per thread, launch_megakernel_restir.
bool megakernel_blocks(Variant v, bool gi);
uint64_t megakernel_items(uint32_t w, uint32_t h);
cudaError_t launch_megakernel(Variant v, const BlockGrid& g, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w,
                              uint32_t* pixels, uint32_t* next);
cudaError_t launch_megakernel_restir(Variant v, uint32_t w, uint32_t h, cudaStream_t s, const vgd::Ctx& c);
// With deferred shadows: finishes every slot live after `wave`; with `q` the radiance cache's paths.
cudaError_t launch_stream_finish(Variant v, const BlockGrid& g, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w,
                                 uint32_t wave, const vgk::CacheWave* q);
cudaError_t launch_wf_shade(Variant v, int blocks, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w, uint32_t d);
int wf_shade_blocks_per_sm(Variant v);

cudaError_t launch_wf_begin(cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w);
cudaError_t launch_wf_select(bool f64, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w);
cudaError_t launch_wf_extend(bool stats, int blocks, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w, uint32_t d);
int wf_extend_blocks_per_sm();
// Streaming wavefront (path regeneration); see kernels.cuh.
cudaError_t launch_stream_start(Variant v, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w);
cudaError_t launch_stream_extend(bool stats, int blocks, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w,
                                 uint32_t wave);
cudaError_t launch_stream_shade(Variant v, int blocks, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w,
                                uint32_t wave);
int stream_shade_blocks_per_sm(Variant v);
// Three-stage wave (lighting split off): shade without traversal, then the shadow stage.
cudaError_t launch_stream_cache_start(bool f64, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w,
                                      const vgk::CacheWave& q);
cudaError_t launch_stream_cache_shade(bool sorted, int blocks, cudaStream_t s, const vgd::Ctx& c,
                                      const vgk::Wave& w, uint32_t wave, const vgk::CacheWave& q);
int stream_cache_shade_blocks_per_sm();
// With `sorted` the resolve stage also fills the class queues and the shade stage takes the wave's slots
// class by class.
cudaError_t launch_stream_shade_deferred(bool sorted, int blocks, cudaStream_t s, const vgd::Ctx& c,
                                         const vgk::Wave& w, uint32_t wave);
cudaError_t launch_stream_resolve(bool f64, bool sorted, int blocks, cudaStream_t s, const vgd::Ctx& c,
                                  const vgk::Wave& w, uint32_t wave);
int stream_resolve_blocks_per_sm(bool f64);
cudaError_t launch_stream_shadow_layers(int blocks, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w,
                                        uint32_t wave);
int stream_shadow_layers_blocks_per_sm();
int stream_deferred_blocks_per_sm();
// Dynamic-fetch traversal stages: a wave's path and shadow rays in one launch, or each in its own.
// With `coop` the warp-cooperative leaf testing of traverse.cuh (the same hits).
cudaError_t launch_stream_trace(int blocks, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w, uint32_t wave);
cudaError_t launch_stream_extend_dyn(bool stats, bool coop, int blocks, cudaStream_t s, const vgd::Ctx& c,
                                     const vgk::Wave& w, uint32_t wave);
cudaError_t launch_stream_shadow_trace(bool stats, bool coop, int blocks, cudaStream_t s, const vgd::Ctx& c,
                                       const vgk::Wave& w, uint32_t wave);
int stream_trace_blocks_per_sm();
int stream_shadow_trace_blocks_per_sm();
// The same streaming stages compiled with ReSTIR (kern_wf_restir.cu); the host runs them one
// sample per launch sequence.
cudaError_t launch_stream_shade_restir(Variant v, int blocks, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w,
                                       uint32_t wave);
int stream_shade_restir_blocks_per_sm(Variant v);
cudaError_t launch_stream_tail_restir(Variant v, uint32_t max_slots, cudaStream_t s, const vgd::Ctx& c,
                                      const vgk::Wave& w, uint32_t wave);
cudaError_t launch_stream_shade_deferred_restir(bool sorted, int blocks, cudaStream_t s, const vgd::Ctx& c,
                                                const vgk::Wave& w, uint32_t wave);
int stream_deferred_restir_blocks_per_sm();
cudaError_t launch_stream_resolve_restir(bool f64, bool sorted, int blocks, cudaStream_t s, const vgd::Ctx& c,
                                         const vgk::Wave& w, uint32_t wave);
// The deferred stages with the lighting split (kern_wf_light.cu).
cudaError_t launch_stream_shade_deferred_light(bool sorted, int blocks, cudaStream_t s, const vgd::Ctx& c,
                                               const vgk::Wave& w, uint32_t wave);
int stream_deferred_light_blocks_per_sm();
cudaError_t launch_stream_resolve_light(bool f64, bool sorted, int blocks, cudaStream_t s, const vgd::Ctx& c,
                                        const vgk::Wave& w, uint32_t wave);
// Without deferred shadows: finishes every slot still live after `wave` (at most max_slots of them) in one launch.
cudaError_t launch_stream_tail(Variant v, uint32_t max_slots, cudaStream_t s, const vgd::Ctx& c, const vgk::Wave& w,
                               uint32_t wave);
// Primary-hit AOVs (normals.slang, aov.slang); camera18 is the reference's camera record.
cudaError_t launch_aov_normals(cudaStream_t s, const vgd::Ctx& c, const float* camera18, float* out);
size_t aov_scratch_bytes(uint32_t w, uint32_t h); // device memory for launch_aov_main's `scratch`, 256-byte aligned
cudaError_t launch_aov_main(int sms, cudaStream_t s, const vgd::Ctx& c, const float* camera18, float* albedo,
                            uint32_t albedo_stride, float* depth, uint32_t depth_stride, uint32_t* object_ids,
                            uint32_t* material_ids, float* coverage, void* scratch);
cudaError_t launch_emitter_aux(cudaStream_t s, const float* emitters, uint32_t n, float4* out);
// `fetch`: a cleared device word.
cudaError_t launch_trace_rays(int sms, cudaStream_t s, const vgd::Ctx& c, const float* rays, uint4* out, uint32_t n,
                              uint32_t* fetch);
cudaError_t launch_occlusion_rays(int sms, cudaStream_t s, const vgd::Ctx& c, const float* rays, uint32_t* out, uint32_t n,
                                  uint32_t* fetch);

} // namespace vgx
