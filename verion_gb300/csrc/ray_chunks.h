// How a ray query of up to 2^32 - 1 rays is split into launches. The dynamic fetch counts rays in 32 bits, and each
// warp adds up to 32 more when the rays have run out: near 2^32 the counter would wrap and the rays be traced
// again without end.
#pragma once
#include <stdint.h>

namespace vgx {

constexpr uint32_t RAY_CHUNK = 1u << 30;       // rays of one launch
constexpr uint32_t RAY_QUERY_WARPS = 1u << 16; // most warps of one launch
static_assert((uint64_t)RAY_CHUNK + 32ull * RAY_QUERY_WARPS < 1ull << 32, "a launch's work counter cannot wrap");

struct RayChunk {
    uint32_t at, n;
};

inline uint32_t ray_chunks(uint32_t n) { return n / RAY_CHUNK + (n % RAY_CHUNK ? 1u : 0u); }

inline RayChunk ray_chunk(uint32_t n, uint32_t k)
{
    uint32_t at = k * RAY_CHUNK, left = n - at;
    return RayChunk{at, left < RAY_CHUNK ? left : RAY_CHUNK};
}

} // namespace vgx
