// icp_batch_chunk.hpp -- ray ids per work-queue chunk of a batched launch (host code only; the host
// test compiles it with g++).
#pragma once
#include <algorithm>
#include <cstdint>

namespace icp::host {

// By ray count: about eight chunks per resident warp, within 64..1024.  A warp drains its lanes at
// the end of every chunk, which costs one ray's chain; a batch with fewer chunks than warps leaves
// the chip idle, which costs more.  32 drops at 180 x 360, chains of 10 (1.6e7 rays):
// 18.9 ms at 8192, 9.9 at 1024, 9.3 at 256; 1.1e8 rays: 57, 51 and 51 ms; 1.6e5 rays: 16.2, 3.7, 2.2 ms.
constexpr uint32_t kChunkMin = 64u, kChunkMax = 1024u, kChunksPerWarp = 8u;

// `most`: the caller's or the tuner's largest chunk, 0 for the default of kChunkMax.  It is a bound,
// because a size that suits one batch starves the warps of a smaller one (see the figures).
inline uint32_t batch_chunk(uint32_t most, uint64_t rays, uint64_t warps)
{
    const uint64_t share = std::max<uint64_t>(kChunkMin, rays / (std::max<uint64_t>(warps, 1u) * kChunksPerWarp));
    return (uint32_t)std::min<uint64_t>(most ? most : kChunkMax, share);
}

} // namespace icp::host
