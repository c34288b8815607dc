// Spike compaction operator shared by the C-ABI entry points.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace dtb {

constexpr int kCompactWordsPerTile = 128;                  // 4096 neurons per tile
constexpr uint32_t kCompactTileNeurons = kCompactWordsPerTile * 32;
// Largest bitmap the operator takes: the last tile boundary below 2^32, so the tile
// count, the word count (n + 31) / 32 and every neuron index stay in 32 bits.
constexpr uint32_t kCompactMaxNeurons = 0xFFFFFFFFu / kCompactTileNeurons * kCompactTileNeurons;

inline uint32_t compact_tiles(uint32_t n) {
    return static_cast<uint32_t>((static_cast<uint64_t>(n) + kCompactTileNeurons - 1) / kCompactTileNeurons);
}

// Bitmaps up to kDirectNeurons are compacted by one launch that re-reads its prefixes and uses
// no scratch: 1024 words a CTA, or one CTA an SM (kDirectCtas) where those would be more CTAs than
// SMs.  The time is the longest prefix and the writes of one SM.  Tiled form / 1024 words a CTA
// throughout / this, us a call among others, 2 and 40 % of the neurons spiking:
//   5.0M neurons   12.4 / 10.3 / 10.3 and 21.9 / 22.6 / 18.5
//   6.5M           12.5 / 15.4 / 12.3 and 24.7 / 29.0 / 22.6
//   8.4M           14.3 / 18.5 / 14.4 and 29.3 / 32.7 / 27.7
constexpr int kDirectThreads = 1024;
constexpr uint32_t kDirectCtas = 148;
constexpr uint32_t kDirectNeurons = 8u << 20;
static_assert(kDirectNeurons / 32u / kDirectCtas + 4u <= 2u * kDirectThreads, "two words a thread cover a CTA's share");

// Count, scan and write (tile_scratch unused up to kDirectNeurons); `tile_scratch` holds compact_tiles(n) words.
cudaError_t compact_launch(const uint32_t* bits, uint32_t n, uint32_t* idx, uint32_t* count, uint32_t* tile_scratch,
                           cudaStream_t s);

}  // namespace dtb
