// Sizes of the hash grid's staged insert (hashgrid.cu), in plain C++.
#pragma once
#include <stdint.h>

namespace rtpg {

// A bucket's list is as long as the distinct new keys that fall into it, walked once per key: with at
// most kStagePerSlot points per slot that is at most 128 on average.
constexpr uint64_t kStagePerSlot = 4;
// Entries of the temporary table, a power of two above the points, are numbered in 32 bits.
constexpr uint64_t kStagePoints = 1ull << 30;

inline bool stage_fits(uint64_t points, uint64_t slots) {
    return points <= kStagePoints && points <= slots * kStagePerSlot;
}
// points of the largest batch that a grid of `slots` slots stages, of up to max_batch
inline uint32_t stage_cap(uint64_t max_batch, uint64_t slots) {
    uint64_t cap = max_batch < kStagePoints ? max_batch : kStagePoints;
    if (cap > slots * kStagePerSlot) cap = slots * kStagePerSlot;
    return (uint32_t)cap;
}
// entries of the table for that many points: a power of two, at least 1.5 points
inline uint32_t stage_size(uint32_t points) {
    uint64_t h = 32;
    while (h < uint64_t(points) + points / 2) h <<= 1;
    return (uint32_t)h;
}

}  // namespace rtpg
