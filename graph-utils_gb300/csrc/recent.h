// recent.h -- slot and tag of a vertex in the per-source engine's table of recent claims
// (local.cu).
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define GU_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define GU_HOST_DEVICE inline
#endif

namespace gu {

constexpr int RECENT_BITS = 14;
constexpr int RECENT_SLOTS = 1 << RECENT_BITS;
constexpr unsigned RECENT_EMPTY = 0xFFFFu;  // a vertex with this tag always goes to the global claim
static_assert(RECENT_BITS + 16 == 30, "slot and tag cover the 30-bit hash");

// Slot in the upper bits, tag in the lower 16: a bijection of the ids below 2^30, so that
// a tag that matches is this vertex and no other.  Ids from 2^30 up do not fit slot and
// tag: they have the tag of an empty slot, and with it no entry.
GU_HOST_DEVICE uint32_t recent_hash(int32_t v)
{
    const uint32_t h = ((uint32_t)v * 0x2C1B3C6Du) & 0x3FFFFFFFu;
    return (uint32_t)v >> 30 ? RECENT_EMPTY : h;
}

}  // namespace gu
