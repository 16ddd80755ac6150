// What k_solo's lanes and warps are given: plain arithmetic, for the kernel, its launcher and the checks
// that run without a GPU.
#pragma once
#include <cstdint>

#include "tiles.cuh"

namespace lmz {

constexpr uint32_t S_TILE = 512;                       // symbols a warp stages, then gives out 16 a lane
constexpr uint32_t S_LANES = 0x377u;                   // the lanes that own states: 0-2, 4-6, 8, 9

// A lane of a warp that decodes one stream.  The lanes that own no state run along: they vote for nothing and
// write nothing, as their symbols are nobody's.
struct SoloLane {
    uint32_t owner;      // 1 for a lane of S_LANES
    uint32_t k;          // the state it owns
    uint32_t below;      // the owners before it
};
LMZ_HD constexpr SoloLane solo_lane(uint32_t lane)
{
    const uint32_t owner = S_LANES >> lane & 1u;
    return {owner, owner ? 3 * (lane >> 2) + (lane & 3u) : 0u, S_LANES & ((1u << (owner ? lane : 0u)) - 1u)};
}

// A step's symbols go to the eight bytes of the stage from `at` on, each from the one lane that has it:
// put(on, address) stores where `on`.
template <class Put>
LMZ_HD inline void solo_put(const SoloLane &me, uint32_t at, bool active, Put put)
{
    put(me.owner & (uint32_t)active, at + me.k);
}

}  // namespace lmz
