// What k_solo's lanes and warps are given: plain arithmetic, for the kernel, its launcher and the checks
// that run without a GPU.
#pragma once
#include <cstdint>

#include "geometry.cuh"

namespace lmz {

constexpr uint32_t S_TILE = 512;                       // symbols a warp stages, then gives out 16 a lane
constexpr uint32_t S_LANES = 0x377u;                   // the lanes that own states: 0-2, 4-6, 8, 9

constexpr uint32_t S_ENTRY = 8;                        // bytes of a table's or the ring's entry
// (a copy of the ring's first round lies behind it)
constexpr uint32_t S_RING = 128 * S_ENTRY, S_ROUND = 32 * S_ENTRY;
constexpr uint32_t S_WIDE_BYTES = PROB_SCALE * S_ENTRY, S_REC_BYTES = 256 * S_ENTRY;

struct SoloSmem {
    uint32_t crc, tab, rec, ring, stage, end;
};
LMZ_HD constexpr SoloSmem solo_smem(bool crc, bool wide, uint32_t W)
{
    // tables on boundaries of their size, behind the checksum's 32 KiB on theirs; below them what fits
    SoloSmem m{};
    uint32_t low = F_SMEM_BASE, high = crc ? 2 * F_CRC_BYTES : wide ? F_CRC_BYTES : 2 * PROB_SCALE;
    const uint32_t low_end = crc || wide ? F_CRC_BYTES : 2 * PROB_SCALE;
    m.crc = F_CRC_BYTES;
    m.tab = high; high += W * (wide ? S_WIDE_BYTES : PROB_SCALE);
    const uint32_t rec = wide ? 0u : W * S_REC_BYTES, ring = W * (S_RING + S_ROUND), stage = W * S_TILE;
    if (rec <= low_end - low) { m.rec = low; low += rec; } else { m.rec = high; high += rec; }
    if (ring <= low_end - low) { m.ring = low; low += ring; } else { m.ring = high; high += ring; }
    if (stage <= low_end - low) { m.stage = low; low += stage; } else { m.stage = high; high += stage; }
    m.end = high;
    return m;
}
LMZ_HD constexpr uint32_t solo_warps(bool crc, bool wide)
{
    uint32_t w = wide ? 7 : 28;
    while (solo_smem(crc, wide, w).end > F_SMEM_BASE + F_SMEM_DYN) w--;
    return w;
}

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

// A launch of `njobs` streams on `room` SMs: at most one CTA each, its warps just enough for as many rounds as the
// fullest would need.  Tables: an entry per slot where that is one round (-1), or as the caller has it.
struct SoloLaunch {
    bool wide;
    uint32_t grid, warps;
};
LMZ_HD constexpr SoloLaunch solo_launch(uint32_t njobs, uint32_t room, bool crc, int tables = -1)
{
    const uint32_t grid = njobs < room ? njobs : room, per = (njobs + grid - 1) / grid;
    const bool wide = tables < 0 ? per <= solo_warps(crc, true) : tables != 0;
    const uint32_t most = solo_warps(crc, wide), rounds = (per + most - 1) / most;
    return {wide, grid, (per + rounds - 1) / rounds};
}
// CTAs of it that an SM has room for.
LMZ_HD constexpr uint32_t solo_resident(const SoloLaunch &l, bool crc) { return F_SMEM_SM / solo_smem(crc, l.wide, l.warps).end; }

}  // namespace lmz
