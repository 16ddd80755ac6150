// Where k_encode's CTA, a warp with four streams, keeps what in shared memory: plain arithmetic, for the kernel, its launcher
// and the checks that run without a GPU.
#pragma once
#include <cstdint>

#include "geometry.cuh"

namespace lmz {

constexpr uint32_t E_TABLE = 4096;                    // 256 entries of 16 bytes; until then the group's share of the counters
// The group's buffer of words: a piece of 128 bytes and what a tile can add to it.  A tile's symbols lie in its first 128
// bytes: they are in registers before the tile's first word, and by the next tile less than a piece is left, at the buffer's end.
constexpr uint32_t E_BUF = 384, E_TILE = 128;
// The groups' buffers lie four banks apart: side by side, all four would read the same two banks at every step.
constexpr uint32_t E_BUF_STRIDE = E_BUF + 16;
LMZ_HD constexpr uint32_t encode_buffer(uint32_t g) { return 4 * E_TABLE + g * E_BUF_STRIDE; }
LMZ_HD constexpr uint32_t encode_smem_bytes() { return encode_buffer(4); }
// CTAs that an SM has room for.
LMZ_HD constexpr uint32_t encode_resident() { return F_SMEM_SM / (F_SMEM_BASE + encode_smem_bytes()); }

}  // namespace lmz
