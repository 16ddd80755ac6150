// Sizes and arithmetic that kernels share with the host and with the checks that run without a GPU.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define LMZ_HD __host__ __device__
#else
#define LMZ_HD
#endif

namespace lmz {

constexpr uint32_t PROB_BITS = 12;
constexpr uint32_t PROB_SCALE = 1u << PROB_BITS;
constexpr uint32_t TILE = 128;        // symbols one 8-lane group retires per tile (16 steps)

constexpr uint32_t F_CRC_BYTES = 32768;             // four tables of a byte's 256 entries, eight copies (CrcQuarters)
// The launch's shared memory starts F_SMEM_BASE bytes into the CTA's window (the launcher checks
// that reservation); at most F_SMEM_DYN bytes of it are to be had, and F_SMEM_SM by all CTAs of an SM, reservations
// counted.
constexpr uint32_t F_SMEM_BASE = 1024, F_SMEM_DYN = 232448, F_SMEM_SM = F_SMEM_BASE + F_SMEM_DYN;

// Dynamic shared memory of a CTA that needs `bytes`, where no SM is to take two of them while another has none: more than half
// of what an SM has.
LMZ_HD constexpr uint32_t alone_on_sm(uint32_t bytes) { return bytes < F_SMEM_SM / 2 ? F_SMEM_SM / 2 : bytes; }
static_assert(2 * (F_SMEM_BASE + alone_on_sm(0)) > F_SMEM_SM && alone_on_sm(0) <= F_SMEM_DYN, "one, and it can be had");

// Tiles of `tile` symbols that n symbols take.  A plane may have any n of 32 bits, so a kernel counts tiles: n + tile - 1
// and the offset behind the last tile can be more than 32 bits hold.
LMZ_HD constexpr uint32_t tiles_of(uint32_t n, uint32_t tile) { return n / tile + (n % tile != 0); }

}  // namespace lmz
