// Arithmetic that kernels share with the host and with the checks that run without a GPU.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define LMZ_HD __host__ __device__
#else
#define LMZ_HD
#endif

namespace lmz {

constexpr uint32_t TILE = 128;        // symbols one 8-lane group retires per tile (16 steps)

// Tiles of `tile` symbols that n symbols take.  A plane may have any n of 32 bits, so a kernel counts tiles: n + tile - 1
// and the offset behind the last tile can be more than 32 bits hold.
LMZ_HD constexpr uint32_t tiles_of(uint32_t n, uint32_t tile) { return n / tile + (n % tile != 0); }

}  // namespace lmz
