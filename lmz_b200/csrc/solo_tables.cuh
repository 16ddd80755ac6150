// Tables of 8-byte entries, {frequency << 8 | symbol, c} (what they are for: solo_kernel.cuh).
#pragma once
#include "common.cuh"
#include "solo_layout.cuh"

namespace lmz {

// The stream's tables from its 256 frequencies, eight per lane.  False if the frequencies do not sum
// to 4096.
template <bool WIDE>
__device__ __forceinline__ bool solo_tables(const uint32_t (&f)[8], uint32_t tab_sa, uint32_t rec_sa, uint32_t lane)
{
    uint32_t tot = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) tot += f[i];
    if (!__all_sync(0xffffffffu, tot <= PROB_SCALE)) return false;
    if (__reduce_add_sync(0xffffffffu, tot) != PROB_SCALE) return false;
    uint32_t incl = tot;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= (uint32_t)d) incl += v;
    }
    uint32_t start = incl - tot;
    // the cnt slots from st on of symbol s, by threads i, i + n, ... (bytes: whole words, and the bytes at the ends)
    auto fill = [&](uint32_t st, uint32_t cnt, uint32_t s, uint32_t i, uint32_t n) {
        if (WIDE) {
            for (uint32_t j = i; j < cnt; j += n) sts_u64_if(1, tab_sa + S_ENTRY * (st + j), cnt << 8 | s, j);
            return;
        }
        const uint32_t end = st + cnt;
        for (uint32_t w = (st & ~3u) + 4 * i; w < end; w += 4 * n) {
            if (w >= st && w + 4 <= end) {
                sts_u32(tab_sa + w, s * 0x01010101u);
            } else {
#pragma unroll
                for (uint32_t b = 0; b < 4; b++)
                    if (w + b >= st && w + b < end) sts_u8(tab_sa + w + b, s);
            }
        }
    };
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t s = lane * 8 + i, fi = f[i], st = start;
        start += fi;
        // (the table's address goes with start: c = -(tab_sa + start) + the address of the slot)
        if (!WIDE) sts_u64_if(1, rec_sa + S_ENTRY * s, fi << 8 | s, 0u - (st + tab_sa));
        const bool big = fi >= (WIDE ? 8u : 32u);
        if (fi && !big) fill(st, fi, s, 0, 1);
        for (uint32_t m = __ballot_sync(0xffffffffu, big); m; m &= m - 1) {
            const int src = __ffs(m) - 1;
            fill(__shfl_sync(0xffffffffu, st, src), __shfl_sync(0xffffffffu, fi, src), (uint32_t)src * 8 + i, lane, 32);
        }
    }
    __syncwarp();
    return true;
}

}  // namespace lmz
