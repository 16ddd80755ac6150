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
    if constexpr (!WIDE) {
        // A symbol's first slot gets what the symbol is above the one before it, every other slot zero: a slot's symbol is the sum up
        // to it.  Lane k sums words 36 k .. 36 k + 35 (sixteen bytes at a time, eight lanes' in different banks; the last three lanes have
        // none), four bytes by one multiplication, as no sum is above 255.  What this takes does not depend on the alphabet, where
        // the lanes or the warp filling the symbols' slots one symbol after the other did.  (One B200, us, compact tables / filled
        // / summed up: four to a warp, 24 planes per SM of 256 uniform bytes 19 / 52 / 15, of 4 KiB 72 / 80 / 66, of 256
        // exponents 19 / 21 / 15, of 4 KiB 70 / 66 / 55; a warp each, 20 per SM, of 256 uniform bytes - / 19 / 11.)
        for (uint32_t i = 0; i < PROB_SCALE; i += 512) sts_u128_if(1, tab_sa + i + 16 * lane, 0, 0, 0, 0);
        uint32_t last = 0;
#pragma unroll
        for (uint32_t i = 0; i < 8; i++)
            if (f[i]) last = lane * 8 + i;
        const uint32_t lower = __ballot_sync(0xffffffffu, tot != 0) & ((1u << lane) - 1u);
        uint32_t before = __shfl_sync(0xffffffffu, last, lower ? 31 - __clz(lower) : lane);
        if (!lower) before = 0;
        __syncwarp();
#pragma unroll
        for (uint32_t i = 0; i < 8; i += 2) {
            const uint32_t s = lane * 8 + i, f0 = f[i], f1 = f[i + 1];
            // (the table's address goes with start: c = -(tab_sa + start) + the address of the slot)
            sts_u128_if(1, rec_sa + S_ENTRY * s, f0 << 8 | s, 0u - (start + tab_sa), f1 << 8 | (s + 1), 0u - (start + f0 + tab_sa));
            sts_u8_if(f0, tab_sa + start, s - before);
            if (f0) before = s;
            sts_u8_if(f1, tab_sa + start + f0, s + 1 - before);
            if (f1) before = s + 1;
            start += f0 + f1;
        }
        __syncwarp();
        const uint32_t first = 36 * lane, mine = tab_sa + 4 * first;
        uint32_t sum = 0;
#pragma unroll
        for (uint32_t j = 0; j < 36; j += 4)
            if (first + j < PROB_SCALE / 4) {
                const uint4 w = lds_u128(mine + 4 * j);
                sum = byte_mad(w.w, 0x01010101u, byte_mad(w.z, 0x01010101u, byte_mad(w.y, 0x01010101u, byte_mad(w.x, 0x01010101u, sum))));
            }
        uint32_t upto = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, upto, d);
            if (lane >= (uint32_t)d) upto += v;
        }
        uint32_t at = (upto - sum) * 0x01010101u;
#pragma unroll
        for (uint32_t j = 0; j < 36; j += 4)
            if (first + j < PROB_SCALE / 4) {
                uint4 w = lds_u128(mine + 4 * j);
                w.x = w.x * 0x01010101u + at;
                w.y = w.y * 0x01010101u + __byte_perm(w.x, 0u, 0x3333);
                w.z = w.z * 0x01010101u + __byte_perm(w.y, 0u, 0x3333);
                w.w = w.w * 0x01010101u + __byte_perm(w.z, 0u, 0x3333);
                sts_u128_if(1, mine + 4 * j, w.x, w.y, w.z, w.w);
                at = __byte_perm(w.w, 0u, 0x3333);
            }
        __syncwarp();
        return true;
    }
    // the cnt slots from st on of symbol s, by threads i, i + n, ...
    auto fill = [&](uint32_t st, uint32_t cnt, uint32_t s, uint32_t i, uint32_t n) {
        for (uint32_t j = i; j < cnt; j += n) sts_u64_if(1, tab_sa + S_ENTRY * (st + j), cnt << 8 | s, j);
    };
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t s = lane * 8 + i, fi = f[i], st = start;
        start += fi;
        const bool big = fi >= 8u;
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
