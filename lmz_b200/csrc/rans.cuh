// Decode tables of a rANS stream.
//
// One stream is decoded by one group of 8 lanes (lane k owns state k, reference
// lmz/native/lmzcore.c:1409-1530); a warp carries four streams.  The step itself is
// in fused_kernel.cuh.
//
// Two layouts, both in shared memory:
//   compact  per stream, 1 KiB + one word per live symbol: level 1 has one word per 16
//            slots -- in the low half a bit per in-bucket position t where another live
//            symbol starts (bit t), in the high half the byte offset in level 2 of the live
//            symbol that covers the bucket's first slot.  Shifting the word left by
//            31 - (slot & 15) leaves exactly the bits at or below the slot's position, so
//            a popcount of it counts the symbols to skip.  Level 2 holds one entry per live
//            symbol.  Two dependent loads and a popcount.  Level-1 words may be strided (L1S)
//            so that several streams interleave.
//   wide     16 KiB, slot -> entry: one load; for a table shared by a whole CTA, or for
//            launches with so few streams that the space does not matter.
// An entry is (4096 - freq) << 20 | start << 8 | symbol: 4096 - freq fits 12 bits even for
// a single-symbol stream, and turns the state update into x - (x >> 12) * (4096 - f) - start
// with no separate slot term.
#pragma once
#include "common.cuh"

namespace lmz {

// lmz_gpu_set_table_mode's numbers: k_stream's compact tables (0 is an earlier layout's), k_solo's two kinds.
enum : int { T_NARROW = 0, T_COMPACT = 2, T_SOLO_WIDE = 3, T_SOLO_BYTES = 4 };

// This lane's eight frequencies (symbols 8 * lane ..) of the table whose magic is at `hdr`.
__device__ __forceinline__ void load_freqs(const uint8_t *hdr, uint32_t lane, uint32_t (&f)[8])
{
    const uintptr_t at = reinterpret_cast<uintptr_t>(hdr + 4 + 16 * lane);
    const uint32_t *q = reinterpret_cast<const uint32_t *>(at & ~uintptr_t(3));
    const uint32_t sh = (uint32_t)(at & 3u) * 8u;
    uint32_t v[5];
#pragma unroll
    for (int i = 0; i < 4; i++) v[i] = __ldg(q + i);
    v[4] = sh ? __ldg(q + 4) : 0u;                 // (the last lane's table ends where its aligned words do)
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t w = __funnelshift_r(v[i], v[i + 1], sh);
        f[2 * i] = w & 0xffffu;
        f[2 * i + 1] = w >> 16;
    }
}

// Warp-cooperative table build for ONE stream from its 256 frequencies, eight per lane.
// Every lane of the warp calls this; returns false (on all lanes) if the frequencies do
// not sum to 4096.  Symbols that cover eight table entries or more are written by the whole
// warp, the others by the lane that owns them.
// Compact layout only: `rot` is added to every live-symbol index, in level 1 and
// in the position of the level-2 entry (streams that share a warp rotate their
// level 2 apart so that their popular entries fall in different banks);
// `nlive_out`, when not NULL, receives the number of live symbols, and a stream
// with more than `max_live` of them is refused before anything is written.
template <bool WIDE, int L1S = 1>
__device__ __forceinline__ bool build_table(const uint32_t (&f)[8], uint32_t *tab, uint32_t *cf, uint32_t lane,
                                            uint32_t rot = 0, uint32_t *nlive_out = nullptr, uint32_t max_live = 256)
{
    uint32_t tot = 0, nlive = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        tot += f[i];
        nlive += f[i] != 0;
    }
    // one scan carries both prefix sums: frequencies (<= 4096 each lane once
    // sane) in the low half, live-symbol counts in the high half
    uint32_t both = (tot & 0xffffu) | (nlive << 16), incl = both;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= (uint32_t)d) incl += v;
    }
    // A frequency above the scale would index past the tables, and a lane total
    // above 16 bits would corrupt the packed scan: reject before any fill.
    bool lane_ok = tot <= PROB_SCALE;
    uint32_t total = __shfl_sync(0xffffffffu, incl, 31) & 0xffffu;
    uint32_t lanes_sum = __reduce_add_sync(0xffffffffu, lane_ok ? tot : PROB_SCALE + 1);
    if (!__all_sync(0xffffffffu, lane_ok) || lanes_sum != PROB_SCALE || total != PROB_SCALE)
        return false;
    const uint32_t all_live = __shfl_sync(0xffffffffu, incl, 31) >> 16;
    if (nlive_out) *nlive_out = all_live;
    if (all_live > max_live) return false;
    uint32_t start = (incl - both) & 0xffffu, live = ((incl - both) >> 16) + rot;
    if (!WIDE) {
#pragma unroll
        for (int i = 0; i < 8; i++) tab[(lane * 8 + i) * L1S] = 0;
        __syncwarp();
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        uint32_t s = lane * 8 + i, fi = f[i], st = start, li = live;
        start += fi;
        live += fi != 0;
        uint32_t packed = ((PROB_SCALE - fi) << 20) | (st << 8) | s;
        if (!WIDE && fi) {
            cf[li] = packed;
            if (st & 15u) atomicOr(&tab[(st >> 4) * L1S], 1u << (st & 15u));
        }
        // work items of this symbol: slots (wide) or covered bucket heads (compact)
        uint32_t lo = WIDE ? st : (st + 15) >> 4;
        uint32_t cnt = WIDE ? fi : (fi ? ((st + fi - 1) >> 4) + 1 - lo : 0);
        if (!WIDE && fi && ((st + fi - 1) >> 4) + 1 < lo) cnt = 0;
        const uint32_t put = WIDE ? packed : li << 18;
        bool big = cnt >= 8;
        if (!big) {
            for (uint32_t t = 0; t < cnt; t++) {
                if (WIDE) tab[lo + t] = put;
                else atomicOr(&tab[(lo + t) * L1S], put);
            }
        }
        uint32_t m = __ballot_sync(0xffffffffu, big);
        while (m) {
            int src = __ffs(m) - 1;
            m &= m - 1;
            uint32_t bc = __shfl_sync(0xffffffffu, cnt, src);
            uint32_t bl = __shfl_sync(0xffffffffu, lo, src);
            uint32_t bp = __shfl_sync(0xffffffffu, put, src);
            for (uint32_t t = lane; t < bc; t += 32) {
                if (WIDE) tab[bl + t] = bp;
                else atomicOr(&tab[(bl + t) * L1S], bp);
            }
        }
    }
    __syncwarp();
    return true;
}

}  // namespace lmz
