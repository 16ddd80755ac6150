// k_encode: the 8-lane interleaved rANS *encoder* for a batch of byte planes, the
// inverse of the batch decode.  Stream i is byte-identical to what the reference's
// CPU encoder writes for plane i with the plane's own histogram
// (lmz/native/lmzcore.c:882-937 rans_normalize, :808-841 rans_enc_put, :958-979
// rans_enc_body, :1318-1383 rans_encode_impl).
//
// One 8-lane group per stream, four streams per warp:
//   1. histogram of the plane in shared memory, a copy per lane ([bin][lane], two 16-bit counters
//      to a word): whatever the bytes, a warp's 32 additions go to 32 banks and never meet on a
//      counter, where one histogram per stream had its eight lanes queue on the popular symbols;
//   2. the reference's normalisation to 12-bit frequencies, by the whole warp for one
//      stream at a time (floor(c * 4096 / n) at least 1, the remainder given to the most
//      common symbol, an overshoot taken back from the largest frequency, first index
//      winning every tie);
//   3. the walk from the last symbol to the first.  Lane k owns state k.  Within a group
//      of eight symbols the reference visits lane 7 first, so a lane's 16-bit word lands
//      below those of the lanes above it: one vote and a popcount give its place.  Words
//      grow down through a buffer that a piece of 128 bytes of the slot ends; whole pieces leave
//      it after every tile of 16 steps, and what is left of one moves up to its end;
//   4. the eight states (lane 0 lowest) and the 516-byte table in front of the words.
// The stream ends exactly at the end of its slot; its length is reported, so it starts
// at slot_bytes - length.
//
// A batch of 4096 planes is seven warps per SM, so what bounds it is latency: in the walk the chain
// through the state (compare, shift, divide, multiply-add) and, as long as that, the one from the
// vote to a word's place, of which a step's is worked out beside the next step's state; in the
// histogram the loads, the next of which are on their way while these are counted.  A tile's symbols
// and, two steps ahead, their table entries are loaded before the state needs them, and the division
// by the symbol's frequency is exact in one multiply-add and a shift (a multiplier and an addend per
// frequency: N. Robison's choice between rounding the reciprocal up and rounding it down, of which one
// always works), with no correction after it.  A warp is a CTA: 17.6 KiB of shared memory (encode_layout.cuh), twelve
// to an SM, dealt out one by one, so that a batch spreads evenly.
//
// One B200, with places and states in one chain and the loads waited for: 4096 planes of 32 KiB of BF16
// exponents 485 -> 309 us, 592 of them 376 -> 219, 28000 of 1 KiB 218 -> 162.  With the groups' tiles in different banks (a third of
// the load/store unit's wavefronts were conflicts, most of them there) and one popcount a step instead of two, through the
// public call: 4096 planes 411 -> 384 us, 8288 of them 786 -> 750, 8288 of 4 KiB of uniform bytes 318 -> 289.  (Tiles of their own
// beside the buffers left room for eleven CTAs per SM: 6800 planes, a round of twelve, 528 us of kernel instead of 369.)
#pragma once
#include "common.cuh"
#include "encode_layout.cuh"

namespace lmz {

struct EncodeArgs {
    const uint8_t *src;     // nstr planes of `plane` bytes, back to back
    uint32_t plane;
    uint32_t nstr;
    uint8_t *slots;         // nstr slots of slot_bytes each, 512-byte aligned
    uint32_t slot_bytes;    // multiple of 512, at least HDR + 32 + 2 * plane
    uint32_t *lengths;      // per stream: bytes written at the end of its slot, 0 = failed
};

constexpr uint32_t E_COUNT_MAX = 8u * 64000u;         // symbols counted before the lanes' 16-bit counters are summed
__host__ __device__ constexpr uint32_t encode_slot_bytes(uint32_t plane)
{
    return (HDR_BYTES + STATE_BYTES + 2u * plane + 64u + 511u) & ~511u;
}

// v / f for every v < f << 20, as (v * mul + add) >> (32 + shift).
struct Reciprocal {
    uint32_t mul, add, shift;
};
__host__ __device__ inline Reciprocal reciprocal_of(uint32_t f)
{
    if (f <= 1) return {0xffffffffu, 0xffffffffu, 0};
    uint32_t s = 0;                                   // floor(log2 f)
#ifdef __CUDA_ARCH__
    s = 31u - (uint32_t)__clz((int)f);
#else
    while ((2u << s) <= f) s++;
#endif
    if ((f & (f - 1)) == 0) return {1u << 31, 0, s - 1};
    // floor(2^(32 + s) / f), below 2^32 as f > 2^s, sixteen bits at a time
    const uint32_t top = (1u << (16 + s)) / f, down = (top << 16) + (((1u << (16 + s)) - top * f) << 16) / f;
    const uint32_t rest = 0u - down * f;              // 2^(32 + s) - down * f, below f
    if (f - rest <= (1u << s)) return {down + 1, 0, s};
    return {down, down, s};
}

__global__ void __launch_bounds__(32) k_encode(EncodeArgs a)
{
    extern __shared__ __align__(512) uint8_t esm[];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t k = lane & 7u, g = lane >> 3;
    // counters of the whole warp, then the four groups' tables, in the same 16 KiB; their buffers behind
    uint32_t *counters = reinterpret_cast<uint32_t *>(esm);
    uint8_t *const gp = esm + (size_t)g * E_TABLE;
    uint8_t *buf = esm + encode_buffer(g);
    const uint32_t buf_sa = smem_addr(buf), tile_sa = buf_sa, tab_sa = smem_addr(gp);

    const uint32_t job = blockIdx.x * 4 + g;
    const bool have = job < a.nstr;
    const uint32_t n = have ? a.plane : 0;
    const uint8_t *src = a.src + (size_t)job * a.plane;

    // ---- 1. histogram ------------------------------------------------------------------
    uint32_t c[4][8];                               // [stream of the warp][symbol_of(j)]
    auto symbol_of = [&](uint32_t j) { return 4 * lane + j + (j >= 4 ? 124u : 0u); };
#pragma unroll
    for (int gg = 0; gg < 4; gg++)
#pragma unroll
        for (int j = 0; j < 8; j++) c[gg][j] = 0;
    // (symbol b: word b & 127 of the lane's, its low half for b < 128)
    const uint32_t mine_sa = smem_addr(counters) + 4 * lane;
    auto count = [&](uint32_t b) { red_shared_add(mine_sa + 128 * (b & 0x7fu), 1u << (16 * (b >> 7))); };
    auto count4 = [&](uint32_t w) {
        // a dot product with one byte of 128 picks a byte, scales it and adds the base
        const uint32_t low = w & 0x7f7f7f7fu, high = (w >> 3) & 0x10101010u;
        red_shared_add(__dp4a(low, 0x00000080u, mine_sa), 1u << (high & 0xffu));
        red_shared_add(__dp4a(low, 0x00008000u, mine_sa), 1u << __byte_perm(high, 0u, 0x4441u));
        red_shared_add(__dp4a(low, 0x00800000u, mine_sa), 1u << __byte_perm(high, 0u, 0x4442u));
        red_shared_add(__dp4a(low, 0x80000000u, mine_sa), 1u << (high >> 24));
    };
    for (uint32_t at = 0; at < a.plane; at += E_COUNT_MAX) {
        for (uint32_t i = lane; i < 4096; i += 32) counters[i] = 0;
        __syncwarp();
        const uint32_t m = n > at ? min(n - at, E_COUNT_MAX) : 0u;
        // bytes up to the first 16-byte boundary, whole 16-byte units (four per lane are counted
        // while the next four load), then the tail; the lanes' shares differ by a unit and two bytes at most,
        // which the last stretch of E_COUNT_MAX leaves room for
        const uint8_t *p = src + at;
        const uint32_t head = min(m, (uint32_t)((16u - (reinterpret_cast<uintptr_t>(p) & 15u)) & 15u));
        const uint32_t units = (m - head) / 16;
        for (uint32_t i = k; i < head; i += 8) count(p[i]);
        const uint4 *u4 = reinterpret_cast<const uint4 *>(p + head);
        auto count16 = [&](const uint4 &v) { count4(v.x); count4(v.y); count4(v.z); count4(v.w); };
        // the next four units are on their way while these are counted
        uint32_t u = k;
        uint4 v[4] = {};
        auto load4 = [&](uint32_t at4, uint4 (&to)[4]) {
#pragma unroll
            for (uint32_t i = 0; i < 4; i++) to[i] = __ldg(u4 + at4 + 8 * i);
        };
        if (u + 24 < units) load4(u, v);
        for (; u + 24 < units; u += 32) {
            uint4 w[4] = {};
            if (u + 56 < units) load4(u + 32, w);
#pragma unroll
            for (int i = 0; i < 4; i++) { count16(v[i]); v[i] = w[i]; }
        }
        for (; u < units; u += 8) count16(__ldg(u4 + u));
        for (uint32_t i = head + units * 16 + k; i < m; i += 8) count(p[i]);
        __syncwarp();
        // lane l sums symbols 4 l .. 4 l + 3 and 128 more of every stream over that stream's eight lanes;
        // the lanes start at different copies, which keeps them apart in the banks
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int gg = 0; gg < 4; gg++) {
                uint32_t lo = 0, hi = 0;
#pragma unroll
                for (uint32_t r = 0; r < 8; r++) {
                    const uint32_t w = counters[(lane * 4 + j) * 32 + ((8 * gg + ((r + lane) & 7u) + 8 * (lane >> 3)) & 31u)];
                    lo += w & 0xffffu;
                    hi += w >> 16;
                }
                // (the rotation by 8 * (lane >> 3) reads stream (gg + lane / 8) & 3)
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (((gg + (lane >> 3)) & 3u) == (uint32_t)q) { c[q][j] += lo; c[q][j + 4] += hi; }
            }
        __syncwarp();
    }

    // ---- 2. frequencies, one stream at a time by the whole warp ---------------------------
    bool ok = n != 0, single = false;
#pragma unroll
    for (uint32_t gg = 0; gg < 4; gg++) {
        const uint32_t nn = __shfl_sync(0xffffffffu, n, gg * 8);
        if (!nn) continue;
        uint32_t f[8], sum = 0;
        uint64_t best = 0;                              // (count << 8) | (255 - symbol): first index wins
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const uint32_t s = symbol_of(j), cj = c[gg][j];
            uint64_t q = nn < (1u << 20) ? (cj * PROB_SCALE) / nn : (uint64_t)cj * PROB_SCALE / nn;
            if (cj && q < 1) q = 1;
            if (q > PROB_SCALE) q = PROB_SCALE;
            f[j] = (uint32_t)q;
            sum += f[j];
            const uint64_t key = ((uint64_t)cj << 8) | (255u - s);
            if (cj && key > best) best = key;
        }
        sum = __reduce_add_sync(0xffffffffu, sum);
#pragma unroll
        for (int d = 16; d; d >>= 1) {
            const uint64_t o = __shfl_xor_sync(0xffffffffu, best, d);
            if (o > best) best = o;
        }
        const uint32_t top = 255u - (uint32_t)(best & 0xffu);
        bool good = true;
        if (sum < PROB_SCALE) {
#pragma unroll
            for (int j = 0; j < 8; j++)
                if (symbol_of(j) == top) f[j] += PROB_SCALE - sum;
        } else {
            uint32_t excess = sum - PROB_SCALE;
            for (uint32_t it = 0; excess && it < 512; it++) {
                uint32_t bk = 0;                        // (freq << 8) | (255 - symbol), freq > 1 only
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const uint32_t key = (f[j] << 8) | (255u - symbol_of(j));
                    if (f[j] > 1 && key > bk) bk = key;
                }
                bk = __reduce_max_sync(0xffffffffu, bk);
                if (!bk) { good = false; break; }
                const uint32_t bi = 255u - (bk & 0xffu), bf = bk >> 8;
                const uint32_t take = bf - 1 < excess ? bf - 1 : excess;
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (symbol_of(j) == bi) f[j] -= take;
                excess -= take;
            }
            if (excess) good = false;
        }
        // cumulative starts, then the entries the walk reads: multiplier, addend, the state from
        // which a word leaves first, and shift | (4096 - f) << 8 | start << 20
        // (one scan for both halves of the alphabet)
        uint32_t mine = 0;
#pragma unroll
        for (int j = 0; j < 8; j++) mine += f[j] << (j < 4 ? 0 : 16);
        uint32_t incl = mine;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= (uint32_t)d) incl += v;
        }
        const uint32_t all = __shfl_sync(0xffffffffu, incl, 31);
        if ((all & 0xffffu) + (all >> 16) != PROB_SCALE) good = false;
        const uint32_t low_start = (incl - mine) & 0xffffu, high_start = (all & 0xffffu) + ((incl - mine) >> 16);
        uint32_t start = low_start;
        const uint32_t t_sa = smem_addr(esm) + gg * E_TABLE;
        bool whole = false;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const uint32_t s = symbol_of(j);
            if (j == 4) start = high_start;
            if ((c[gg][j] != 0) != (f[j] != 0)) good = false;
            const Reciprocal r = reciprocal_of(f[j] ? f[j] : 1u);
            sts_u128_if(1, t_sa + 16 * s, r.mul, r.add, f[j] << 20, r.shift | ((PROB_SCALE - f[j]) << 8) | (start << 20));
            start += f[j];
            whole = whole || f[j] == PROB_SCALE;
        }
        good = __all_sync(0xffffffffu, good);
        whole = __any_sync(0xffffffffu, whole);
        if (!good && g == gg) ok = false;
        if (whole && g == gg) single = true;            // one symbol only: states stay, no words
    }
    __syncwarp();

    // ---- 3. the walk, last symbol first ---------------------------------------------------
    uint8_t *slot = a.slots + (size_t)job * a.slot_bytes;
    const uint32_t T = ok && !single ? (n + 7) / 8 : 0; // groups of eight symbols
    const uint32_t tiles = (T + 15) / 16;
    const uint32_t warp_tiles = __reduce_max_sync(0xffffffffu, tiles);
    uint32_t x = RANS_LOW, flushed = 0, pos = buf_sa + E_BUF;   // words grow down from `pos`; bytes counted back from the slot's end
    const uint32_t above = 0xffffff00u | (0xfeu << k & 0xffu);
    // a tile's 128 symbols (lane k: bytes 16 k .. 16 k + 15), requested a tile ahead
    const bool aligned = (reinterpret_cast<uintptr_t>(src) & 15u) == 0;
    auto fetch = [&](uint32_t tt) {
        uint4 v = make_uint4(0, 0, 0, 0);
        const uint32_t at = tt * 128 + 16 * k;
        if (tt < tiles && at < n) {
            if (at + 16 <= n) {
                if (aligned) {
                    v = __ldg(reinterpret_cast<const uint4 *>(src + at));
                } else {
                    const uintptr_t p = reinterpret_cast<uintptr_t>(src + at);
                    const uint32_t *q = reinterpret_cast<const uint32_t *>(p & ~uintptr_t(3));
                    const uint32_t sh = (uint32_t)(p & 3u) * 8u;
                    const uint32_t w0 = __ldg(q), w1 = __ldg(q + 1), w2 = __ldg(q + 2), w3 = __ldg(q + 3), w4 = sh ? __ldg(q + 4) : 0u;
                    v = make_uint4(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh), __funnelshift_r(w2, w3, sh), __funnelshift_r(w3, w4, sh));
                }
            } else {
                uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
                for (uint32_t j = 0; j < 16; j++)
                    if (at + j < n) w[j >> 2] |= (uint32_t)src[at + j] << (8 * (j & 3));
                v = make_uint4(w[0], w[1], w[2], w[3]);
            }
        }
        return v;
    };
    uint4 next = warp_tiles ? fetch(warp_tiles - 1) : make_uint4(0, 0, 0, 0);
#pragma unroll 1
    for (uint32_t tt = warp_tiles; tt-- > 0;) {
        const bool mine_tile = tt < tiles;
        __syncwarp();
        sts_u128_if(1, tile_sa + 16 * k, next.x, next.y, next.z, next.w);
        if (tt) next = fetch(tt - 1);
        if (tt >= 8 && tt < tiles) prefetch_l2(src + (tt - 8) * 128 + 16 * k);
        __syncwarp();
        uint32_t at[16];
#pragma unroll
        for (int s = 15; s >= 0; s--) at[s] = tab_sa + 16 * lds_u8(tile_sa + s * 8 + k);
        __syncwarp();                                    // (words may lie where the tile did)
        uint4 e0 = lds_u128(at[15]), e1 = lds_u128(at[14]);
        const bool full = __all_sync(0xffffffffu, mine_tile && tt * 128 + 128 <= n);
        // A step's words are placed while the next step's states are worked out: the vote's byte, its
        // popcount and the address are a chain as long as the state's own.  `hist` collects the votes of four steps, the newest
        // in byte 0: the words before this lane's, counted back from `pos`, are the older bytes' and the lanes' above it.
        uint32_t hist = 0, word = 0;
        bool out = false;
        auto place = [&](bool last) {
            sts_u16_if(out, pos - 2 * __popc(hist & above) - 2, word);
            if (last) pos -= 2 * __popc(hist);
        };
        auto step = [&](int s, bool active) {
            const uint4 e = e0;
            e0 = e1;
            if (s >= 2) e1 = lds_u128(at[s - 2]);
            uint32_t v = x;
            const bool need = active && v >= e.z;
            const uint32_t vote = __ballot_sync(0xffffffffu, need);
            if (need) v >>= 16;
            const uint64_t p = (uint64_t)v * e.x + e.y;
            if (s < 15) place((s & 3) == 3);
            word = x;
            out = need;
            const uint32_t q = __funnelshift_r((uint32_t)(p >> 32), 0u, e.w);          // (by the low five bits)
            const uint32_t nx = v + (e.w >> 20) + q * ((e.w >> 8) & 0xfffu);
            if (active) x = nx;
            hist = __byte_perm(vote, (s & 3) == 3 ? 0u : hist, 0x6540u + g);
        };
        if (full) {
#pragma unroll
            for (int s = 15; s >= 0; s--) step(s, true);
        } else {
#pragma unroll
            for (int s = 15; s >= 0; s--) step(s, mine_tile && tt * 128 + s * 8 + k < n);
        }
        place(true);
        // whole 128-byte pieces leave the buffer, what is left of one moves up to its end
        const uint32_t whole = (buf_sa + E_BUF - pos) / 128;
        if (__any_sync(0xffffffffu, whole != 0)) {
            __syncwarp();
            uint8_t *const to = slot + a.slot_bytes - flushed - 128 + 16 * k;
            const uint4 v0 = lds_u128(buf_sa + 256 + 16 * k), v1 = lds_u128(buf_sa + 128 + 16 * k), v2 = lds_u128(buf_sa + 16 * k);
            if (whole >= 1) *reinterpret_cast<uint4 *>(to) = v0;
            if (whole >= 2) *reinterpret_cast<uint4 *>(to - 128) = v1;
            __syncwarp();
            const uint4 rest = whole >= 2 ? v2 : v1;
            sts_u128_if(whole != 0, buf_sa + 256 + 16 * k, rest.x, rest.y, rest.z, rest.w);
            flushed += 128 * whole;
            pos += 128 * whole;
        }
    }
    const uint32_t emitted = flushed + buf_sa + E_BUF - pos;
    __syncwarp();
    if (ok) {
        // the pending tail of the words, byte by byte
        for (uint32_t j = k; j < buf_sa + E_BUF - pos; j += 8) slot[a.slot_bytes - 1 - flushed - j] = buf[E_BUF - 1 - j];
        // ---- 4. states (lane 0 lowest) and the table, in front of the words -------------
        // (an even number of bytes from the slot's end: half words)
        uint16_t *p = reinterpret_cast<uint16_t *>(slot + a.slot_bytes - emitted - STATE_BYTES), *h = p - HDR_BYTES / 2;
        p[2 * k] = (uint16_t)x;
        p[2 * k + 1] = (uint16_t)(x >> 16);
        if (k == 0) { h[0] = 'R' | '1' << 8; h[1] = 0; }
#pragma unroll 4
        for (uint32_t s = k; s < 256; s += 8) {
            // (f << 20 is zero for no frequency and for all of it; only the latter leaves the field above the shift empty)
            const uint4 w = lds_u128(tab_sa + 16 * s);
            h[2 + s] = (uint16_t)(w.z ? w.z >> 20 : (w.w >> 8 ? 0u : PROB_SCALE));
        }
    }
    if (have && k == 0) a.lengths[job] = ok ? HDR_BYTES + STATE_BYTES + emitted : 0u;
}

// Where every stream goes when they are packed back to back: offs[2 i] = sum of the lengths before
// it, offs[2 i + 1] = its length; sum[0] = all of them, sum[1] = how many could not be coded
// (length 0).  One CTA: a batch has tens of thousands of streams at most.
__global__ void __launch_bounds__(1024) k_pack_offsets(const uint32_t *lengths, uint32_t nstr, uint64_t *offs, uint64_t *sum)
{
    __shared__ uint64_t part[32];
    __shared__ uint32_t failed;
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t == 0) failed = 0;
    __syncthreads();
    uint64_t run = 0;
    uint32_t bad = 0;
    for (uint32_t at = 0; at < nstr; at += 4096) {
        // four lengths a thread, then an exclusive scan over the threads
        uint32_t v[4];
        uint64_t mine = 0;
#pragma unroll
        for (uint32_t j = 0; j < 4; j++) {
            const uint32_t i = at + 4 * t + j;
            v[j] = i < nstr ? lengths[i] : 0u;
            bad += i < nstr && v[j] == 0;
            mine += v[j];
        }
        uint64_t incl = mine;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint64_t o = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= (uint32_t)d) incl += o;
        }
        if (lane == 31) part[warp] = incl;
        __syncthreads();
        uint64_t before = run, all = 0;
        for (uint32_t w = 0; w < 32; w++) {
            if (w < warp) before += part[w];
            all += part[w];
        }
        uint64_t pos = before + incl - mine;
#pragma unroll
        for (uint32_t j = 0; j < 4; j++) {
            const uint32_t i = at + 4 * t + j;
            if (i < nstr) { offs[2 * (size_t)i] = pos; offs[2 * (size_t)i + 1] = v[j]; }
            pos += v[j];
        }
        run += all;
        __syncthreads();
    }
    if (bad) atomicAdd(&failed, bad);
    __syncthreads();
    if (t == 0) { sum[0] = run; sum[1] = failed; }
}

// `len` bytes from anywhere to anywhere by `nt` threads, 16 aligned bytes per store: the source is
// read as aligned words and shifted (up to three bytes either side of it, within its words).
__device__ __forceinline__ void copy_bytes(uint8_t *d, const uint8_t *s, uint64_t len, uint32_t t, uint32_t nt)
{
    const uint64_t head = min(len, (uint64_t)((16u - (reinterpret_cast<uintptr_t>(d) & 15u)) & 15u));
    const uint64_t units = (len - head) / 16;
    for (uint64_t i = t; i < head; i += nt) d[i] = s[i];
    const uintptr_t from = reinterpret_cast<uintptr_t>(s + head);
    const uint32_t *q = reinterpret_cast<const uint32_t *>(from & ~uintptr_t(3));
    const uint32_t sh = (uint32_t)(from & 3u) * 8u;
    uint4 *d4 = reinterpret_cast<uint4 *>(d + head);
    for (uint64_t u = t; u < units; u += nt) {
        uint32_t v[5];
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = __ldg(q + 4 * u + i);
        v[4] = sh ? __ldg(q + 4 * u + 4) : 0u;
        d4[u] = make_uint4(__funnelshift_r(v[0], v[1], sh), __funnelshift_r(v[1], v[2], sh),
                           __funnelshift_r(v[2], v[3], sh), __funnelshift_r(v[3], v[4], sh));
    }
    for (uint64_t i = head + units * 16 + t; i < len; i += nt) d[i] = s[i];
}

// Streams out of their slots into one buffer, stream i at offs[2 i] (the layout the batch
// decode reads): one CTA per stream.  offs[2 i + 1] must hold the length.
__global__ void k_pack_streams(const uint8_t *slots, uint32_t slot_bytes, const uint64_t *offs,
                               uint32_t nstr, uint8_t *out)
{
    const uint32_t i = blockIdx.x;
    if (i >= nstr) return;
    uint64_t len = offs[2 * i + 1];
    if (len > slot_bytes) len = slot_bytes;        // a stream never outgrows its slot
    const uint8_t *s = slots + (size_t)(i + 1) * slot_bytes - len;
    uint8_t *d = out + offs[2 * i];
    copy_bytes(d, s, len, threadIdx.x, blockDim.x);
}

}  // namespace lmz
