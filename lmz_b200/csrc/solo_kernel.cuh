// k_solo: the decode kernel for launches of few streams.  A warp decodes ONE stream, with eight of
// its lanes, and the rest of the stream's work with all thirty-two.
//
// What bounds such a launch is how long a step takes, so a step here is the shortest chain there is:
// multiply-add, compare, vote, count the lanes below, load.  A state is never put together.  What a
// step needs of it is kept as three values, of which the next (unrefilled) state is y * f + c:
//
//   not refilled   y = x >> 12, f = the slot's frequency, c = slot - start
//   refilled       y = x >> 12 without the word's bits, c = slot - start + (word >> 12) * f: all of the
//                  word's own, so it is worked out before the word is asked for (32 words at a time,
//                  one a lane) and waits in a ring
//
// Ring and tables hold the same 8-byte entries, {f << 8 | symbol, c}.
//
//   WIDE      an entry per slot: 32 KiB a stream.  A lane without a refill loads its entry while the vote is under way, one with a
//             refill behind it: two loads, of which a lane takes part in one, into the same registers, with nothing to pick
//             between them
//   else      a byte per slot, its symbol (4 KiB), looked up while the vote is under way, and an entry
//             per symbol whose c is -start: the slot is added to what was loaded.  One load serves both kinds of lanes, from an
//             address picked behind the vote, as warps are many enough here for a load's slot to count (12 streams
//             per SM 316 us, 329 with two)
//
// Measured on one B200, cycles: multiply-add 4, compare and vote 17, and 4, permute 4, dot product 4,
// load 23; a popcount is 17, so the lanes below are counted by a byte permute that looks three votes
// up at a time and a dot product that adds them.  For that the eight lanes sit three to a nibble of
// the vote; the other twenty-four run along, vote for nothing and write nothing.
//
// One B200, k_stream's wide tables against this: a lone stream 61.5 -> 38.5 ns a step (41.9 with one load behind a pick), a
// 4096 x 14336 BF16 tensor in 64 KiB chunks 480 -> 381 us (issue slots 67 % busy, 31 instructions a stream's step), in 8 MiB
// chunks 34.1 -> 22.4 ms (23.1 with one load), seven planes of 4 KiB between host buffers 78 -> 55 us.  Uniform bytes, four words a
// step, cost no more than exponents with one and a third.  Where the store of a step's symbols stands matters: behind the
// vote, or behind the load, a lone stream's 8 MiB took 24.6 ms instead of 23.1.
//
// Sinks as in fused_kernel.cuh, a tile being 512 symbols: 16 a lane.
#pragma once
#include "fused_kernel.cuh"

namespace lmz {

// A call: in line it makes the compiler's loop over the steps a slower one (12 planes of 32 KiB of exponents per SM 249 us, 257 in
// line; 20 per SM 336 and 345).
__device__ __noinline__ bool solo_byte_tables(const uint32_t (&f)[8], uint32_t tab_sa, uint32_t rec_sa, uint32_t lane)
{
    return solo_tables<false>(f, tab_sa, rec_sa, lane);
}

template <int SINK, bool CRC, bool WIDE>
__global__ void __launch_bounds__(solo_warps(CRC, WIDE) * 32, 1) k_solo(StreamArgs a)
{
    constexpr uint32_t LEAD = HDR_BYTES + STATE_BYTES;
    constexpr int NRA = SINK == SINK_F32 ? 16 : 8;         // words of a row that one lane emits
    constexpr uint32_t ROW = SINK == SINK_F32 ? 4 * S_TILE : 2 * S_TILE, ROWS = PIECE_BYTES / ROW;
    extern __shared__ __align__(16) uint8_t ssm[];
    const uint32_t lane = threadIdx.x & 31u, W = blockDim.x >> 5;
    const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);       // (the compiler sees that it is the warp's)
    const SoloLane me = solo_lane(lane);
    const bool owner = me.owner;
    const uint32_t k = me.k, below = me.below;

    const uint32_t s0 = smem_addr(ssm);
    const SoloSmem m_ = solo_smem(CRC, WIDE, W);
    const bool fits = s0 == F_SMEM_BASE && m_.end <= s0 + dynamic_smem_bytes();
    const uint32_t tab_sa = m_.tab + warp * (WIDE ? S_WIDE_BYTES : PROB_SCALE), rec_sa = m_.rec + warp * S_REC_BYTES;
    const uint32_t ring_sa = m_.ring + warp * (S_RING + S_ROUND), stage_sa = m_.stage + warp * S_TILE;
    CrcQuarters cq;
    if (CRC) {
        const uint32_t cg = lane >> 3;
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) cq.b[i] = m_.crc + 32u * (3u - (i ^ cg)) + 4u * (lane & 7u);
        cq.rot = 0x3210u ^ (0x1111u * cg);
        if (fits) {
            // "multiply by x^(8 * ROW)", byte m of a value through table m, eight copies (CrcQuarters)
            uint32_t *ts = reinterpret_cast<uint32_t *>(ssm + (m_.crc - s0));
            const uint32_t(*mul)[256] = SINK == SINK_F32 ? a.tabs->mul_row2048 : a.tabs->mul_row1024;
            for (uint32_t i = threadIdx.x; i < F_CRC_BYTES / 4; i += blockDim.x) ts[i] = mul[3u - ((i >> 3) & 3u)][i >> 5];
        }
        __syncthreads();
    }

#pragma unroll 1
    for (uint32_t job = blockIdx.x + gridDim.x * warp; job < a.njobs; job += gridDim.x * W) {
        uint64_t soff, doff, moff = 0;
        uint32_t slen, n, piece0 = 0;
        bool open = false;
        if (a.jobs) {
            const FusedJob j = a.jobs[job];
            soff = j.src_off; doff = j.dst_off; moff = j.mant_off;
            slen = j.src_len; n = j.n; piece0 = j.piece0;
        } else if (a.sjobs) {
            const StreamJob j = a.sjobs[job];
            soff = j.src_off; doff = j.dst_off; slen = j.src_len; n = j.n;
            open = SINK == SINK_OPEN && (j.flags & STREAM_OPEN);
        } else {
            soff = a.offs[2 * (size_t)job]; slen = (uint32_t)a.offs[2 * (size_t)job + 1];
            n = a.plane; doff = (uint64_t)job * a.plane;
        }
        const bool was_open = open;
        uint32_t st = ST_OK;
        if (!fits) { st = ST_BAD_SHAPE; n = 0; }
        if (n != 0 && slen < LEAD) { st = ST_BAD_HEADER; n = 0; }
        const uint8_t *sbase = a.src + soff;

        // ---- words: this lane's of a round of 32, two rounds ahead of the round that is translated --
        const uintptr_t wat = reinterpret_cast<uintptr_t>(sbase + LEAD) + 2 * lane;
        const uint32_t wsh = (uint32_t)(wat & 3u) * 8u;
        const uint32_t *next = reinterpret_cast<const uint32_t *>(wat & ~uintptr_t(3));
        const uint32_t words = n ? (slen - LEAD) / 2 : 0;
        const int32_t rounds = (int32_t)(words / 32 + (words % 32 != 0));
        int32_t left = rounds;                          // rounds that have not been requested
        const int32_t skip = words % 32 != 0 && lane >= words % 32;       // this lane has no word in the last one
        uint32_t lo[2] = {0, 0}, hi[2] = {0, 0};
        // the next round into lo[1], hi[1], where `want`
        auto request = [&](bool want) {
            const int32_t go = want ? left - skip : 0;
            if (want) { lo[0] = lo[1]; hi[0] = hi[1]; }
            // (no branch; the second word only where a word of the stream straddles two)
            asm volatile("{\n\t.reg .pred p, q;\n\tsetp.gt.s32 p, %3, 0;\n\tsetp.eq.and.u32 q, %4, 24, p;\n\t"
                         "@p ld.global.nc.u32 %0, [%2];\n\t@q ld.global.nc.u32 %1, [%2+4];\n\t}"
                         : "+r"(lo[1]), "+r"(hi[1]) : "l"(next), "r"(go), "r"(wsh));
            if (go > 10 && lane == 0) prefetch_l2(next + 128);        // 512 bytes ahead, eight rounds
            next += want ? 16 : 0;
            left -= want ? 1 : 0;
        };
        uint32_t first[2][2];
#pragma unroll
        for (int j = 0; j < 2; j++) {
            request(true);
            first[j][0] = lo[1]; first[j][1] = hi[1];
        }
        request(true);
        request(true);
        uint32_t x = 0;
        bool ok = true;
        if (n) {
            uint32_t f[8], w1[1];
            load_words_nc<1>(sbase + HDR_BYTES + 4 * k, w1);
            x = w1[0];
            load_freqs(sbase, lane, f);
            ok = WIDE ? solo_tables<true>(f, tab_sa, rec_sa, lane) : solo_byte_tables(f, tab_sa, rec_sa, lane);
            ok = ok && sbase[0] == 'R' && sbase[1] == '1';
        }
        if (!ok) { st = ST_BAD_HEADER; n = 0; }
        n = __shfl_sync(0xffffffffu, n, 0);

        uint8_t *out = a.dst + doff;
        uint32_t rd = 0, wr = 0;                        // words consumed / translated, in bytes of ring entries
        if (n) {
            // where a state's slot lies in the table; the entry of a slot, from its own table or (the
            // byte looked up) from its symbol's, whose c wants the slot's address added
            auto slot_at = [&](uint32_t v) { return WIDE ? (v * S_ENTRY & (S_WIDE_BYTES - S_ENTRY)) | tab_sa : (v & (PROB_SCALE - 1)) | tab_sa; };
            auto byte_at = [&](uint32_t ta) { return WIDE ? 0u : lds_u8(ta); };
            auto entry_at = [&](uint32_t ta, uint32_t s) { return WIDE ? ta : rec_sa + S_ENTRY * s; };
            // a round of words into the ring, in three parts, so that steps can run between them
            uint32_t tv, tt, ts;
            uint2 te;
            bool room;
            auto part1 = [&]() {
                room = wr - rd <= S_RING - S_ROUND;
                tv = __funnelshift_r(lo[0], hi[0], wsh) & 0xffffu;
                tt = slot_at(tv);
                ts = byte_at(tt);
            };
            auto part2 = [&]() { te = lds_u64(entry_at(tt, ts)); };
            auto part3 = [&]() {
                const uint32_t c = (tv >> PROB_BITS) * (te.x >> 8) + (WIDE ? te.y : tt + te.y), at = ring_sa + (wr & (S_RING - 1)) + S_ENTRY * lane;
                sts_u64_if(room, at, te.x, c);
                sts_u64_if(room && !(wr & (S_RING - 1)), at + S_RING, te.x, c);      // (a block reads on behind the ring's end)
                wr += room ? S_ROUND : 0;
                request(room);
                __syncwarp();
            };
            const uint32_t lo1 = lo[1], hi1 = hi[1], lo0 = lo[0], hi0 = hi[0];
            const uint32_t *next0 = next;
            const int32_t left0 = left;
            left = 0;
#pragma unroll
            for (int j = 0; j < 2; j++) {
                lo[0] = first[j][0]; hi[0] = first[j][1];
                part1(); part2(); part3();
            }
            lo[0] = lo0; hi[0] = hi0; lo[1] = lo1; hi[1] = hi1; next = next0; left = left0;
            // words taken so far
            auto taken_now = [&]() { return 32u * (uint32_t)(rounds - left - 2) - (wr - rd) / S_ENTRY; };

            uint32_t y = x >> PROB_BITS, x2 = x, c;
            uint32_t e;                                     // frequency << 8 | symbol
            {
                const uint32_t ta = slot_at(x);
                const uint2 r = lds_u64(entry_at(ta, byte_at(ta)));
                e = r.x;
                c = WIDE ? r.y : ta + r.y;
            }
            uint32_t base = 0;
            auto put = [&](uint32_t at_stage, bool active) {
                solo_put(me, at_stage, active, [&](uint32_t on, uint32_t at) { sts_u8_if(on, at, e); });
            };
            auto step = [&](uint32_t at_stage) {
                put(at_stage, true);
                x2 = y * (e >> 8) + c;
                const uint32_t ta = slot_at(x2), s = byte_at(ta);
                const bool need = owner && x2 < RANS_LOW;
                uint2 r = {0, 0};
                if (WIDE) lds_u64_if(!need, ta, r);             // (on its way while the vote is)
                const uint32_t vote = __ballot_sync(0xffffffffu, need);
                const uint32_t at = __dp4a(__byte_perm(0x02010100u, 0x03020201u, vote & below), S_ENTRY * 0x01010101u, base);
                if (WIDE) lds_u64_if(need, at, r);
                else r = lds_u64(need ? at : entry_at(ta, s));
                y = need ? x2 * 16 : x2 >> PROB_BITS;
                e = r.x;
                c = WIDE ? r.y : r.y + (need ? 0u : ta);
                base += S_ENTRY * __popc(vote);
            };

            uint32_t m[5] = {0, 0, 0, 0, 0};
            const uint8_t *mant = a.src + moff + 16 * lane;
            const uint32_t msh = (uint32_t)(reinterpret_cast<uintptr_t>(mant) & 3u) * 8u;
            const uint32_t *mq = reinterpret_cast<const uint32_t *>(reinterpret_cast<uintptr_t>(mant) & ~uintptr_t(3));
            if (SINK == SINK_BF16 && n > 16 * lane) {
#pragma unroll
                for (int i = 0; i < 5; i++) m[i] = __ldg(mq + i);
            }
            const uint32_t al = (uint32_t)(reinterpret_cast<uintptr_t>(out) & 15u);
            uint32_t ra[NRA];
#pragma unroll
            for (int i = 0; i < NRA; i++) ra[i] = 0;

#pragma unroll 1
            for (uint32_t t = 0, tiles = tiles_of(n, S_TILE); t < tiles; t++) {
                const uint32_t done = t * S_TILE;
                uint32_t rem = min(n - done, S_TILE);
                uint32_t pr[SINK == SINK_F32 ? 3 : 1][5];
                if constexpr (SINK == SINK_F32) {
                    const bool mine = rem > 16 * lane;
#pragma unroll
                    for (int j = 0; j < 3; j++) {
                        const uint8_t *pp = a.src + moff + (size_t)j * n + done + 16 * lane;
                        const uint32_t *pq = reinterpret_cast<const uint32_t *>(reinterpret_cast<uintptr_t>(pp) & ~uintptr_t(3));
#pragma unroll
                        for (int i = 0; i < 5; i++) pr[j][i] = mine ? __ldg(pq + i) : 0u;
                    }
                }
                // ---- up to 64 steps: eight at a time while they are whole (and, of an open stream, while
                // its words are sure to be enough: `left` > 0 means 64 more than are translated).
                // Eight steps take 64 words at most, four 32.  With 32 in the ring at their start, and a round
                // more where the ring has room, the second four have theirs; the check for the next eight
                // looks at the count behind the first four, which nothing waits for by then.
                uint32_t s = 0;
                const uint32_t whole = rem / 64 * 8;
#pragma unroll 1
                for (; s < whole && !(SINK == SINK_OPEN && open && left <= 0); s += 8) {
                    const uint32_t at = stage_sa + s * NLANES;
                    base = ring_sa + (rd & (S_RING - 1));
                    uint32_t base0 = base;
                    part1();
                    step(at);
                    part2();
                    step(at + 8);
                    part3();
                    step(at + 16);
                    step(at + 24);
                    rd += base - base0;
                    const bool low = wr - rd < 2 * S_ROUND;
                    base = ring_sa + (rd & (S_RING - 1));
                    base0 = base;
                    step(at + 32);
                    step(at + 40);
                    if (low) { part1(); part2(); part3(); }
                    step(at + 48);
                    step(at + 56);
                    rd += base - base0;
                }
                // one step at a time, of any mix of lanes: those past the end keep what they have
#pragma unroll 1
                for (; s * NLANES < rem; s++) {
                    if (wr - rd < S_ROUND) { part1(); part2(); part3(); }
                    base = ring_sa + (rd & (S_RING - 1));
                    const bool active = s * NLANES + k < rem;
                    put(stage_sa + s * NLANES, active);
                    const uint32_t nx = y * (e >> 8) + c;
                    const bool need = owner && active && nx < RANS_LOW;
                    const uint32_t vote = __ballot_sync(0xffffffffu, need), before = __popc(vote & below);
                    const uint32_t ta = slot_at(nx), sn = byte_at(ta);
                    const uint2 r = lds_u64(need ? base + S_ENTRY * before : entry_at(ta, sn));
                    if (active) {
                        x2 = nx;
                        y = need ? nx * 16 : nx >> PROB_BITS;
                        e = r.x;
                        c = WIDE ? r.y : r.y + (need ? 0u : ta);
                    }
                    if (SINK == SINK_OPEN && open) {
                        // the first lane that took a word the stream has not got ends it
                        const uint32_t outs = __ballot_sync(0xffffffffu, need && taken_now() + before >= words);
                        if (outs) {
                            n = done + s * NLANES + __popc(S_LANES & ((outs & (0u - outs)) - 1u));
                            rem = n - done;
                            tiles = t + 1;
                            open = false;
                        }
                    }
                    rd += S_ENTRY * __popc(vote);
                }
                __syncwarp();
                if (rem == 0) break;                     // (an open stream that ended with the tile before)

                // ---- 16 symbols a lane
                const uint4 ev = lds_u128(stage_sa + 16 * lane);
                __syncwarp();
                const uint32_t ew[4] = {ev.x, ev.y, ev.z, ev.w};
                const uint32_t ve = rem > 16 * lane ? min(rem - 16 * lane, 16u) : 0u;
                if constexpr (SINK == SINK_BYTES || SINK == SINK_OPEN) {
                    uint8_t *d = out + done + 16 * lane;
                    if (ve == 16 && al == 0) {
                        *reinterpret_cast<uint4 *>(d) = ev;
                    } else {
#pragma unroll
                        for (uint32_t i = 0; i < 16; i++)
                            if (i < ve) d[i] = (uint8_t)(ew[i >> 2] >> (8 * (i & 3)));
                    }
                } else {
                    uint32_t v[NRA];
                    if constexpr (SINK == SINK_BF16) {
#pragma unroll
                        for (int h = 0; h < 4; h++)
                            bf16_merge4(ew[h], __funnelshift_r(m[h], m[h + 1], msh), v[2 * h], v[2 * h + 1]);
                        if (n - done > S_TILE + 16 * lane) {            // the next tile's stored bytes
#pragma unroll
                            for (int i = 0; i < 5; i++) m[i] = __ldg(mq + (size_t)(t + 1) * (S_TILE / 4) + i);
                        }
                    } else {
                        uint32_t pw[3][4];
#pragma unroll
                        for (int j = 0; j < 3; j++) {
                            const uint32_t sh = (uint32_t)((reinterpret_cast<uintptr_t>(a.src) + moff + (size_t)j * n + done) & 3u) * 8u;
#pragma unroll
                            for (int h = 0; h < 4; h++) pw[j][h] = __funnelshift_r(pr[j][h], pr[j][h + 1], sh);
                        }
#pragma unroll
                        for (int h = 0; h < 4; h++) {
                            const uint32_t u0 = __byte_perm(pw[0][h], pw[1][h], 0x5140), u1 = __byte_perm(pw[0][h], pw[1][h], 0x7362);
                            const uint32_t v0 = __byte_perm(pw[2][h], ew[h], 0x5140), v1 = __byte_perm(pw[2][h], ew[h], 0x7362);
                            v[4 * h + 0] = __byte_perm(u0, v0, 0x5410); v[4 * h + 1] = __byte_perm(u0, v0, 0x7632);
                            v[4 * h + 2] = __byte_perm(u1, v1, 0x5410); v[4 * h + 3] = __byte_perm(u1, v1, 0x7632);
                        }
                    }
                    constexpr uint32_t ES = SINK == SINK_F32 ? 4 : 2, UNIT = 16 * ES;
                    uint8_t *d = out + (size_t)done * ES + UNIT * lane;
                    if (ve == 16) {
                        if (al == 0) {
#pragma unroll
                            for (int i = 0; i < NRA / 4; i++)
                                reinterpret_cast<uint4 *>(d)[i] = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                        } else if ((al & 7) == 0) {
#pragma unroll
                            for (int i = 0; i < NRA / 2; i++) reinterpret_cast<uint2 *>(d)[i] = make_uint2(v[2 * i], v[2 * i + 1]);
                        } else if ((al & 3) == 0) {
#pragma unroll
                            for (int i = 0; i < NRA; i++) reinterpret_cast<uint32_t *>(d)[i] = v[i];
                        } else {
#pragma unroll
                            for (uint32_t i = 0; i < UNIT; i++) d[i] = (uint8_t)(v[i >> 2] >> (8 * (i & 3)));
                        }
                    } else {
                        // (bytes past the end count as zeros for the checksum)
                        const uint32_t vb = ES * ve;
#pragma unroll
                        for (uint32_t i = 0; i < UNIT; i++)
                            if (i < vb) d[i] = (uint8_t)(v[i >> 2] >> (8 * (i & 3)));
#pragma unroll
                        for (int i = 0; i < NRA; i++) {
                            const uint32_t keep = vb > 4u * i ? min(vb - 4u * i, 4u) : 0u;
                            v[i] = keep >= 4 ? v[i] : (keep ? v[i] & ((1u << (8 * keep)) - 1u) : 0u);
                        }
                    }
                    if (CRC) {
#pragma unroll
                        for (int i = 0; i < NRA; i++) ra[i] = crc_feed4q(cq, ra[i]) ^ v[i];
                        if (t % ROWS == ROWS - 1 || n - done <= S_TILE) {
                            // close the 64 KiB piece: every running value to the row's end, XOR over the lanes
                            uint32_t r = 0;
#pragma unroll 1
                            for (int i = 0; i < NRA; i++) {
                                const uint32_t q = ra[0];
#pragma unroll
                                for (int j = 0; j + 1 < NRA; j++) ra[j] = ra[j + 1];
                                ra[NRA - 1] = 0;
                                r ^= crc_mulmod(a.tabs->word_pow[ROW / 4 - NRA * lane - i], q);
                            }
                            r = __reduce_xor_sync(0xffffffffu, r);
                            if (lane == 0) {
                                const uint32_t p = t / ROWS, rows = t % ROWS + 1;
                                const uint32_t plen = min(PIECE_BYTES, ES * n - p * PIECE_BYTES);
                                if (rows * ROW != plen) r = crc_unshift(a.tabs->x2, r, rows * ROW - plen);
                                a.piece_crc[piece0 + p] = r;
                            }
                        }
                    }
                }
            }
            // ---- verdict.  A sound stream's states end as 2^16: unrefilled, or as 1 with a word of zeros,
            // whose entry is slot 0's.
            const uint32_t t0 = slot_at(0), f0 = lds_u64(entry_at(t0, byte_at(t0))).x;
            const bool rests = x2 == RANS_LOW || (x2 == 1 && e == f0 && c == 0) || !owner;
            const uint64_t used = LEAD + 2 * (uint64_t)taken_now();
            if (!was_open) {
                const bool rest = __all_sync(0xffffffffu, rests);
                if (used > slen) st = ST_OVERRUN;
                else if (used != slen || !rest) st = ST_SLACK;
            }
        }
        if (lane == 0) {
            if (was_open) const_cast<StreamJob *>(a.sjobs)[job].aux = st == ST_OK ? n : 0u;
            if (a.status) a.status[job] = st;
            if (a.any_bad && st != ST_OK && st != ST_SLACK) atomicOr(a.any_bad, 1u);
        }
        __syncwarp();
    }
}

}  // namespace lmz
