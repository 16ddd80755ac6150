// k_stream: the decode kernel of launches of many streams (few: solo_kernel.cuh).  One 8-lane group per
// rANS stream and the stream's consumer fused into the decode loop:
//
//   SINK_BYTES  the decoded plane is written as is (decode_batch, scratch planes)
//   SINK_OPEN   the same where open streams (STREAM_OPEN) may be among them; an instance of its own, as
//               the watch for their ends costs the others 8 %
//   SINK_BF16   a CODEC_BF16 chunk whose exponent plane is rANS and whose
//               sign/mantissa plane is stored: each 128-symbol tile is merged with
//               128 stored bytes (lmz/native/lmzcore.c:439-447), written once as
//               256 bytes of BF16, and folded into the chunk's CRC-32 -- no
//               scratch plane, no second pass
//   SINK_F32    a CODEC_SPLIT chunk of 4-byte elements whose top byte plane is rANS
//               and whose three lower planes are stored back to back: each tile is
//               interleaved with 3 x 128 stored bytes (lmz/native/lmzcore.c:289-347),
//               written once as 512 bytes and folded into the chunk's CRC-32
//   SINK_DELTA  a delta chunk (lmz/codec.py:1012-1057) whose difference is a CODEC_BF16
//               chunk with both planes rANS: two neighbouring groups of a warp decode the two
//               planes in step, the merged difference is XOR-ed with the base bytes already
//               in the output space, written once and checksummed (CFN = 192: a 128-entry
//               level 2 for the first plane, a 256-entry one for the second)
//
// What bounds it: a symbol depends on the one before it, so the time of a launch is (steps of
// a stream) x (latency of a step) x (waves of streams), and the chip is filled with as many
// streams as shared memory and registers hold.  A step is a table lookup on the state's low
// 12 bits, the state update, and -- for the lanes whose state fell below 2^16 -- a refill with
// the next 16-bit word of the stream, whose place a vote over the group gives.  Done in that
// order a refilled lane's lookup waits for update, vote, popcount, word and then the table.
// Here the words are looked up before anyone asks for them: while the group decodes, each of its
// lanes also translates two of the next sixteen words (their place in the table is known: a
// refilled state's low 12 bits ARE the word's) and leaves word and lookup result together in a
// ring in shared memory.  A refilled lane finds its next table entry in the word it fetches, the
// other lanes look theirs up meanwhile, and the two halves of the old chain run side by side.
//
//   * compressed words come straight from global memory into registers, two aligned 32-bit
//     loads per lane and 16 words (any byte alignment: a funnel shift), one round ahead
//   * the ring holds 64 translated words and a copy of its first 32 behind them, so a block of
//     four steps reads linearly; a round of 16 is translated every eight steps where there is
//     room, and a loop before each block tops up streams that consume more than that
//   * refill offsets come from a 4-step history of the group's votes: one
//     byte-permute and one popcount per step instead of two popcounts
//   * a warp's four level-1 tables interleave word by word: the lookup address is the state's
//     bits 4-11 unshifted, and the four streams' lookups stay in different banks
//   * CFN = 128: level 2 has 128 slots, the four streams of a warp rotated 8
//     entries apart so their popular symbols sit in different banks; streams with
//     more than 104 live symbols must be given to the CFN = 256 instance
//   * a ring entry is word and table entry (8 bytes), or word and level-2 offset (TR_4: 4 bytes, half
//     the space: more streams per SM for one more lookup in a refilled lane's step)
//   * CFN = 1 (F_BYTE_CFN), up to 24 or 28 streams per SM: k_solo's tables of a byte per slot and its 8-byte entries, 7.6 KiB a
//     stream; a step is two lookups without a popcount between them, and half as many instructions of the integer
//     pipe, of which a warp that has a scheduler to itself issues one in two cycles
//   * CFN = 0 (few delta chunks): a 16 KiB slot -> entry table per stream; CFN = -1: one such table per CTA, for
//     batches whose streams share one 516-byte table (lmz_gpu_decode_batch's d_hdr) or for the
//     chunks of a shared-table archive (StreamArgs.tables); a stream is then states + words
//   * warps are independent: each takes four streams, then the next four, ...; a launch is
//     at most one CTA per SM, with no more warps than its streams need
#pragma once
#include "chunk_kernels.cuh"
#include "rans.cuh"
#include "solo_tables.cuh"

namespace lmz {

enum : int { SINK_BYTES = 0, SINK_BF16 = 1, SINK_F32 = 2, SINK_DELTA = 3, SINK_OPEN = 4 };
// How a kernel instance keeps its translated words, and how many warps it is for (see Words):
//   TR_FEW  8-byte ring entries, data brought to the L2 early: up to 16 warps
//   TR_8    8-byte ring entries
//   TR_4    4-byte ring entries: the most warps
enum : int { TR_4 = 0, TR_8 = 1, TR_FEW = 2 };
constexpr uint32_t TR_N = 64, TR_MIRROR = 32;      // ring of translated words; a block of four steps reads at most 32
constexpr uint32_t TR_ROUND = 16;                  // words translated at a time, two per lane
constexpr uint32_t F_ROW = 256;                    // bytes of BF16 one group emits per tile
constexpr int F_SMALL_CFN = 128;                   // level-2 slots of the dense instance
constexpr int F_BYTE_CFN = 1;                      // a byte per slot, its symbol, and k_solo's 8-byte entries: a middling number of streams
constexpr int F_HYBRID_CFN = 192;                  // delta sink: 128-entry tables for first planes, 256-entry for second planes
constexpr uint32_t F_SMALL_LIVE = F_SMALL_CFN - 24; // largest alphabet it takes (the warp's streams sit 0, 8, 16, 24 entries in)

// F_BYTE_CFN: a stream's 256 entries, and the next one's sixteen banks on, so that two streams' popular symbols lie apart
// (28 streams of bytes per SM 379 -> 370 us through the public call, tables filled one symbol after the other).
constexpr uint32_t F_REC_STRIDE = S_REC_BYTES + 64;

// Bytes of a stream's stage, a tile's 128 symbols and some: groups land four banks apart, or, where a lane takes a word from
// each of four places, eight.  (With 160 for all, 28577 streams of 32 KiB 1536 -> 1560 us.)
__host__ __device__ constexpr uint32_t stage_bytes(int sink) { return sink == SINK_BF16 || sink == SINK_F32 ? 160u : 144u; }

struct FusedJob {
    uint64_t src_off;    // rANS stream, bytes from the source base
    uint64_t mant_off;   // SINK_BF16: the stored sign/mantissa plane, bytes from the source base;
                         // SINK_F32: stored plane 0, planes 1 and 2 follow at n and 2n
    uint64_t dst_off;    // first output byte
    uint32_t src_len;
    uint32_t n;          // symbols (= elements)
    uint32_t piece0;     // first piece id of the chunk (for piece_crc)
    uint32_t flags;
};
static_assert(sizeof(FusedJob) == 40, "FusedJob layout is shared with the host");

// SINK_DELTA: a delta chunk (lmz/codec.py:1012-1057) whose difference is a CODEC_BF16 chunk
// with both planes rANS-coded.  Two neighbouring stream groups of a warp decode the two
// planes in step; the merged difference is XOR-ed with the base bytes, which are already in
// the output space, and written once.
struct DeltaJob {
    uint64_t src_a, src_b;   // the exponent plane's and the sign/mantissa plane's streams
    uint64_t dst_off;        // first output byte
    uint64_t base_off;       // the chunk this one is a difference against, in the output space
    uint32_t len_a, len_b;
    uint32_t n;              // elements
    uint32_t piece0;
};
static_assert(sizeof(DeltaJob) == 48, "DeltaJob layout is shared with the host");

struct StreamArgs {
    const uint8_t *src;
    const FusedJob *jobs;       // SINK_BF16 jobs, or NULL
    const StreamJob *sjobs;     // plain stream jobs, or NULL
    const DeltaJob *djobs;      // SINK_DELTA: njobs counts streams, two per job
    const uint64_t *offs;       // neither: reference layout, (offset, length) pairs + plane
    uint32_t plane;
    uint32_t njobs;
    uint8_t *dst;
    uint32_t *status;
    uint32_t *any_bad;
    uint32_t *piece_crc;        // SINK_BF16 with checksums: R() per 64 KiB piece
    const CrcTables *tabs;
    const uint8_t *shared_hdr;  // CFN = -1: the 516-byte table every stream of the launch shares
    const uint8_t *tables;      // CFN = -1, or NULL: the 516-byte tables of a shared-table archive, F_TABLE_STRIDE
                                // bytes apart; a CTA's streams all use table number `flags` of its first job
    // Optional indirection, filled on the device by k_classify: the launch covers the
    // first *count entries of `order` (read from its end backwards when order_from_back),
    // each the index of a job; CTAs past the count leave at once.
    const uint32_t *order;
    const uint32_t *count;
    uint32_t order_from_back;
    uint32_t most_ctas;         // for the launcher: fewer CTAs than there are SMs (0 = one per SM), as something
                                // else runs beside this launch
};

constexpr uint32_t F_WIDE_BYTES = PROB_SCALE * 4;   // a slot -> entry table
constexpr uint32_t F_TABLE_STRIDE = 528;            // 516 rounded up to 16
constexpr uint32_t F_SHARED_SINK_WARPS = 20;        // chunks of a shared-table archive: 80 per CTA share its table

// Where a CTA of W warps keeps what, as addresses in the shared window.  The CRC tables sit on a
// 32 KiB boundary (a table index is OR-ed onto the base) and level-1 tables on 4 KiB boundaries;
// what fits goes below the CRC tables, chosen so that the whole is shortest.
struct StreamSmem {
    uint32_t cf, stage, tr, l1, crc, poison, end;
};
__host__ __device__ constexpr uint32_t tr_entry(int mode) { return mode == TR_4 ? 4u : 8u; }
__host__ __device__ constexpr uint32_t tr_words(int cfn) { return cfn == F_BYTE_CFN ? 2 * TR_N : TR_N; }
__host__ __device__ constexpr uint32_t tr_group(int cfn, int mode) { return (tr_words(cfn) + TR_MIRROR) * tr_entry(mode); }
__host__ __device__ constexpr StreamSmem stream_smem_with(int cfn, bool crc, int sink, int mode, uint32_t W, bool low_stage, bool low_tr)
{
    StreamSmem m{};
    uint32_t p = F_SMEM_BASE;
    m.poison = p; p += cfn < 0 ? 16u : 0u;
    const uint32_t cf = cfn == F_BYTE_CFN ? W * 4u * F_REC_STRIDE : cfn > 0 ? W * 16u * (uint32_t)cfn : 0u, stage = W * 4u * stage_bytes(sink), tr = W * 4u * tr_group(cfn, mode);
    m.cf = p; p += cf;
    if (low_stage) { m.stage = p; p += stage; }
    if (low_tr) { m.tr = p; p += tr; }
    if (crc) {
        p = (p + F_CRC_BYTES - 1) & ~(F_CRC_BYTES - 1);
        m.crc = p; p += F_CRC_BYTES;
    }
    const uint32_t align = cfn > 0 ? 4096u : F_WIDE_BYTES;
    p = (p + align - 1) & ~(align - 1);
    m.l1 = p; p += cfn == F_BYTE_CFN ? W * 4u * PROB_SCALE : cfn > 0 ? W * 4096u : cfn == 0 ? W * 4u * F_WIDE_BYTES : F_WIDE_BYTES;
    if (!low_tr) { m.tr = p; p += tr; }
    if (!low_stage) { m.stage = p; p += stage; }
    m.end = p;
    return m;
}
__host__ __device__ constexpr StreamSmem stream_smem(int cfn, bool crc, int sink, int mode, uint32_t W)
{
    StreamSmem best = stream_smem_with(cfn, crc, sink, mode, W, false, false);
    for (int i = 1; i < 4; i++) {
        const StreamSmem m = stream_smem_with(cfn, crc, sink, mode, W, (i & 1) != 0, (i & 2) != 0);
        if (m.end < best.end) best = m;
    }
    return best;
}
// The most warps of an instance: what shared memory holds, and registers (128 a thread up to 16
// warps, 96 up to 20, 80 up to 24).
__host__ __device__ constexpr uint32_t stream_warps(int cfn, bool crc, int sink, int mode)
{
    if (cfn < 0 && sink == SINK_BF16) return F_SHARED_SINK_WARPS;
    uint32_t w = cfn < 0 ? 32u : mode == TR_FEW ? 16u : 24u;
    while (stream_smem(cfn, crc, sink, mode, w).end > F_SMEM_BASE + F_SMEM_DYN) w--;
    return w;
}

// ---- the ring of translated words ------------------------------------------------------------
// A slot's table entry (wide: its address), `from` bytes on.  Compact: from its byte offset from the stream's first entry.
template <int CFN>
__device__ __forceinline__ uint32_t slot_ref(uint32_t x, uint32_t l1_sa, uint32_t from)
{
    if (CFN <= 0) return ((x << 2) & 0x3ffcu) | l1_sa;         // the table is 16 KiB aligned
    // the warp's four level-1 tables are interleaved word by word, so bucket b of this group
    // sits 16 * b bytes in -- the slot's bits 4-11, unshifted
    const uint32_t e1 = lds_u32((x & 0xff0u) | l1_sa);
    return high_half_add(e1, from + 4u * __popc(e1 << ((~x & 15u) | 16u)));
}
// Its address.  One B200: TR_4 adds the tables' address last, as a ring entry's is added (four 8B layers 1711 us, 1800 with a sum
// of three); TR_8 first (28577 streams of 32 KiB 1535 us, 1576 with it last); TR_FEW, whose warps have the integer pipe almost to
// themselves, takes the offset by a shift (44 BF16 chunks per SM 586 us, 603 by a dot product).  The delta sink's mixed tables are
// the other way round: TR_4 by a shift (a chain of 14.9 K chunks 1934 us, 1945 by a dot product), TR_FEW by a dot product (a chain of
// 10.3 K 1493 us, 1499 by a shift; one of 6.1 K 936 and 934).
template <int CFN, int MODE>
__device__ __forceinline__ uint32_t slot_addr(uint32_t x, uint32_t l1_sa, uint32_t cf_sa)
{
    if (CFN > 0 && MODE == (CFN == F_HYBRID_CFN ? TR_4 : TR_FEW)) {
        const uint32_t e1 = lds_u32((x & 0xff0u) | l1_sa);
        return cf_sa + ((e1 >> 16) + 4u * __popc(e1 << ((~x & 15u) | 16u)));
    }
    if (CFN > 0 && MODE == TR_4) return cf_sa + slot_ref<CFN>(x, l1_sa, 0u);
    return slot_ref<CFN>(x, l1_sa, cf_sa);
}

// Positions are in bytes of ring entries and only grow; the ring index is the position modulo the ring.
//
// A warp that waits for one load waits for all that the compiler counts on the same counter, however
// long ago they were requested, so where warps are few every load in flight is a stall (one B200, 12
// streams per SM: a third of the time; bulk copies through a raw ring cost as much as they saved).
// TR_FEW has the L2 fetch words 512 bytes ahead, and the stored bytes that a sink merges four tiles
// ahead.  On one B200: a 4096 x 14336 BF16 tensor's kernel 581 -> 458 us, the delta kernel of a
// three-checkpoint chain 1189 -> 1083 us.
template <int CFN, int MODE>
struct Words {
    static constexpr bool TR8 = MODE != TR_4;
    static constexpr int AHEAD = MODE == TR_FEW ? 2 : 1;
    static constexpr bool BYTES = CFN == F_BYTE_CFN;
    static constexpr uint32_t ES = tr_entry(MODE), RB = tr_words(CFN) * ES, LOW = TR_MIRROR * ES;
    static_assert(TR8 || CFN > 0, "a wide table's entry does not fit a 4-byte ring entry");
    uint32_t sa;             // the ring
    uint32_t rd, wr;         // words consumed / translated so far
    uint32_t lo, hi, sh;     // this lane's next two words: aligned loads and the shift between them
    uint32_t lo2, hi2;       // TR_FEW: and the two after those
    const uint32_t *next;
    int32_t left;            // rounds of the stream that have not been requested

    // This lane's next two words, if the stream has them and `want`.  No branch: the loads are
    // predicated.  A stream is read front to back in 32-byte pieces: the L2 is asked for 256 bytes
    // at a time, so that most requests wait for the L2 and not for HBM.
    __device__ __forceinline__ void request(bool want)
    {
        const int32_t go = want ? left : 0;
        if constexpr (MODE == TR_FEW) {
            if (want) { lo = lo2; hi = hi2; }
            asm volatile("{\n\t.reg .pred p;\n\tsetp.gt.s32 p, %3, 0;\n\t"
                         "@p ld.global.nc.u32 %0, [%2];\n\t@p ld.global.nc.u32 %1, [%2+4];\n\t}"
                         : "+r"(lo2), "+r"(hi2) : "l"(next), "r"(go));
            if (go > 20 && !(reinterpret_cast<uintptr_t>(next) & 64u)) prefetch_l2(next + 128);
        } else {
            asm volatile("{\n\t.reg .pred p;\n\tsetp.gt.s32 p, %3, 0;\n\t"
                         "@p ld.global.nc.L2::256B.u32 %0, [%2];\n\t@p ld.global.nc.u32 %1, [%2+4];\n\t}"
                         : "+r"(lo), "+r"(hi) : "l"(next), "r"(go));
        }
        next += want ? TR_ROUND / 2 : 0;
        left -= want ? 1 : 0;
    }
    __device__ __forceinline__ uint32_t block() const { return sa + (rd & (RB - 1)); }
    // Fewer than `blocks` of four steps can take.
    __device__ __forceinline__ bool low(uint32_t blocks = 1) const { return wr - rd < blocks * LOW; }
    // Words consumed so far of a stream of that many bytes.  (Positions are 32-bit bytes of ring entries
    // and wrap in a stream of half a Gi words; the rounds do not.  AHEAD rounds are loaded ahead of `wr`.)
    __device__ __forceinline__ uint32_t taken(uint32_t bytes) const
    {
        const int32_t rounds = (int32_t)((bytes / 2 + TR_ROUND - 1) / TR_ROUND) - left - AHEAD;
        return TR_ROUND * (uint32_t)rounds - (wr - rd) / ES;
    }
    // A group that only runs along asks for no more words (and writes none: there is never room).
    __device__ __forceinline__ void retire() { wr = rd + 0x40000000u; }

    // A round in three parts, so that the steps of the decode run between them.
    uint32_t v, r0, r1;
    uint2 b0, b1;            // F_BYTE_CFN: the entries of the symbols r0, r1
    bool room;
    __device__ __forceinline__ void part1()
    {
        room = wr - rd <= RB - TR_ROUND * ES;
        v = __funnelshift_r(lo, hi, sh);
    }
    __device__ __forceinline__ void part2(uint32_t l1_sa, uint32_t cf_sa)
    {
        if constexpr (BYTES) {
            r0 = lds_u8((v & (PROB_SCALE - 1)) | l1_sa);
            r1 = lds_u8((v >> 16 & (PROB_SCALE - 1)) | l1_sa);
            return;
        }
        r0 = slot_ref<CFN>(v, l1_sa, TR8 ? cf_sa : 0u);          // (a 4-byte ring entry has the offset alone)
        r1 = slot_ref<CFN>(v >> 16, l1_sa, TR8 ? cf_sa : 0u);
    }
    __device__ __forceinline__ void part2b(uint32_t cf_sa)
    {
        b0 = lds_u64(cf_sa + S_ENTRY * r0);
        b1 = lds_u64(cf_sa + S_ENTRY * r1);
    }
    __device__ __forceinline__ void part3(uint32_t l1_sa, uint32_t cf_sa, uint32_t k)
    {
        const uint32_t at = sa + (wr & (RB - 1)) + 2u * ES * k;
        const uint32_t keep = room, again = room && !(wr & (RB - LOW));
        if constexpr (BYTES) {
            const uint2 e0 = b0, e1 = b1;
            const uint32_t c0 = (v >> PROB_BITS & 15u) * (e0.x >> 8) + e0.y + ((v & (PROB_SCALE - 1)) | l1_sa);
            const uint32_t c1 = (v >> 28) * (e1.x >> 8) + e1.y + ((v >> 16 & (PROB_SCALE - 1)) | l1_sa);
            sts_u128_if(keep, at, e0.x, c0, e1.x, c1);
            sts_u128_if(again, at + RB, e0.x, c0, e1.x, c1);
        } else if (TR8) {
            const uint32_t e0 = lds_u32(r0), e1 = lds_u32(r1);
            sts_u128_if(keep, at, e0, v, e1, v >> 16);
            sts_u128_if(again, at + RB, e0, v, e1, v >> 16);
        } else {
            const uint32_t t0 = __byte_perm(v, r0, 0x5410), t1 = __byte_perm(v, r1, 0x5432);
            sts_u64_if(keep, at, t0, t1);
            sts_u64_if(again, at + RB, t0, t1);
        }
        wr += room ? TR_ROUND * ES : 0;
        request(room);
    }
    __device__ __forceinline__ void round(uint32_t l1_sa, uint32_t cf_sa, uint32_t k)
    {
        part1();
        part2(l1_sa, cf_sa);
        if constexpr (BYTES) part2b(cf_sa);
        part3(l1_sa, cf_sa, k);
    }
};

// MULT: the start field is e >> 8 less the bits above it, taken off by the multiplier's pipe, as the integer
// pipe is the busy one where warps are many.  One B200: four 8B layers 1825 -> 1796 us, 28577 streams of 32 KiB
// 1588 -> 1574; a delta chain, whose merge keeps the multiplier busy, 1534 -> 1547, so not there.
template <bool MULT>
__device__ __forceinline__ uint32_t rans_update(uint32_t x, uint32_t e)
{
    // f * (x >> 12) + slot - start  ==  x - (x >> 12) * (4096 - f) - start
    if constexpr (MULT) {
        const uint32_t g = e >> 20;
        uint32_t start, u;
        asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(start) : "r"(g), "r"(0u - PROB_SCALE), "r"(e >> 8));
        asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(u) : "r"(x >> PROB_BITS), "r"(g), "r"(start));
        return x - u;
    } else {
        return x - ((x >> PROB_BITS) * (e >> 20) + ((e >> 8) & 0xfffu));
    }
}

// The second half of a step: x2 is the updated state; a lane that needs a refill takes the ring
// entry at word_sa, the others look their slot up.  `e` leaves as the entry of the new state's slot.
template <int CFN, int MODE>
__device__ __forceinline__ void refill(uint32_t &x, uint32_t &e, uint32_t x2, bool need, uint32_t word_sa, uint32_t l1_sa,
                                       uint32_t cf_sa)
{
    uint32_t a = slot_addr<CFN, MODE>(x2, l1_sa, cf_sa);
    if (MODE != TR_4) {
        e = lds_u32(a);
        const uint2 w = lds_u64(word_sa);
        if (need) { e = w.x; x2 = __byte_perm(w.y, x2, 0x5410); }
    } else {
        const uint32_t w = lds_u32(word_sa);
        if (need) { a = cf_sa + (w >> 16); x2 = __byte_perm(w, x2, 0x5410); }
        e = lds_u32(a);
    }
    x = x2;
}

// One step of a full tile, four to a block.  `hist` collects the group's votes of
// the block, newest in byte 0 (vsel = 0x6540 + group picks this group's byte of
// the warp vote and shifts the older ones up); refills consumed before this
// lane's = bits of the older bytes plus the lanes below it in the newest, so one
// popcount of hist & below (= 0xffffff00 | lanes below) gives the offset from
// the block's start.
template <int CFN, int MODE, bool FIRST, bool MULT>
__device__ __forceinline__ void stream_step4(uint32_t &x, uint32_t &e, uint32_t &hist, uint32_t base, uint32_t l1_sa,
                                             uint32_t cf_sa, uint32_t below, uint32_t vsel)
{
    const uint32_t x2 = rans_update<MULT>(x, e);
    const bool need = x2 < RANS_LOW;
    const uint32_t vote = __ballot_sync(0xffffffffu, need);
    hist = __byte_perm(vote, FIRST ? 0u : hist, vsel);
    refill<CFN, MODE>(x, e, x2, need, base + tr_entry(MODE) * __popc(hist & below), l1_sa, cf_sa);
}

// One step of a ragged tile, any lane mix: lanes past the end keep their state.  `base` is where the
// block's next word lies; returns how many of the block's words had been taken when this lane took
// one, NONE32 if it took none.
constexpr uint32_t NONE32 = 0xffffffffu;
template <int CFN, int MODE, bool MULT>
__device__ __forceinline__ uint32_t stream_step(uint32_t &x, uint32_t &e, uint32_t &base, uint32_t base0, uint32_t l1_sa, uint32_t cf_sa,
                                                uint32_t lt_mask, uint32_t grp_mask, bool active)
{
    const uint32_t x2 = rans_update<MULT>(x, e);
    const bool need = active && x2 < RANS_LOW;
    const uint32_t vote = __ballot_sync(0xffffffffu, need);
    const uint32_t at = base + tr_entry(MODE) * __popc(vote & lt_mask);
    uint32_t nx = x, ne = e;
    refill<CFN, MODE>(nx, ne, x2, need, at, l1_sa, cf_sa);
    if (active) { x = nx; e = ne; }
    base += tr_entry(MODE) * __popc(vote & grp_mask);
    return need ? (at - base0) / tr_entry(MODE) : NONE32;
}

// F_BYTE_CFN's steps, as k_solo's: of a state x only y, e and c are kept, of which the next (unrefilled) one is
// y * (e >> 8) + c.  (One B200, planes of 32 KiB: 278 us up to 16 streams per SM, 303 with 24, where the compact tables take 379.
// With two predicated loads instead of the picked one, as k_solo has them, it took a tenth longer.)
struct ByteState {
    uint32_t y, c;
};
__device__ __forceinline__ void byte_next(uint32_t &x, uint32_t &e, ByteState &b, uint32_t x2, bool need, uint32_t word_sa,
                                          uint32_t ta, uint32_t sym, uint32_t rec_sa)
{
    const uint2 r = lds_u64(need ? word_sa : rec_sa + S_ENTRY * sym);
    x = x2;
    b.y = need ? x2 * 16 : x2 >> PROB_BITS;
    e = r.x;
    b.c = r.y + (need ? 0u : ta);
}
template <bool FIRST>
__device__ __forceinline__ void byte_step4(uint32_t &x, uint32_t &e, ByteState &b, uint32_t &hist, uint32_t base, uint32_t tab_sa,
                                           uint32_t rec_sa, uint32_t below, uint32_t vsel)
{
    const uint32_t x2 = b.y * (e >> 8) + b.c;
    const uint32_t ta = (x2 & (PROB_SCALE - 1)) | tab_sa, sym = lds_u8(ta);
    const bool need = x2 < RANS_LOW;
    const uint32_t vote = __ballot_sync(0xffffffffu, need);
    hist = __byte_perm(vote, FIRST ? 0u : hist, vsel);
    byte_next(x, e, b, x2, need, base + S_ENTRY * __popc(hist & below), ta, sym, rec_sa);
}
__device__ __forceinline__ uint32_t byte_step(uint32_t &x, uint32_t &e, ByteState &b, uint32_t &base, uint32_t base0, uint32_t tab_sa,
                                              uint32_t rec_sa, uint32_t lt_mask, uint32_t grp_mask, bool active)
{
    const uint32_t x2 = b.y * (e >> 8) + b.c;
    const uint32_t ta = (x2 & (PROB_SCALE - 1)) | tab_sa, sym = lds_u8(ta);
    const bool need = active && x2 < RANS_LOW;
    const uint32_t vote = __ballot_sync(0xffffffffu, need);
    const uint32_t at = base + S_ENTRY * __popc(vote & lt_mask);
    uint32_t nx = x, ne = e;
    ByteState nb = b;
    byte_next(nx, ne, nb, x2, need, at, ta, sym, rec_sa);
    if (active) { x = nx; e = ne; b = nb; }
    base += S_ENTRY * __popc(vote & grp_mask);
    return need ? (at - base0) / S_ENTRY : NONE32;
}

template <int SINK, bool CRC, int CFN, int MODE>
__global__ void __launch_bounds__(stream_warps(CFN, CRC, SINK, MODE) * 32, 1) k_stream(StreamArgs a)
{
    // Checksums: lane k keeps one running value for each word that it emits of a row (a tile; SINK_F32: a quarter of one),
    // ra[i] = sum over the piece's rows so far of word i * x^(8 * row * rows since); a row
    // costs each of them one multiplication by x^(8 * row) (the same four lookups as feeding a
    // word) with no chain between them and no per-row advance; the constants
    // word_pow[], word_mul16[] carry them to the piece's end.
    constexpr int NRA = SINK == SINK_BF16 ? 8 : 4;        // running values per lane: words of its unit of a row
    extern __shared__ __align__(16) uint8_t ssm[];
    constexpr bool WIDE = CFN <= 0, SHARED = CFN < 0, BYTES = CFN == F_BYTE_CFN, MULT = SINK != SINK_DELTA;
    // SINK_DELTA with CFN = 192: the two planes of a chunk have level-2 tables of different sizes, 128
    // entries for the exponent differences (a handful of symbols) and 256 for the sign/mantissa
    // differences, 768 bytes a stream on average.
    constexpr bool HYB = SINK == SINK_DELTA && CFN == F_HYBRID_CFN;
    static_assert(CFN != F_HYBRID_CFN || SINK == SINK_DELTA, "mixed table sizes are the delta sink's");
    constexpr uint32_t LEAD = (SHARED ? 0u : HDR_BYTES) + STATE_BYTES;
    constexpr uint32_t TS = TILE;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, W = blockDim.x >> 5, G = W * 4;
    const uint32_t k = lane & 7u, g = lane >> 3, gi = warp * 4 + g;
    const uint32_t grp_mask = 0xffu << (g * 8), lt_mask = ((1u << k) - 1u) << (g * 8);
    const uint32_t below = 0xffffff00u | ((1u << k) - 1u), vsel = 0x6540u + g;

    constexpr uint32_t F_STAGE = stage_bytes(SINK);
    // ---- shared memory (addresses are 32-bit shared-space addresses) ----------------------
    const uint32_t s0 = smem_addr(ssm);
    const StreamSmem m_ = stream_smem(CFN, CRC, SINK, MODE, W);
    const bool fits = s0 == F_SMEM_BASE && m_.end <= s0 + dynamic_smem_bytes();
    auto gen = [&](uint32_t sa) { return ssm + (sa - s0); };
    const uint32_t tab0 = m_.crc;
    const uint32_t l1_sa = BYTES ? m_.l1 + gi * PROB_SCALE : SHARED ? m_.l1 : WIDE ? m_.l1 + gi * F_WIDE_BYTES : m_.l1 + warp * 4096u + g * 4;
    // (mixed sizes: the 1 KiB tables of the second planes first, then the half-KiB tables of the first planes)
    auto cf_of = [&](uint32_t grp) { return HYB ? ((grp & 1u) ? m_.cf + (grp >> 1) * 1024u : m_.cf + (G / 2) * 1024u + (grp >> 1) * 512u)
                                               : m_.cf + grp * (WIDE ? 0u : BYTES ? F_REC_STRIDE : 4u * CFN); };
    const uint32_t cf_sa = cf_of(gi);
    const uint32_t stage_sa = m_.stage + gi * F_STAGE;
    // SINK_BF16, SINK_F32: a tile is given out in units of four elements, unit u by lane u & 7, so that what a group loads
    // and stores at a time lies in a row; unit u's symbols lie at 16 (u & 7) + 4 (u >> 3), a lane's four units side by side.
    // (With sixteen consecutive elements to a lane, a warp's 4-byte load took 4.2 wavefronts of the load/store unit and its 8-byte
    // store 8.2, of 4-byte elements 14.8, where these take 3.4, 3.9 and 4.5: that unit was 83 and 78 % busy, now 76 and 77.
    // One B200: four 8B layers 1785 -> 1761 us, twelve FP32 layers 893 -> 679; 1704 and 665 with what the multiplier's pipe does
    // for the addresses.  Rows given out by all 32 lanes take still fewer, and as many more instructions: 1838 instead of 1761.)
    constexpr bool UNITS = SINK == SINK_BF16 || SINK == SINK_F32;
    const uint32_t put_sa = stage_sa + 16 * (k >> 2) + (k & 3u);
    // byte i ^ g of a state word goes through table 3 - (i ^ g)
    CrcQuarters cq;
#pragma unroll
    for (uint32_t i = 0; i < 4; i++) cq.b[i] = tab0 + 32u * (3u - (i ^ g)) + 4u * k;
    cq.rot = 0x3210u ^ (0x1111u * g);

    uint32_t limit = a.njobs;
    if (a.count) limit = SINK == SINK_DELTA ? 2u * *a.count : *a.count;     // (delta: the count is of chunks, two streams each)
    // A CTA of a shared-table archive takes one table's next 80 jobs; every other launch deals
    // fours of jobs to warps, over the CTAs first.
    const bool by_table = SHARED && a.tables != nullptr;
    if (blockIdx.x * (by_table ? G : 4u) >= limit) return;          // the whole CTA has nothing to do

    if (CRC && fits) {
        // "multiply by a row", eight copies in the bank-quartered layout of CrcQuarters (crc_feed4q sends byte m of a
        // value through table 3 - m)
        uint32_t *ts = reinterpret_cast<uint32_t *>(gen(tab0));
        const uint32_t(*mul)[256] = SINK == SINK_F32 ? a.tabs->mul_row128 : a.tabs->mul_row;
        for (uint32_t i = threadIdx.x; i < F_CRC_BYTES / 4; i += blockDim.x) ts[i] = mul[3u - ((i >> 3) & 3u)][i >> 5];
    }
    if (SHARED && fits && warp == 0) {
        // one table for the CTA, built by its first warp: the launch's, or the one this CTA's chunks
        // name (a shared-table archive); a table that does not validate fails every stream of the CTA
        const uint8_t *h = by_table ? a.tables + (size_t)a.jobs[blockIdx.x * G].flags * F_TABLE_STRIDE : a.shared_hdr;
        uint32_t f[8];
        load_freqs(h, lane, f);
        bool ok = build_table<true>(f, reinterpret_cast<uint32_t *>(gen(m_.l1)), nullptr, lane);
        if (lane == 0) *reinterpret_cast<uint32_t *>(gen(m_.poison)) = (ok && h[0] == 'R' && h[1] == '1') ? 0u : 1u;
    }
    __syncthreads();
    const bool poisoned = SHARED && fits && lds_u32(m_.poison) != 0;

    const uint32_t quads = limit / 4 + ((limit & 3u) != 0), q_step = gridDim.x * W;       // (a by-table launch has one each)
#pragma unroll 1
    for (uint32_t quad = by_table ? blockIdx.x * W + warp : blockIdx.x + gridDim.x * warp; quad < quads; quad += q_step) {
    // ---- this group's stream ------------------------------------------------------
    const uint32_t idx = quad * 4 + g;
    const bool have = idx < limit;
    // (SINK_DELTA: `order` lists chunks; stream 2c + p is plane p of chunk c)
    const uint32_t job = !(have && a.order) ? idx
                       : SINK == SINK_DELTA ? 2u * a.order[a.order_from_back ? a.njobs / 2 - 1 - (idx >> 1) : idx >> 1] + (idx & 1u)
                                            : a.order[a.order_from_back ? a.njobs - 1 - idx : idx];
    uint64_t soff = 0, doff = 0, moff = 0;
    uint32_t slen = 0, n = 0, piece0 = 0;
    bool open = false;
    if (have) {
        if (SINK == SINK_DELTA) {
            // groups 2c and 2c + 1 of the warp take the two planes of its chunk c
            const DeltaJob j = a.djobs[job >> 1];
            soff = (job & 1u) ? j.src_b : j.src_a; slen = (job & 1u) ? j.len_b : j.len_a;
            doff = j.dst_off; moff = j.base_off; n = j.n; piece0 = j.piece0;
        } else if (a.jobs) {
            FusedJob j = a.jobs[job];
            soff = j.src_off; doff = j.dst_off; moff = j.mant_off;
            slen = j.src_len; n = j.n; piece0 = j.piece0;
        } else if (a.sjobs) {
            StreamJob j = a.sjobs[job];
            soff = j.src_off; doff = j.dst_off; slen = j.src_len; n = j.n;
            open = SINK == SINK_OPEN && (j.flags & STREAM_OPEN);
        } else {
            soff = a.offs[2 * job]; slen = (uint32_t)a.offs[2 * job + 1];
            n = a.plane; doff = (uint64_t)job * a.plane;
        }
    }
    uint32_t st = ST_OK;
    if (!fits) { st = ST_BAD_SHAPE; n = 0; }          // the launch gave less shared memory than the layout needs
    if (n != 0 && (slen < LEAD || poisoned)) { st = ST_BAD_HEADER; n = 0; }
    if (n == 0) slen = 0;
    const uint8_t *sbase = a.src + soff;

    // the words follow table and states; the first four rounds are requested before the table is
    // built, which hides their latency
    Words<CFN, MODE> wd;
    wd.sa = m_.tr + gi * tr_group(CFN, MODE);
    wd.rd = wd.wr = 0;
    wd.lo = wd.hi = wd.lo2 = wd.hi2 = 0;
    uint32_t first[4][2];
    uint32_t x = 0;
    {
        const uintptr_t at = reinterpret_cast<uintptr_t>(sbase + LEAD);
        wd.sh = (uint32_t)(at & 3u) * 8u;
        wd.next = reinterpret_cast<const uint32_t *>(at & ~uintptr_t(3)) + k;
        const uint32_t words = n ? (slen - LEAD) / 2 : 0;
        wd.left = (int32_t)((words + TR_ROUND - 1) / TR_ROUND);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            wd.request(true);
            first[j][0] = MODE == TR_FEW ? wd.lo2 : wd.lo; first[j][1] = MODE == TR_FEW ? wd.hi2 : wd.hi;
        }
        for (int j = 0; j < wd.AHEAD; j++) wd.request(true);
        if (n) {
            uint32_t s[1];
            load_words_nc<1>(sbase + LEAD - STATE_BYTES + 4 * k, s);
            x = s[0];
        }
    }

    // ---- per-stream tables, built by the whole warp one stream at a time ------------
    if (!SHARED) {
        uint32_t fr[4][8], magic[4];
#pragma unroll
        for (uint32_t gg = 0; gg < 4; gg++) {
            const uint32_t on = __shfl_sync(0xffffffffu, n, gg * 8);
            const uint8_t *h = reinterpret_cast<const uint8_t *>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(sbase), gg * 8));
            magic[gg] = 0;
#pragma unroll
            for (int i = 0; i < 8; i++) fr[gg][i] = 0;
            if (on) {
                load_freqs(h, lane, fr[gg]);
                magic[gg] = (uint32_t)h[0] | ((uint32_t)h[1] << 8);
            }
        }
#pragma unroll
        for (uint32_t gg = 0; gg < 4; gg++) {
            const uint32_t on = __shfl_sync(0xffffffffu, n, gg * 8);
            uint32_t nlive = 0, max_live = 256;
            bool ok = false;
            uint32_t *tab = reinterpret_cast<uint32_t *>(gen(WIDE ? m_.l1 + (warp * 4 + gg) * F_WIDE_BYTES : m_.l1 + warp * 4096u + gg * 4));
            if (BYTES) {
                if (on) ok = solo_tables<false>(fr[gg], m_.l1 + (warp * 4 + gg) * PROB_SCALE, cf_of(warp * 4 + gg), lane);
            } else if (WIDE) {
                if (on) ok = build_table<true>(fr[gg], tab, nullptr, lane);
            } else {
                const bool small = HYB ? !(gg & 1u) : CFN < 256;
                max_live = small ? F_SMALL_LIVE : 256u;
                if (on)
                    ok = build_table<false, 4>(fr[gg], tab, reinterpret_cast<uint32_t *>(gen(cf_of(warp * 4 + gg))), lane,
                                               small ? 8u * gg : 0u, &nlive, max_live);
                // a group without a stream runs along in full tiles: its lookups must stay in its tables
                if (!ok && fits)
                    for (uint32_t i = lane; i < 256; i += 32) tab[i * 4] = 0;
            }
            ok = ok && magic[gg] == ('R' | ('1' << 8));
            // an alphabet too large for this instance is the caller's mistake, not the stream's
            if (on && !ok && g == gg) { st = nlive > max_live ? ST_BAD_SHAPE : ST_BAD_HEADER; n = 0; }
        }
        __syncwarp();
    }
    if (SINK == SINK_DELTA) {
        // The two groups of a chunk walk its tiles together (they share the merge, and the
        // checksum is folded over both with shuffles): when one plane has been refused, the
        // other is not decoded either.  The refused plane's status reports the chunk.
        const uint32_t partner_n = __shfl_xor_sync(0xffffffffu, n, 8);
        if (partner_n == 0) n = 0;
    }
    uint32_t e = 0;
    ByteState by{};
    if (__any_sync(0xffffffffu, n != 0)) {
        // the whole ring, so that a group without a stream finds nothing but bounded entries in it.  (F_BYTE_CFN: half of it; such a
        // group's addresses come from bytes and masked slots alone, whatever its ring and tables hold.)
        const uint32_t lo = wd.lo, hi = wd.hi, lo2 = wd.lo2, hi2 = wd.hi2;
        const uint32_t *next = wd.next;
        const int32_t left = wd.left;
        wd.left = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            wd.lo = first[j][0]; wd.hi = first[j][1];
            wd.round(l1_sa, cf_sa, k);
        }
        wd.lo = lo; wd.hi = hi; wd.lo2 = lo2; wd.hi2 = hi2; wd.next = next; wd.left = left;
        if (n == 0) wd.retire();
        if constexpr (BYTES) byte_next(x, e, by, x, false, 0u, (x & (PROB_SCALE - 1)) | l1_sa, lds_u8((x & (PROB_SCALE - 1)) | l1_sa), cf_sa);
        else e = lds_u32(slot_addr<CFN, MODE>(x, l1_sa, cf_sa));
        __syncwarp();
    }
    uint8_t *out = a.dst + doff;
    const uint32_t al = (uint32_t)(reinterpret_cast<uintptr_t>(out) & 15u);

    // SINK_BF16: the stored plane, read as aligned words and funnel-shifted.
    // SINK_DELTA: the base bytes in the output space, likewise; a tile of a chunk is 256 bytes
    // of output, of which lane k of the chunk's first group takes the 16 from 16 k and lane k
    // of its second group the 16 from 128 + 16 k.
    const uint32_t j16 = 8u * (g & 1u) + k;
    const uint8_t *mant = SINK == SINK_DELTA ? a.dst + moff + 16 * j16 : a.src + moff + 4 * k;
    const uint32_t msh = (uint32_t)(reinterpret_cast<uintptr_t>(mant) & 3u) * 8u;
    const uint32_t *mq = reinterpret_cast<const uint32_t *>(reinterpret_cast<uintptr_t>(mant) & ~uintptr_t(3));
    uint32_t m[5] = {0, 0, 0, 0, 0};
    // (a plane of bytes may have any n; a chunk's elements are two bytes or more of fewer than 2^32, and its sink
    // measured 0.7 % slower with the other count: four 8B layers 1796 -> 1809 us)
    uint32_t my_tiles = SINK == SINK_BYTES ? tiles_of(n, TS) : (n + TS - 1) / TS;
    const bool has_base = SINK == SINK_DELTA && moff != NONE64;      // (a plain two-plane chunk has none: m stays zero)
    auto fetch = [&](uint32_t tt) {
#pragma unroll
        for (int i = 0; i < 4; i++) m[i] = __ldg(mq + (size_t)tt * (TILE / 4) + 8 * i);
        if (k == 0) m[4] = __ldg(mq + (size_t)tt * (TILE / 4) + 32);
    };
    if (SINK == SINK_BF16 && my_tiles) fetch(0);
    if (has_base && n > 8 * j16) {
#pragma unroll
        for (int i = 0; i < 5; i++) m[i] = __ldg(mq + i);
    }
    // SINK_BF16 checksum: the eight running values ra[] are multiplied by x^2048 while the
    // NEXT tile decodes (32 independent table lookups that hide behind the decode chain),
    // then that tile's words are XORed in.
    uint32_t ra[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    const bool was_open = open;
    uint32_t last_x = x, taken = 0;               // state and words consumed at the stream's end
    // (F_BYTE_CFN: as 2^16 unrefilled, or as 1 with a word of zeros, whose entry is slot 0's)
    auto rest = [&]() {
        if (!BYTES) return x;
        return x == RANS_LOW || (x == 1 && by.c == 0 && e == lds_u64(cf_sa + S_ENTRY * lds_u8(l1_sa)).x) ? RANS_LOW : 0u;
    };

    // ---- tiles of 128 symbols ---------------------------------------------------------
    // FULL: every group of the warp that has symbols left has a whole tile of them.  (A group that has no
    // stream, or is done with it, runs along; nothing of its is kept.)
    uint32_t t = 0;
    bool scarce = true;                           // some stream of the warp may have too few words for the next block
    auto tile = [&](auto full_c) {
        constexpr bool FULL = decltype(full_c)::value;
        const uint32_t done = t * TS;
        uint32_t rem = n > done ? n - done : 0;
        __syncwarp();
        // SINK_F32: the tile's stored bytes are requested before the decode, which hides
        // their latency: of each plane's 33 words around them every eighth from k on, the last by lane 0.  (A plane may start
        // three bytes into a word: `rem` bytes of it reach into word w where rem + 3 > 4 w.)
        uint32_t pr[SINK == SINK_F32 ? 3 : 1][5];
        if constexpr (SINK == SINK_F32) {
#pragma unroll
            for (int j = 0; j < 3; j++) {
                const uint8_t *pp = a.src + moff + (size_t)j * n + done;
                const uint32_t *pq = reinterpret_cast<const uint32_t *>(reinterpret_cast<uintptr_t>(pp) & ~uintptr_t(3)) + k;
#pragma unroll
                for (int i = 0; i < 4; i++) pr[j][i] = rem && (FULL || rem + 3 > 4 * (k + 8 * i)) ? __ldg(pq + 8 * i) : 0u;
                pr[j][4] = k == 0 && rem + 3 > TS ? __ldg(pq + 32) : 0u;
                if (MODE == TR_FEW && rem > 5 * TS) prefetch_l2(pq + 4 * TS / 4 + 3 * k);
            }
        }
        auto top_up = [&](uint32_t blocks = 1) {
            while (__any_sync(0xffffffffu, wd.low(blocks))) {
                wd.round(l1_sa, cf_sa, k);
                __syncwarp();
            }
        };
        auto step4 = [&](auto first_c, uint32_t &hist, uint32_t base) {
            constexpr bool FIRST = decltype(first_c)::value;
            if constexpr (BYTES) byte_step4<FIRST>(x, e, by, hist, base, l1_sa, cf_sa, below, vsel);
            else stream_step4<CFN, MODE, FIRST, MULT>(x, e, hist, base, l1_sa, cf_sa, below, vsel);
        };
        auto put = [&](uint32_t step) { sts_u8(UNITS ? put_sa + 32 * (step & 3u) + 4 * (step >> 2) : stage_sa + step * NLANES + k, e); };
        // (the delta sink with many warps adds up addresses on both pipes: a chain of 14.9 K chunks 1934 -> 1922 us)
        auto fold = [&](uint32_t i) {
            if (CRC && i < NRA) ra[i] = crc_feed4q<SINK == SINK_DELTA && MODE == TR_4>(cq, ra[i]);
        };
        if constexpr (FULL) {
#pragma unroll
            for (uint32_t s8 = 0; s8 < TS / NLANES; s8 += 8) {
                // eight steps: two blocks, and where warps are few a round of translation between the
                // steps of the first (where they are many, top_up does all of them: fewer instructions)
                constexpr bool WOVEN = MODE != TR_4;
                // (F_BYTE_CFN has words for two blocks in its ring, and whether that will do for the block behind is asked
                // while a block runs)
                if (!BYTES) top_up();
                else if (scarce) top_up(2);
                if (BYTES) scarce = __any_sync(0xffffffffu, wd.low(2));
                uint32_t base = wd.block(), hist = 0;
                if (WOVEN) wd.part1();
                put(s8);
                step4(std::true_type{}, hist, base);
                if (WOVEN) wd.part2(l1_sa, cf_sa);
                put(s8 + 1);
                step4(std::false_type{}, hist, base);
                if (BYTES) wd.part2b(cf_sa);
                fold(s8 / 2);
                put(s8 + 2);
                step4(std::false_type{}, hist, base);
                if (WOVEN) wd.part3(l1_sa, cf_sa, k);
                put(s8 + 3);
                step4(std::false_type{}, hist, base);
                fold(s8 / 2 + 1);
                wd.rd += tr_entry(MODE) * __popc(hist);
                __syncwarp();
                if (!BYTES) top_up();
                else if (scarce) top_up(2);
                if (BYTES) scarce = __any_sync(0xffffffffu, wd.low(2));
                base = wd.block();
                hist = 0;
                put(s8 + 4);
                step4(std::true_type{}, hist, base);
                put(s8 + 5);
                step4(std::false_type{}, hist, base);
                fold(s8 / 2 + 2);
                put(s8 + 6);
                step4(std::false_type{}, hist, base);
                put(s8 + 7);
                step4(std::false_type{}, hist, base);
                fold(s8 / 2 + 3);
                wd.rd += tr_entry(MODE) * __popc(hist);
            }
        } else {
#pragma unroll
            for (int i = 0; i < NRA; i++) fold(i);
#pragma unroll 1
            for (uint32_t s4 = 0; s4 < TS / NLANES; s4 += 4) {
                top_up();
                uint32_t base = wd.block();
                const uint32_t base0 = base;
#pragma unroll 1
                for (uint32_t s = s4; s < s4 + 4; s++) {
                    const bool active = s * NLANES + k < rem;
                    if (active) put(s);
                    uint32_t ahead;
                    if constexpr (BYTES) ahead = byte_step(x, e, by, base, base0, l1_sa, cf_sa, lt_mask, grp_mask, active);
                    else ahead = stream_step<CFN, MODE, MULT>(x, e, base, base0, l1_sa, cf_sa, lt_mask, grp_mask, active);
                    if (SINK == SINK_OPEN) {
                        // the first lane that took a word the stream has not got ends an open stream:
                        // `ahead` words had been taken in this block before it took its own
                        const bool out = open && ahead != NONE32 && wd.taken(slen - LEAD) + ahead >= (slen - LEAD) / 2;
                        const uint32_t outs = __ballot_sync(0xffffffffu, out) & grp_mask;
                        if (outs) {
                            n = done + s * NLANES + (uint32_t)__ffs((int)(outs >> (8 * g))) - 1;
                            rem = n - done;
                            my_tiles = t + 1;
                            open = false;
                        }
                    }
                }
                wd.rd += base - base0;
            }
            scarce = true;
        }
        __syncwarp();
        uint32_t pw[SINK == SINK_F32 ? 4 : 1][3];
        if constexpr (SINK == SINK_F32) {
            // (unit i of this lane: elements 4 (k + 8 i) .. + 3; the words behind are the next lane's, lane 0's of the next unit)
#pragma unroll
            for (int j = 0; j < 3; j++) {
                const uint32_t sh = (uint32_t)((reinterpret_cast<uintptr_t>(a.src) + moff + (size_t)j * n) & 3u) * 8u;
#pragma unroll
                for (int i = 0; i < 4; i++)
                    pw[i][j] = __funnelshift_r(pr[j][i], __shfl_sync(0xffffffffu, k == 0 ? pr[j][i + 1] : pr[j][i], (lane & 24u) | ((k + 1) & 7u)), sh);
            }
        }
        uint32_t mw[SINK == SINK_BF16 ? 4 : 1];
        if constexpr (SINK == SINK_BF16) {
#pragma unroll
            for (int i = 0; i < 4; i++)
                mw[i] = __funnelshift_r(m[i], __shfl_sync(0xffffffffu, k == 0 ? m[i + 1] : m[i], (lane & 24u) | ((k + 1) & 7u)), msh);
        }
        if (!rem) return;
        if (SINK == SINK_DELTA) {
            // ---- both planes' symbols of this lane's eight elements, merge, XOR the base, write, checksum
            const uint32_t pair_sa = m_.stage + (gi & ~1u) * F_STAGE + 8u * j16;
            const uint2 ea = lds_u64(pair_sa), eb = lds_u64(pair_sa + F_STAGE);
            uint32_t w[4];
            bf16_merge4(ea.x, eb.x, w[0], w[1]);
            bf16_merge4(ea.y, eb.y, w[2], w[3]);
#pragma unroll
            for (int h = 0; h < 4; h++) w[h] ^= __funnelshift_r(m[h], m[h + 1], msh);
            if (has_base && n > (t + 1) * TS + 8u * j16) {         // next tile's base bytes, if this lane has any
#pragma unroll
                for (int i = 0; i < 5; i++) m[i] = __ldg(mq + (size_t)(t + 1) * (2 * TS / 4) + i);
                if (MODE == TR_FEW && t + 4 < my_tiles) prefetch_l2(mq + (size_t)(t + 4) * (2 * TS / 4));
            }
            uint8_t *d = out + (size_t)done * 2 + 16u * j16;
            const uint32_t ve = FULL ? 8u : rem > 8u * j16 ? min(rem - 8u * j16, 8u) : 0u;   // valid elements of this lane
            if (ve == 8) {
                if (al == 0) *reinterpret_cast<uint4 *>(d) = make_uint4(w[0], w[1], w[2], w[3]);
                else if ((al & 3) == 0) {
#pragma unroll
                    for (int i = 0; i < 4; i++) reinterpret_cast<uint32_t *>(d)[i] = w[i];
                } else {
#pragma unroll
                    for (int i = 0; i < 16; i++) d[i] = (uint8_t)(w[i >> 2] >> (8 * (i & 3)));
                }
            } else {
                const uint32_t vb = 2 * ve;
#pragma unroll
                for (int i = 0; i < 16; i++)
                    if ((uint32_t)i < vb) d[i] = (uint8_t)(w[i >> 2] >> (8 * (i & 3)));
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const uint32_t keep = vb > 4u * i ? min(vb - 4u * i, 4u) : 0u;
                    w[i] = keep >= 4 ? w[i] : (keep ? w[i] & ((1u << (8 * keep)) - 1u) : 0u);
                }
            }
            if (CRC) {
#pragma unroll
                for (int i = 0; i < 4; i++) ra[i] ^= w[i];
                if ((t & 255u) == 255u || t + 1 == my_tiles) {
                    // close the 64 KiB piece: every running value to the row's end, XOR over the chunk's 16 lanes
                    uint32_t v = 0;
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        v ^= crc_mulmod(a.tabs->word_mul16[j16][i], ra[i]);
                        ra[i] = 0;
                    }
                    const uint32_t pair_mask = 0xffffu << (16u * (g >> 1));
                    v ^= __shfl_xor_sync(pair_mask, v, 1);
                    v ^= __shfl_xor_sync(pair_mask, v, 2);
                    v ^= __shfl_xor_sync(pair_mask, v, 4);
                    v ^= __shfl_xor_sync(pair_mask, v, 8);
                    if (j16 == 0) {
                        const uint32_t p = t >> 8, rows = (t & 255u) + 1;
                        const uint32_t plen = min(PIECE_BYTES, 2 * n - p * PIECE_BYTES);
                        if (rows * F_ROW != plen) v = crc_unshift(a.tabs->x2, v, rows * F_ROW - plen);
                        a.piece_crc[piece0 + p] = v;
                    }
                }
            }
            return;
        }
        const uint4 ev = lds_u128(stage_sa + 16 * k);
        const uint32_t ew[4] = {ev.x, ev.y, ev.z, ev.w};
        if constexpr (SINK == SINK_F32) {
            // ---- interleave with the three stored planes, write, checksum: eight lanes' units in a row at a time
#pragma unroll
            for (uint32_t i = 0; i < 4; i++) {
                const uint32_t u = k + 8 * i, ve = FULL ? 4u : rem > 4 * u ? min(rem - 4 * u, 4u) : 0u;
                uint32_t w[4];
                interleave4(pw[i][0], pw[i][1], pw[i][2], ew[i], w);
                row_store<4>(out + (size_t)done * 4 + 16 * u, w, ve);
                if (CRC) {
#pragma unroll
                    for (int h = 0; h < 4; h++) ra[h] = (i ? crc_feed4q(cq, ra[h]) : ra[h]) ^ w[h];
                }
            }
            if (CRC && ((t & 127u) == 127u || t + 1 == my_tiles)) {
                // close the 64 KiB piece: every running value to the row's end, XOR over the group
                uint32_t v = 0;
#pragma unroll
                for (int h = 0; h < 4; h++) {
                    v ^= crc_mulmod(a.tabs->word_pow[32 - 4 * k - h], ra[h]);
                    ra[h] = 0;
                }
                v ^= __shfl_xor_sync(grp_mask, v, 1);
                v ^= __shfl_xor_sync(grp_mask, v, 2);
                v ^= __shfl_xor_sync(grp_mask, v, 4);
                if (k == 0) {
                    const uint32_t p = t >> 7, tiles = (t & 127u) + 1;
                    const uint32_t plen = min(PIECE_BYTES, 4 * n - p * PIECE_BYTES);
                    if (tiles * 512u != plen) v = crc_unshift(a.tabs->x2, v, tiles * 512u - plen);
                    a.piece_crc[piece0 + p] = v;
                }
            }
            return;
        }
        if (SINK == SINK_BYTES || SINK == SINK_OPEN) {
            if ((FULL || rem >= TS) && al == 0) {
                *reinterpret_cast<uint4 *>(out + done + 16 * k) = ev;
            } else {
                const uint32_t cnt = FULL || rem >= TS ? TS : rem;
#pragma unroll
                for (uint32_t i = 0; i < 16; i++)
                    if (16 * k + i < cnt) out[done + 16 * k + i] = (uint8_t)(ew[i >> 2] >> (8 * (i & 3)));
            }
            return;
        }

        // ---- SINK_BF16: merge with the stored plane, write, checksum, units as above -----
        if (t + 1 < my_tiles) {                                // next tile's stored bytes
            fetch(t + 1);
            if (MODE == TR_FEW && t + 5 < my_tiles) prefetch_l2(mq + (size_t)(t + 5) * (TILE / 4) + 3 * k);
        }
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) {
            const uint32_t u = k + 8 * i, ve = FULL ? 4u : rem > 4 * u ? min(rem - 4 * u, 4u) : 0u;
            uint32_t w[2];
            bf16_merge4(ew[i], mw[i], w[0], w[1]);
            row_store<2>(out + (size_t)done * 2 + 8 * u, w, ve);
            if (CRC) { ra[2 * i] ^= w[0]; ra[2 * i + 1] ^= w[1]; }
        }
        if (CRC) {
            if ((t & 255u) == 255u || t + 1 == my_tiles) {
                // close the 64 KiB piece: every running value to the row's end, XOR over the group
                uint32_t v = 0;
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    v ^= crc_mulmod(a.tabs->word_pow[64 - 16 * (i / 2) - 2 * k - i % 2], ra[i]);
                    ra[i] = 0;
                }
                v ^= __shfl_xor_sync(grp_mask, v, 1);
                v ^= __shfl_xor_sync(grp_mask, v, 2);
                v ^= __shfl_xor_sync(grp_mask, v, 4);
                if (k == 0) {
                    const uint32_t p = t >> 8, rows = (t & 255u) + 1;
                    const uint32_t plen = min(PIECE_BYTES, 2 * n - p * PIECE_BYTES);
                    if (rows * F_ROW != plen) v = crc_unshift(a.tabs->x2, v, rows * F_ROW - plen);
                    a.piece_crc[piece0 + p] = v;
                }
            }
        }
    };
    // Streams of bytes alone look at every tile whether it is whole: with runs they measured slower (a lone
    // warp's step 78 against 64 ns, 28577 streams of 32 KiB 1600 against 1495 us), and so do the warps
    // of a launch with open streams that have none.
    if (SINK == SINK_BYTES || (SINK == SINK_OPEN && !__any_sync(0xffffffffu, open))) {
        const uint32_t warp_tiles = __reduce_max_sync(0xffffffffu, my_tiles);
#pragma unroll 1
        for (; t < warp_tiles;) {
            const uint32_t done = t * TS;
            if (__all_sync(0xffffffffu, n <= done || n - done >= TS)) tile(std::true_type{});
            else tile(std::false_type{});
            t++;
            if (t == my_tiles) { last_x = rest(); taken = wd.taken(slen - LEAD); wd.retire(); }
        }
    } else {
    // Tiles are decoded in runs of whole ones, with nothing to watch inside a run: as many as the
    // group with the fewest has, and what an open stream's unloaded rounds of sixteen words are sure to be
    // enough for (a tile takes eight of them at most).  Where there is none, one tile step by step.
    for (;;) {
        const uint32_t done = t * TS;
        uint32_t whole = n > done ? (n - done) / TS : 0xffffffffu;
        if (SINK == SINK_OPEN && open && n > done) whole = min(whole, wd.left > 0 ? (uint32_t)wd.left / 8 : 0u);
        const uint32_t run = __reduce_min_sync(0xffffffffu, whole);
        if (run == 0xffffffffu) break;                            // nobody has anything left
        const uint32_t stop = t + max(run, 1u);
        if (run) {
#pragma unroll 1
            for (; t < stop; t++) tile(std::true_type{});
        } else {
            tile(std::false_type{});
            t++;
        }
        if (t == my_tiles) { last_x = rest(); taken = wd.taken(slen - LEAD); wd.retire(); }
    }
    }

    // ---- verdict -----------------------------------------------------------------------
    const uint32_t all_rest = __ballot_sync(0xffffffffu, last_x == RANS_LOW) & grp_mask;
    if (have && k == 0) {
        if (SINK == SINK_OPEN && was_open) {
            const_cast<StreamJob *>(a.sjobs)[job].aux = st == ST_OK ? n : 0u;
        } else if (st == ST_OK && n) {
            const uint64_t used = LEAD + 2 * (uint64_t)taken;
            if (used > slen) st = ST_OVERRUN;
            else if (used != slen || all_rest != grp_mask) st = ST_SLACK;
        }
        if (a.status) a.status[job] = st;
        if (a.any_bad && st != ST_OK && st != ST_SLACK) atomicOr(a.any_bad, 1u);
    }
    __syncwarp();
    }   // the warp's next four streams
}

// Sort a launch's streams by alphabet size, on the device: one warp per stream counts the
// non-zero frequencies of its table; streams with at most `small_live` go to the front of
// `order` (counts[0] of them), the others to its back (counts[1]).
__global__ void k_classify(StreamArgs a, uint32_t small_live, uint32_t *order, uint32_t *counts)
{
    const uint32_t job = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (job >= a.njobs) return;
    // (delta jobs: njobs counts chunks here, and the first plane's alphabet decides: the instance for
    // small ones gives the second plane a full-size table)
    uint64_t soff;
    uint32_t slen;
    if (a.djobs) { soff = a.djobs[job].src_a; slen = a.djobs[job].len_a; }
    else if (a.jobs) { soff = a.jobs[job].src_off; slen = a.jobs[job].src_len; }
    else if (a.sjobs) { soff = a.sjobs[job].src_off; slen = a.sjobs[job].src_len; }
    else { soff = a.offs[2 * job]; slen = (uint32_t)a.offs[2 * job + 1]; }
    uint32_t live = 257;                               // too short: the large instance reports it
    if (slen >= HDR_BYTES + STATE_BYTES) {
        // this lane's eight frequencies: 16 bytes at any alignment, as aligned words
        uint32_t w[4], mine = 0;
        load_words_nc<4>(a.src + soff + 4 + 16 * lane, w);
#pragma unroll
        for (int i = 0; i < 4; i++) mine += ((w[i] & 0xffffu) != 0) + ((w[i] >> 16) != 0);
        live = __reduce_add_sync(0xffffffffu, mine);
    }
    if (lane == 0) {
        const bool small = live <= small_live;
        const uint32_t pos = atomicAdd(&counts[small ? 0 : 1], 1u);
        order[small ? pos : a.njobs - 1 - pos] = job;
    }
}

// (offset, length) pairs -> stream jobs of `plane` symbols each, in order in the output.  A stream
// outside the `nbytes` of the buffer gets an empty job and bit 1 of *bad.
__global__ void k_batch_jobs(const uint64_t *pairs, uint64_t nbytes, uint32_t nstr, uint32_t plane, StreamJob *jobs, uint32_t *bad)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nstr) return;
    const uint64_t at = pairs[2 * (size_t)i], len = pairs[2 * (size_t)i + 1];
    const bool inside = at <= nbytes && len <= nbytes - at && len >> 32 == 0;
    StreamJob j{};
    j.src_off = inside ? at : 0;
    j.dst_off = (uint64_t)i * plane;
    j.src_len = inside ? (uint32_t)len : 0u;
    j.n = inside ? plane : 0u;
    jobs[i] = j;
    if (!inside) atomicOr(bad, 2u);
}

}  // namespace lmz
