// Chunk records -> job arrays for the chunks most archives consist of (included by lmz_b200.cu):
// stored, one-stream, byte-plane and BF16 chunks, no references to other chunks.  The planner
// (lmz_b200/plan.py, build_plan) does every kind with numpy, some forty passes over columns of all
// records; this is one pass in order, with the same results.  A record of another kind, or
// anything irregular, makes it answer 1: the planner then does the archive itself and says what is
// wrong with it.

namespace {

struct Record {                  // lmz/format.py:53-56
    uint64_t off, dst;
    uint32_t clen, rlen, crc;
    uint8_t codec, esize;
    uint16_t flags;
};
static_assert(sizeof(Record) == 32, "chunk record");

constexpr unsigned PLAN_HEAD = 32;           // bytes of every chunk's payload the caller fetched: up to eight plane lengths
enum : unsigned { C_STORED = 0, C_ONE = 1, C_SPLIT = 2, C_BF16 = 3, M_STORED = 0, M_RANS = 3 };

}  // namespace

API int lmz_host_plan_head_bytes(void) { return (int)PLAN_HEAD; }

static int plan_chunks(const void *records, const int64_t *select, size_t n, const uint64_t *ranges /* payload lo, hi, output lo, hi */,
                      const void *heads, int fuse /* 0 no, 1 yes, 2 every chunk that can be */, unsigned fuse_f32_min,
                      void *chunks_v, void *fused_v, void *delta_v, void *streams_v, int64_t *owner, uint32_t *piece_chunk,
                      int64_t *general, uint64_t *counts)
{
    const Record *all = static_cast<const Record *>(records);
    const uint8_t *head = static_cast<const uint8_t *>(heads);
    auto rec = [&](size_t i) -> const Record & { return all[select ? (size_t)select[i] : i]; };
    const uint64_t pay_lo = ranges[0], pay = ranges[1] - ranges[0], out_lo = ranges[2], outs = ranges[3] - ranges[2];
    ChunkJob *chunks = static_cast<ChunkJob *>(chunks_v);
    FusedJob *fused = static_cast<FusedJob *>(fused_v);
    DeltaJob *delta = static_cast<DeltaJob *>(delta_v);
    StreamJob *streams = static_cast<StreamJob *>(streams_v);

    // ---- every record: what it is, and whether all is as it should be -------------------------
    enum : uint8_t { PLAIN, FUSED, FUSED4, PAIR };
    struct Shape {
        uint32_t start[8], len[8];       // planes, from the chunk's payload
        uint8_t coded, planes, way;
    };
    std::vector<Shape> shapes(n);
    size_t fused4 = 0;
    uint64_t coded_bytes = 0;
    for (size_t i = 0; i < n; i++) {
        const Record &r = rec(i);
        Shape &s = shapes[i];
        s.coded = 0; s.planes = 1; s.way = PLAIN;
        s.start[0] = 0; s.len[0] = r.clen;
        if (r.off < pay_lo || r.off - pay_lo > pay || r.clen > pay - (r.off - pay_lo)) return 1;
        if (r.dst < out_lo || r.dst - out_lo > outs || r.rlen > outs - (r.dst - out_lo)) return 1;
        if (!r.rlen) return 1;
        coded_bytes += r.clen;
        const unsigned m = r.flags & 3u;
        if (r.codec == C_STORED || (r.codec == C_ONE && m == M_STORED)) {
            if (r.clen != r.rlen) return 1;
        } else if (r.codec == C_ONE) {
            if (m == M_RANS) s.coded = 1;
        } else if (r.codec == C_SPLIT || r.codec == C_BF16) {
            const unsigned p = r.esize;
            if (p != 2 && (p != 4 || r.codec == C_BF16) && (p != 8 || r.codec == C_BF16)) return 1;
            if (r.rlen % p || r.clen < 4 * p) return 1;
            const uint32_t elems = r.rlen / p;
            uint64_t at = 4 * p;
            for (unsigned k = 0; k < p; k++) {
                uint32_t len;
                memcpy(&len, head + i * PLAN_HEAD + 4 * k, 4);
                const unsigned how = r.flags >> (2 * k) & 3u;
                if (how != M_STORED && how != M_RANS) return 1;
                if (how == M_STORED && len != elems) return 1;
                s.start[k] = (uint32_t)at;
                s.len[k] = len;
                s.coded |= (how == M_RANS) << k;
                at += len;
                if (at > r.clen) return 1;
            }
            s.planes = (uint8_t)p;
            if (fuse && r.codec == C_BF16) s.way = s.coded == 1 ? FUSED : s.coded == 3 ? PAIR : PLAIN;
            if (fuse && r.codec == C_SPLIT && p == 4 && s.coded == 8) { s.way = FUSED4; fused4++; }
        } else {
            return 1;
        }
    }
    if (fuse != 2 && fused4 < fuse_f32_min) {
        for (Shape &s : shapes)
            if (s.way == FUSED4) s.way = PLAIN;
        fused4 = 0;
    }

    // ---- launch order: plain chunks, then those written by kernels of their own ----------------
    std::vector<uint32_t> place(n);
    size_t pos = 0;
    uint64_t pieces = 0, plain_pieces = 0;
    uint64_t extra = pay;                    // host-inflated chunks travel behind the payload
    size_t ngeneral = 0, nfused = 0, nfused4 = 0, npair = 0, nbf = 0;
    for (const Shape &s : shapes) nbf += s.way == FUSED;
    for (int own = 0; own < 2; own++) {
        for (size_t i = 0; i < n; i++) {
            const Shape &s = shapes[i];
            if ((s.way != PLAIN) != (own != 0)) continue;
            const Record &r = rec(i);
            const uint64_t at = r.off - pay_lo, to = r.dst - out_lo;
            place[i] = (uint32_t)pos;
            ChunkJob c{};
            c.dst_off = to; c.base_off = NONE64;
            for (unsigned k = 0; k < s.planes; k++) c.plane_off[k] = at + s.start[k];
            c.rlen = r.rlen; c.crc = r.crc; c.piece0 = (uint32_t)pieces;
            c.kind = r.codec == C_BF16 ? K_BF16 : r.codec == C_SPLIT ? K_SPLIT : K_COPY;
            c.esize = r.esize;
            c.scratch_mask = own ? 0 : s.coded;
            c.record = (uint32_t)i;
            for (uint64_t q = 0; q < ((uint64_t)r.rlen + PIECE_BYTES - 1) / PIECE_BYTES; q++) piece_chunk[pieces++] = (uint32_t)pos;
            chunks[pos++] = c;
            if (s.way == FUSED || s.way == FUSED4) {
                FusedJob f{};
                const unsigned k = s.way == FUSED ? 0 : 3;
                f.src_off = at + s.start[k]; f.src_len = s.len[k];
                f.mant_off = at + s.start[s.way == FUSED ? 1 : 0];
                f.dst_off = to; f.n = r.rlen / r.esize; f.piece0 = c.piece0;
                fused[s.way == FUSED ? nfused++ : nbf + nfused4++] = f;
            } else if (s.way == PAIR) {
                DeltaJob d{};
                d.src_a = at + s.start[0]; d.len_a = s.len[0];
                d.src_b = at + s.start[1]; d.len_b = s.len[1];
                d.dst_off = to; d.base_off = NONE64; d.n = r.rlen / 2; d.piece0 = c.piece0;
                delta[npair++] = d;
            }
        }
        if (!own) plain_pieces = pieces;
    }
    for (size_t i = 0; i < n; i++) {
        const Record &r = rec(i);
        if (r.codec == C_ONE && (r.flags & 3u) != M_STORED && (r.flags & 3u) != M_RANS) {
            chunks[place[i]].plane_off[0] = extra;
            extra += r.rlen;
            general[ngeneral++] = (int64_t)i;
        }
    }

    // ---- streams that are decoded to scratch: one-stream chunks, byte planes by width, BF16 ----
    size_t nstreams = 0;
    uint64_t scratch = 0;
    auto collect = [&](unsigned codec, unsigned planes) {
        for (size_t i = 0; i < n; i++) {
            const Shape &s = shapes[i];
            const Record &r = rec(i);
            if (s.way != PLAIN || !s.coded || r.codec != codec || s.planes != planes) continue;
            for (unsigned k = 0; k < planes; k++) {
                if (!(s.coded >> k & 1)) continue;
                StreamJob j{};
                j.src_off = r.off - pay_lo + s.start[k]; j.src_len = s.len[k];
                j.n = r.rlen / (codec == C_ONE ? 1 : planes);
                j.dst_off = scratch;
                chunks[place[i]].plane_off[k] = scratch;
                scratch += ((uint64_t)j.n + 15) & ~(uint64_t)15;
                owner[nstreams] = (int64_t)i;
                streams[nstreams++] = j;
            }
        }
    };
    collect(C_ONE, 1);
    collect(C_SPLIT, 2); collect(C_SPLIT, 4); collect(C_SPLIT, 8);
    collect(C_BF16, 2);
    if (nstreams > 1) {                      // long streams first
        std::vector<uint32_t> by(nstreams);
        for (size_t i = 0; i < nstreams; i++) by[i] = (uint32_t)i;
        std::stable_sort(by.begin(), by.end(), [&](uint32_t a, uint32_t b) { return streams[a].n > streams[b].n; });
        std::vector<StreamJob> js(nstreams);
        std::vector<int64_t> os(nstreams);
        for (size_t i = 0; i < nstreams; i++) { js[i] = streams[by[i]]; os[i] = owner[by[i]]; }
        std::copy(js.begin(), js.end(), streams);
        std::copy(os.begin(), os.end(), owner);
    }
    const uint64_t c[] = {nfused + nfused4, nfused4, npair, nstreams, pieces, plain_pieces, ngeneral, extra - pay, scratch, coded_bytes};
    memcpy(counts, c, sizeof c);
    return LMZ_GPU_OK;
}

API int lmz_host_plan(const void *records, const int64_t *select, size_t n, const uint64_t *ranges /* payload lo, hi, output lo, hi */,
                      const void *heads, int fuse /* 0 no, 1 yes, 2 every chunk that can be */, unsigned fuse_f32_min,
                      void *chunks_v, void *fused_v, void *delta_v, void *streams_v, int64_t *owner, uint32_t *piece_chunk,
                      int64_t *general, uint64_t *counts)
{
    return guarded(1, [&] {
        return plan_chunks(records, select, n, ranges, heads, fuse, fuse_f32_min, chunks_v, fused_v, delta_v, streams_v, owner,
                           piece_chunk, general, counts);
    });
}
