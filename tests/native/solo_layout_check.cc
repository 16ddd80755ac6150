// Checks of csrc/solo_layout.cuh.  argv[1] names the check; exit status 0 = it held.
#include <cstdio>
#include <string>
#include <vector>

#include "../../lmz_b200/csrc/solo_layout.cuh"

using namespace lmz;

#define NEED(c)                                                          \
    do {                                                                 \
        if (!(c)) {                                                      \
            fprintf(stderr, "line %d: %s\n", __LINE__, #c);             \
            return 1;                                                    \
        }                                                                \
    } while (0)

// The lanes of a step store one after another, in any order: every byte has one writer, the lane that owns the state.
static int stores()
{
    for (uint32_t s = 0; s < 64; s++)
        for (uint32_t active = 0; active < 256; active++) {           // (the states a cut-off step still has)
            std::vector<int> writer(512 + 64, -1);
            for (uint32_t lane = 0; lane < 32; lane++) {
                const SoloLane me = solo_lane(lane);
                int clash = 0;
                solo_put(me, 8 * s, active >> me.k & 1u, [&](uint32_t on, uint32_t at) {
                    if (!on) return;
                    clash = writer[at] >= 0;
                    writer[at] = (int)lane;
                });
                NEED(!clash);
            }
            for (uint32_t b = 0; b < writer.size(); b++) {
                const bool due = b / 8 == s && (active >> (b & 7u) & 1u);
                NEED((writer[b] >= 0) == due);
                if (due) NEED(solo_lane((uint32_t)writer[b]).owner && solo_lane((uint32_t)writer[b]).k == (b & 7u));
            }
        }
    // states in order of lanes, each lane's `below` the owners of the states before its own
    for (uint32_t lane = 0; lane < 32; lane++) {
        const SoloLane me = solo_lane(lane);
        NEED(me.owner == (S_LANES >> lane & 1u) && (me.below & ~S_LANES) == 0);
        if (me.owner) NEED((uint32_t)__builtin_popcount(me.below) == me.k && me.below < (1u << lane));
    }
    return 0;
}

// Tiles of any plane of 32 bits: each begins inside the plane, the last one reaches its end, and there are so many.
static int tiles()
{
    for (uint32_t tile : {TILE, S_TILE})
        for (uint64_t edge : {0ull, 1ull << 12, 1ull << 31, 1ull << 32})
            for (int64_t off = -3 * (int64_t)tile; off <= 3 * (int64_t)tile; off++) {
                const int64_t n64 = (int64_t)edge + off;
                if (n64 < 0 || n64 > 0xffffffffll) continue;
                const uint32_t n = (uint32_t)n64, count = tiles_of(n, tile);
                NEED((uint64_t)count * tile >= n && (n == 0 ? count == 0 : (uint64_t)(count - 1) * tile < n));
                NEED(n == 0 || n - (count - 1) * tile <= tile);         // (as the kernels work it out, in 32 bits)
            }
    return 0;
}

int main(int argc, char **argv)
{
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "stores") return stores();
    if (what == "tiles") return tiles();
    fprintf(stderr, "no such check\n");
    return 2;
}
