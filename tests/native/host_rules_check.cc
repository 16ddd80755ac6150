// Checks of csrc/host_rules.inl.  argv[1] names the check; exit status 0 = it held.
#include <cstdio>
#include <string>

#include "../../lmz_b200/csrc/host_rules.inl"
#include "../../lmz_b200/csrc/solo_layout.cuh"

#define NEED(c)                                                          \
    do {                                                                 \
        if (!(c)) {                                                      \
            fprintf(stderr, "line %d: %s\n", __LINE__, #c);             \
            return 1;                                                    \
        }                                                                \
    } while (0)

static int size_classes()
{
    size_t last = 0, classes = 0;
    for (size_t n = 1; n < ((size_t)1 << 33); n += n / 37 + 1) {
        const size_t c = size_class(n);
        NEED(c >= n && c >= last && c % 4096 == 0);
        NEED(c <= n + n / 8 || c < n + 4096);
        NEED(size_class(c) == c && size_class(c + 1) > c);
        classes += c != last;
        last = c;
    }
    NEED(classes <= 8 * 34);
    for (int k = 12; k < 63; k++) NEED(size_class((size_t)1 << k) == (size_t)1 << k);
    for (size_t back = 0; back < 3; back++) NEED(size_class(SIZE_MAX - back) >= SIZE_MAX - back);
    NEED(size_class(((size_t)1 << 63) + 1) > (size_t)1 << 63);
    return 0;
}

// Streams of `plane` symbols, a byte in for each byte out: slices share one stream's time or hide it.
static int slices()
{
    constexpr unsigned SMS = 148;
    for (unsigned nstr : {1u, 2u, 7u, 8u, 9u, 16u, 63u, 64u, 257u, 512u, 1183u, 1184u, 1185u, 1600u, 3199u, 3200u, 11248u, 40000u})
        for (uint64_t plane : {1ull, 640ull, 32768ull, 65537ull, 1ull << 20, 1ull << 22, 1ull << 29}) {
            const unsigned s = batch_slices(2 * nstr * plane, nstr, SMS);
            NEED(s >= 1 && s <= MOST_SLICES && s <= nstr);
            if (s == 1) continue;
            NEED(2 * nstr * plane / s >= SLICE_BYTES);
            // the launcher's CTAs: how many wait for how many others, in chains one after the other
            unsigned ctas = 0, resident = ~0u, warps = 0;
            for (unsigned j = 0; j < s; j++) {
                const lmz::SoloLaunch l = lmz::solo_launch((uint32_t)((uint64_t)nstr * (j + 1) / s - (uint64_t)nstr * j / s), SMS, false);
                ctas += l.grid;
                resident = std::min(resident, lmz::solo_resident(l, false));
                warps = std::max(warps, l.warps);
            }
            const unsigned chains = (ctas + SMS * resident - 1) / (SMS * resident);
            const double chain = plane / 8 * 42e-9, out = (double)nstr / s * plane / 50e9;
            NEED(chains <= (warps == 1 ? 3 : 4) || out >= chain);
        }
    // what the rule's comment says of the room on an SM
    NEED(lmz::solo_resident(lmz::solo_launch(SMS, SMS, false), false) == 3);
    NEED(lmz::solo_resident(lmz::solo_launch(SMS + 1, SMS, false), false) == 2);
    NEED(lmz::solo_smem(false, true, 1).end == 64 << 10);
    NEED(batch_slices(2ull * 16 << 22, 16, SMS) == 8);
    NEED(batch_slices(28ull << 20, 512, SMS) == 7);
    NEED(batch_slices(2ull * 1500 << 20, 1500, SMS) == 3);
    return 0;
}

int main(int argc, char **argv)
{
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "size classes") return size_classes();
    if (what == "slices") return slices();
    fprintf(stderr, "no such check\n");
    return 2;
}
