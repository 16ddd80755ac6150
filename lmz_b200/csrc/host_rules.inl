// Sizes that the host side chooses by (included by lmz_b200.cu): plain arithmetic, no CUDA.
#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace {

// Kept memory comes in classes an eighth of a power of two apart (a page at least), so that a call finds
// memory of one a little smaller or larger and no block is an eighth larger than what was asked for.
size_t size_class(size_t bytes)
{
    if (bytes <= 4096) return 4096;
    size_t p = 4096;                                       // the power of two at or below `bytes`
    while (p <= bytes / 2) p <<= 1;
    const size_t step = std::max<size_t>(4096, p / 8), up = bytes + (step - 1);
    return up < bytes ? bytes : up - up % step;
}

// A large host batch runs in slices of its streams, so that streams go in, are decoded and plaintext comes
// out at the same time: at most MOST_SLICES, of at least SLICE_BYTES in and out.  One B200, BF16 exponent
// planes, ms a call with slices of at least 1, 2, 4, 8 MiB: 256 of 64 KiB 1.18, 1.14, 1.06, 1.11; 2000 of
// 16 KiB 1.61, 1.65, 1.29, 1.28.  With at most 1, 2, 4, 8, 16 of them: 512 of 32 KiB 1.00, 0.86, 0.85, 0.87, 0.88;
// 1500 of 256 KiB 52.7, 32.8, 27.8, 26.0, 35.0.
constexpr unsigned MOST_SLICES = 8;
constexpr size_t SLICE_BYTES = (size_t)4 << 20;

// How many slices, for `nstr` streams and `bytes` in and out.  A slice takes as long as one of its streams,
// plane / 8 steps of some 39 ns, however few they are.  Up to eight streams per SM the slices go side by side: each is
// a launch of its own, of one CTA per SM at most, of which an SM has room for three of one warp (64 KiB: a table of
// 32 KiB on a boundary of its size) or two of two, and a CTA that finds none waits for one of an earlier slice to
// end, which came in with an earlier copy.  At most three chains in turn for slices of one-warp CTAs, four for the others,
// most of them under the copies.  (One B200, steps of 42 ns, us, new inputs, as here against slices only where all are
// resident: 444 of 32 KiB 840 either way, 600 of 32 KiB 1100 against 1190, 600 of 64 KiB 1830 against 2300, 1184 of 64 KiB
// 3400 against 3800, 600 of 256 KiB 7200 against 9500.)  Beyond that slices take their chains in turn, and one must hide under
// the copies: a slice's plaintext takes plane * streams / 50 GB/s to come out, its chain plane * 4.8 ns, and more
// where streams share an SM, so 400 streams and more.  (With four slices at a time, by bytes alone, and steps of
// 64 ns: 16 planes of 4 Mi symbols 66.9 ms, two chains; as here 35.1, in one piece 36.4.)
unsigned batch_slices(uint64_t bytes, unsigned nstr, unsigned sms)
{
    unsigned s = (unsigned)std::min<uint64_t>(std::min(MOST_SLICES, nstr), bytes / SLICE_BYTES);
    if (s < 2) return 1;
    const uint64_t quads = ((uint64_t)(nstr + s - 1) / s + 3) / 4;
    if (s * quads > 2ull * sms) s = std::min(s, nstr / 400);
    return std::max(s, 1u);
}

}  // namespace
