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
// plane / 8 steps of some 41 ns, however few they are.  Where the slices fit on the device beside each
// other they share that time (each is a launch of its own, of CTAs of a warp or two with 34 KiB of tables a warp: six
// warps to an SM, and a slice that finds no room starts a copy or two later than one that does); else they take it in turn, and it must hide under the copies: a slice's plaintext takes plane * streams /
// 50 GB/s to come out, its chain plane * 8 ns, so 400 streams and more.  (With four slices at a time, by bytes
// alone: 16 planes of 4 Mi symbols 66.9 ms, two chains; as here 35.1, in one piece 36.4.)
unsigned batch_slices(uint64_t bytes, unsigned nstr, unsigned sms)
{
    unsigned s = (unsigned)std::min<uint64_t>(std::min(MOST_SLICES, nstr), bytes / SLICE_BYTES);
    if (s < 2) return 1;
    const uint64_t quads = ((uint64_t)(nstr + s - 1) / s + 3) / 4;
    if (s * quads > 2ull * sms) s = std::min(s, nstr / 400);
    return std::max(s, 1u);
}

}  // namespace
