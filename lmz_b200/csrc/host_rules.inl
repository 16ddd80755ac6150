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

}  // namespace
