// Checks of csrc/encode_layout.cuh.  argv[1] names the check; exit status 0 = it held.
#include <cstdint>
#include <cstdio>
#include <string>

#include "../../lmz_b200/csrc/encode_layout.cuh"

using namespace lmz;

#define NEED(c)                                             \
    do {                                                    \
        if (!(c)) {                                         \
            fprintf(stderr, "line %d: %s\n", __LINE__, #c); \
            return 1;                                       \
        }                                                   \
    } while (0)

// Twelve warps, three to a scheduler, are resident on an SM.
static int residents()
{
    NEED(encode_resident() == 12);
    NEED(12 * (F_SMEM_BASE + encode_smem_bytes()) <= F_SMEM_SM);
    return 0;
}

// A tile lies clear of the words that are left (less than a piece, at the buffer's end), a tile's words (a word of two
// bytes a symbol at most) and those fit, and the groups' buffers, read sixteen bytes at a time, lie apart.
static int buffers()
{
    NEED(E_TILE <= E_BUF - 128);
    NEED(126 + 2 * E_TILE <= E_BUF);
    for (uint32_t g = 0; g < 4; g++) {
        NEED(encode_buffer(g) % 16 == 0 && encode_buffer(g) >= 4 * E_TABLE);
        NEED(encode_buffer(g) + E_BUF <= (g < 3 ? encode_buffer(g + 1) : encode_smem_bytes()));
    }
    return 0;
}

// The eight bytes of a step that each of the four groups reads lie in banks of their own.
static int banks()
{
    for (uint32_t s = 0; s < 16; s++) {
        int32_t owner[32];
        for (auto &o : owner) o = -1;
        for (uint32_t g = 0; g < 4; g++)
            for (uint32_t k = 0; k < 8; k++) {
                int32_t &o = owner[(encode_buffer(g) + 8 * s + k) / 4 % 32];
                NEED(o < 0 || o == (int32_t)g);
                o = (int32_t)g;
            }
    }
    return 0;
}

int main(int argc, char **argv)
{
    const std::string check = argc > 1 ? argv[1] : "";
    if (check == "residents") return residents();
    if (check == "buffers") return buffers();
    if (check == "banks") return banks();
    fprintf(stderr, "no such check\n");
    return 2;
}
