// Checks of csrc/host_pool.inl over a stand-in for the CUDA runtime (cuda_runtime.h beside this file).
// argv[1] names the check; exit status 0 = it held.
#include <cstdint>
#include <cstdio>
#include <string>

#include "cuda_runtime.h"
#include "../../include/lmz_b200.h"

#define API extern "C"
#include "../../lmz_b200/csrc/host_error.inl"
#include "../../lmz_b200/csrc/host_rules.inl"
#include "../../lmz_b200/csrc/host_pool.inl"

#define NEED(c)                                                          \
    do {                                                                 \
        if (!(c)) {                                                      \
            fprintf(stderr, "line %d: %s\n", __LINE__, #c);             \
            return 1;                                                    \
        }                                                                \
    } while (0)

constexpr size_t MIB = (size_t)1 << 20;
static size_t held()
{
    size_t n = 0;
    for (auto &kv : fake::host) n += kv.second;
    return n;
}

// Sizes that are asked for no more give way to those that are.
static int old_sizes_make_room()
{
    void *a = lmz_gpu_host_alloc(200 * MIB), *b = lmz_gpu_host_alloc(250 * MIB), *c = lmz_gpu_host_alloc(17);
    lmz_gpu_host_free(a);
    lmz_gpu_host_free(b);
    lmz_gpu_host_free(c);
    NEED(fake::host.size() == 3);
    for (int i = 0; i < 5; i++) {
        void *q = lmz_gpu_host_alloc(400 * MIB);
        NEED(q && lmz_gpu_host_lent(q, 400 * MIB) && !lmz_gpu_host_lent(q, 600 * MIB) && !lmz_gpu_host_lent((char *)q + 1, 1));
        lmz_gpu_host_free(q);
        NEED(!lmz_gpu_host_lent(q, 1));
        NEED(held() <= KEPT_HOST_BYTES);
    }
    NEED(fake::host_allocs == 4);                        // the fifth to the first 400 MiB are one block
    lmz_gpu_host_free(lmz_gpu_host_alloc(17));           // the youngest of the small ones is still there
    NEED(fake::host_allocs == 4);
    lmz_gpu_host_free(lmz_gpu_host_alloc(KEPT_HOST_BYTES));      // too large to be kept: nothing makes room for it
    NEED(fake::host_allocs == 5 && held() >= 400 * MIB && held() <= KEPT_HOST_BYTES);
    lmz_gpu_host_free(nullptr);
    lmz_gpu_trim();
    NEED(fake::host.empty());
    return 0;
}

// Random use: no block is lent twice, the idle ones stay within the bound, all is given back.
static int random_use()
{
    std::vector<std::pair<uint8_t *, size_t>> out;
    uint64_t x = 7;
    for (int i = 0; i < 20000; i++) {
        x = x * 6364136223846793005ull + 1442695040888963407ull;
        const size_t n = ((size_t)1 << (x >> 59)) / 2 * (1 + (x >> 33) % 7) % (90 * MIB) + 1;
        if (out.size() < 12 && (x >> 20 & 1)) {
            uint8_t *q = static_cast<uint8_t *>(lmz_gpu_host_alloc(n));
            NEED(q && lmz_gpu_host_lent(q, n));
            for (auto &o : out) NEED(q + n <= o.first || o.first + o.second <= q);
            q[0] = q[n - 1] = 1;
            out.push_back({q, n});
        } else if (!out.empty()) {
            const size_t at = (x >> 40) % out.size();
            lmz_gpu_host_free(out[at].first);
            out.erase(out.begin() + at);
        }
        size_t lent = 0;
        for (auto &o : out) lent += size_class(o.second + LENT_HEAD);
        NEED(held() - lent <= KEPT_HOST_BYTES);
    }
    for (auto &o : out) lmz_gpu_host_free(o.first);
    lmz_gpu_trim();
    NEED(fake::host.empty());
    return 0;
}

int main(int argc, char **argv)
{
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "old sizes make room") return old_sizes_make_room();
    if (what == "random use") return random_use();
    fprintf(stderr, "no such check\n");
    return 2;
}
