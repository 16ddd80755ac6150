// Checks of csrc/host_io.inl over a stand-in for the CUDA runtime (cuda_runtime.h beside this file).
// argv[1] names the check; exit status 0 = it held.
#include <cstdint>
#include <cstdio>
#include <string>
#include <vector>

#include <sys/resource.h>

#include "cuda_runtime.h"
#include "../../include/lmz_b200.h"

#define API extern "C"
#include "../../lmz_b200/csrc/host_error.inl"
#include "../../lmz_b200/csrc/host_io.inl"

#define NEED(c)                                                          \
    do {                                                                 \
        if (!(c)) {                                                      \
            fprintf(stderr, "line %d: %s\n", __LINE__, #c);             \
            return 1;                                                    \
        }                                                                \
    } while (0)

// The memory uploaded to may go once the transfer is freed, whether or not anybody waited for the range.
static int freed_transfer_has_arrived(bool waited)
{
    void *staging = lmz_gpu_staging_new(1000, 4, 2);
    NEED(staging);
    std::vector<uint8_t> from(9999), to(9999);
    for (size_t i = 0; i < from.size(); i++) from[i] = (uint8_t)(i * 7 + 1);
    void *t = lmz_gpu_transfer_new(staging, nullptr);
    NEED(t);
    const int r = lmz_gpu_transfer_upload(t, -1, from.data(), 0, from.size(), to.data());
    NEED(r == 0);
    if (waited) NEED(lmz_gpu_transfer_wait(t, r, nullptr) == LMZ_GPU_OK);
    NEED(lmz_gpu_transfer_free(t) == LMZ_GPU_OK);
    NEED(to == from);
    NEED(fake::dropped == 0);
    lmz_gpu_staging_free(staging);
    return 0;
}

// A range that could not be opened is not waited for, and those before and after it are whole.
static int failed_range_is_not_waited_for(bool up, int *call)
{
    void *staging = lmz_gpu_staging_new(1000, 4, 2);
    NEED(staging);
    FILE *f = tmpfile();
    NEED(f);
    std::vector<uint8_t> from(4567), to(3 * 4567);
    for (size_t i = 0; i < from.size(); i++) from[i] = (uint8_t)(i * 5 + 3);
    void *t = lmz_gpu_transfer_new(staging, nullptr);
    NEED(t);
    for (int i = 0; i < 3; i++) {
        const uint64_t at = (uint64_t)i * from.size();
        if (i == 1) *call = 1;
        const int r = up ? lmz_gpu_transfer_upload(t, -1, from.data(), 0, from.size(), to.data() + at)
                         : lmz_gpu_transfer_download(t, from.data(), from.size(), fileno(f), nullptr, at, nullptr);
        NEED(i == 1 ? r < 0 && strstr(g_err, "made to fail") : r >= 0);
        if (r >= 0) NEED(lmz_gpu_transfer_wait(t, r, nullptr) == LMZ_GPU_OK);
    }
    NEED(lmz_gpu_transfer_free(t) == LMZ_GPU_OK);
    if (!up) NEED(pread(fileno(f), to.data(), to.size(), 0) == (ssize_t)to.size());
    for (int i = 0; i < 3; i++)
        NEED((memcmp(to.data() + i * from.size(), from.data(), from.size()) == 0) == (i != 1));
    lmz_gpu_staging_free(staging);
    return 0;
}

// Threads that cannot be started (no room for their stacks) are an error, or the caller's own work; never
// the end of the process.
static int no_room_for_threads()
{
    constexpr size_t N = 4096, WIDTH = 32;
    std::vector<uint8_t> from(N * 40), got(N * WIDTH);
    std::vector<uint64_t> offs(N);
    for (size_t i = 0; i < from.size(); i++) from[i] = (uint8_t)(i * 11);
    for (size_t i = 0; i < N; i++) offs[i] = i * 40;
    struct rlimit was, now;
    NEED(getrlimit(RLIMIT_AS, &was) == 0);
    long pages = 0;
    FILE *f = fopen("/proc/self/statm", "r");
    NEED(f && fscanf(f, "%ld", &pages) == 1);
    fclose(f);
    now = was;
    now.rlim_cur = (rlim_t)pages * 4096 + (20 << 20);        // two stacks of eight MiB
    NEED(setrlimit(RLIMIT_AS, &now) == 0);
    void *staging = lmz_gpu_staging_new(64, 200, 100);
    const bool said = strstr(g_err, "host resources") != nullptr;
    const int rc = lmz_host_gather(-1, from.data(), from.size(), offs.data(), N, WIDTH, got.data());
    NEED(setrlimit(RLIMIT_AS, &was) == 0);
    NEED(!staging && said);
    NEED(rc == LMZ_GPU_OK);
    for (size_t i = 0; i < N; i++) NEED(memcmp(got.data() + i * WIDTH, from.data() + i * 40, WIDTH) == 0);
    return 0;
}

int main(int argc, char **argv)
{
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "arrived unwaited") return freed_transfer_has_arrived(false);
    if (what == "arrived waited") return freed_transfer_has_arrived(true);
    if (what == "upload without an event") return failed_range_is_not_waited_for(true, &fake::fail_event_create);
    if (what == "download without an event") return failed_range_is_not_waited_for(false, &fake::fail_event_create);
    if (what == "download without a record") return failed_range_is_not_waited_for(false, &fake::fail_event_record);
    if (what == "no room for threads") return no_room_for_threads();
    fprintf(stderr, "no such check\n");
    return 2;
}
