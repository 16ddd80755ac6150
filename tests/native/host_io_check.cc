// Checks of csrc/host_io.inl over a stand-in for the CUDA runtime (cuda_runtime.h beside this file).
// argv[1] names the check; exit status 0 = it held.
#include <atomic>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <mutex>
#include <string>
#include <vector>

#include "cuda_runtime.h"
#include "../../include/lmz_b200.h"

#define API extern "C"
static thread_local char g_err[256];
static int report(int code, const char *fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof g_err, fmt, ap);
    va_end(ap);
    return code;
}
static int fail_msg(int rc, const char *what) { return report(rc, "%s", what); }
static int fail_cuda(const char *what, cudaError_t e) { return report(LMZ_GPU_ECUDA, "%s: %s", what, cudaGetErrorString(e)); }
#define CK(what, x)                                                                    \
    if (cudaError_t status_of_call = (x); status_of_call != cudaSuccess)               \
        return fail_cuda(what, status_of_call)

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

int main(int argc, char **argv)
{
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "arrived unwaited") return freed_transfer_has_arrived(false);
    if (what == "arrived waited") return freed_transfer_has_arrived(true);
    if (what == "upload without an event") return failed_range_is_not_waited_for(true, &fake::fail_event_create);
    if (what == "download without an event") return failed_range_is_not_waited_for(false, &fake::fail_event_create);
    if (what == "download without a record") return failed_range_is_not_waited_for(false, &fake::fail_event_record);
    fprintf(stderr, "no such check\n");
    return 2;
}
