// How an entry point says what went wrong (included by lmz_b200.cu).
#include <cstdarg>
#include <cstdio>
#include <exception>

// Why the last call on this thread failed (lmz_gpu_last_error).
static thread_local char g_err[256];

// Record a reason and hand back the code to return.
static int report(int code, const char *fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof g_err, fmt, ap);
    va_end(ap);
    return code;
}

static int fail_msg(int rc, const char *what) { return report(rc, "%s", what); }

static int fail_cuda(const char *what, cudaError_t e)
{
    return report(LMZ_GPU_ECUDA, "%s: %s", what, cudaGetErrorString(e));
}

// A CUDA call inside a function that returns a code: leave with ECUDA when it fails.
#define CK(what, x)                                                                    \
    if (cudaError_t status_of_call = (x); status_of_call != cudaSuccess)               \
        return fail_cuda(what, status_of_call)

// What may throw (memory for a vector, a thread that cannot be started) stays inside the entry point: its
// callers are C, where an exception ends the process.
template <class R, class F>
static R guarded(R failed, F f)
{
    try {
        return f();
    } catch (const std::exception &e) {
        report(LMZ_GPU_EUNSUPPORTED, "host resources: %s", e.what());
    } catch (...) {
        report(LMZ_GPU_EUNSUPPORTED, "host resources");
    }
    return failed;
}
