// A stand-in for the CUDA runtime that needs no GPU: what csrc/host_io.inl calls, over ordinary memory.
// Work on a stream is queued and runs only when somebody waits for it, as late as a real device
// might run it; a call can be told to fail.
#pragma once
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <mutex>
#include <set>

typedef int cudaError_t;
enum { cudaSuccess = 0, cudaErrorUnknown = 999 };
enum { cudaEventDisableTiming = 2, cudaStreamNonBlocking = 1, cudaHostAllocPortable = 1 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1, cudaMemcpyDeviceToHost = 2 };
struct FakeStream { std::deque<std::function<void()>> queue; };
struct FakeEvent { FakeStream *on = nullptr; size_t upto = 0; };
typedef FakeStream *cudaStream_t;
typedef FakeEvent *cudaEvent_t;

namespace fake {
inline std::recursive_mutex mu;
inline FakeStream legacy;
inline std::map<FakeStream *, size_t> ran;              // operations of a stream that have run
inline std::set<FakeStream *> streams;                  // alive
inline std::map<void *, size_t> host;                   // page-locked blocks that are alive
inline size_t host_allocs = 0;
inline size_t dropped = 0;                              // operations queued when their stream was destroyed
inline int fail_event_create = 0, fail_event_record = 0;     // calls from now until one fails, 0 = never
inline bool due(int &n) { return n > 0 && --n == 0; }
inline FakeStream *of(cudaStream_t s) { return s ? s : &legacy; }
inline void run(FakeStream *s, size_t upto)
{
    while (ran[s] < upto && !s->queue.empty()) {
        auto op = std::move(s->queue.front());
        s->queue.pop_front();
        ran[s]++;
        op();
    }
}
inline size_t queued(FakeStream *s) { return ran[s] + s->queue.size(); }
}  // namespace fake

#define FAKE_LOCK std::lock_guard<std::recursive_mutex> lock_(fake::mu)
inline const char *cudaGetErrorString(cudaError_t) { return "made to fail"; }
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
inline cudaError_t cudaSetDevice(int) { return cudaSuccess; }
inline cudaError_t cudaHostAlloc(void **p, size_t n, unsigned)
{
    FAKE_LOCK;
    *p = malloc(n);                                      // (pages nobody touches cost nothing)
    if (!*p) return cudaErrorUnknown;
    fake::host[*p] = n;
    fake::host_allocs++;
    return cudaSuccess;
}
inline cudaError_t cudaMallocHost(void **p, size_t n) { return cudaHostAlloc(p, n, 0); }
inline cudaError_t cudaFreeHost(void *p)
{
    FAKE_LOCK;
    fake::host.erase(p);
    free(p);
    return cudaSuccess;
}
inline cudaError_t cudaMalloc(void **p, size_t n) { *p = malloc(n); return *p ? cudaSuccess : cudaErrorUnknown; }
inline cudaError_t cudaFree(void *p) { free(p); return cudaSuccess; }
inline cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned)
{
    FAKE_LOCK;
    *s = new FakeStream;
    fake::streams.insert(*s);
    return cudaSuccess;
}
inline cudaError_t cudaStreamDestroy(cudaStream_t s)     // (what is queued still runs, later: nobody has waited)
{
    FAKE_LOCK;
    fake::dropped += s->queue.size();
    fake::streams.erase(s);
    return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t s)
{
    FAKE_LOCK;
    fake::run(fake::of(s), ~(size_t)0);
    return cudaSuccess;
}
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned)
{
    FAKE_LOCK;
    if (fake::due(fake::fail_event_create)) return cudaErrorUnknown;
    *e = new FakeEvent;
    return cudaSuccess;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s)
{
    FAKE_LOCK;
    if (fake::due(fake::fail_event_record)) return cudaErrorUnknown;
    e->on = fake::of(s);
    e->upto = fake::queued(e->on);
    return cudaSuccess;
}
inline cudaError_t cudaEventSynchronize(cudaEvent_t e)
{
    FAKE_LOCK;
    if (e->on) fake::run(e->on, e->upto);
    return cudaSuccess;
}
inline cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned)
{
    FAKE_LOCK;
    FakeStream *on = e->on;
    const size_t upto = e->upto;
    if (on) fake::of(s)->queue.push_back([=] { fake::run(on, upto); });
    return cudaSuccess;
}
inline cudaError_t cudaMemcpyAsync(void *to, const void *from, size_t n, cudaMemcpyKind, cudaStream_t s)
{
    FAKE_LOCK;
    fake::of(s)->queue.push_back([=] { memcpy(to, from, n); });
    return cudaSuccess;
}
