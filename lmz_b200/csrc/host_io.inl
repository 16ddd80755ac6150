// Bytes between files (or host memory) and HBM (included by lmz_b200.cu).
//
// A file's pages are not page-locked, so its bytes cross through a ring of page-locked blocks.  What
// bounds that is the host copy: one thread moves 5 GB/s out of the page cache, eight to twelve
// about 36 (16 cores), against 54 GB/s of the link.  The threads, their blocks
// and the CUDA calls are all here: a thread takes a free block, fills it (pread, or memcpy from
// memory), starts its copy on the transfer's stream and takes the next, so several blocks are
// being filled while others are on the link and no interpreter lock is involved.  Writing a file
// is the same backwards.
#include <atomic>
#include <cerrno>
#include <condition_variable>
#include <deque>
#include <functional>
#include <memory>
#include <mutex>
#include <new>
#include <thread>
#include <vector>
#include <fcntl.h>
#include <sys/mman.h>
#include <sys/stat.h>
#include <sys/vfs.h>
#include <unistd.h>

namespace {

// Threads that take jobs in order.
struct Workers {
    std::mutex mu;
    std::condition_variable wake;
    std::deque<std::function<void()>> jobs;
    std::vector<std::thread> threads;
    bool stop = false;

    explicit Workers(unsigned n)
    {
        threads.reserve(n);
        try {
            for (unsigned i = 0; i < n; i++) threads.emplace_back([this] { run(); });
        } catch (...) {
            end();                       // (those that were started must be joined)
            throw;
        }
    }
    ~Workers() { end(); }
    void run()
    {
        for (;;) {
            std::function<void()> job;
            {
                std::unique_lock<std::mutex> lock(mu);
                wake.wait(lock, [this] { return stop || !jobs.empty(); });
                if (jobs.empty()) return;
                job = std::move(jobs.front());
                jobs.pop_front();
            }
            job();
        }
    }
    void end()
    {
        {
            std::lock_guard<std::mutex> lock(mu);
            stop = true;
        }
        wake.notify_all();
        for (std::thread &t : threads) t.join();
    }
    void add(std::function<void()> job)
    {
        {
            std::lock_guard<std::mutex> lock(mu);
            jobs.push_back(std::move(job));
        }
        wake.notify_one();
    }
};

struct Block {
    uint8_t *p = nullptr;
    cudaEvent_t left = nullptr;      // the block's last copy to the device
    int device = -1;                 // of that event
    bool busy = false;
};

struct StagingPool {
    size_t block;
    std::mutex mu;
    std::condition_variable freed;
    std::deque<Block *> free_blocks;               // the one whose copy was started first is in front
    std::vector<std::unique_ptr<Block>> blocks;
    std::unique_ptr<Workers> workers;

    Block *take()
    {
        std::unique_lock<std::mutex> lock(mu);
        freed.wait(lock, [this] { return !free_blocks.empty(); });
        Block *b = free_blocks.front();
        free_blocks.pop_front();
        return b;
    }
    void give(Block *b)
    {
        {
            std::lock_guard<std::mutex> lock(mu);
            free_blocks.push_back(b);
        }
        freed.notify_one();
    }
    ~StagingPool()
    {
        workers.reset();
        for (auto &b : blocks) {
            if (b->left) {
                if (b->busy) cudaEventSynchronize(b->left);
                cudaEventDestroy(b->left);
            }
            if (b->p) cudaFreeHost(b->p);
        }
    }
};

struct Transfer {
    StagingPool *pool;
    int device = 0;
    cudaStream_t stream = nullptr;                 // of this transfer's copies
    std::mutex issue;                              // one issuer at a time: stream order = event order
    std::mutex mu;
    std::condition_variable done;
    struct Range {
        size_t left = 0;
        cudaEvent_t event = nullptr;
        bool to_device = true;
    };
    std::deque<Range> ranges;
    size_t open = 0;                               // blocks of all ranges not finished
    char error[200] = "";

    void finish(size_t r, const char *what)
    {
        std::lock_guard<std::mutex> lock(mu);
        if (what && !error[0]) snprintf(error, sizeof error, "%s", what);
        ranges[r].left--;
        open--;
        done.notify_all();
    }
    bool failed()
    {
        std::lock_guard<std::mutex> lock(mu);
        return error[0] != 0;
    }
};

bool read_fully(int fd, uint8_t *to, uint64_t at, size_t n)
{
    while (n) {
        const ssize_t got = pread(fd, to, n, (off_t)at);
        if (got < 0 && errno == EINTR) continue;
        if (got <= 0) return false;
        to += got; at += (uint64_t)got; n -= (size_t)got;
    }
    return true;
}

bool write_fully(int fd, const uint8_t *from, uint64_t at, size_t n)
{
    while (n) {
        const ssize_t put = pwrite(fd, from, n, (off_t)at);
        if (put < 0 && errno == EINTR) continue;
        if (put <= 0) return false;
        from += put; at += (uint64_t)put; n -= (size_t)put;
    }
    return true;
}

// A block whose last copy has left it, with an event of `device`'s.
cudaError_t block_ready(Block *b, int device)
{
    cudaError_t e = cudaSuccess;
    if (b->busy) e = cudaEventSynchronize(b->left);
    b->busy = false;
    if (e == cudaSuccess && b->device != device) {
        if (b->left) cudaEventDestroy(b->left);
        b->left = nullptr;
        e = cudaEventCreateWithFlags(&b->left, cudaEventDisableTiming);
        b->device = e == cudaSuccess ? device : -1;
    }
    return e;
}

void upload_block(Transfer *t, size_t r, int fd, const uint8_t *host, uint64_t off, size_t n, uint8_t *dst)
{
    const char *bad = nullptr;
    cudaSetDevice(t->device);
    Block *b = t->pool->take();
    cudaError_t e = t->failed() ? cudaErrorUnknown : block_ready(b, t->device);
    if (e != cudaSuccess) bad = "an upload block failed";
    else if (fd >= 0) {
        if (!read_fully(fd, b->p, off, n)) bad = "reading the file failed";
    } else {
        memcpy(b->p, host + off, n);
    }
    if (!bad) {
        std::lock_guard<std::mutex> lock(t->issue);
        e = cudaMemcpyAsync(dst, b->p, n, cudaMemcpyHostToDevice, t->stream);
        if (e == cudaSuccess) {
            e = cudaEventRecord(b->left, t->stream);
            if (e != cudaSuccess) cudaStreamSynchronize(t->stream);      // (the block is not to be had before its copy has left it)
        }
        b->busy = e == cudaSuccess;
        if (e == cudaSuccess) {
            // whichever block of the range is issued last records the range's event
            std::lock_guard<std::mutex> state(t->mu);
            if (t->ranges[r].left == 1) e = cudaEventRecord(t->ranges[r].event, t->stream);
            t->ranges[r].left--;
            t->open--;
            if (e != cudaSuccess && !t->error[0]) snprintf(t->error, sizeof t->error, "%s", cudaGetErrorString(e));
            t->done.notify_all();
            t->pool->give(b);
            return;
        }
        bad = cudaGetErrorString(e);
    }
    t->pool->give(b);
    t->finish(r, bad);
}

void download_block(Transfer *t, size_t r, const uint8_t *src, size_t n, int fd, uint8_t *map, uint64_t off, cudaEvent_t after)
{
    const char *bad = nullptr;
    cudaSetDevice(t->device);
    Block *b = t->pool->take();
    cudaError_t e = t->failed() ? cudaErrorUnknown : block_ready(b, t->device);
    if (e == cudaSuccess) {
        std::lock_guard<std::mutex> lock(t->issue);
        e = cudaStreamWaitEvent(t->stream, after, 0);
        if (e == cudaSuccess) e = cudaMemcpyAsync(b->p, src, n, cudaMemcpyDeviceToHost, t->stream);
        if (e == cudaSuccess) e = cudaEventRecord(b->left, t->stream);
    }
    if (e == cudaSuccess) e = cudaEventSynchronize(b->left);
    if (e != cudaSuccess) bad = "a download block failed";
    else if (map) memcpy(map + off, b->p, n);
    else if (!write_fully(fd, b->p, off, n)) bad = "writing the file failed";
    t->pool->give(b);
    t->finish(r, bad);
}

}  // namespace

API void *lmz_gpu_staging_new(size_t block, unsigned depth, unsigned threads)
{
    if (!block || !threads || threads >= depth) {
        fail_msg(LMZ_GPU_EUNSUPPORTED, "staging needs more blocks than threads");
        return nullptr;
    }
    return guarded<void *>(nullptr, [&]() -> void * {
        std::unique_ptr<StagingPool> p(new StagingPool);
        p->block = block;
        for (unsigned i = 0; i < depth; i++) {
            p->blocks.emplace_back(new Block);
            cudaError_t e = cudaHostAlloc((void **)&p->blocks.back()->p, block, cudaHostAllocPortable);
            if (e != cudaSuccess) {
                cudaGetLastError();
                fail_cuda("page-locked staging", e);
                return nullptr;
            }
            p->free_blocks.push_back(p->blocks.back().get());
        }
        p->workers.reset(new Workers(threads));
        return p.release();
    });
}

API void lmz_gpu_staging_free(void *staging) { delete static_cast<StagingPool *>(staging); }

API void *lmz_gpu_transfer_new(void *staging, void *cuda_stream)
{
    std::unique_ptr<Transfer> t(new (std::nothrow) Transfer);
    if (!t) {
        fail_msg(LMZ_GPU_EUNSUPPORTED, "host resources");
        return nullptr;
    }
    t->pool = static_cast<StagingPool *>(staging);
    cudaEvent_t ev = nullptr;
    cudaError_t e = cudaGetDevice(&t->device);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&t->stream, cudaStreamNonBlocking);
    // what the caller's stream still does with the memory comes first
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventRecord(ev, (cudaStream_t)cuda_stream);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(t->stream, ev, 0);
    if (ev) cudaEventDestroy(ev);
    if (e != cudaSuccess) {
        cudaGetLastError();
        if (t->stream) cudaStreamDestroy(t->stream);
        fail_cuda("a transfer's stream", e);
        return nullptr;
    }
    return t.release();
}

// A range of `n` blocks with its event.  Its blocks count as open from here on, so this comes after every
// call that can fail: transfer_free waits for each of them.
// -1: no memory, and the event is gone.
static int open_range(Transfer *t, size_t n, cudaEvent_t event, bool to_device)
{
    const int r = guarded(-1, [&] {
        std::lock_guard<std::mutex> lock(t->mu);
        t->ranges.emplace_back();
        Transfer::Range &range = t->ranges.back();
        range.left = n;
        range.event = event;
        range.to_device = to_device;
        t->open += n;
        return (int)t->ranges.size() - 1;
    });
    if (r < 0) cudaEventDestroy(event);
    return r;
}

// A range's block for the workers; one that cannot be handed over ends the transfer like one that failed.
template <class F>
static void queue_block(Transfer *t, size_t r, F job)
{
    try {
        t->pool->workers->add(job);
    } catch (...) {
        t->finish(r, "no memory for a transfer's block");
    }
}

API int lmz_gpu_transfer_upload(void *transfer, int fd, const void *host, uint64_t off, uint64_t len, void *d_dst)
{
    Transfer *t = static_cast<Transfer *>(transfer);
    const size_t B = t->pool->block, n = (size_t)((len + B - 1) / B);
    cudaEvent_t arrived = nullptr;
    CK("cudaEventCreate", cudaEventCreateWithFlags(&arrived, cudaEventDisableTiming));
    const int r = open_range(t, n, arrived, true);
    if (r < 0) return LMZ_GPU_EUNSUPPORTED;
    for (uint64_t at = 0; at < len; at += B) {
        const size_t m = (size_t)(len - at < B ? len - at : B);
        uint8_t *dst = static_cast<uint8_t *>(d_dst) + at;
        queue_block(t, r, [=] { upload_block(t, r, fd, static_cast<const uint8_t *>(host), off + at, m, dst); });
    }
    return r;
}

API int lmz_gpu_transfer_download(void *transfer, const void *d_src, uint64_t len, int fd, void *map, uint64_t off, void *cuda_stream)
{
    Transfer *t = static_cast<Transfer *>(transfer);
    const size_t B = t->pool->block, n = (size_t)((len + B - 1) / B);
    cudaEvent_t after = nullptr;
    CK("cudaEventCreate", cudaEventCreateWithFlags(&after, cudaEventDisableTiming));
    if (cudaError_t e = cudaEventRecord(after, (cudaStream_t)cuda_stream); e != cudaSuccess) {
        cudaEventDestroy(after);
        return fail_cuda("cudaEventRecord", e);
    }
    const int r = open_range(t, n, after, false);
    if (r < 0) return LMZ_GPU_EUNSUPPORTED;
    for (uint64_t at = 0; at < len; at += B) {
        const size_t m = (size_t)(len - at < B ? len - at : B);
        const uint8_t *src = static_cast<const uint8_t *>(d_src) + at;
        queue_block(t, r, [=] { download_block(t, r, src, m, fd, static_cast<uint8_t *>(map), off + at, after); });
    }
    return r;
}

API int lmz_gpu_transfer_wait(void *transfer, int range, void *cuda_stream)
{
    Transfer *t = static_cast<Transfer *>(transfer);
    std::unique_lock<std::mutex> lock(t->mu);
    if (range < 0 || (size_t)range >= t->ranges.size()) return fail_msg(LMZ_GPU_EUNSUPPORTED, "no such range");
    Transfer::Range &r = t->ranges[(size_t)range];
    t->done.wait(lock, [&] { return r.left == 0; });
    if (t->error[0]) return fail_msg(LMZ_GPU_ECUDA, t->error);
    if (r.to_device) CK("wait for an upload", cudaStreamWaitEvent((cudaStream_t)cuda_stream, r.event, 0));
    return LMZ_GPU_OK;
}

API int lmz_gpu_transfer_free(void *transfer)
{
    Transfer *t = static_cast<Transfer *>(transfer);
    int rc = LMZ_GPU_OK;
    {
        std::unique_lock<std::mutex> lock(t->mu);
        t->done.wait(lock, [&] { return t->open == 0; });
        if (t->error[0]) rc = fail_msg(LMZ_GPU_ECUDA, t->error);
    }
    { std::lock_guard<std::mutex> lock(t->issue); }          // the last issuer has let go
    // Issued is not arrived: a caller that has not waited for every range (an error on its way) gives
    // the memory back right after this.
    const cudaError_t e = cudaStreamSynchronize(t->stream);
    if (e != cudaSuccess && rc == LMZ_GPU_OK) rc = fail_cuda("the copies of a transfer", e);
    for (Transfer::Range &r : t->ranges)
        if (r.event) cudaEventDestroy(r.event);
    cudaStreamDestroy(t->stream);
    delete t;
    return rc;
}

// `n` pieces of `width` bytes at offs[i] of a file (fd >= 0) or of memory, one after the other into
// `out`: the small headers in front of every chunk, one page each, which a few threads fetch in a
// tenth of the time that faulting their pages in takes.  Bytes past `size` read as zero.
API int lmz_host_gather(int fd, const void *host, uint64_t size, const uint64_t *offs, size_t n, unsigned width, void *out)
{
    if ((fd < 0 && !host) || (n && (!offs || !out))) return fail_msg(LMZ_GPU_EUNSUPPORTED, "null argument");
    std::atomic<bool> bad{false};
    auto run = [&](size_t lo, size_t hi) {
        for (size_t i = lo; i < hi && !bad.load(std::memory_order_relaxed); i++) {
            uint8_t *to = static_cast<uint8_t *>(out) + i * width;
            const uint64_t at = offs[i] < size ? offs[i] : size;
            const size_t m = size - at < width ? (size_t)(size - at) : width;
            if (m < width) memset(to + m, 0, width - m);
            if (fd < 0) memcpy(to, static_cast<const uint8_t *>(host) + at, m);
            else if (!read_fully(fd, to, at, m)) bad.store(true);
        }
    };
    const size_t threads = n < 512 ? 1 : 8, per = (n + threads - 1) / threads;
    std::thread crew[8];
    for (size_t i = 1; i < threads; i++) {
        const size_t lo = i * per < n ? i * per : n, hi = (i + 1) * per < n ? (i + 1) * per : n;
        try {
            crew[i] = std::thread(run, lo, hi);
        } catch (...) {
            run(lo, hi);                 // no thread to be had: this one's work
        }
    }
    run(0, per < n ? per : n);
    for (std::thread &t : crew)
        if (t.joinable()) t.join();
    return bad.load() ? fail_msg(LMZ_GPU_EBADSTREAM, "reading the file failed") : LMZ_GPU_OK;
}

// [off, off + len) of a file on a memory-backed file system (tmpfs) as writable memory, its pages reserved
// first so that no store can find the file system full.  There write() is one thread's work whatever
// the number of writers (the file's lock: 300 MB in 80 ms), stores through a
// mapping are not (38 ms with eight threads, the reservation included; 21 ms over an existing file).
// NULL: not such a file, or no room -- write() then.
API void *lmz_host_map_file(int fd, uint64_t off, uint64_t len)
{
    constexpr long TMPFS = 0x01021994;
    struct statfs fs;
    if (!len || fstatfs(fd, &fs) != 0 || (long)fs.f_type != TMPFS || (off & 4095)) return nullptr;
    if (posix_fallocate(fd, (off_t)off, (off_t)len) != 0) return nullptr;
    void *p = mmap(nullptr, len, PROT_READ | PROT_WRITE, MAP_SHARED, fd, (off_t)off);
    return p == MAP_FAILED ? nullptr : p;
}
API int lmz_host_unmap_file(void *p, uint64_t len) { return munmap(p, len) == 0 ? LMZ_GPU_OK : LMZ_GPU_EUNSUPPORTED; }
