// Memory that host calls keep (included by lmz_b200.cu).
//
// A call of a few planes decodes in tens of microseconds, while allocating and freeing its
// buffers took 0.8 ms (one B200, 7 streams of 4 KiB: 830 us a call, of which 60 us kernel).
// So a call borrows a workspace -- a stream, a device buffer, a small page-locked block -- and
// gives it back; results that this library's callers do not bring a buffer for come in
// page-locked memory that the copy engine writes itself.  Both are bounded: at most
// KEPT_WORKSPACES idle workspaces per device with device buffers of at most KEPT_DEVICE_BYTES,
// at most KEPT_HOST_BYTES of idle result memory, which what has been idle longest leaves first (one B200,
// results of 500 MiB among smaller ones: 225 ms a call while the smaller ones kept the room, 37 now); what is
// over goes back to the driver at once, and lmz_gpu_trim() returns the rest.  A workspace belongs to one
// call at a time.
#include <list>
#include <mutex>
#include <unordered_map>
#include <vector>

namespace {

constexpr size_t KEPT_DEVICE_BYTES = (size_t)256 << 20;
constexpr size_t KEPT_HOST_BYTES = (size_t)512 << 20;
constexpr size_t KEPT_WORKSPACES = 4;
// Result memory has this much in front of what the caller sees, where a small call's verdict lands.
constexpr size_t LENT_HEAD = 64;

struct Workspace {
    int device = -1;
    cudaStream_t stream = nullptr;
    uint8_t *dev = nullptr;
    size_t dev_bytes = 0;
    uint8_t *pin = nullptr;          // offsets in, verdict out
    size_t pin_bytes = 0;
    cudaStream_t lane[MOST_SLICES] = {};     // sliced calls: decode and copy out, each slice on its own
    cudaEvent_t here[MOST_SLICES] = {}, done[MOST_SLICES] = {};

    cudaError_t need_lanes(size_t slices)
    {
        cudaError_t e = cudaSuccess;
        for (size_t i = 0; i < slices && e == cudaSuccess; i++) {
            if (!lane[i]) e = cudaStreamCreateWithFlags(&lane[i], cudaStreamNonBlocking);
            if (e == cudaSuccess && !done[i]) e = cudaEventCreateWithFlags(&done[i], cudaEventDisableTiming);
            if (e == cudaSuccess && !here[i]) e = cudaEventCreateWithFlags(&here[i], cudaEventDisableTiming);
        }
        return e;
    }
    void idle()
    {
        if (stream) cudaStreamSynchronize(stream);
        for (cudaStream_t l : lane)
            if (l) cudaStreamSynchronize(l);
    }

    cudaError_t need(size_t device_bytes, size_t pinned_bytes)
    {
        cudaError_t e = cudaSuccess;
        if (!stream) e = cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking);
        if (e == cudaSuccess && dev_bytes < device_bytes) {
            if (dev) cudaFree(dev);
            dev = nullptr; dev_bytes = 0;
            const size_t c = device_bytes <= KEPT_DEVICE_BYTES ? size_class(device_bytes) : device_bytes;
            e = cudaMalloc((void **)&dev, c);
            if (e == cudaSuccess) dev_bytes = c;
        }
        if (e == cudaSuccess && pin_bytes < pinned_bytes) {
            if (pin) cudaFreeHost(pin);
            pin = nullptr; pin_bytes = 0;
            const size_t c = size_class(pinned_bytes);
            e = cudaMallocHost((void **)&pin, c);
            if (e == cudaSuccess) pin_bytes = c;
        }
        return e;
    }
    void drop()
    {
        if (dev) cudaFree(dev);
        if (pin) cudaFreeHost(pin);
        if (stream) cudaStreamDestroy(stream);
        for (cudaStream_t l : lane)
            if (l) cudaStreamDestroy(l);
        for (cudaEvent_t e : here)
            if (e) cudaEventDestroy(e);
        for (cudaEvent_t e : done)
            if (e) cudaEventDestroy(e);
        *this = Workspace{};
    }
};

struct HostPool {
    std::mutex mu;
    std::vector<Workspace> idle;
    std::unordered_map<void *, size_t> lent;               // result memory in callers' hands
    struct Spare { size_t bytes; void *block; };
    std::list<Spare> spare;                                // idle result memory, the longest idle first,
    std::unordered_multimap<size_t, std::list<Spare>::iterator> by_class;      // and by size class
    size_t spare_bytes = 0;

    // Take an idle block out of the books.
    void *take(std::unordered_multimap<size_t, std::list<Spare>::iterator>::iterator it)
    {
        void *block = it->second->block;
        spare_bytes -= it->second->bytes;
        spare.erase(it->second);
        by_class.erase(it);
        return block;
    }
    // ... the one that has been idle longest.
    void *take_oldest()
    {
        auto range = by_class.equal_range(spare.front().bytes);
        while (range.first->second != spare.begin()) ++range.first;
        return take(range.first);
    }
    void put(size_t bytes, void *block)
    {
        spare.push_back({bytes, block});
        try {
            by_class.emplace(bytes, std::prev(spare.end()));
        } catch (...) {
            spare.pop_back();
            throw;
        }
        spare_bytes += bytes;
    }
};
HostPool &host_pool()
{
    static HostPool *p = new HostPool;      // (never destroyed: calls may still run while the process exits)
    return *p;
}

// A workspace for one call, given back when the call ends -- with its stream idle.
struct Borrowed {
    Workspace w;
    bool sound = false;
    explicit Borrowed(int device)
    {
        HostPool &p = host_pool();
        std::lock_guard<std::mutex> lock(p.mu);
        for (size_t i = 0; i < p.idle.size(); i++)
            if (p.idle[i].device == device) {
                w = p.idle[i];
                p.idle.erase(p.idle.begin() + i);
                break;
            }
        w.device = device;
    }
    ~Borrowed()
    {
        w.idle();
        if (sound && w.dev_bytes <= KEPT_DEVICE_BYTES) {
            HostPool &p = host_pool();
            std::lock_guard<std::mutex> lock(p.mu);
            size_t mine = 0;
            for (const Workspace &o : p.idle) mine += o.device == w.device;
            if (mine < KEPT_WORKSPACES) {
                try {
                    p.idle.push_back(w);
                    return;
                } catch (...) {          // no memory to remember it by
                }
            }
        }
        w.drop();
    }
};

bool is_lent(const void *p, size_t bytes)
{
    HostPool &pool = host_pool();
    std::lock_guard<std::mutex> lock(pool.mu);
    auto it = pool.lent.find(const_cast<void *>(p));
    return it != pool.lent.end() && it->second - LENT_HEAD >= bytes;
}

}  // namespace

API void *lmz_gpu_host_alloc(size_t bytes)
{
    if (bytes > SIZE_MAX - LENT_HEAD) return nullptr;
    // (what is too large to be kept is taken as large as it is)
    const size_t c = bytes + LENT_HEAD <= KEPT_HOST_BYTES ? size_class(bytes + LENT_HEAD) : bytes + LENT_HEAD;
    return guarded<void *>(nullptr, [&]() -> void * {
        HostPool &p = host_pool();
        {
            std::lock_guard<std::mutex> lock(p.mu);
            auto it = p.by_class.find(c);
            if (it != p.by_class.end()) {
                void *q = static_cast<uint8_t *>(it->second->block) + LENT_HEAD;
                p.lent[q] = c;
                p.take(it);
                return q;
            }
        }
        void *block = nullptr;
        if (cudaHostAlloc(&block, c, cudaHostAllocPortable) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        void *q = static_cast<uint8_t *>(block) + LENT_HEAD;
        std::lock_guard<std::mutex> lock(p.mu);
        try {
            p.lent[q] = c;
        } catch (...) {
            cudaFreeHost(block);
            throw;
        }
        return q;
    });
}

API void lmz_gpu_host_free(void *q)
{
    HostPool &p = host_pool();
    std::unique_lock<std::mutex> lock(p.mu);
    auto it = p.lent.find(q);
    if (it == p.lent.end()) return;
    const size_t c = it->second;
    p.lent.erase(it);
    q = static_cast<uint8_t *>(q) - LENT_HEAD;
    if (c <= KEPT_HOST_BYTES) {
        // what has been idle longest makes room (sizes that are asked for no more would fill it for good)
        while (p.spare_bytes + c > KEPT_HOST_BYTES) {
            void *oldest = p.take_oldest();
            lock.unlock();
            cudaFreeHost(oldest);
            lock.lock();
        }
        try {
            p.put(c, q);
            return;
        } catch (...) {                  // no memory to remember it by
        }
    }
    lock.unlock();
    cudaFreeHost(q);
}

API int lmz_gpu_host_lent(const void *q, size_t bytes) { return is_lent(q, bytes); }

API void lmz_gpu_trim(void)
{
    HostPool &p = host_pool();
    std::vector<Workspace> idle;
    std::list<HostPool::Spare> spare;
    {
        std::lock_guard<std::mutex> lock(p.mu);
        idle.swap(p.idle);
        p.by_class.clear();
        spare.swap(p.spare);
        p.spare_bytes = 0;
    }
    int dev = 0;
    const bool had = cudaGetDevice(&dev) == cudaSuccess;
    for (Workspace &w : idle) {
        cudaSetDevice(w.device);
        w.drop();
    }
    if (had) cudaSetDevice(dev);
    for (const HostPool::Spare &s : spare) cudaFreeHost(s.block);
}
