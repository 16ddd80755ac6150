// lmz_gpu_decode_batch for host memory (included by lmz_b200.cu), and the memory it keeps.
//
// A call of a few planes decodes in tens of microseconds, while allocating and freeing its
// buffers took 0.8 ms (one B200, 7 streams of 4 KiB: 830 us a call, of which 60 us kernel).
// So a call borrows a workspace -- a stream, a device buffer, a small page-locked block -- and
// gives it back; results that this library's callers do not bring a buffer for come in
// page-locked memory that the copy engine writes itself.  Both are bounded: at most
// KEPT_WORKSPACES idle workspaces per device with device buffers of at most KEPT_DEVICE_BYTES,
// at most KEPT_HOST_BYTES of idle result memory; what is over goes back to the driver at once,
// and lmz_gpu_trim() returns the rest.  A workspace belongs to one call at a time.

namespace {

constexpr size_t KEPT_DEVICE_BYTES = (size_t)256 << 20;
constexpr size_t KEPT_HOST_BYTES = (size_t)512 << 20;
constexpr size_t KEPT_WORKSPACES = 4;
// Result memory has this much in front of what the caller sees, where a small call's verdict lands.
constexpr size_t LENT_HEAD = 64, VERDICT = 16;
// Calls up to here go in by one copy from page-locked memory and out by one, verdict and plaintext
// together.  (One B200: 64 planes of 1 KiB 95 -> 69 us, 16 of 16 KiB, 170 KB in, 195 -> 189; 1.2 MB in 156 -> 151, 1.6 MB
// in 641 -> 653.)
constexpr size_t SMALL_BYTES = (size_t)256 << 10;

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
    std::unordered_multimap<size_t, void *> spare;         // idle result memory by size class
    size_t spare_bytes = 0;
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
            auto it = p.spare.find(c);
            if (it != p.spare.end()) {
                void *q = static_cast<uint8_t *>(it->second) + LENT_HEAD;
                p.lent[q] = c;
                p.spare.erase(it);
                p.spare_bytes -= c;
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
    {
        std::lock_guard<std::mutex> lock(p.mu);
        auto it = p.lent.find(q);
        if (it == p.lent.end()) return;
        const size_t c = it->second;
        p.lent.erase(it);
        q = static_cast<uint8_t *>(q) - LENT_HEAD;
        if (p.spare_bytes + c <= KEPT_HOST_BYTES) {
            try {
                p.spare.emplace(c, q);
                p.spare_bytes += c;
                return;
            } catch (...) {              // no memory to remember it by
            }
        }
    }
    cudaFreeHost(q);
}

API int lmz_gpu_host_lent(const void *q, size_t bytes) { return is_lent(q, bytes); }

API void lmz_gpu_trim(void)
{
    HostPool &p = host_pool();
    std::vector<Workspace> idle;
    std::unordered_multimap<size_t, void *> spare;
    {
        std::lock_guard<std::mutex> lock(p.mu);
        idle.swap(p.idle);
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
    for (auto &kv : spare) cudaFreeHost(kv.second);
}

API int lmz_gpu_decode_batch(const void *hdr, const void *streams, size_t nbytes, const void *off,
                             unsigned nstr, unsigned plane, void *out)
{
    if (nstr == 0) return LMZ_GPU_OK;
    if (plane == 0) return fail_msg(LMZ_GPU_EUNSUPPORTED, "plane is zero");
    if (int rc = device_ready()) return rc;
    // every (offset, length) pair must lie inside the buffer, and a length must fit the
    // 32 bits the kernels carry it in
    const uint64_t *pairs = static_cast<const uint64_t *>(off);
    bool in_order = true;
    for (unsigned i = 0; i < nstr; i++) {
        const uint64_t at = pairs[2 * i], len = pairs[2 * i + 1];
        if (at > nbytes || len > nbytes - at) return fail_msg(LMZ_GPU_EBADSTREAM, "a stream lies outside the buffer");
        if (len >> 32) return fail_msg(LMZ_GPU_EUNSUPPORTED, "a stream is 4 GiB or longer");
        in_order = in_order && (i == 0 || pairs[2 * (size_t)i - 2] + pairs[2 * (size_t)i - 1] <= at);
    }
    int device = 0;
    CK("cudaGetDevice", cudaGetDevice(&device));

    // device buffer: offsets | shared table | verdict | streams + slack | plaintext + its verdict
    auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
    const size_t out_bytes = (size_t)nstr * plane, table_bytes = (size_t)nstr * 16;
    const size_t at_hdr = table_bytes, at_verdict = (at_hdr + (hdr ? HDR_BYTES : 0) + 15) & ~(size_t)15;
    const size_t head_bytes = at_verdict + 16, at_src = up(head_bytes), at_out = up(at_src + nbytes + PAD_BYTES + VERDICT);
    // memory of this library's own takes the plaintext at once; a caller's buffer only if all is well
    const bool direct = is_lent(out, out_bytes);
    // slices want each its own stretch of the streams, and plaintext that may leave before the verdict
    int sms = 0;
    if (int rc = sm_count(&sms)) return rc;
    const size_t slices = direct && in_order ? batch_slices(nbytes + out_bytes, nstr, (unsigned)sms) : 1;
    const bool small = direct && slices == 1 && at_out <= SMALL_BYTES;
    Borrowed b(device);
    Workspace &w = b.w;
    if (cudaError_t e = w.need(at_out + out_bytes, (small ? at_out : head_bytes) + 16)) {
        cudaGetLastError();
        return fail_cuda("memory for the batch", e);
    }
    uint8_t *d = w.dev;
    memcpy(w.pin, off, table_bytes);
    if (hdr) memcpy(w.pin + at_hdr, hdr, HDR_BYTES);
    memset(w.pin + at_verdict, 0, 16);
    // the device's verdict: in the head, or (small) right in front of the plaintext
    uint8_t *const d_verdict = small ? d + at_out - VERDICT : d + at_verdict;
    uint32_t *verdict = reinterpret_cast<uint32_t *>(small ? static_cast<uint8_t *>(out) - VERDICT : w.pin + head_bytes);
    if (small) {
        memcpy(w.pin + at_src, streams, nbytes);
        memset(w.pin + at_src + nbytes, 0, at_out - at_src - nbytes);
        CK("copy the batch in", cudaMemcpyAsync(d, w.pin, at_out, cudaMemcpyHostToDevice, w.stream));
    } else {
        *verdict = 0;
        CK("copy offsets in", cudaMemcpyAsync(d, w.pin, head_bytes, cudaMemcpyHostToDevice, w.stream));
    }
    RansArgs a{};
    a.src = d + at_src;
    a.plane = plane;
    a.shared_hdr = hdr ? d + at_hdr : nullptr;
    a.any_bad = reinterpret_cast<uint32_t *>(d_verdict);
    if (slices > 1) CK("streams for the batch", w.need_lanes(slices));
    size_t from = 0;
    for (size_t j = 0; j < slices; j++) {
        const size_t first = nstr * j / slices, last = nstr * (j + 1) / slices;
        const size_t upto = last == nstr ? nbytes : (size_t)pairs[2 * last];
        if (upto > from && !small)
            CK("copy streams in", cudaMemcpyAsync(d + at_src + from, static_cast<const uint8_t *>(streams) + from, upto - from,
                                                  cudaMemcpyHostToDevice, w.stream));
        from = upto;
        cudaStream_t cs = w.stream;
        if (slices > 1) {
            cs = w.lane[j];
            CK("slice of the batch", cudaEventRecord(w.here[j], w.stream));
            CK("slice of the batch", cudaStreamWaitEvent(cs, w.here[j], 0));
        }
        a.offs = reinterpret_cast<const uint64_t *>(d) + 2 * first;
        a.njobs = (uint32_t)(last - first);
        const size_t at = first * plane, bytes = (size_t)a.njobs * plane;
        a.dst = d + at_out + at;
        if (int rc = launch_rans(a, cs)) return rc;
        if (small) {
            CK("copy verdict and plaintext out", cudaMemcpyAsync(verdict, d_verdict, VERDICT + out_bytes, cudaMemcpyDeviceToHost, cs));
        } else if (direct) {
            CK("copy plaintext out", cudaMemcpyAsync(static_cast<uint8_t *>(out) + at, d + at_out + at, bytes, cudaMemcpyDeviceToHost, cs));
        }
    }
    for (size_t l = 0; slices > 1 && l < slices; l++) {
        CK("end of the batch", cudaEventRecord(w.done[l], w.lane[l]));
        CK("end of the batch", cudaStreamWaitEvent(w.stream, w.done[l], 0));
    }
    if (!small) CK("copy the verdict out", cudaMemcpyAsync(verdict, d_verdict, 4, cudaMemcpyDeviceToHost, w.stream));
    CK("decode", cudaStreamSynchronize(w.stream));
    b.sound = true;
    if (*verdict) {
        // (the device's word is enough to refuse the batch; the host looks again for the reason)
        if (!hdr)
            if (int rc = lmz_gpu_validate(streams, off, nstr)) return rc;
        return fail_msg(LMZ_GPU_EBADSTREAM, "a stream is malformed or truncated");
    }
    if (!direct) {
        CK("copy plaintext out", cudaMemcpyAsync(out, d + at_out, out_bytes, cudaMemcpyDeviceToHost, w.stream));
        CK("copy plaintext out", cudaStreamSynchronize(w.stream));
    }
    return LMZ_GPU_OK;
}

// ---- batches in device memory, with the answer ------------------------------------------------

API int lmz_gpu_batch_work_bytes(unsigned nstr)
{
    const uint64_t b = (uint64_t)nstr * sizeof(StreamJob) + 256;
    return b > 0x7fffffffu ? 0 : (int)b;
}

API int lmz_gpu_decode_batch_checked_dev(const void *d_hdr, const void *d_streams, uint64_t nbytes, const void *d_off,
                                         unsigned nstr, unsigned plane, void *d_out, void *d_work, void *cuda_stream)
{
    if (nstr == 0) return LMZ_GPU_OK;
    if (plane == 0) return fail_msg(LMZ_GPU_EUNSUPPORTED, "plane is zero");
    if (int rc = device_ready()) return rc;
    int device = 0;
    CK("cudaGetDevice", cudaGetDevice(&device));
    cudaStream_t cs = (cudaStream_t)cuda_stream;
    uint32_t *d_verdict = static_cast<uint32_t *>(d_work);
    StreamJob *jobs = reinterpret_cast<StreamJob *>(static_cast<uint8_t *>(d_work) + 256);
    Borrowed b(device);
    CK("a page-locked word", b.w.need(0, 64));
    volatile uint32_t *verdict = reinterpret_cast<volatile uint32_t *>(b.w.pin);
    CK("clear the verdict", cudaMemsetAsync(d_verdict, 0, 4, cs));
    k_batch_jobs<<<(nstr + 255) / 256, 256, 0, cs>>>(static_cast<const uint64_t *>(d_off), nbytes, nstr, plane, jobs, d_verdict);
    cudaError_t le = cudaGetLastError();
    if (le != cudaSuccess) return fail_cuda("launch k_batch_jobs", le);
    RansArgs a{};
    a.src = static_cast<const uint8_t *>(d_streams);
    a.jobs = jobs;
    a.njobs = nstr;
    a.dst = static_cast<uint8_t *>(d_out);
    a.shared_hdr = static_cast<const uint8_t *>(d_hdr);
    a.any_bad = d_verdict;
    if (int rc = launch_rans(a, cs)) return rc;
    CK("copy the verdict out", cudaMemcpyAsync(b.w.pin, d_verdict, 4, cudaMemcpyDeviceToHost, cs));
    CK("decode", cudaStreamSynchronize(cs));
    b.sound = true;
    if (*verdict & 2u) return fail_msg(LMZ_GPU_EBADSTREAM, "a stream lies outside the buffer");
    if (*verdict) return fail_msg(LMZ_GPU_EBADSTREAM, "a stream is malformed or truncated");
    return LMZ_GPU_OK;
}

API int lmz_gpu_pack_offsets_dev(const void *d_lengths, unsigned nstr, void *d_offsets, void *d_work, uint64_t *h_total,
                                 unsigned *h_failed, void *cuda_stream)
{
    if (int rc = device_ready()) return rc;
    *h_total = 0;
    *h_failed = 0;
    if (nstr == 0) return LMZ_GPU_OK;
    if (!d_lengths || !d_offsets || !d_work) return fail_msg(LMZ_GPU_EUNSUPPORTED, "null argument");
    int device = 0;
    CK("cudaGetDevice", cudaGetDevice(&device));
    cudaStream_t cs = (cudaStream_t)cuda_stream;
    Borrowed b(device);
    CK("a page-locked block", b.w.need(0, 64));
    k_pack_offsets<<<1, 1024, 0, cs>>>(static_cast<const uint32_t *>(d_lengths), nstr, static_cast<uint64_t *>(d_offsets),
                                       static_cast<uint64_t *>(d_work));
    cudaError_t le = cudaGetLastError();
    if (le != cudaSuccess) return fail_cuda("launch k_pack_offsets", le);
    CK("copy the sizes out", cudaMemcpyAsync(b.w.pin, d_work, 16, cudaMemcpyDeviceToHost, cs));
    CK("encode", cudaStreamSynchronize(cs));
    b.sound = true;
    const volatile uint64_t *got = reinterpret_cast<const volatile uint64_t *>(b.w.pin);
    *h_total = got[0];
    *h_failed = (unsigned)got[1];
    return LMZ_GPU_OK;
}
