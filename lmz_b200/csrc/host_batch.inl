// lmz_gpu_decode_batch for host memory, and checked batches in device memory (included by lmz_b200.cu).

namespace {

constexpr size_t VERDICT = 16;           // what a verdict takes where it is copied with the plaintext
// Calls up to here go in by one copy from page-locked memory and out by one, verdict and plaintext
// together.  (One B200: 64 planes of 1 KiB 95 -> 69 us, 16 of 16 KiB, 170 KB in, 195 -> 189; 1.2 MB in 156 -> 151, 1.6 MB
// in 641 -> 653.)
constexpr size_t SMALL_BYTES = (size_t)256 << 10;

}  // namespace

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
