// C-ABI shared library: sm_100a decode of lmz rANS byte-plane streams.
//
// The first nine exports are the boundary the reference's Python binds
// (lmz/gpu/lmzgpu.cu:341-527, ctypes signatures at lmz/gpu/__init__.py:130-148)
// with the same names, argument meaning, return codes and error behaviour; the
// rest are additive entry points for whole-archive decode.  Declarations and
// the per-function contract live in include/lmz_b200.h.
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "../../include/lmz_b200.h"
#include "chunk_kernels.cuh"
#include "cond_kernels.cuh"
#include "fused_kernel.cuh"
#include "solo_kernel.cuh"
#include "encode_kernel.cuh"
#include "save_kernels.cuh"

using namespace lmz;

#define API extern "C" __attribute__((visibility("default")))

#include "host_error.inl"

static int device_ready()
{
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n < 1) {
        cudaGetLastError();
        return fail_msg(LMZ_GPU_ENODEV, "no CUDA device");
    }
    return LMZ_GPU_OK;
}

// Kernels ask for more dynamic shared memory than the default 48 KiB; the
// opt-in is per device and is made once.
template <class K>
static int opt_in_smem(K kernel, uint32_t bytes, bool *done /* [64] by device */)
{
    int dev = 0;
    CK("cudaGetDevice", cudaGetDevice(&dev));
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 0 && dev < 64 && done[dev]) return LMZ_GPU_OK;
    CK("cudaFuncSetAttribute",
       cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    if (dev >= 0 && dev < 64) done[dev] = true;
    return LMZ_GPU_OK;
}

// k_stream takes all the shared memory one CTA may have and lays its tables out from
// both ends, counting on the window starting F_SMEM_BASE bytes in (what the
// driver reserves per CTA on this architecture).
static int stream_smem_ok()
{
    static int state[64];                       // 0 unknown, 1 good, -1 bad
    int dev = 0;
    CK("cudaGetDevice", cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail_msg(LMZ_GPU_EUNSUPPORTED, "device index out of range");
    if (state[dev] == 0) {
        int reserved = 0, optin = 0;
        CK("cudaDeviceGetAttribute", cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev));
        CK("cudaDeviceGetAttribute", cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
        state[dev] = (reserved == (int)F_SMEM_BASE && optin >= (int)F_SMEM_DYN) ? 1 : -1;
    }
    if (state[dev] < 0)
        return fail_msg(LMZ_GPU_EUNSUPPORTED, "this GPU's shared memory per CTA is not the 1 KiB + 227 KiB k_stream is laid out for");
    return LMZ_GPU_OK;
}

static int sm_count(int *out);

// Kernels this thread has launched for the plan it was last given (lmz_gpu_plan_launches).
static thread_local unsigned g_launches;

template <int SINK, bool CRC, int CFN, int MODE>
static int launch_stream_as(const StreamArgs &a, uint32_t grid, uint32_t W, cudaStream_t cs)
{
    static bool done[64];
    // A launch is of one CTA per SM at most, and as long as its fullest SM.  Beside the kernel for an archive's other chunks, whose
    // CTAs with checksum tables hold an SM when this one starts, CTAs of up to seven warps went two to another SM.  (One B200,
    // chunks with checksums, 28 per SM: BF16 634 -> 491 us, FP32 455 -> 366; 32 per SM, whose CTAs are larger, 494 and 370
    // either way.  Without checksums, and of planes alone, none were seen to, and launches of several threads may share an SM.)
    uint32_t shm = stream_smem(CFN, CRC, SINK, MODE, W).end - F_SMEM_BASE;
    if (CRC && CFN > 0 && SINK != SINK_DELTA) shm = alone_on_sm(shm);
    int rc = opt_in_smem(k_stream<SINK, CRC, CFN, MODE>, F_SMEM_DYN, done);
    if (rc) return rc;
    k_stream<SINK, CRC, CFN, MODE><<<grid, W * 32, shm, cs>>>(a);
    g_launches++;
    cudaError_t le = cudaGetLastError();
    if (le != cudaSuccess) return fail_cuda("launch k_stream", le);
    return LMZ_GPU_OK;
}

// Streams per SM that the delta sink's wide-table instance takes in one round.
template <bool CRC>
constexpr uint32_t wide_per_sm() { return 4 * stream_warps(0, CRC, SINK_DELTA, TR_FEW); }

// lmz_gpu_set_table_mode's; -1 picks by batch size.
static std::atomic<int> g_force_table_mode{-1};

template <int SINK, bool CRC, bool WIDE>
static int launch_solo_as(const StreamArgs &a, uint32_t grid, uint32_t W, cudaStream_t cs)
{
    static bool done[64];
    int rc = opt_in_smem(k_solo<SINK, CRC, WIDE>, F_SMEM_DYN, done);
    if (rc) return rc;
    k_solo<SINK, CRC, WIDE><<<grid, W * 32, solo_smem(CRC, WIDE, W).end - F_SMEM_BASE, cs>>>(a);
    g_launches++;
    cudaError_t le = cudaGetLastError();
    if (le != cudaSuccess) return fail_cuda("launch k_solo", le);
    return LMZ_GPU_OK;
}

// A warp per stream, whatever the alphabets.
template <int SINK, bool CRC>
static int launch_solo(const StreamArgs &a, cudaStream_t cs)
{
    if (a.njobs == 0) return LMZ_GPU_OK;
    int rc = stream_smem_ok();
    if (rc) return rc;
    int sms = 0;
    rc = sm_count(&sms);
    if (rc) return rc;
    const int forced = g_force_table_mode.load(std::memory_order_relaxed);
    const SoloLaunch l = solo_launch(a.njobs, a.most_ctas ? a.most_ctas : (uint32_t)sms, CRC,
                                     forced == T_SOLO_WIDE ? 1 : forced == T_SOLO_BYTES ? 0 : -1);
    return l.wide ? launch_solo_as<SINK, CRC, true>(a, l.grid, l.warps, cs) : launch_solo_as<SINK, CRC, false>(a, l.grid, l.warps, cs);
}

// Launches of few streams, with nothing to sort by: a warp each up to so many per SM, then four to a warp as long as
// byte tables (F_BYTE_CFN) take the launch in one round.  1 when they are more.
//
// One B200, us, compact tables / a warp each / byte tables.  Exponent planes of 32 KiB: 16 per SM - / 291 / 278, 20 per SM
// - / 338 / 301, 24 per SM 379 / - / 303, 28 per SM 381 / - / 303; uniform bytes 16 per SM - / 297 / 383, 20 per SM - / 352 / 395,
// 24 per SM 418 / - / 397, 28 per SM 420 / - / 399; planes of 4 KiB, exponents 20 per SM - / 53 / 53, 24 per SM 68 / - / 55, uniform
// bytes - / 55 / 66 and 72 / - / 66: a warp each up to 20.
// With the sinks' own work in the same issue slots, 64 KiB BF16 chunks with checksums: 12 per SM - / 327 / 403, 16 per SM
// - / 376 / 405, 17 per SM 483 / - / 411, 24 per SM 489 / - / 417; FP32 ones: 12 per SM - / 255 / 264, 16 per SM - / 294 / 264,
// 17 per SM 358 / - / 269, 24 per SM 362 / - / 284; without checksums 28 per SM, BF16 463 / - / 374, FP32 325 / - / 239: a warp each up
// to 16 (FP32 chunks, which come here only where a caller has few of them fused, share the line of BF16's).
// Open streams have no byte-table instance.
template <int SINK, bool CRC>
static int launch_few(const StreamArgs &a, cudaStream_t cs)
{
    if (a.njobs == 0) return LMZ_GPU_OK;
    int rc = stream_smem_ok();
    if (rc) return rc;
    int sms = 0;
    rc = sm_count(&sms);
    if (rc) return rc;
    const int forced = g_force_table_mode.load(std::memory_order_relaxed);
    const uint64_t room = a.most_ctas ? a.most_ctas : (uint32_t)sms;
    constexpr uint32_t solo = SINK == SINK_BYTES || SINK == SINK_OPEN ? 20 : 16;
    if (forced >= 0 ? forced == T_SOLO_WIDE || forced == T_SOLO_BYTES : a.njobs <= solo * room) return launch_solo<SINK, CRC>(a, cs);
    if constexpr (SINK != SINK_OPEN) {
        if (forced < 0 && a.njobs <= 4 * stream_warps(F_BYTE_CFN, CRC, SINK, TR_FEW) * room) {
            const uint32_t quads = (a.njobs + 3) / 4, grid = quads < room ? quads : (uint32_t)room;
            return launch_stream_as<SINK, CRC, F_BYTE_CFN, TR_FEW>(a, grid, (quads + grid - 1) / grid, cs);
        }
    }
    return 1;
}

// CFN = 128 is for streams the caller knows to have at most F_SMALL_LIVE live symbols;
// CFN = -1 is one wide table per CTA.
template <int SINK, bool CRC, int CFN>
static int launch_stream(const StreamArgs &a, cudaStream_t cs)
{
    if (a.njobs == 0) return LMZ_GPU_OK;
    int rc = stream_smem_ok();
    if (rc) return rc;
    int sms = 0;
    rc = sm_count(&sms);
    if (rc) return rc;
    if constexpr (CFN < 0 && SINK == SINK_BF16)     // the job list is laid out 80 to a CTA
        return launch_stream_as<SINK, CRC, CFN, TR_8>(a, a.njobs / (F_SHARED_SINK_WARPS * 4), F_SHARED_SINK_WARPS, cs);
    // Else at most one CTA per SM; its warps take four streams at a time.  As many rounds of fours as the
    // fullest CTA would need, the warps of a CTA just enough for them (when the device holds the count,
    // as if every job of the launch were of this class).
    const uint32_t quads = (a.njobs + 3) / 4, room = a.most_ctas ? a.most_ctas : (uint32_t)sms;
    const uint32_t grid = quads < room ? quads : room;
    auto waves = [&](uint32_t most) { return (quads + grid * most - 1) / (grid * most); };
    auto warps = [&](uint32_t most) { return (quads + grid * waves(most) - 1) / (grid * waves(most)); };
    // TR_FEW makes the shortest step, TR_4 has room for the most warps: that is taken where it saves a
    // round (one B200, 64 KiB BF16 chunks with checksums, TR_8 against TR_4: 180 chunks per SM
    // 2160 against 1880 us, 34 per SM 605 against 675).  Streams of bytes alone, with no checksum tables to
    // make room for, run as many warps of TR_8 as of TR_4, and faster (193 streams per SM 1490 against
    // 1535 us).
    // Up to eight of the delta sink's streams per SM (twelve without checksums) a wide table each fits (CFN = 0): a
    // step is one lookup and five instructions shorter, whatever the alphabet.
    if constexpr (CFN > 0 && SINK == SINK_DELTA)
        if (quads * 4 <= grid * wide_per_sm<CRC>())
            return launch_stream_as<SINK, CRC, 0, TR_FEW>(a, grid, warps(wide_per_sm<CRC>() / 4), cs);
    if constexpr (CFN > 0) {
        constexpr uint32_t few = stream_warps(CFN, CRC, SINK, TR_FEW), most4 = stream_warps(CFN, CRC, SINK, TR_4);
        if constexpr (SINK == SINK_BYTES) {
            constexpr uint32_t most8 = stream_warps(CFN, CRC, SINK, TR_8);
            if (waves(most8) <= waves(most4) && waves(most8) < waves(few))
                return launch_stream_as<SINK, CRC, CFN, TR_8>(a, grid, warps(most8), cs);
        }
        if (waves(most4) < waves(few)) return launch_stream_as<SINK, CRC, CFN, TR_4>(a, grid, warps(most4), cs);
        return launch_stream_as<SINK, CRC, CFN, TR_FEW>(a, grid, warps(few), cs);
    } else {
        return launch_stream_as<SINK, CRC, CFN, TR_8>(a, grid, warps(stream_warps(CFN, CRC, SINK, TR_8)), cs);
    }
}

// A batch of streams to decode to bytes.
struct RansArgs {
    const uint8_t *src;         // compressed bytes (16-byte aligned base, PAD_BYTES of slack after)
    const StreamJob *jobs;      // njobs descriptors, or NULL to use `offs`/`plane`
    const uint64_t *offs;       // reference layout: (offset, length) pairs
    uint32_t plane;             // symbols per stream when `offs` is used
    uint32_t njobs;
    uint8_t *dst;
    const uint8_t *shared_hdr;  // 516-byte table shared by every stream
    uint32_t *status;           // one word per job, may be NULL
    uint32_t *any_bad;          // set non-zero when a job fails hard, may be NULL
    bool open;                  // open streams may be among the jobs
};

static StreamArgs as_stream_args(const RansArgs &a)
{
    StreamArgs sa{};
    sa.src = a.src; sa.sjobs = a.jobs; sa.offs = a.offs; sa.plane = a.plane;
    sa.njobs = a.njobs; sa.dst = a.dst; sa.status = a.status; sa.any_bad = a.any_bad;
    sa.shared_hdr = a.shared_hdr;
    return sa;
}

// A large batch whose tables the host cannot see: sort the streams by alphabet size on the
// device and give the small ones to the denser 128-entry instance.  The index list lives in
// stream-ordered memory for the duration of the two launches.  Returns 1 when that memory
// is not to be had (the caller then runs everything on the 256-entry instance).
// A memory pool of this library's own per device, which keeps what is freed into it: the
// default pool hands memory back to the driver at every synchronisation, and getting it
// again costs more than the index list's kernels.
static cudaMemPool_t scratch_pool()
{
    static cudaMemPool_t pools[64];
    static bool tried[64];
    static std::mutex mu;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    std::lock_guard<std::mutex> lock(mu);
    if (!tried[dev]) {
        tried[dev] = true;
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.handleTypes = cudaMemHandleTypeNone;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        if (cudaMemPoolCreate(&pool, &props) == cudaSuccess) {
            uint64_t keep = ~0ull;
            cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
            pools[dev] = pool;
        } else {
            cudaGetLastError();
        }
    }
    return pools[dev];
}

static int launch_compact_sorted(const RansArgs &a, cudaStream_t cs)
{
    uint32_t *buf = nullptr;
    const size_t bytes = ((size_t)a.njobs + 2) * sizeof(uint32_t);
    cudaMemPool_t pool = scratch_pool();
    if (!pool || cudaMallocFromPoolAsync((void **)&buf, bytes, pool, cs) != cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    uint32_t *counts = buf, *order = buf + 2;
    StreamArgs sa = as_stream_args(a);
    int rc = LMZ_GPU_OK;
    do {
        if (cudaMemsetAsync(counts, 0, 8, cs) != cudaSuccess) { rc = fail_msg(LMZ_GPU_ECUDA, "cudaMemsetAsync failed"); break; }
        k_classify<<<(a.njobs + 7) / 8, 256, 0, cs>>>(sa, F_SMALL_LIVE, order, counts);
        g_launches++;
        cudaError_t le = cudaGetLastError();
        if (le != cudaSuccess) { rc = fail_cuda("launch k_classify", le); break; }
        sa.order = order;
        sa.count = counts;
        sa.order_from_back = 0;
        rc = launch_stream<SINK_BYTES, false, F_SMALL_CFN>(sa, cs);
        if (rc) break;
        sa.count = counts + 1;
        sa.order_from_back = 1;
        rc = launch_stream<SINK_BYTES, false, 256>(sa, cs);
    } while (0);
    cudaFreeAsync(buf, cs);
    return rc;
}

// Streams that carry their own table.  Few of them: launch_few; up to 76 per SM the full-size compact
// tables take the launch in one round, whatever the alphabets; above that small alphabets go to the denser instance.
constexpr unsigned COMPACT_PER_SM = 4 * stream_warps(256, false, SINK_BYTES, TR_8);

static int launch_rans(const RansArgs &a, cudaStream_t cs, bool may_alloc = true)
{
    if (a.njobs == 0) return LMZ_GPU_OK;
    int sms = 0;
    int rc = sm_count(&sms);
    if (rc) return rc;
    const StreamArgs sa = as_stream_args(a);
    if (a.shared_hdr) return launch_stream<SINK_BYTES, false, -1>(sa, cs);
    const int forced = g_force_table_mode.load(std::memory_order_relaxed);
    rc = a.open ? launch_few<SINK_OPEN, false>(sa, cs) : launch_few<SINK_BYTES, false>(sa, cs);
    if (rc != 1) return rc;
    if (a.open) return launch_stream<SINK_OPEN, false, 256>(sa, cs);
    if (may_alloc && forced < 0 && a.njobs > (unsigned)sms * COMPACT_PER_SM) {
        rc = launch_compact_sorted(a, cs);
        if (rc != 1) return rc;
    }
    return launch_stream<SINK_BYTES, false, 256>(sa, cs);
}

// ------------------------------------------------------- the reference's nine

API int lmz_gpu_abi_version(void) { return 1; }
API const char *lmz_gpu_last_error(void) { return g_err; }
API int lmz_gpu_grain(void) { return 1; }
API int lmz_gpu_header_bytes(void) { return (int)HDR_BYTES; }
API int lmz_gpu_pad_bytes(void) { return (int)PAD_BYTES; }

API int lmz_gpu_device_name(char *buf, int cap)
{
    if (!buf || cap <= 0) return fail_msg(LMZ_GPU_EUNSUPPORTED, "no room for the device name");
    if (int rc = device_ready()) return rc;
    int dev = 0, cc_major = 0, cc_minor = 0, sms = 0;
    CK("cudaGetDevice", cudaGetDevice(&dev));
    cudaDeviceProp prop;
    CK("cudaGetDeviceProperties", cudaGetDeviceProperties(&prop, dev));
    cc_major = prop.major; cc_minor = prop.minor; sms = prop.multiProcessorCount;
    snprintf(buf, (size_t)cap, "%s sm_%d%d %d SMs", prop.name, cc_major, cc_minor, sms);
    return LMZ_GPU_OK;
}

// What is wrong with the stream at `p` of `len` bytes as far as its first 516 bytes can
// tell (NULL = nothing): the checks lmz_rans_decode makes before it touches a state
// (lmz/native/lmzcore.c:1413-1427).
static const char *header_defect(const uint8_t *p, uint64_t len)
{
    if (len < HDR_BYTES + STATE_BYTES) return "a stream is shorter than its own header";
    if (p[0] != 'R' || p[1] != '1') return "a stream does not start with the rANS magic";
    uint32_t total = 0;
    for (const uint8_t *f = p + 4; f < p + HDR_BYTES; f += 2) total += f[0] | ((uint32_t)f[1] << 8);
    return total == PROB_SCALE ? nullptr : "a stream's frequencies do not sum to 4096";
}

API int lmz_gpu_validate(const void *streams_v, const void *off_v, unsigned nstr)
{
    const uint8_t *base = static_cast<const uint8_t *>(streams_v);
    const uint64_t *pairs = static_cast<const uint64_t *>(off_v);
    for (const uint64_t *e = pairs; e != pairs + 2 * (size_t)nstr; e += 2)
        if (const char *defect = header_defect(base + e[0], e[1])) return fail_msg(LMZ_GPU_EBADSTREAM, defect);
    return LMZ_GPU_OK;
}

API int lmz_gpu_decode_batch_dev(const void *d_hdr, const void *d_streams, const void *d_off,
                                 unsigned nstr, unsigned plane, void *d_out, void *cuda_stream,
                                 unsigned tpb)
{
    (void)tpb;  // block shape is fixed by the shared-memory layout
    if (nstr == 0) return LMZ_GPU_OK;
    if (plane == 0) return fail_msg(LMZ_GPU_EUNSUPPORTED, "plane is zero");
    int rc = device_ready();
    if (rc) return rc;
    RansArgs a{};
    a.src = (const uint8_t *)d_streams;
    a.offs = (const uint64_t *)d_off;
    a.plane = plane;
    a.njobs = nstr;
    a.dst = (uint8_t *)d_out;
    a.shared_hdr = (const uint8_t *)d_hdr;
    return launch_rans(a, (cudaStream_t)cuda_stream);
}

#include "host_rules.inl"
#include "host_pool.inl"
#include "host_batch.inl"
#include "host_io.inl"
#include "host_plan.inl"

// ------------------------------------------------------------------- additive

API int lmz_gpu_set_table_mode(int mode)
{
    if (mode != -1 && mode != T_NARROW && mode != T_COMPACT && mode != T_SOLO_WIDE && mode != T_SOLO_BYTES)
        return fail_msg(LMZ_GPU_EUNSUPPORTED,
                        "table mode must be -1 (auto), 0 or 2 (compact), 3 or 4 (a warp per stream)");
    g_force_table_mode.store(mode, std::memory_order_relaxed);
    return LMZ_GPU_OK;
}

// ---- batch encode (no counterpart in the reference's GPU library) -------------------

constexpr unsigned ENCODE_MAX_PLANE = 1u << 29;      // slot sizes stay below 2^31

API int lmz_gpu_encode_slot_bytes(unsigned plane)
{
    return plane == 0 || plane > ENCODE_MAX_PLANE ? 0 : (int)encode_slot_bytes(plane);
}

API int lmz_gpu_encode_batch_dev(const void *d_planes, unsigned nstr, unsigned plane, void *d_slots,
                                 void *d_lengths, void *cuda_stream)
{
    int rc = device_ready();
    if (rc) return rc;
    if (nstr == 0) return LMZ_GPU_OK;
    if (!d_planes || !d_slots || !d_lengths) return fail_msg(LMZ_GPU_EUNSUPPORTED, "null argument");
    if (plane == 0 || plane > ENCODE_MAX_PLANE) return fail_msg(LMZ_GPU_EUNSUPPORTED, "plane must be 1 .. 2^29 bytes");
    if ((uintptr_t)d_slots & 511u) return fail_msg(LMZ_GPU_EUNSUPPORTED, "the slot buffer must be 512-byte aligned");
    constexpr uint32_t shm = encode_smem_bytes();
    EncodeArgs a{};
    a.src = (const uint8_t *)d_planes;
    a.plane = plane;
    a.nstr = nstr;
    a.slots = (uint8_t *)d_slots;
    a.slot_bytes = encode_slot_bytes(plane);
    a.lengths = (uint32_t *)d_lengths;
    k_encode<<<(nstr + 3) / 4, 32, shm, (cudaStream_t)cuda_stream>>>(a);
    cudaError_t le = cudaGetLastError();
    if (le != cudaSuccess) return fail_cuda("launch k_encode", le);
    return LMZ_GPU_OK;
}

API int lmz_gpu_pack_streams_dev(const void *d_slots, unsigned plane, const void *d_offsets, unsigned nstr,
                                 void *d_out, void *cuda_stream)
{
    int rc = device_ready();
    if (rc) return rc;
    if (nstr == 0) return LMZ_GPU_OK;
    if (!d_slots || !d_offsets || !d_out) return fail_msg(LMZ_GPU_EUNSUPPORTED, "null argument");
    if (plane == 0 || plane > ENCODE_MAX_PLANE) return fail_msg(LMZ_GPU_EUNSUPPORTED, "plane must be 1 .. 2^29 bytes");
    k_pack_streams<<<nstr, 128, 0, (cudaStream_t)cuda_stream>>>((const uint8_t *)d_slots, encode_slot_bytes(plane),
                                                              (const uint64_t *)d_offsets, nstr, (uint8_t *)d_out);
    cudaError_t le = cudaGetLastError();
    if (le != cudaSuccess) return fail_cuda("launch k_pack_streams", le);
    return LMZ_GPU_OK;
}

// ---- chunk framing for the save path (no counterpart in the reference's GPU library) --------

static int framing_args(const void *d_src, uint64_t nbytes, unsigned chunk)
{
    if (!d_src) return fail_msg(LMZ_GPU_EUNSUPPORTED, "null argument");
    if (chunk < 2 || (chunk & 1u) || (nbytes & 1u))
        return fail_msg(LMZ_GPU_EUNSUPPORTED, "chunk size and byte count must be even (whole BF16 elements)");
    if (nbytes > (uint64_t)chunk * 0x7fffffffu) return fail_msg(LMZ_GPU_EUNSUPPORTED, "too many chunks for one call");
    return LMZ_GPU_OK;
}

API int lmz_gpu_split_bf16_dev(const void *d_src, uint64_t nbytes, unsigned chunk, void *d_planes, void *cuda_stream)
{
    int rc = device_ready();
    if (rc) return rc;
    if (nbytes == 0) return LMZ_GPU_OK;
    rc = framing_args(d_src, nbytes, chunk);
    if (rc) return rc;
    if (!d_planes) return fail_msg(LMZ_GPU_EUNSUPPORTED, "null argument");
    const unsigned nchunks = (unsigned)((nbytes + chunk - 1) / chunk);
    k_split_bf16<<<nchunks, 256, 0, (cudaStream_t)cuda_stream>>>((const uint8_t *)d_src, nbytes, chunk, (uint8_t *)d_planes);
    cudaError_t le = cudaGetLastError();
    if (le != cudaSuccess) return fail_cuda("launch k_split_bf16", le);
    return LMZ_GPU_OK;
}

API int lmz_gpu_frame_bf16_dev(const void *d_src, uint64_t nbytes, unsigned chunk, const void *d_lengths,
                               void *d_meta, const void *d_planes, const void *d_slots, const void *d_offsets,
                               void *d_out, void *cuda_stream)
{
    int rc = device_ready();
    if (rc) return rc;
    if (nbytes == 0) return LMZ_GPU_OK;
    rc = framing_args(d_src, nbytes, chunk);
    if (rc) return rc;
    if (!d_lengths || !d_meta) return fail_msg(LMZ_GPU_EUNSUPPORTED, "null argument");
    const unsigned nchunks = (unsigned)((nbytes + chunk - 1) / chunk), nfull = (unsigned)(nbytes / chunk);
    cudaStream_t cs = (cudaStream_t)cuda_stream;
    if (!d_out) {
        k_frame_decide<<<(nchunks + 127) / 128, 128, 0, cs>>>(nbytes, chunk, nchunks, (const uint32_t *)d_lengths,
                                                             (FrameMeta *)d_meta);
    } else {
        if (!d_planes || !d_slots || !d_offsets) return fail_msg(LMZ_GPU_EUNSUPPORTED, "null argument");
        const unsigned tail = (unsigned)(nbytes - (uint64_t)nfull * chunk);
        k_frame_pack<<<nchunks, 256, 0, cs>>>((const uint8_t *)d_src, nbytes, chunk, (const uint32_t *)d_lengths,
                                              (const FrameMeta *)d_meta, (const uint8_t *)d_planes,
                                              (const uint8_t *)d_slots, encode_slot_bytes(chunk / 2),
                                              tail ? encode_slot_bytes(tail / 2) : 0u, nfull,
                                              (const uint64_t *)d_offsets, (uint8_t *)d_out);
    }
    cudaError_t le = cudaGetLastError();
    if (le != cudaSuccess) return fail_cuda("launch chunk framing", le);
    return LMZ_GPU_OK;
}

API int lmz_gpu_crc32_chunks_dev(const void *d_src, uint64_t nbytes, unsigned chunk, const void *d_crc_tables,
                                 void *d_meta, void *cuda_stream)
{
    int rc = device_ready();
    if (rc) return rc;
    if (nbytes == 0) return LMZ_GPU_OK;
    if (!d_src || !d_crc_tables || !d_meta || chunk == 0) return fail_msg(LMZ_GPU_EUNSUPPORTED, "null argument");
    static bool done[64];
    constexpr uint32_t shm = 5u * (1024u << 4);       // four tables replicated 16x, and room to align them
    rc = opt_in_smem(k_crc32_chunks, shm, done);
    if (rc) return rc;
    const unsigned nchunks = (unsigned)((nbytes + chunk - 1) / chunk);
    k_crc32_chunks<<<nchunks, 256, shm, (cudaStream_t)cuda_stream>>>((const uint8_t *)d_src, nbytes, chunk,
                                                                     (const CrcTables *)d_crc_tables, (FrameMeta *)d_meta);
    cudaError_t le = cudaGetLastError();
    if (le != cudaSuccess) return fail_cuda("launch k_crc32_chunks", le);
    return LMZ_GPU_OK;
}

API int lmz_gpu_set_device(int device)
{
    int rc = device_ready();
    if (rc) return rc;
    CK("cudaSetDevice", cudaSetDevice(device));
    return LMZ_GPU_OK;
}

API int lmz_gpu_decode_streams_dev(const void *d_jobs, unsigned njobs, const void *d_src,
                                   void *d_dst, const void *d_shared_hdr, void *d_status,
                                   void *d_any_bad, void *cuda_stream)
{
    if (njobs == 0) return LMZ_GPU_OK;
    int rc = device_ready();
    if (rc) return rc;
    RansArgs a{};
    a.src = (const uint8_t *)d_src;
    a.jobs = (const StreamJob *)d_jobs;
    a.njobs = njobs;
    a.dst = (uint8_t *)d_dst;
    a.shared_hdr = (const uint8_t *)d_shared_hdr;
    a.status = (uint32_t *)d_status;
    a.any_bad = (uint32_t *)d_any_bad;
    return launch_rans(a, (cudaStream_t)cuda_stream);
}

#include "chunk_abi.inl"

// ------------------------------------------------- checked decode, no allocation

// Some hosts cannot let a plug-in allocate device memory: an inference server or
// training job whose own pool has already claimed all of HBM (cudaMalloc then fails
// or fragments the pool), or a loader that runs where the embedding framework
// forbids driver allocations.  lmz_gpu_decode_batch_dev serves them but cannot say
// whether a stream was truncated, because its per-stream verdicts need memory the
// reference's signature has no argument for.  This entry point keeps those verdicts
// in a fixed device array that is part of the library image instead.
//
// The array costs LMZ_GPU_NOALLOC_MAX_STREAMS * 4 + 256 bytes on every GPU that
// loads the library, until the process exits.  Every call on a device shares it:
// calls that overlap on the GPU (different CUDA streams, different host threads)
// race on the verdicts and must be serialised by the caller.
static __device__ __align__(256) uint32_t g_noalloc_verdicts[64 + LMZ_GPU_NOALLOC_MAX_STREAMS];

// In host code the array's name only stands for the symbol; the address a kernel
// can use comes from cudaGetSymbolAddress, per device, with that device current.
static int noalloc_scratch(uint32_t **out)
{
    static uint32_t *ptr_of[64];
    static std::mutex mu;
    int dev = 0;
    CK("cudaGetDevice", cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail_msg(LMZ_GPU_EUNSUPPORTED, "device index above 63");
    std::lock_guard<std::mutex> lock(mu);
    if (!ptr_of[dev]) {
        void *p = nullptr;
        CK("cudaGetSymbolAddress(verdicts)", cudaGetSymbolAddress(&p, g_noalloc_verdicts));
        ptr_of[dev] = static_cast<uint32_t *>(p);
    }
    *out = ptr_of[dev];
    return LMZ_GPU_OK;
}

API int lmz_gpu_decode_batch_dev_noalloc(const void *d_hdr, const void *d_streams,
                                         const void *d_off, unsigned nstr, unsigned plane,
                                         void *d_out, void *cuda_stream, uint32_t *h_status)
{
    if (nstr == 0) return LMZ_GPU_OK;
    if (plane == 0) return fail_msg(LMZ_GPU_EUNSUPPORTED, "plane is zero");
    if (nstr > LMZ_GPU_NOALLOC_MAX_STREAMS) {
        snprintf(g_err, sizeof g_err,
                 "lmz_gpu_decode_batch_dev_noalloc takes at most %u streams per call, got %u; "
                 "split the batch", (unsigned)LMZ_GPU_NOALLOC_MAX_STREAMS, nstr);
        return LMZ_GPU_EUNSUPPORTED;
    }
    int rc = device_ready();
    if (rc) return rc;
    uint32_t *scratch = nullptr;
    rc = noalloc_scratch(&scratch);          // first call on a device resolves the symbol
    if (rc) return rc;
    cudaStream_t cs = (cudaStream_t)cuda_stream;
    // the summary word keeps the previous call's value: it must start at zero
    CK("cudaMemsetAsync(verdict summary)", cudaMemsetAsync(scratch, 0, 256, cs));
    RansArgs a{};
    a.src = (const uint8_t *)d_streams;
    a.offs = (const uint64_t *)d_off;
    a.plane = plane;
    a.njobs = nstr;
    a.dst = (uint8_t *)d_out;
    a.shared_hdr = (const uint8_t *)d_hdr;
    a.status = scratch + 64;                 // every job writes its own word
    a.any_bad = scratch;
    rc = launch_rans(a, cs, /*may_alloc=*/false);
    if (rc) return rc;
    uint32_t bad = 0;
    CK("cudaMemcpyAsync(verdict summary)",
       cudaMemcpyAsync(&bad, scratch, sizeof bad, cudaMemcpyDeviceToHost, cs));
    if (h_status)
        CK("cudaMemcpyAsync(verdicts)", cudaMemcpyAsync(h_status, scratch + 64, (size_t)nstr * 4,
                                                        cudaMemcpyDeviceToHost, cs));
    CK("cudaStreamSynchronize", cudaStreamSynchronize(cs));
    if (bad) return fail_msg(LMZ_GPU_EBADSTREAM, "a stream is malformed or truncated");
    return LMZ_GPU_OK;
}
