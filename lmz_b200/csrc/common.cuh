// Shared definitions for the sm_100a lmz decode library: format constants,
// job descriptors handed over by the host, status codes, and the thin PTX
// wrappers for loads and stores by shared-space address.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "geometry.cuh"

namespace lmz {

// ---- stream format (reference: lmz/native/lmzcore.c:755-767) ---------------
constexpr uint32_t RANS_LOW = 1u << 16;
constexpr uint32_t NLANES = 8;        // interleaved states per stream
constexpr uint32_t HDR_BYTES = 516;   // 'R','1',0,0 + 256 x u16 frequencies
constexpr uint32_t STATE_BYTES = 32;  // 8 x u32 initial states

// ---- kernel geometry --------------------------------------------------------
constexpr uint32_t PAD_BYTES = 576;   // readable slack owed after the last stream

// ---- per-stream status words -------------------------------------------------
constexpr uint32_t ST_OK = 0;
constexpr uint32_t ST_BAD_HEADER = 1;   // magic, frequency sum or minimum length
constexpr uint32_t ST_OVERRUN = 2;      // a refill was needed past the stream's end
                                        // (3 is the reference's input timeout; no kernel here waits for a copy)
constexpr uint32_t ST_BAD_SHAPE = 4;    // lengths in a payload disagree with the record
constexpr uint32_t ST_BAD_CRC = 5;      // decoded chunk does not match the record's crc32
constexpr uint32_t ST_SLACK = 0x100;    // soft: final states != 2^16 or cursor != length

// One rANS stream to decode.  Written by the host planner (numpy structured
// array with the same layout) or by a device planning kernel.
struct StreamJob {
    uint64_t src_off;   // stream start, bytes from the source base
    uint64_t dst_off;   // first output byte, bytes from the destination base
    uint32_t src_len;   // stream length in bytes
    uint32_t n;         // symbols to produce
    uint32_t flags;     // STREAM_OPEN: see below
    uint32_t aux;       // written for STREAM_OPEN: how many symbols the stream's words were good for
};
// A stream whose length is not known yet, only a bound (`n`): decoded until it asks for a word it has
// not got, which a sound one does right behind its last symbol.  Running out is no failure; who
// learns the length compares it with `aux`.
constexpr uint32_t STREAM_OPEN = 1;
static_assert(sizeof(StreamJob) == 32, "StreamJob layout is shared with the host");

// ---- PTX wrappers ------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void *p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

// Bytes of dynamic shared memory this launch was given.
__device__ __forceinline__ uint32_t dynamic_smem_bytes()
{
    uint32_t v;
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(v));
    return v;
}

// Loads and stores by 32-bit shared-space address (no generic-pointer arithmetic).
__device__ __forceinline__ uint32_t lds_u32(uint32_t saddr)
{
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(saddr));
    return v;
}
__device__ __forceinline__ uint32_t lds_u8(uint32_t a)
{
    uint32_t v;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts_u8(uint32_t a, uint32_t v)
{
    asm volatile("st.shared.u8 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ uint4 lds_u128(uint32_t a)
{
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t lds_u16(uint32_t a)
{
    uint32_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts_u32(uint32_t a, uint32_t v)
{
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ uint2 lds_u64(uint32_t a)
{
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}

// Sums of products of a's bytes, or a's two halves, with constants, plus c: one instruction of the multiplier's pipe picks a
// byte or the upper half out of a word, scales it and adds it, where a shift or a permute would be the integer pipe's.
__device__ __forceinline__ uint32_t byte_mad(uint32_t a, uint32_t weights, uint32_t c)
{
    uint32_t v;
    asm("dp4a.u32.u32 %0, %1, %2, %3;" : "=r"(v) : "r"(a), "r"(weights), "r"(c));
    return v;
}
__device__ __forceinline__ uint32_t high_half_add(uint32_t a, uint32_t c)
{
    uint32_t v;
    asm("dp2a.lo.u32.u32 %0, %1, %2, %3;" : "=r"(v) : "r"(a), "r"(0x0100u), "r"(c));
    return v;
}

__device__ __forceinline__ void red_shared_add(uint32_t a, uint32_t v)
{
    asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

__device__ __forceinline__ void prefetch_l2(const void *p)
{
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// The same where `on`, without a branch.
__device__ __forceinline__ void lds_u64_if(uint32_t on, uint32_t a, uint2 &v)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t@p ld.shared.v2.u32 {%0,%1}, [%2];\n\t}"
                 : "+r"(v.x), "+r"(v.y) : "r"(a), "r"(on));
}
__device__ __forceinline__ void sts_u8_if(uint32_t on, uint32_t a, uint32_t v)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p st.shared.u8 [%0], %1;\n\t}"
                 ::"r"(a), "r"(v), "r"(on) : "memory");
}
__device__ __forceinline__ void sts_u16_if(uint32_t on, uint32_t a, uint32_t v)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p st.shared.u16 [%0], %1;\n\t}"
                 ::"r"(a), "r"(v), "r"(on) : "memory");
}
__device__ __forceinline__ void sts_u64_if(uint32_t on, uint32_t a, uint32_t x, uint32_t y)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t@p st.shared.v2.u32 [%0], {%1,%2};\n\t}"
                 ::"r"(a), "r"(x), "r"(y), "r"(on) : "memory");
}
__device__ __forceinline__ void sts_u128_if(uint32_t on, uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %5, 0;\n\t@p st.shared.v4.u32 [%0], {%1,%2,%3,%4};\n\t}"
                 ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w), "r"(on) : "memory");
}

}  // namespace lmz
