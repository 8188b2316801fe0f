// What the streaming expert kernels share (stream.cu: decode; wide.cu: blocks of rows): the order of the activations, their
// split into fp16 numbers and the unpacking of the codes for mma.sync.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace mfb {

constexpr float CODE_UNIT = 1.0f / 16777216.0f;  // 2^-24
constexpr float REST = 1.0f / 2048.0f;           // weight of the remainder


// How a lane takes codes out of a 16-byte piece of a row, and with that the order of the activations:
//   0  4-bit: word t of the piece (32 codes)
//   1  2-bit: word t of the piece (64 codes)
//   2  2-bit, scale groups of 32: the 16-bit half t of either 8-byte half of the piece
enum { L4 = 0, L2 = 1, L2H = 2 };

// Place and factor of element e (0..15) of a 16-element run.
__host__ __device__ inline uint32_t s_pos(uint32_t e, int layout) {
    if (layout == L4) return (e & 8u) | ((e & 3u) << 1) | ((e >> 2) & 1u);
    if (layout == L2) return ((e & 7u) << 1) | (e >> 3);
    return e;
}
__host__ __device__ inline float s_scale(uint32_t e, int layout) {
    const uint32_t i = e & 7u;
    const uint32_t bit = layout == L4 ? 6u : layout == L2 ? (0xDAu >> i & 1u ? 8u : 6u) : 6u + 2u * (i & 1u);   // see s_unpack4 ...
    return 1.0f / (float)(1u << bit);
}

__device__ __forceinline__ void head_and_rest(float v, __half& head, __half& rest) {
    head = __float2half_rn(v);
    rest = __float2half_rn((v - __half2float(head)) * 2048.0f);
}

// Power of two that brings a row whose largest magnitude has these bits below 2^20, and its inverse.  A row of zeros or
// denormals takes 2^126; infinities and NaN pass through any factor.
__device__ __forceinline__ float s_factor(uint32_t max_bits, float& inverse) {
    const int e = (int)min(max_bits >> 23, 254u) - 127, shift = min(19 - e, 126);
    inverse = __uint_as_float((uint32_t)(127 - shift) << 23);
    return __uint_as_float((uint32_t)(127 + shift) << 23);
}

// Whether a 16-bit row times `factor` (s_factor of its largest element) has an element that the head does not hold.  As an fp16 subnormal
// it loses the bits below 2^-24; that takes one 2^28 (bf16 rows; at 4 bits 2^30) or 2^25 (2^27) times below the largest, and of
// fp16 rows, whose own bits end at 2^-24, a largest one of 2^12 (2^14).  smallest: of those that are not zero.
__device__ __forceinline__ bool s_inexact(float smallest, float largest, float factor, int dtype, bool four) {
    if (dtype == MFB_DT_BF16) return smallest < largest * (four ? 0x1p-30f : 0x1p-28f);
    return factor < (four ? 64.0f : 256.0f) && smallest < largest * (four ? 0x1p-27f : 0x1p-25f);
}
// Then: whether it matters, and if so the row's remainders, in one or two orders, and its mark.  It does not matter beside a neighbour of
// 2^-13 of the largest, since what is lost is below 2^-24 of that one, as is what the fp32 sums over a scale group lose; a run of 32 without
// one makes a marked row.  Called by the whole block, whose first 256 threads take part; k is a multiple of 256.
template <typename Element>
__device__ __forceinline__ void s_rests(Element element, uint32_t k, float factor, float back, int layout, __half* xr_rest, int layout_s, __half* xs_rest, float* unit) {
    bool found = false;
    for (uint32_t i = threadIdx.x; i < k && threadIdx.x < 256; i += 256) {
        const float most = __uint_as_float(__reduce_max_sync(0xFFFFFFFFu, __float_as_uint(element(i)) & 0x7FFFFFFFu));
        found = found || (most != 0.0f && most * factor < 128.0f);
    }
    if (!__syncthreads_or(found)) return;
    if (threadIdx.x == 0) *unit = -back;
    for (uint32_t i = threadIdx.x; i < k && threadIdx.x < 256; i += 256) {
        const float v = element(i) * factor;
        const auto put = [&](__half* row, int l) {
            __half head, rest;
            head_and_rest(v * s_scale(i & 15u, l), head, rest);
            row[(i & ~15u) + s_pos(i & 15u, l)] = rest;
        };
        put(xr_rest, layout);
        if (xs_rest) put(xs_rest, layout_s);
    }
}

// The fixed factor of hidden rows, and the maxima it suits: below 2^11 the heads stay finite, from 2^-13 on the remainders' last bit
// (2^-37) is below fp32's of the maximum.
constexpr float HIDDEN_FACTOR = 1024.0f;
__device__ __forceinline__ bool s_plain(uint32_t max_bits) { return (max_bits >> 23) - 114u < 24u; }

__device__ __forceinline__ uint32_t s_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
template <int BYTES>
__device__ __forceinline__ void s_copy(uint32_t dst, const void* src) {
    if (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
// Sixteen bytes with a cache hint (l2_policy).
__device__ __forceinline__ void s_copy(uint32_t dst, const void* src, uint64_t policy) {
    asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "l"(policy) : "memory");
}
// Loads from shared memory at 32-bit addresses: an address is a register and a constant.
__device__ __forceinline__ uint4 s_load128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ uint2 s_load64(uint32_t a) {
    uint2 v;
    asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t s_load32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t s_load16(uint32_t a) {
    uint16_t v;
    asm volatile("ld.shared.b16 %0, [%1];" : "=h"(v) : "r"(a));
    return v;
}
// Two fp32 numbers at a time, each rounded as by the scalar instructions.
__device__ __forceinline__ uint64_t s_pair(float a, float b) { return (uint64_t)__float_as_uint(b) << 32 | __float_as_uint(a); }
__device__ __forceinline__ float2 s_unpair(uint64_t v) { return make_float2(__uint_as_float((uint32_t)v), __uint_as_float((uint32_t)(v >> 32))); }
__device__ __forceinline__ uint64_t s_fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t s_mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t s_add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ void s_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <int SDT>
__device__ __forceinline__ float s_widen(uint32_t packed, int i) {   // i-th 16-bit half
    if (SDT == MFB_DT_BF16) return __uint_as_float(i ? (packed & 0xFFFF0000u) : (packed << 16));
    const __half2 h = *reinterpret_cast<const __half2*>(&packed);
    return i ? __high2float(h) : __low2float(h);
}

// Registers of one word: pairs of codes as fp16 subnormals.  Every code lies at bit 6 or 8 of the mantissa: the tensor core lines
// products up by the exponents of the operands as they stand, and every subnormal has the same one, so a code at bit 0 cost
// its sum ten bits (rows of 4096 two-bit codes: 7e-6 off the 64-bit sum, now 2.3e-7; the fp32 kernels in decode.cu
// 2.8e-7).  What bounds the kernels is the pipe that masks and shifts, so shifts to the left are made as products, which
// another pipe takes; mul = {4, 64} is opaque to the compiler, which would turn constants back into shifts.  Against codes where
// they lie (one shift per word): eight layers of 64 rows 1126 -> 1211 us, of 8 rows 441 -> 476, two layers of 13 rows of
// the 2-bit family 395 -> 412.  Products that shift to the right (mul.hi): 1349, 510, 457.
__device__ __forceinline__ uint32_t s_mul(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.lo.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ void s_unpack4(uint32_t w, const uint32_t (&m)[2], uint32_t (&p)[4]) {
    constexpr uint32_t B6 = 0x03C003C0u;
    p[0] = s_mul(w, m[1]) & B6; p[1] = s_mul(w, m[0]) & B6; p[2] = (w >> 2) & B6; p[3] = (w >> 6) & B6;
}
__device__ __forceinline__ void s_unpack2(uint32_t w, const uint32_t (&m)[2], uint32_t (&p)[8]) {
    constexpr uint32_t B6 = 0x00C000C0u, B8 = 0x03000300u;
    const uint32_t l6 = s_mul(w, m[1]), l2 = s_mul(w, m[0]), r4 = w >> 4;
    p[0] = l6 & B6; p[1] = l6 & B8; p[2] = l2 & B6; p[3] = l2 & B8;
    p[4] = w & B8; p[5] = r4 & B6; p[6] = r4 & B8; p[7] = (w >> 6) & B8;
}
__device__ __forceinline__ void s_unpack2h(uint32_t half, uint32_t (&p)[4]) {
    constexpr uint32_t B = 0x030000C0u;
    const uint32_t w = half * 0x10001u;
    p[0] = (half * 0x400040u) & B; p[1] = (half * 0x40004u) & B; p[2] = (w >> 2) & B; p[3] = (w >> 6) & B;
}

}  // namespace mfb
