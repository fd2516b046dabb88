// Shared device/host helpers for the affine INT4 projection kernels (sm_100a only).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

// ---- status codes returned by every extern "C" entry point -------------------------------
#define MT_OK 0
#define MT_ERR_SHAPE (-1)        // shape outside what the kernels accept
#define MT_ERR_ALIGN (-2)        // pointer not aligned for the vector width the kernel uses
#define MT_ERR_FORMAT (-3)       // quantisation format other than 4-bit, group 64
#define MT_ERR_LAUNCH (-4)       // CUDA reported a launch / API error
#define MT_ERR_DEVICE (-5)       // current device is not compute capability 10.x
#define MT_ERR_NULL (-6)         // required pointer is null
#define MT_ERR_WORKSPACE (-7)    // workspace missing or too small
#define MT_ERR_DEVICE_WAIT (-8)  // a bounded device-side wait gave up (see mt_device_status)
#define MT_ERR_INDEX (-9)        // a kernel met an index outside its table (see mt_device_status)

// ---- flags word ---------------------------------------------------------------------------
#define MT_FLAG_FORCE_GEMV 0x1u   // CUDA-core GEMV regardless of row count (rows <= 8 only)
#define MT_FLAG_FORCE_UMMA 0x2u   // tcgen05 path regardless of row count
#define MT_FLAG_MLP_FUSED_MMA 0x80u  // mt_affine_mlp: insist on the warp-MMA single-launch kernel (M <= 8)
#define MT_FLAG_HOST_PAIR 0x40u    // mt_affine_mlp_host: activations and residual share one host allocation
#define MT_FLAG_MLP_FUSED 0x20u    // mt_affine_mlp: insist on the single-launch kernel (error if it does not apply)
#define MT_FLAG_FIXED_ORDER 0x100u  // tcgen05 sums in an order that does not depend on the row count (FORCE_UMMA implies it)
#define MT_FLAG_GELU 0x10u        // dense activation: x/(1+exp(-1.702x)) instead of SiLU

namespace mt {

// Device-side record of a bounded wait that gave up, or of an index outside its table: word 0 = code, 1 = block, 2 = detail.
// Written with atomicCAS so the first failure wins; zero means that there was none.
// The library is one translation unit, so the definition lives here.
__device__ unsigned int g_device_status[4] = {0, 0, 0, 0};

__device__ __forceinline__ float bf16_bits_to_f32(uint32_t bits16) { return __uint_as_float(bits16 << 16); }
__device__ __forceinline__ float bf16_lo(uint32_t pair) { return __uint_as_float(pair << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t pair) { return __uint_as_float(pair & 0xFFFF0000u); }

__device__ __forceinline__ uint16_t f32_to_bf16_bits(float v) {
    return __bfloat16_as_ushort(__float2bfloat16_rn(v));
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    return (uint32_t)f32_to_bf16_bits(lo) | ((uint32_t)f32_to_bf16_bits(hi) << 16);
}

// One packed word (8 nibbles e0..e7) -> four bf16 pairs (128+e_i, 128+e_{i+4}), i = 0..3: the nibble
// lands in the low mantissa bits of the bf16 value 128.0 (0x4300), so every value is exact.
// (x & mask) | magic as ONE lop3 (truth table 0xEA) with both constants in registers.
__device__ __forceinline__ void unpack_word_offset128(uint32_t w, uint32_t* out) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
        asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(out[i]) : "r"(w >> (4 * i)), "r"(0x000F000Fu), "r"(0x43004300u));
}

// One packed word -> four bf16 pairs ((e_i - 8) / 64, (e_{i+4} - 8) / 64), i = 0..3, exact.  Masked out, a nibble is the
// subnormal bf16 number e 2^-133 (or 16 e 2^-133), which one fma.rn.bf16x2 brings up and centres: nine instructions.
__device__ __forceinline__ void unpack_word_centred64(uint32_t w, uint32_t* out) {
    const uint32_t upper = w >> 8;
#pragma unroll
    for (int i = 0; i < 4; ++i)
        asm("{\n\t.reg .b32 t;\n\tand.b32 t, %1, %2;\n\tfma.rn.bf16x2 %0, t, %3, %4;\n\t}"
            : "=r"(out[i]) : "r"(i < 2 ? w : upper), "r"(i & 1 ? 0x00F000F0u : 0x000F000Fu),
              "r"(i & 1 ? 0x7D007D00u : 0x7F007F00u),  // 2^123, 2^127
              "r"(0xBE00BE00u));                       // -1/8
}

// The eight nibbles of a word as the floats 128+e0 .. 128+e7 (natural order).
__device__ __forceinline__ void unpack_word_f32_offset128(uint32_t w, float (&q)[8]) {
    const uint32_t even = w & 0x0F0F0F0Fu, odd = (w >> 4) & 0x0F0F0F0Fu;
    constexpr uint32_t kMagic = 0x43000000u;  // 128.0f
    q[0] = __uint_as_float(__byte_perm(even, kMagic, 0x7044));
    q[1] = __uint_as_float(__byte_perm(odd, kMagic, 0x7044));
    q[2] = __uint_as_float(__byte_perm(even, kMagic, 0x7144));
    q[3] = __uint_as_float(__byte_perm(odd, kMagic, 0x7144));
    q[4] = __uint_as_float(__byte_perm(even, kMagic, 0x7244));
    q[5] = __uint_as_float(__byte_perm(odd, kMagic, 0x7244));
    q[6] = __uint_as_float(__byte_perm(even, kMagic, 0x7344));
    q[7] = __uint_as_float(__byte_perm(odd, kMagic, 0x7344));
}

__device__ __forceinline__ float warp_sum_xor(float v) {
#pragma unroll
    for (int offset = 16; offset >= 1; offset >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, offset);
    return v;
}

// g/(1+exp(-g)) * u on un-rounded fp32 sums.
__device__ __forceinline__ float swiglu_f32(float gate, float up) { return gate / (1.0f + __expf(-gate)) * up; }

// The same for eight outputs at once, with the same bits.  A float division compiles to a fast path and a branch
// to a slow one, and eight branches in a row leave nothing to overlap: 150 cycles per output, more than a
// whole tile's multiplication takes.  Here the quotient is refined by Markstein's method (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", 1990): an approximate
// reciprocal, one Newton step on it, the quotient, its exact remainder by FMA, one correction.  That rounds as the
// division does while 1 + exp(-g) and its reciprocal are normal numbers; beyond (g below -69) all eight divide.
// The remainder is taken with the other sign, which keeps the sign of a zero.  A test compares it with the division
// over all 2^32 gates.
__device__ __forceinline__ void swiglu8_f32(const float (&gate)[8], const float (&up)[8], float (&out)[8]) {
    float d[8], largest = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        d[i] = 1.0f + __expf(-gate[i]);
        largest = fmaxf(largest, fmaxf(d[i], gate[i]));
    }
    if (largest < 1e30f) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float r0 = __fdividef(1.0f, d[i]);
            const float r = fmaf(fmaf(-d[i], r0, 1.0f), r0, r0);
            const float quotient = gate[i] * r;
            out[i] = fmaf(-fmaf(d[i], quotient, -gate[i]), r, quotient) * up[i];
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) out[i] = gate[i] / d[i] * up[i];
    }
}

inline bool aligned_to(const void* p, size_t bytes) { return (reinterpret_cast<uintptr_t>(p) % bytes) == 0; }

}  // namespace mt
