// The arithmetic of the MXFP4 decode kernels (one matrix: gemv_mxfp4.cu; a mixture layer: moe_dec.cuh).
#pragma once
#include "jl_internal.cuh"

// One warp, one 64-element span of activations (two per lane): x * 2^s = hi + lo in f16, s such that the span's largest
// magnitude sits in [2^14, 2^15) (f16 neither overflows nor flushes). Returns 2^-s.
__device__ __forceinline__ float mx_split_span(float2 v, __half2 &hi, __half2 &lo) {
    float amax = fmaxf(fabsf(v.x), fabsf(v.y));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    int sh = 14 - ((int)((__float_as_uint(amax) >> 23) & 0xFF) - 127);
    if (amax == 0.f || !(amax < __int_as_float(0x7f800000))) sh = 0;
    sh = max(-100, min(100, sh));
    const float scale = __uint_as_float((uint32_t)(127 + sh) << 23);
    const float a = v.x * scale, b = v.y * scale;
    hi = __floats2half2_rn(a, b);
    const float2 back = __half22float2(hi);
    lo = __floats2half2_rn(a - back.x, b - back.y);
    return __uint_as_float((uint32_t)(127 - sh) << 23);
}

__device__ __forceinline__ void mx_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                       uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// four codes in the HIGH nibbles of v's bytes -> the high bytes of their f16 images
__device__ __forceinline__ uint32_t mx_hbytes(uint32_t v) { return ((v & 0x70707070u) >> 3) | (v & 0x80808080u); }

// One 32-element block of 16 rows: the sums of rows g (c[0], c[1]) and g + 8 (c[2], c[3]) against the lane's two B columns.
// a, b: the lane's four code bytes of the two rows; x0, x1: elements 4t..4t+3 and 16+4t..16+4t+3 of its column.
// k-slots (2t, 2t+1 | 2t+8, 2t+9) = elements (4t, 4t+1 | 4t+2, 4t+3), then the same + 16.
__device__ __forceinline__ void mx_block(float (&c)[4], uint32_t a, uint32_t b, uint2 x0, uint2 x1) {
    const uint32_t hla = mx_hbytes(a << 4), hha = mx_hbytes(a);     // low / high nibbles of row g
    const uint32_t hlb = mx_hbytes(b << 4), hhb = mx_hbytes(b);     // ... of row g + 8
    mx_mma(c, __byte_perm(hla, 0u, 0x1404), __byte_perm(hlb, 0u, 0x1404), __byte_perm(hla, 0u, 0x3424), __byte_perm(hlb, 0u, 0x3424), x0.x, x0.y);
    mx_mma(c, __byte_perm(hha, 0u, 0x1404), __byte_perm(hhb, 0u, 0x1404), __byte_perm(hha, 0u, 0x3424), __byte_perm(hhb, 0u, 0x3424), x1.x, x1.y);
}
// 2^(e - 127) * 2^14 as an f32 (an all-zero block may carry any byte: keep the exponent field legal)
__device__ __forceinline__ float mx_block_scale(uint32_t e) { return __uint_as_float((min(e & 0xFFu, 240u) + 14u) << 23); }
