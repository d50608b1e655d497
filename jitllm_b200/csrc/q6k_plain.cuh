// One output of a Q6_K product as a sum over single weights.
#pragma once
#include "jl_internal.cuh"

// The sum over `nsb` super-blocks of one row, each weight formed before it meets its activation, as quant.Dequant32 does
// (format/quant/dequant.go:443-470). The batch kernel multiplies codes by activations first and scales the sums: where an activation,
// a scale or such a sum is not finite the output is formed here instead.
// w: the row's resident blocks, d: their scales, x: the activations that go with them.
static __device__ __noinline__ float q6k_plain(const uint8_t *w, const uint16_t *d, const float *x, int nsb) {
    float acc = 0.f;
    for (int sb = 0; sb < nsb; sb++, w += JL_Q6K_BLOCK, x += 256) {
        const float db = __half2float(__ushort_as_half(d[sb]));
        for (int e = 0; e < 256; e++) {
            const int n = e >> 7, j = (e >> 5) & 3, l = e & 31;
            const int byte = w[n * 64 + l + (j & 1) * 32];
            const int q = (j >= 2 ? byte >> 4 : byte & 0xF) | (((w[128 + n * 32 + l] >> (2 * j)) & 3) << 4);
            const int sc = (int)(int8_t)w[192 + n * 8 + (l >> 4) + 2 * j];
            acc = fmaf(__fmul_rn(__fmul_rn(db, (float)sc), (float)(q - 32)), x[e], acc);
        }
    }
    return acc;
}
