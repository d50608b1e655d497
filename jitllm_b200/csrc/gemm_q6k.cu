// Q6_K for batches (9 tokens and more): out[tok][row] = sum_k W[row][k] x[tok][k] on the integer tensor cores.
//
// A Q6_K weight is d * sc * (q - 32): an integer w = sc (q - 32) of at most 13 bits times the super-block's f16 d. The row
// kernel serves it with f32 weights and f32 activations, and at 203 tokens of 4096 x 14336 that is 3.4 ms of FP32 FMAs
// (7 TFLOP/s); this kernel takes 146 us (163 TFLOP/s), activation planes included. Both sides are integers and nothing
// is rounded inside a super-block:
//
//   weights      w = 256 h + l, both signed bytes (|w| <= 4096): two int8 operands.
//   activations  per (token, super-block) a power-of-two scale takes the largest magnitude into [2^29, 2^30); the rounded
//                32-bit integer is four signed bytes x0 (top) .. x3. An element within 2^-7 of the largest is held
//                exactly, every other one to 2^-30 of the largest.
//   products     tcgen05.mma.kind::i8, s32 accumulators in TMEM, exact, all eight digit products. The four byte planes of
//                G tokens are the N = 4 G columns of one operand, [x0 | x1 | x2 | x3]; h and l multiply it into an
//                accumulator each (8 G columns of TMEM). Column block c of h and c - 1 of l weigh the same, 2^(32 - 8 c).
//   drain        once per super-block: integer shifts-and-adds and three conversions join the eight sums, one FMA adds
//                them, times d and 1/scale, to the token's f32 accumulator in registers. 56 such additions per output
//                at k = 14336.
//
// A super-block where fewer than a quarter of a token's elements that are not zero lie within 2^-8 of its largest (one activation a
// few hundred times the others) is not multiplied here: a row whose weight is zero at the large element sums the small
// ones alone, and 2^-30 of the largest is then more than f32 sums would lose. Neither is one whose largest magnitude is below
// 2^-80 (d over the scale would be denormal) or not finite. The prep kernel leaves its planes zero and marks it, and the CTA adds it
// at its end in f32 (q6g_apart). Against float64, 4096-wide rows of activations of one size: 6e-8 to 8e-8 (the row kernel 1e-7, an
// f32 FMA chain 2e-7); with one element in 256 up to 1e6 times the others and met by zero weights 1.1e-7. (Without
// l x3 and the marks: 4.8e-7 at 100 times, 9e-6 there where the scales are small.)
//
// Work split: a CTA is 128 rows x T tokens (T = 16, 24 .. 64) x a slice of the super-blocks. Up to 32 tokens are one group whose
// two accumulator pairs alternate by super-block; more are two groups of up to 32 with a pair each, and one group drains while the
// other multiplies (the four k-steps of h before those of l: alternating between the accumulators took 203 tokens from 146 to
// 183 us). The slices of a tile are the CTAs of one thread-block cluster, which add their f32 tiles in rank order through
// distributed shared memory (bit-stable; nothing is waited for but the cluster barrier). Roles: warps 0..3 drain, warp 4 copies the activation planes (untiled bulk
// copies: the prep kernel writes them as the swizzled shared-memory image), warp 5 issues the MMAs, warps 6..13 make the
// weight operands, 16 rows x 2 runs of 16 codes a warp, half a super-block (128 k) per stage.
//
// An output that comes out infinite or NaN is formed again weight by weight (q6k_plain.cuh).
#include "q6k_plain.cuh"
#include "tc5.cuh"
#include <cooperative_groups.h>
namespace cg = cooperative_groups;

#define Q6G_ROWS 128
#define Q6G_A_BYTES (Q6G_ROWS * 128)      // one int8 operand of half a super-block: 128 rows x 128 k
#define Q6G_STAGES 3
#define Q6G_THREADS 448
#define Q6G_RED_STRIDE (Q6G_ROWS + 4)

// ------------------------------------------------------------------ activations

// One warp per (super-block, token of the padded batch); lane l converts elements 8 l .. 8 l + 7.
__global__ void __launch_bounds__(256)
q6k_xprep_kernel(const float *__restrict__ X, uint8_t *__restrict__ planes, float *__restrict__ inv, int nsb, int ntok, int T, int G0) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int lane = threadIdx.x & 31, sb = blockIdx.x;
    const int tok = blockIdx.y * 8 + (threadIdx.x >> 5);         // the padded token count is a multiple of 8
    const int tt = tok / T, t = tok - tt * T;
    float v[8];
    uint32_t amax = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = 0.f;
    if (tok < ntok) {
        const float4 *src = reinterpret_cast<const float4 *>(X + ((size_t)tok * nsb + sb) * 256) + lane * 2;
        const float4 a = __ldg(src), b = __ldg(src + 1);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
#pragma unroll
        for (int i = 0; i < 8; i++) amax = max(amax, __float_as_uint(v[i]) & 0x7FFFFFFFu);   // orders NaN above infinity
    }
    amax = __reduce_max_sync(0xffffffffu, amax);
    // marked (see above): not finite, all below 2^-80, or too wide a range for the integers
    const float near = __uint_as_float(amax) * 0.00390625f;
    int count = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) count += (v[i] != 0.f) | (fabsf(v[i]) >= near) << 16;
    count = __reduce_add_sync(0xffffffffu, count);
    const bool apart = amax >= 0x7F800000u || (amax != 0u && amax < (47u << 23)) || 4 * (count >> 16) < (count & 0xFFFF);
    const int p = min(126, 29 - ((int)(amax >> 23) - 127));      // largest magnitude in [2^29, 2^30)
    const float scale = __uint_as_float((uint32_t)(127 + p) << 23);
    uint32_t u[8];
#pragma unroll
    for (int i = 0; i < 8; i++)      // byte j of u is digit j + 128
        u[i] = (uint32_t)(apart ? 0 : __float2int_rn(v[i] * scale)) + 0x80808080u;
    if (lane == 0)
        inv[((size_t)tt * nsb + sb) * T + t] = apart ? -1.f : __uint_as_float((uint32_t)(127 - p) << 23);
    // image of half a super-block: the groups one after the other, each 4 G rows (plane c, token of the group) of 128 bytes,
    // 16-byte chunks swizzled by the row (a multiple of 8 in front of every plane)
    const int G = t < G0 ? G0 : T - G0, row0 = t < G0 ? t : 4 * G0 + t - G0;
    const int half = lane >> 4, chunk = (lane & 15) >> 1;
    uint8_t *img = planes + (((size_t)tt * nsb + sb) * 2 + half) * (size_t)(T * 512) + (((uint32_t)chunk ^ (uint32_t)(t & 7)) << 4) + (lane & 1) * 8;
#pragma unroll
    for (int c = 0; c < 4; c++) {    // plane c = byte 3 - c
        const uint32_t s2 = (uint32_t)(3 - c) | (uint32_t)(7 - c) << 4;
        const uint32_t lo = __byte_perm(__byte_perm(u[0], u[1], s2), __byte_perm(u[2], u[3], s2), 0x5410);
        const uint32_t hi = __byte_perm(__byte_perm(u[4], u[5], s2), __byte_perm(u[6], u[7], s2), 0x5410);
        *reinterpret_cast<uint2 *>(img + (size_t)(c * G + row0) * 128) = make_uint2(lo ^ 0x80808080u, hi ^ 0x80808080u);
    }
}

// ------------------------------------------------------------------------- GEMM

struct q6g_params {
    int nrows, nsb, ntok, slices;
    const uint8_t *w;            // [row][nsb][208]
    const uint16_t *d;           // [row][nsb]
    const float *x;              // [ntok][k]
    const uint8_t *planes;
    const float *inv;            // [token tile][nsb][T]
    float *out;                  // [ntok][nrows]
    int *status;
};

template <int G0, int G1>
struct q6g_smem {
    static constexpr int T = G0 + G1;
    static constexpr int B_BYTES = T * 512;                            // the four planes
    static constexpr int STAGE = 2 * Q6G_A_BYTES + B_BYTES;            // h, l, planes
    static constexpr int BAR_OFS = Q6G_STAGES * STAGE;                 // full[3] empty[3] acc_full[2] acc_empty[2]
    static constexpr int INV_OFS = BAR_OFS + (2 * Q6G_STAGES + 4) * 8; // [4 warps][T] 1 / scale of the drained super-block
    static constexpr int MISC_OFS = INV_OFS + 4 * T * 4;
    static constexpr int TOTAL = MISC_OFS + 16 + 1024;
    static_assert(32768 + 16 * Q6G_ROWS * 4 + T * Q6G_ROWS * 4 + T * 1024 + (T + 1) * 4 <= BAR_OFS, "the marked super-blocks' operands reuse the stages");
    static constexpr int PAIR1 = 8 * G0;                               // columns of the first accumulator pair, where the second begins
    static constexpr int NEED = PAIR1 + 8 * (G1 ? G1 : G0);
    static constexpr int COLS = NEED <= 128 ? 128 : (NEED <= 256 ? 256 : 512);
    static_assert(G0 % 8 == 0 && G1 % 8 == 0 && G1 <= G0 && NEED <= 512 && STAGE % 1024 == 0, "operands start on swizzle atoms, accumulators fit TMEM");
};

__device__ __forceinline__ void q6g_mma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Instruction descriptor, kind::i8: D s32, A and B signed, both K-major.
__host__ __device__ constexpr uint32_t q6g_idesc(int m, int n) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// The sums of one group of tokens: h at columns ta .. ta + 4 G, l behind them.
template <int G>
__device__ __forceinline__ void q6g_drain(uint32_t ta, float d, const float *minv, float *acc) {
#pragma unroll
    for (int t0 = 0; t0 < G; t0 += 8) {
        int hi[8];
        {
            uint32_t h0[8], h1[8], l0[8];
            tc5_ld8(ta + t0, h0);
            tc5_ld8(ta + G + t0, h1);
            tc5_ld8(ta + 4 * G + t0, l0);
            tc5_wait_ld();
#pragma unroll
            for (int t = 0; t < 8; t++) hi[t] = (int)h0[t] * 256 + ((int)h1[t] + (int)l0[t]);      // |h0| < 2^18.1, |h1 + l0| < 2^21.4
        }
        int lo2[8];
        {
            uint32_t h2[8], l1[8];
            tc5_ld8(ta + 2 * G + t0, h2);
            tc5_ld8(ta + 5 * G + t0, l1);
            tc5_wait_ld();
#pragma unroll
            for (int t = 0; t < 8; t++) lo2[t] = ((int)h2[t] + (int)l1[t]) * 256;                  // the sum < 2^22.2
        }
        uint32_t h3[8], l2[8], l3[8];
        tc5_ld8(ta + 3 * G + t0, h3);
        tc5_ld8(ta + 6 * G + t0, l2);
        tc5_ld8(ta + 7 * G + t0, l3);
        tc5_wait_ld();
#pragma unroll
        for (int t = 0; t < 8; t++) {
            const int lo = lo2[t] + ((int)h3[t] + (int)l2[t]);                                     // likewise
            const float v = fmaf((float)hi[t], 65536.f, fmaf((float)(int)l3[t], 0.00390625f, (float)lo));
            acc[t0 + t] = fmaf(v, d * minv[t0 + t], acc[t0 + t]);
        }
    }
}

// What the marked (token, super-block) pairs of a CTA's tile add, by all its threads once the stages are free: per super-block the
// 128 rows' codes as signed bytes (word i of row r: elements 4 i .. 4 i + 3), the marked tokens' activations beside them, and
// a warp takes 32 rows x 8 tokens at a time. Sums as in the row kernel: 16 products, times d sc, 16 of those, added to the
// tile's f32 sums in sum[t][row]. 203 tokens of 4096 x 14336 with every pair marked take 2.5 ms (the row kernel
// 3.4), with one super-block of every token 220 us.
#define Q6G_APART_WARPS (Q6G_THREADS / 32)
#define Q6G_SUM_OFS (32768 + 16 * Q6G_ROWS * 4)
static __device__ __noinline__ void q6g_apart(const q6g_params &p, uint8_t *smem, int T, int rt, int tt, int sb0, int sb1) {
    uint32_t *codes = reinterpret_cast<uint32_t *>(smem);                       // [64][128]
    float *dsc = reinterpret_cast<float *>(smem + 32768);                       // [16][128]
    float *sum = reinterpret_cast<float *>(smem + Q6G_SUM_OFS);                 // [T][128]
    float *xs = sum + T * Q6G_ROWS;                                             // [marked][256]
    int *list = reinterpret_cast<int *>(xs + T * 256);                          // [T] the marked tokens, [T] their number
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int sb = sb0; sb < sb1; sb++) {
        __syncthreads();                                                        // the last super-block's operands are read
        if (warp == 0) {
            const float *inv = p.inv + ((size_t)tt * p.nsb + sb) * T;
            int n = 0;
            for (int t0 = 0; t0 < T; t0 += 32) {
                const bool m = t0 + lane < T && __ldg(inv + t0 + lane) < 0.f;
                const uint32_t mask = __ballot_sync(0xffffffffu, m);
                if (m) list[n + __popc(mask & ((1u << lane) - 1))] = t0 + lane;
                n += __popc(mask);
            }
            if (lane == 0) list[T] = n;
        }
        __syncthreads();
        const int n = list[T];
        if (n == 0) continue;
        for (int i = tid; i < Q6G_ROWS * 16; i += Q6G_THREADS) {                // a run of 16 codes of a row
            const int row = i % Q6G_ROWS, r = i / Q6G_ROWS, h = r >> 3, j = (r >> 1) & 3, l = (r & 1) * 16;
            const size_t b = (size_t)min(rt * Q6G_ROWS + row, p.nrows - 1) * p.nsb + sb;
            const uint8_t *blk = p.w + b * JL_Q6K_BLOCK;
            const uint4 L = ldg_nc16(blk + h * 64 + (j & 1) * 32 + l), H = ldg_nc16(blk + 128 + h * 32 + l);
            const uint32_t lw[4] = {L.x, L.y, L.z, L.w}, hw[4] = {H.x, H.y, H.z, H.w};
#pragma unroll
            for (int q = 0; q < 4; q++)
                codes[(r * 4 + q) * Q6G_ROWS + row] = ((lw[q] >> (4 * (j >> 1))) & 0x0F0F0F0Fu) | (((hw[q] >> (2 * j)) & 0x03030303u) << 4);
            dsc[r * Q6G_ROWS + row] = __half2float(__ushort_as_half(__ldg(p.d + b))) * (float)(int)(int8_t)__ldg(blk + 192 + r);
        }
        for (int i = tid; i < n * 64; i += Q6G_THREADS)
            reinterpret_cast<float4 *>(xs)[i] = __ldg(reinterpret_cast<const float4 *>(p.x + ((size_t)(tt * T + list[i >> 6]) * p.nsb + sb) * 256) + (i & 63));
        __syncthreads();
        for (int task = warp; task < 4 * ((n + 7) / 8); task += Q6G_APART_WARPS) {
            const int row = (task & 3) * 32 + lane, m0 = (task >> 2) * 8;
            float acc[8];
#pragma unroll
            for (int t = 0; t < 8; t++) acc[t] = 0.f;
            for (int r = 0; r < 16; r++) {
                float2 g[8];
#pragma unroll
                for (int t = 0; t < 8; t++) g[t] = make_float2(0.f, 0.f);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const uint32_t c4 = codes[(r * 4 + q) * Q6G_ROWS + row];
                    float w[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) w[e] = __uint_as_float(__byte_perm(c4, 0x4B000000u, 0x7650 + e)) - 8388640.f;
#pragma unroll
                    for (int t = 0; t < 8; t++) {
                        const float4 x = reinterpret_cast<const float4 *>(xs)[min(m0 + t, n - 1) * 64 + r * 4 + q];
                        g[t].x = fmaf(w[0], x.x, g[t].x); g[t].y = fmaf(w[1], x.y, g[t].y);
                        g[t].x = fmaf(w[2], x.z, g[t].x); g[t].y = fmaf(w[3], x.w, g[t].y);
                    }
                }
                const float s = dsc[r * Q6G_ROWS + row];
#pragma unroll
                for (int t = 0; t < 8; t++) acc[t] = fmaf(g[t].x + g[t].y, s, acc[t]);
            }
#pragma unroll
            for (int t = 0; t < 8; t++)
                if (m0 + t < n) sum[list[m0 + t] * Q6G_ROWS + row] += acc[t];   // this task's alone
        }
    }
    __syncthreads();
}

template <int G0, int G1>
__global__ void __launch_bounds__(Q6G_THREADS, 1) gemm_q6k_kernel(const q6g_params p) {
    using L = q6g_smem<G0, G1>;
    constexpr int T = G0 + G1;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t sbase = smem_u32(smem), bars = sbase + L::BAR_OFS;
    const uint32_t full = bars, empty = bars + 8 * Q6G_STAGES, acc_full = bars + 16 * Q6G_STAGES, acc_empty = acc_full + 16;
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(smem + L::MISC_OFS);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + L::MISC_OFS + 4);
    volatile int *apart = reinterpret_cast<volatile int *>(smem + L::MISC_OFS + 12);      // some pair of the tile is marked
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rt = blockIdx.x / p.slices, slice = blockIdx.x - rt * p.slices, tt = blockIdx.y;
    const int sb0 = (int)((long long)slice * p.nsb / p.slices), sb1 = (int)((long long)(slice + 1) * p.nsb / p.slices);
    const int nmine = sb1 - sb0;          // at least 1: slices <= nsb

    if (tid == 0) {
        for (int s = 0; s < Q6G_STAGES; s++) {
            mbar_init(full + 8 * s, 9);           // eight weight warps and the activation copy
            mbar_init(empty + 8 * s, 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(acc_full + 8 * i, 1);
            mbar_init(acc_empty + 8 * i, 4);
        }
        abort_flag[0] = 0;
        abort_flag[1] = p.status[1];
        *apart = 0;
        mbar_init_fence();
    }
    if (warp == 5) tc5_alloc(smem_u32(const_cast<uint32_t *>(tmem_slot)), L::COLS);
    tc5_fence_before();
    __syncthreads();
    tc5_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    float acc[T];
    if (warp == 4) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        if (lane == 0) {
            const uint8_t *src = p.planes + ((size_t)tt * p.nsb + sb0) * 2 * L::B_BYTES;
            for (int i = 0; i < 2 * nmine; i++) {
                const uint32_t s = i % Q6G_STAGES, ph = (i / Q6G_STAGES) & 1;
                if (i >= Q6G_STAGES && !tc5_wait(empty + 8 * s, ph ^ 1, abort_flag)) break;
                mbar_arrive_expect_tx(full + 8 * s, L::B_BYTES);
                bulk_load_1d(sbase + s * L::STAGE + 2 * Q6G_A_BYTES, src + (size_t)i * L::B_BYTES, L::B_BYTES, full + 8 * s);
            }
        }
    } else if (warp == 5) {
        const bool leader = tc5_elect();
        const uint32_t tbase = (uint32_t)tc5_uniform((int)tmem_base), sb_u = (uint32_t)tc5_uniform((int)sbase);
        bool ok = true;
        for (int i = 0; i < 2 * nmine; i++) {
            const uint32_t s = i % Q6G_STAGES, ph = (i / Q6G_STAGES) & 1;
            const int sbi = i >> 1;
            const uint32_t st = sb_u + s * L::STAGE;
            const uint64_t ah = tc5_smem_desc(st), al = tc5_smem_desc(st + Q6G_A_BYTES);
#pragma unroll
            for (int g = 0; g < (G1 ? 2 : 1); g++) {
                // the pair's use u: one group alternates between two pairs, of two groups each has its own
                const int pair = G1 ? g : sbi & 1, u = G1 ? sbi : sbi >> 1;
                const int n = 4 * (g ? G1 : G0);
                if (ok && !(i & 1) && u) ok = __all_sync(0xffffffffu, tc5_wait(acc_empty + 8 * pair, (u & 1) ^ 1, abort_flag));
                if (ok && g == 0) ok = __all_sync(0xffffffffu, tc5_wait(full + 8 * s, ph, abort_flag));
                if (!ok) break;
                tc5_fence_after();
                if (leader) {
                    const uint32_t idesc = q6g_idesc(Q6G_ROWS, n), dh = tbase + pair * L::PAIR1, dl = dh + n;
                    const uint64_t bx = tc5_smem_desc(st + 2 * Q6G_A_BYTES + (g ? G0 * 512 : 0));
#pragma unroll
                    for (int j = 0; j < 4; j++) q6g_mma(dh, ah + 2 * j, bx + 2 * j, idesc, ((i & 1) | j) != 0);     // 32 bytes of k each
#pragma unroll
                    for (int j = 0; j < 4; j++) q6g_mma(dl, al + 2 * j, bx + 2 * j, idesc, ((i & 1) | j) != 0);
                    if (i & 1) tc5_commit(acc_full + 8 * pair);
                }
                __syncwarp();
            }
            if (!ok) break;
            if (leader) tc5_commit(empty + 8 * s);
            __syncwarp();
        }
    } else if (warp >= 6) {
        // lane: row r of the warp's 16, run j (16 positions) of each half
        const int r = (warp - 6) * 16 + (lane & 15), j = lane >> 4;
        const size_t row = (size_t)min(rt * Q6G_ROWS + r, p.nrows - 1);
        const uint8_t *wrow = p.w + (row * p.nsb + sb0) * JL_Q6K_BLOCK;
        const uint32_t swz = (uint32_t)(r & 7);
        // codes of half n of the next super-block; requested after the fence of the same half, since a proxy fence waits for the
        // thread's loads in flight (in front of it they put a DRAM round trip into every stage)
        uint4 A[2], B[2], H[2];
        uint2 S[2];
        auto fetch = [&](int sbi, int n) {
            const uint8_t *blk = wrow + (size_t)sbi * JL_Q6K_BLOCK;
            A[n] = ldg_nc16(blk + n * 64 + 16 * j);
            B[n] = ldg_nc16(blk + n * 64 + 32 + 16 * j);
            H[n] = ldg_nc16(blk + 128 + n * 32 + 16 * j);
            S[n] = __ldg(reinterpret_cast<const uint2 *>(blk + 192 + n * 8));
        };
        fetch(0, 0);
        fetch(0, 1);
        bool ok = true;
        for (int sbi = 0; sbi < nmine && ok; sbi++) {
#pragma unroll
            for (int n = 0; n < 2; n++) {
                const int i = 2 * sbi + n;
                const uint32_t s = i % Q6G_STAGES, ph = (i / Q6G_STAGES) & 1;
                if (i >= Q6G_STAGES) ok = __all_sync(0xffffffffu, tc5_wait(empty + 8 * s, ph ^ 1, abort_flag));
                if (!ok) break;
                const uint32_t la[4] = {A[n].x, A[n].y, A[n].z, A[n].w}, lb[4] = {B[n].x, B[n].y, B[n].z, B[n].w};
                const uint32_t lh[4] = {H[n].x, H[n].y, H[n].z, H[n].w};
                uint8_t *dst = smem + s * L::STAGE + r * 128;
#pragma unroll
                for (int c = 0; c < 4; c++) {     // elements c * 32 + 16 j .. + 15 of the half: 16-byte chunk 2 c + j
                    const int sc = (int)(int8_t)((c < 2 ? S[n].x : S[n].y) >> (16 * (c & 1) + 8 * j));
                    // 16-bit lanes: sc q - 32 sc + 32896 = w + 128 * 257 lies in (0, 65536), so the two products of a word do
                    // not borrow from each other, and its bytes are h + 128 and l + 128
                    const uint32_t bias = (uint32_t)(32896 - 32 * sc) * 0x10001u;
                    uint32_t hw[4], lw[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const uint32_t l4 = (c & 1) ? lb[q] : la[q];
                        const uint32_t h4 = c == 0 ? lh[q] << 4 : c == 1 ? lh[q] << 2 : c == 2 ? lh[q] : lh[q] >> 2;
                        const uint32_t c4 = ((c < 2 ? l4 : l4 >> 4) & 0x0F0F0F0Fu) | (h4 & 0x30303030u);
                        const uint32_t e = (c4 & 0x00FF00FFu) * (uint32_t)sc + bias;
                        const uint32_t o = ((c4 >> 8) & 0x00FF00FFu) * (uint32_t)sc + bias;
                        hw[q] = __byte_perm(e, o, 0x7351) ^ 0x80808080u;
                        lw[q] = __byte_perm(e, o, 0x6240) ^ 0x80808080u;
                    }
                    const uint32_t ofs = ((uint32_t)(2 * c + j) ^ swz) << 4;
                    *reinterpret_cast<uint4 *>(dst + ofs) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
                    *reinterpret_cast<uint4 *>(dst + Q6G_A_BYTES + ofs) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
                }
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(full + 8 * s);
                if (sbi + 1 < nmine) fetch(sbi + 1, n);
            }
        }
    } else {
        asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll
        for (int t = 0; t < T; t++) acc[t] = 0.f;
        const int row = rt * Q6G_ROWS + warp * 32 + lane;
        const uint16_t *drow = p.d + (size_t)min(row, p.nrows - 1) * p.nsb + sb0;
        const float *inv = p.inv + ((size_t)tt * p.nsb + sb0) * T;
        float *minv = reinterpret_cast<float *>(smem + L::INV_OFS) + warp * T;
        bool marked = false;
        constexpr int PER = (T + 31) / 32;
        float inext[PER];
        uint16_t dnext = __ldg(drow);
#pragma unroll
        for (int i = 0; i < PER; i++) inext[i] = lane + 32 * i < T ? __ldg(inv + lane + 32 * i) : 0.f;
        for (int i = 0; i < nmine; i++) {
            const float d = __half2float(__ushort_as_half(dnext)) * 256.f;      // the last column block weighs 2^8
            __syncwarp();
#pragma unroll
            for (int q = 0; q < PER; q++) {
                marked |= inext[q] < 0.f;
                if (lane + 32 * q < T) minv[lane + 32 * q] = fmaxf(inext[q], 0.f);
            }
            __syncwarp();
            if (i + 1 < nmine) {
                dnext = __ldg(drow + i + 1);
#pragma unroll
                for (int q = 0; q < PER; q++)
                    if (lane + 32 * q < T) inext[q] = __ldg(inv + (size_t)(i + 1) * T + lane + 32 * q);
            }
            bool ok = true;
#pragma unroll
            for (int g = 0; g < (G1 ? 2 : 1); g++) {
                const int pair = G1 ? g : i & 1, u = G1 ? i : i >> 1;
                ok = __all_sync(0xffffffffu, tc5_wait(acc_full + 8 * pair, u & 1, abort_flag));
                if (!ok) break;
                tc5_fence_after();
                const uint32_t ta = tmem_base + pair * L::PAIR1 + ((uint32_t)(warp * 32) << 16);
                if (g == 0) q6g_drain<G0>(ta, d, minv, acc);
                else q6g_drain<G1 ? G1 : 8>(ta, d, minv + G0, acc + (G1 ? G0 : 0));
                tc5_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty + 8 * pair);
            }
            if (!ok) break;
        }
        if (marked) *apart = 1;
    }

    tc5_fence_before();
    __syncthreads();             // every MMA of this CTA has been drained (or the CTA has given up): the stages are free
    if (tid == 0 && *abort_flag) atomicExch(p.status, 2);
    if (warp == 5) {
        tc5_fence_after();
        tc5_dealloc(tmem_base, L::COLS);
    }
    // the rare ends, on the sums in shared memory: marked super-blocks, then outputs that are not finite
    float *sum = reinterpret_cast<float *>(smem + Q6G_SUM_OFS) + (warp & 3) * 32 + lane;
    if (*apart && *abort_flag == 0) {
        if (warp < 4)
#pragma unroll
            for (int t = 0; t < T; t++) sum[t * Q6G_ROWS] = acc[t];
        q6g_apart(p, smem, T, rt, tt, sb0, sb1);
#pragma unroll
        for (int t = 0; t < T; t++) acc[t] = sum[t * Q6G_ROWS];      // (in every warp, so that none has to keep its own across the call)
    }
    if (warp < 4) {
        const int row = rt * Q6G_ROWS + warp * 32 + lane;
        bool finite = true;
#pragma unroll
        for (int t = 0; t < T; t++) finite &= fabsf(acc[t]) < __int_as_float(0x7f800000);
        if (!finite && row < p.nrows) {
#pragma unroll
            for (int t = 0; t < T; t++) sum[t * Q6G_ROWS] = acc[t];
#pragma unroll 1
            for (int t = 0; t < T && tt * T + t < p.ntok; t++)
                if (!(fabsf(sum[t * Q6G_ROWS]) < __int_as_float(0x7f800000)))
                    sum[t * Q6G_ROWS] = q6k_plain(p.w + ((size_t)row * p.nsb + sb0) * JL_Q6K_BLOCK, p.d + (size_t)row * p.nsb + sb0,
                                                  p.x + ((size_t)(tt * T + t) * p.nsb + sb0) * 256, nmine);
#pragma unroll
            for (int t = 0; t < T; t++) acc[t] = sum[t * Q6G_ROWS];
        }
        if (p.slices == 1) {
#pragma unroll
            for (int t = 0; t < T; t++)
                if (row < p.nrows && tt * T + t < p.ntok) p.out[(size_t)(tt * T + t) * p.nrows + row] = acc[t];
        }
    }
    __syncthreads();             // those sums are read: the stages take the partial tile
    if (p.slices > 1) {
        cg::cluster_group cluster = cg::this_cluster();
        float *red = reinterpret_cast<float *>(smem);          // [T][Q6G_RED_STRIDE]
        if (warp < 4) {
#pragma unroll
            for (int t = 0; t < T; t++) red[t * Q6G_RED_STRIDE + warp * 32 + lane] = acc[t];
        }
        cluster.sync();
        const int ntok = min(T, p.ntok - tt * T), nvec = ntok * (Q6G_ROWS / 4);
        const int per = (nvec + p.slices - 1) / p.slices, e1 = min(nvec, (slice + 1) * per);
        const float4 *peer[8];
#pragma unroll
        for (int q = 0; q < 8; q++) peer[q] = reinterpret_cast<const float4 *>(cluster.map_shared_rank(red, q < p.slices ? q : 0));
        for (int e = slice * per + tid; e < e1; e += Q6G_THREADS) {
            const int t = e / (Q6G_ROWS / 4), r4 = e - t * (Q6G_ROWS / 4);
            float4 v[8];
#pragma unroll
            for (int q = 0; q < 8; q++)
                if (q < p.slices) v[q] = peer[q][t * (Q6G_RED_STRIDE / 4) + r4];
            float4 sum = v[0];
#pragma unroll
            for (int q = 1; q < 8; q++)
                if (q < p.slices) { sum.x += v[q].x; sum.y += v[q].y; sum.z += v[q].z; sum.w += v[q].w; }
            const float o[4] = {sum.x, sum.y, sum.z, sum.w};
            const int row = rt * Q6G_ROWS + 4 * r4;
            float *dst = p.out + (size_t)(tt * T + t) * p.nrows + row;
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (row + q < p.nrows) dst[q] = o[q];
        }
        cluster.sync();          // no CTA leaves while its tile is being read
    }
}

// ------------------------------------------------------------------------- host

// Tokens of a tile: the batch over the fewest tiles of 64 (8 T columns are all of TMEM there), rounded up to 8. Shared memory is
// what bounds the kernel (82 % of its throughput on the SMs that work, the tensor pipe at 49 %), and the operands read from it grow with T: 203 tokens of 4096 x 14336 as four tiles of 64 took 154 us where tiles of 56 took 141, 140 tokens as
// three of 64 153, of 48 124 (without the eighth digit product and the marks; now 146 and 142).
static int q6g_tile(int ntok) {
    const int tiles = (ntok + 63) / 64, T = ((ntok + tiles - 1) / tiles + 7) & ~7;
    return T < 16 ? 16 : T;
}
static int q6g_first(int T) { return T <= 32 ? T : (T / 2 + 7) & ~7; }     // tokens of its first group

// CTAs that share a tile's super-blocks: only as many as fill SMs that the tiles alone would leave idle.
static int q6g_slices(int nrows, int nsb, int ntok, int sms) {
    const int T = q6g_tile(ntok), tiles = (nrows + Q6G_ROWS - 1) / Q6G_ROWS * ((ntok + T - 1) / T);
    int s = 8;
    while (s > 1 && (s * tiles > sms || s > nsb)) s >>= 1;
    return s;
}

size_t jl_gemm_q6k_scratch_bytes(int k, int ntok) {
    const int T = q6g_tile(ntok);
    const size_t padded = (size_t)(ntok + T - 1) / T * T;
    return padded * k * 4 + padded * (k / 256) * 4 + 256;
}

// Workspace for `ntok` tokens of width `k`, grown at upload, in jl_reserve and before a host-pointer call, never inside a
// device-pointer call. A batch that finds it too small runs on the row kernel, so a refused allocation is no error.
int jl_gemm_q6k_reserve(jl_ctx *ctx, int k, int ntok) {
    const size_t need = jl_gemm_q6k_scratch_bytes(k, ntok);
    if (ntok <= 8 || ctx->q6k_cap >= need) return JL_OK;
    if (!ctx->q6k_done) JL_CUDA(ctx, cudaEventCreateWithFlags(&ctx->q6k_done, cudaEventDisableTiming));
    JL_CUDA(ctx, cudaDeviceSynchronize());   // an earlier launch may still read the old buffer
    if (ctx->q6k_work) cudaFree(ctx->q6k_work);
    ctx->q6k_work = nullptr; ctx->q6k_cap = 0;
    if (cudaMalloc(&ctx->q6k_work, need) != cudaSuccess) { cudaGetLastError(); ctx->q6k_work = nullptr; return JL_OK; }
    ctx->q6k_cap = need;
    return JL_OK;
}

int jl_gemm_q6k_choice(jl_ctx *ctx, int nrows, int k, int ntok, jl_choice *out) {
    if (k % 256 || ctx->opts.pin_kernel != JL_K_AUTO || (ctx->opts.flags & (JL_FLAG_NO_TMA | JL_FLAG_DECODE_CONCURRENT)) ||
        ctx->q6k_cap < jl_gemm_q6k_scratch_bytes(k, ntok))
        return JL_DECLINED;
    jl_choice c = {};
    const int T = q6g_tile(ntok);
    c.kernel = JL_K_TC5; c.warps = Q6G_THREADS / 32; c.rows_per_cta = Q6G_ROWS;
    c.split_k = q6g_slices(nrows, k / 256, ntok, ctx->sm_count);
    c.tile_m = Q6G_ROWS; c.tile_n = 4 * q6g_first(T); c.tile_k = 128;
    c.grid = (nrows + Q6G_ROWS - 1) / Q6G_ROWS * ((ntok + T - 1) / T) * c.split_k;
    c.launches = 2;
    *out = c;
    return JL_OK;
}

template <int G0, int G1>
static int q6g_launch(jl_ctx *ctx, const q6g_params &p, int tok_tiles, cudaStream_t s) {
    using L = q6g_smem<G0, G1>;
    static_assert(L::TOTAL <= 227 * 1024, "shared memory budget");
    static_assert(L::T * Q6G_RED_STRIDE * 4 <= L::BAR_OFS, "the partial tile reuses the stages");
    if (!(ctx->q6k_ready >> (L::T / 8) & 1)) {       // once per context and form, not on every call
        JL_CUDA(ctx, cudaFuncSetAttribute(gemm_q6k_kernel<G0, G1>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL));
        ctx->q6k_ready |= 1u << (L::T / 8);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((p.nrows + Q6G_ROWS - 1) / Q6G_ROWS * p.slices, tok_tiles); cfg.blockDim = dim3(Q6G_THREADS);
    cfg.dynamicSmemBytes = L::TOTAL; cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = p.slices; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = (ctx->opts.flags & JL_FLAG_NO_PDL) ? 1 : 2;
    JL_CUDA(ctx, cudaLaunchKernelEx(&cfg, gemm_q6k_kernel<G0, G1>, p));
    ctx->st.launches++;
    return JL_OK;
}

// JL_DECLINED: no workspace for this call, the row kernel takes it.
int jl_launch_gemm_q6k(jl_ctx *ctx, float *out_dev, const jl_weight *w, int expert, const float *x_dev, int ntok, cudaStream_t s) {
    const int nsb = w->k / 256, T = q6g_tile(ntok), tok_tiles = (ntok + T - 1) / T;
    // Plain calls share the context's workspace: those of one stream follow each other, one on another stream waits for
    // the call before it. A captured call works in memory of its graph's own, since nothing orders a replay against the rest.
    const size_t need = jl_gemm_q6k_scratch_bytes(w->k, ntok);
    jl_stream_state st;
    if (!jl_stream_query(s, &st)) return JL_DECLINED;
    uint8_t *planes = (uint8_t *)(st.graph ? jl_capture_place(ctx, st, need) : ctx->q6k_cap >= need ? ctx->q6k_work : nullptr);
    if (!planes) return JL_DECLINED;
    if (!st.graph && ctx->q6k_recorded && ctx->q6k_stream != st.stream) JL_CUDA(ctx, cudaStreamWaitEvent(s, ctx->q6k_done, 0));
    const size_t rows_off = (size_t)expert * w->nrows;
    q6g_params p;
    p.nrows = w->nrows; p.nsb = nsb; p.ntok = ntok; p.slices = q6g_slices(w->nrows, nsb, ntok, ctx->sm_count);
    p.w = w->data + rows_off * nsb * JL_Q6K_BLOCK;
    p.d = reinterpret_cast<const uint16_t *>(w->scales) + rows_off * nsb;
    p.x = x_dev; p.out = out_dev; p.status = ctx->dev_status;
    float *inv = (float *)(planes + (size_t)tok_tiles * T * w->k * 4);
    p.planes = planes; p.inv = inv;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3(nsb, tok_tiles * T / 8); cfg.blockDim = dim3(256); cfg.stream = s;
    cfg.attrs = at; cfg.numAttrs = (ctx->opts.flags & JL_FLAG_NO_PDL) ? 0 : 1;
    JL_CUDA(ctx, cudaLaunchKernelEx(&cfg, q6k_xprep_kernel, x_dev, planes, inv, nsb, ntok, T, q6g_first(T)));
    ctx->st.launches++;
    int rc;
    switch (T) {
    case 16: rc = q6g_launch<16, 0>(ctx, p, tok_tiles, s); break;
    case 24: rc = q6g_launch<24, 0>(ctx, p, tok_tiles, s); break;
    case 32: rc = q6g_launch<32, 0>(ctx, p, tok_tiles, s); break;
    case 40: rc = q6g_launch<24, 16>(ctx, p, tok_tiles, s); break;
    case 48: rc = q6g_launch<24, 24>(ctx, p, tok_tiles, s); break;
    case 56: rc = q6g_launch<32, 24>(ctx, p, tok_tiles, s); break;
    default: rc = q6g_launch<32, 32>(ctx, p, tok_tiles, s); break;
    }
    if (!st.graph) {          // also where the second launch was refused: the first one writes the planes
        JL_CUDA(ctx, cudaEventRecord(ctx->q6k_done, s));
        ctx->q6k_stream = st.stream;
        ctx->q6k_recorded = true;
    }
    return rc;
}
