// Q6_K for batches (9 tokens and more): out[tok][row] = sum_k W[row][k] x[tok][k] on the integer tensor cores.
//
// A Q6_K weight is d * sc * (q - 32): an integer w = sc (q - 32) of at most 13 bits times the super-block's f16 d. The row
// kernel serves it with f32 weights and f32 activations, and at 203 tokens of 4096 x 14336 that is 3.4 ms of FP32 FMAs
// (7 TFLOP/s); this kernel takes 141 us (169 TFLOP/s), activation planes included. Both sides are integers and nothing
// is rounded inside a super-block:
//
//   weights      w = 256 h + l, both signed bytes (|w| <= 4096): two int8 operands.
//   activations  per (token, super-block) a power-of-two scale takes the largest magnitude into [2^29, 2^30); the rounded
//                32-bit integer is four signed bytes x0 (top) .. x3. An element within 2^-7 of the largest is held
//                exactly, every other one to 2^-31 of the largest: finer than the f32 sums of the row kernel.
//   products     tcgen05.mma.kind::i8, s32 accumulators in TMEM, exact. The four byte planes of T tokens are the N = 4 T
//                columns of one operand, [x0 | x1 | x2 | x3], with T rows of zeros in front of it. h multiplies it from
//                its start, l from the zeros on (the same shape and accumulator): column block c then collects
//                h x_c + l x_(c-1), all of weight 2^(32 - 8 c). (l x3 is left out: 2^-31 of the largest magnitude.)
//   drain        once per super-block: two integer shifts-and-adds and two conversions join the four sums, one FMA adds
//                them, times d and 1/scale, to the token's f32 accumulator in registers. 56 such additions per output
//                at k = 14336, where the row kernel makes one per element.
//
// Work split: a CTA is 128 rows x T tokens (T = 16, 24 .. 64) x a slice of the super-blocks; the slices of a tile are the
// CTAs of one thread-block cluster, which add their f32 tiles in rank order through distributed shared memory (bit-stable;
// nothing is waited for but the cluster barrier). Roles: warps 0..3 drain, warp 4 copies the activation planes (untiled bulk
// copies: the prep kernel writes them as the swizzled shared-memory image), warp 5 issues the MMAs, warps 6..13 make the
// weight operands, 16 rows x 2 runs of 16 codes a warp, half a super-block (128 k) per stage.
//
// Activations that are not finite have no such integers: the prep kernel gives their super-block a NaN scale, the f32
// accumulator becomes NaN, and the drain then computes that output as both Q6_K kernels do, weight by weight (q6k_plain.cuh).
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
q6k_xprep_kernel(const float *__restrict__ X, uint8_t *__restrict__ planes, float *__restrict__ inv, int nsb, int ntok, int T) {
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
    const bool finite = amax < 0x7F800000u;
    const int p = min(126, 29 - ((int)(amax >> 23) - 127));      // largest magnitude in [2^29, 2^30); 2^-p stays normal
    const float scale = __uint_as_float((uint32_t)(127 + p) << 23);
    uint32_t u[8];
#pragma unroll
    for (int i = 0; i < 8; i++)      // byte j of u is digit j + 128
        u[i] = (uint32_t)(finite ? __float2int_rn(v[i] * scale) : 0) + 0x80808080u;
    if (lane == 0)
        inv[((size_t)tt * nsb + sb) * T + t] = !finite ? __uint_as_float(0x7FC00000u) : __uint_as_float((uint32_t)(127 - p) << 23);
    // image of half a super-block: 4 T rows (plane c, token t) of 128 bytes, 16-byte chunks swizzled by the row
    const int half = lane >> 4, chunk = (lane & 15) >> 1;
    uint8_t *img = planes + (((size_t)tt * nsb + sb) * 2 + half) * (size_t)(T * 512) + (((uint32_t)chunk ^ (uint32_t)(t & 7)) << 4) + (lane & 1) * 8;
#pragma unroll
    for (int c = 0; c < 4; c++) {    // plane c = byte 3 - c
        const uint32_t s2 = (uint32_t)(3 - c) | (uint32_t)(7 - c) << 4;
        const uint32_t lo = __byte_perm(__byte_perm(u[0], u[1], s2), __byte_perm(u[2], u[3], s2), 0x5410);
        const uint32_t hi = __byte_perm(__byte_perm(u[4], u[5], s2), __byte_perm(u[6], u[7], s2), 0x5410);
        *reinterpret_cast<uint2 *>(img + (size_t)(c * T + t) * 128) = make_uint2(lo ^ 0x80808080u, hi ^ 0x80808080u);
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

template <int T>
struct q6g_smem {
    static constexpr int B_BYTES = T * 512;                            // the four planes
    static constexpr int STAGE = 2 * Q6G_A_BYTES + T * 128 + B_BYTES;  // h, l, zeros, planes
    static constexpr int BAR_OFS = Q6G_STAGES * STAGE;                 // full[3] empty[3] acc_full[2] acc_empty[2]
    static constexpr int INV_OFS = BAR_OFS + (2 * Q6G_STAGES + 4) * 8; // [4 warps][T] 1 / scale of the drained super-block
    static constexpr int MISC_OFS = INV_OFS + 4 * T * 4;
    static constexpr int TOTAL = MISC_OFS + 16 + 1024;
    static constexpr int COLS = T <= 16 ? 128 : (T <= 32 ? 256 : 512); // two accumulators of 4 T columns, a power of two allocated
    static_assert(T % 8 == 0 && STAGE % 1024 == 0, "operands start on swizzle atoms");
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

template <int T>
__global__ void __launch_bounds__(Q6G_THREADS, 1) gemm_q6k_kernel(const q6g_params p) {
    using L = q6g_smem<T>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t sbase = smem_u32(smem), bars = sbase + L::BAR_OFS;
    const uint32_t full = bars, empty = bars + 8 * Q6G_STAGES, acc_full = bars + 16 * Q6G_STAGES, acc_empty = acc_full + 16;
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(smem + L::MISC_OFS);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + L::MISC_OFS + 4);
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
        mbar_init_fence();
    }
    if (warp == 5) tc5_alloc(smem_u32(const_cast<uint32_t *>(tmem_slot)), L::COLS);
    // the zero rows in front of each stage's planes
    for (int i = tid; i < Q6G_STAGES * T * 8; i += Q6G_THREADS)
        *reinterpret_cast<uint4 *>(smem + (i / (T * 8)) * L::STAGE + 2 * Q6G_A_BYTES + (i % (T * 8)) * 16) = make_uint4(0, 0, 0, 0);
    fence_async_smem();
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
                bulk_load_1d(sbase + s * L::STAGE + 2 * Q6G_A_BYTES + T * 128, src + (size_t)i * L::B_BYTES, L::B_BYTES, full + 8 * s);
            }
        }
    } else if (warp == 5) {
        constexpr uint32_t idesc = q6g_idesc(Q6G_ROWS, 4 * T);
        const bool leader = tc5_elect();
        const uint32_t tbase = (uint32_t)tc5_uniform((int)tmem_base), sb_u = (uint32_t)tc5_uniform((int)sbase);
        bool ok = true;
        for (int i = 0; i < 2 * nmine; i++) {
            const uint32_t s = i % Q6G_STAGES, ph = (i / Q6G_STAGES) & 1;
            const int sbi = i >> 1, ab = sbi & 1;
            if (!(i & 1) && sbi >= 2) ok = __all_sync(0xffffffffu, tc5_wait(acc_empty + 8 * ab, ((sbi >> 1) & 1) ^ 1, abort_flag));
            if (ok) ok = __all_sync(0xffffffffu, tc5_wait(full + 8 * s, ph, abort_flag));
            if (!ok) break;
            tc5_fence_after();
            if (leader) {
                const uint32_t st = sb_u + s * L::STAGE, d_tmem = tbase + ab * 4 * T;
                const uint64_t ah = tc5_smem_desc(st), al = tc5_smem_desc(st + Q6G_A_BYTES);
                const uint64_t bz = tc5_smem_desc(st + 2 * Q6G_A_BYTES), bx = tc5_smem_desc(st + 2 * Q6G_A_BYTES + T * 128);
#pragma unroll
                for (int j = 0; j < 4; j++) {     // 32 bytes of k per instruction
                    q6g_mma(d_tmem, ah + 2 * j, bx + 2 * j, idesc, ((i & 1) | j) != 0);
                    q6g_mma(d_tmem, al + 2 * j, bz + 2 * j, idesc, 1);
                }
                tc5_commit(empty + 8 * s);
                if (i & 1) tc5_commit(acc_full + 8 * ab);
            }
            __syncwarp();
        }
    } else if (warp >= 6) {
        // lane: row r of the warp's 16, run j (16 positions) of each half
        const int r = (warp - 6) * 16 + (lane & 15), j = lane >> 4;
        const size_t row = (size_t)min(rt * Q6G_ROWS + r, p.nrows - 1);
        const uint8_t *wrow = p.w + (row * p.nsb + sb0) * JL_Q6K_BLOCK;
        const uint32_t swz = (uint32_t)(r & 7);
        uint4 A, B, H;
        uint2 S;
        auto fetch = [&](int i) {
            const uint8_t *blk = wrow + (size_t)(i >> 1) * JL_Q6K_BLOCK;
            const int n = i & 1;
            A = ldg_nc16(blk + n * 64 + 16 * j);
            B = ldg_nc16(blk + n * 64 + 32 + 16 * j);
            H = ldg_nc16(blk + 128 + n * 32 + 16 * j);
            S = __ldg(reinterpret_cast<const uint2 *>(blk + 192 + n * 8));
        };
        fetch(0);
        for (int i = 0; i < 2 * nmine; i++) {
            const uint32_t s = i % Q6G_STAGES, ph = (i / Q6G_STAGES) & 1;
            const uint32_t la[4] = {A.x, A.y, A.z, A.w}, lb[4] = {B.x, B.y, B.z, B.w}, lh[4] = {H.x, H.y, H.z, H.w};
            const uint2 sc8 = S;
            if (i + 1 < 2 * nmine) fetch(i + 1);
            if (i >= Q6G_STAGES && !__all_sync(0xffffffffu, tc5_wait(empty + 8 * s, ph ^ 1, abort_flag))) break;
            uint8_t *dst = smem + s * L::STAGE + r * 128;
#pragma unroll
            for (int c = 0; c < 4; c++) {         // elements c * 32 + 16 j .. + 15 of the half: 16-byte chunk 2 c + j
                const int sc = (int)(int8_t)((c < 2 ? sc8.x : sc8.y) >> (16 * (c & 1) + 8 * j));
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
        }
    } else {
        asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll
        for (int t = 0; t < T; t++) acc[t] = 0.f;
        const int row = rt * Q6G_ROWS + warp * 32 + lane;
        const uint16_t *drow = p.d + (size_t)min(row, p.nrows - 1) * p.nsb + sb0;
        const float *inv = p.inv + ((size_t)tt * p.nsb + sb0) * T;
        float *minv = reinterpret_cast<float *>(smem + L::INV_OFS) + warp * T;
        constexpr int PER = (T + 31) / 32;
        float inext[PER];
        uint16_t dnext = __ldg(drow);
#pragma unroll
        for (int i = 0; i < PER; i++) inext[i] = lane + 32 * i < T ? __ldg(inv + lane + 32 * i) : 0.f;
        for (int i = 0; i < nmine; i++) {
            const int ab = i & 1;
            const float d = __half2float(__ushort_as_half(dnext)) * 256.f;      // the last column block weighs 2^8
            __syncwarp();
#pragma unroll
            for (int q = 0; q < PER; q++)
                if (lane + 32 * q < T) minv[lane + 32 * q] = inext[q];
            __syncwarp();
            if (i + 1 < nmine) {
                dnext = __ldg(drow + i + 1);
#pragma unroll
                for (int q = 0; q < PER; q++)
                    if (lane + 32 * q < T) inext[q] = __ldg(inv + (size_t)(i + 1) * T + lane + 32 * q);
            }
            if (!__all_sync(0xffffffffu, tc5_wait(acc_full + 8 * ab, (i >> 1) & 1, abort_flag))) break;
            tc5_fence_after();
            const uint32_t ta = tmem_base + ab * 4 * T + ((uint32_t)(warp * 32) << 16);
#pragma unroll
            for (int t0 = 0; t0 < T; t0 += 8) {
                uint32_t c0[8], c1[8], c2[8], c3[8];
                tc5_ld8(ta + t0, c0);
                tc5_ld8(ta + T + t0, c1);
                tc5_ld8(ta + 2 * T + t0, c2);
                tc5_ld8(ta + 3 * T + t0, c3);
                tc5_wait_ld();
#pragma unroll
                for (int t = 0; t < 8; t++) {
                    // |c0| < 2^18.1, |c1| < 2^21.4, |c2|, |c3| < 2^22.2: both joined sums fit 32 bits
                    const int hi = (int)c0[t] * 256 + (int)c1[t], lo = (int)c2[t] * 256 + (int)c3[t];
                    const float v = fmaf((float)hi, 65536.f, (float)lo);
                    acc[t0 + t] = fmaf(v, d * minv[t0 + t], acc[t0 + t]);
                }
            }
            tc5_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty + 8 * ab);
        }
#pragma unroll
        for (int t = 0; t < T; t++)
            if (!(fabsf(acc[t]) < __int_as_float(0x7f800000)) && row < p.nrows && tt * T + t < p.ntok)
                acc[t] = q6k_plain(p.w + ((size_t)row * p.nsb + sb0) * JL_Q6K_BLOCK, drow, p.x + ((size_t)(tt * T + t) * p.nsb + sb0) * 256, nmine);
        if (p.slices == 1) {
#pragma unroll
            for (int t = 0; t < T; t++)
                if (row < p.nrows && tt * T + t < p.ntok) p.out[(size_t)(tt * T + t) * p.nrows + row] = acc[t];
        }
    }

    tc5_fence_before();
    __syncthreads();             // every MMA of this CTA has been drained (or the CTA has given up): the stages are free
    if (tid == 0 && *abort_flag) atomicExch(p.status, 2);
    if (warp == 5) {
        tc5_fence_after();
        tc5_dealloc(tmem_base, L::COLS);
    }
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

// Tokens of a tile: the batch over the fewest tiles of 64 (8 T columns are all of TMEM there), rounded up to 8. The MMAs
// are what bounds the kernel and their N is 4 T: 203 tokens of 4096 x 14336 as four tiles of 64 took 154 us, of 56 take 141; 140
// tokens as three of 64 153, of 48 124.
static int q6g_tile(int ntok) {
    const int tiles = (ntok + 63) / 64, T = ((ntok + tiles - 1) / tiles + 7) & ~7;
    return T < 16 ? 16 : T;
}

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
    c.tile_m = Q6G_ROWS; c.tile_n = 4 * T; c.tile_k = 128;
    c.grid = (nrows + Q6G_ROWS - 1) / Q6G_ROWS * ((ntok + T - 1) / T) * c.split_k;
    c.launches = 2;
    *out = c;
    return JL_OK;
}

template <int T>
static int q6g_launch(jl_ctx *ctx, const q6g_params &p, int tok_tiles, cudaStream_t s) {
    using L = q6g_smem<T>;
    static_assert(L::TOTAL <= 227 * 1024, "shared memory budget");
    static_assert(T * Q6G_RED_STRIDE * 4 <= L::BAR_OFS, "the partial tile reuses the stages");
    JL_CUDA(ctx, cudaFuncSetAttribute(gemm_q6k_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((p.nrows + Q6G_ROWS - 1) / Q6G_ROWS * p.slices, tok_tiles); cfg.blockDim = dim3(Q6G_THREADS);
    cfg.dynamicSmemBytes = L::TOTAL; cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = p.slices; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = (ctx->opts.flags & JL_FLAG_NO_PDL) ? 1 : 2;
    JL_CUDA(ctx, cudaLaunchKernelEx(&cfg, gemm_q6k_kernel<T>, p));
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
    JL_CUDA(ctx, cudaLaunchKernelEx(&cfg, q6k_xprep_kernel, x_dev, planes, inv, nsb, ntok, T));
    ctx->st.launches++;
    int rc;
    switch (T) {
    case 16: rc = q6g_launch<16>(ctx, p, tok_tiles, s); break;
    case 24: rc = q6g_launch<24>(ctx, p, tok_tiles, s); break;
    case 32: rc = q6g_launch<32>(ctx, p, tok_tiles, s); break;
    case 40: rc = q6g_launch<40>(ctx, p, tok_tiles, s); break;
    case 48: rc = q6g_launch<48>(ctx, p, tok_tiles, s); break;
    case 56: rc = q6g_launch<56>(ctx, p, tok_tiles, s); break;
    default: rc = q6g_launch<64>(ctx, p, tok_tiles, s); break;
    }
    if (!st.graph) {          // also where the second launch was refused: the first one writes the planes
        JL_CUDA(ctx, cudaEventRecord(ctx->q6k_done, s));
        ctx->q6k_stream = st.stream;
        ctx->q6k_recorded = true;
    }
    return rc;
}
