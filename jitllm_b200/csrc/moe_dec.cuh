// The mixture layer for a few (token, expert) pairs: each pair is a matrix-vector product of the expert's three matrices,
// bound by the bytes of the chosen experts (13 MB each at 2880 x 2880), with the decode kernel's arithmetic (mxfp4_dot.cuh:
// exact weights, activations as f16 hi + lo per 64 elements, f32 sums). The grouped GEMM it stands in for walks all
// experts' units with 128- and 256-row tiles: at 4 pairs it keeps 90 CTAs busy on four experts and spends 150 us in eight
// launches. Where the lines lie (one layer of 2880 x 2880, grouped GEMM against this path): 4 pairs 145 / 40 us, 32 pairs of 32
// experts 270 / 148. With few experts the GEMM reads each once while every pair here fetches its own: 16 pairs of 8 experts 142 / 81,
// 32 pairs 140 / 138 to 176. So up to 32 pairs and two per expert in the exact arm; in the three-digit arm up to 8 pairs (98 / 59 of 32
// experts, 67 / 61 of 8; at 12 119 / 118).
// Three launches, each fetching as soon as its input allows:
//   route + split   the router (moe_route_token) and the hidden rows as f16 hi / lo, side by side
//   gate | up       a CTA is 64 gate rows and the same 64 up rows of one pair, k split in two: its 64 gated values are one
//                   span, so it writes them as the next kernel's hi / lo operand itself
//   down            a CTA is 16 rows of one token for ALL its experts, k split over the warps; the sums meet in shared
//                   memory in fixed order and are added into the row in ascending expert id. Its first weights are asked
//                   for before it waits for the gate | up kernel: the ids come from the launch before that one, which is
//                   complete (gate | up allows its dependents only after its own wait).
#pragma once
#include "mxfp4_dot.cuh"
#include "tc5.cuh"      // ldg_nc16

#define MXD_U 1          // units of four blocks (128 elements) a warp asks for ahead; 2 spill at two CTAs an SM (47 against 40 us)
#define MXD_WARPS 16

// 16 rows of one expert matrix against one token. Lane (g, t) takes block 4 u + t of rows g and g + 8 in unit u: its 16 code
// bytes are ONE 16-byte load (a quad reads 64 contiguous bytes of a row), and the four blocks of a quad stay apart in the
// MMA because B is block-diagonal: column 2 t carries the hi halves of block t's activations and column 2 t + 1 the lo
// halves, in the lanes with g >> 1 == t, and every other lane feeds zeros. Lane (g, t) so ends with its own block's two sums
// for its two rows, and applies its own block's scale. (With a block spread over the quad, 4 bytes a lane, and one token
// in two of the eight columns, the layer took 57 us at four pairs; now 40. What bounds it now: 50 000 instructions a CTA, 80 a unit of
// them turning codes into f16, on the SMs that hold two of the 180 CTAs.)
//
// ca, ea: code and scale rows of the lane's row g, c8, e8: bytes from there to those of row g + 8; x: the row of the lane's
// column (hi or lo); isc: 1 / scale of each 64-element span. The warp takes part `part` of `parts` of the row. `ready` runs after the first weights have been asked for and before the operand is read.
template <typename Ready>
__device__ __forceinline__ void mxd_dot(const uint8_t *ca, uint32_t c8, const uint8_t *ea, uint32_t e8, const __half *x, int g, int t,
                                        const float *isc, int nblk, int part, int parts, float &acc_a, float &acc_b, Ready ready) {
    uint4 wa[MXD_U], wb[MXD_U], xv[4];
    uint32_t sa[MXD_U], sb[MXD_U];
    const int units = (nblk + 3) / 4, first = units * part / parts, last = units * (part + 1) / parts;
    const bool live = (g >> 1) == t;
    const uint8_t *pc = ca + (first * 4 + t) * 16, *pe = ea + first * 4 + t;      // of the next unit to ask for
    auto load = [&](int slot, bool in) {
        wa[slot] = in ? ldg_nc16(pc) : make_uint4(0, 0, 0, 0);
        wb[slot] = in ? ldg_nc16(pc + c8) : make_uint4(0, 0, 0, 0);
        sa[slot] = in ? __ldg(pe) : 0u;
        sb[slot] = in ? __ldg(pe + e8) : 0u;
        pc += 64;
        pe += 4;
    };
    int ask = first * 4 + t;                           // its block of this lane; blocks past the row weigh nothing
#pragma unroll
    for (int i = 0; i < MXD_U; i++, ask += 4) load(i, first + i < last && ask < nblk);
    ready();
    acc_a = acc_b = 0.f;
    const __half *px = x + (first * 4 + t) * 32;
    const float *pi = isc + first * 2 + (t >> 1);
#pragma unroll
    for (int j = 0; j < 4; j++) xv[j] = make_uint4(0, 0, 0, 0);
    for (int base = first; base < last; base += MXD_U) {
#pragma unroll
        for (int i = 0; i < MXD_U; i++) {
            const int unit = base + i;
            if (unit >= last) break;
            const bool in = unit * 4 + t < nblk;
            if (live) {                                // the other lanes' columns stay zero
#pragma unroll
                for (int j = 0; j < 4; j++) xv[j] = in ? *reinterpret_cast<const uint4 *>(px + 8 * j) : make_uint4(0, 0, 0, 0);
            }
            const float is = in ? *pi : 0.f;
            px += 128;
            pi += 2;
            const uint32_t qa[4] = {wa[i].x, wa[i].y, wa[i].z, wa[i].w}, qb[4] = {wb[i].x, wb[i].y, wb[i].z, wb[i].w};
            const uint32_t ea8 = sa[i], eb8 = sb[i];
            load(i, unit + MXD_U < last && ask < nblk);
            ask += 4;
            float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int q = 0; q < 4; q++) {     // word q: elements 4q..4q+3 (low nibbles) and 16+4q..16+4q+3 (high nibbles)
                const uint4 lo = xv[q >> 1], hi = xv[2 + (q >> 1)];
                mx_block(c, qa[q], qb[q], (q & 1) ? make_uint2(lo.z, lo.w) : make_uint2(lo.x, lo.y), (q & 1) ? make_uint2(hi.z, hi.w) : make_uint2(hi.x, hi.y));
            }
            acc_a = fmaf((c[0] + c[1]) * mx_block_scale(ea8), is, acc_a);
            acc_b = fmaf((c[2] + c[3]) * mx_block_scale(eb8), is, acc_b);
        }
    }
    acc_a += __shfl_xor_sync(0xffffffffu, acc_a, 1); acc_b += __shfl_xor_sync(0xffffffffu, acc_b, 1);
    acc_a += __shfl_xor_sync(0xffffffffu, acc_a, 2); acc_b += __shfl_xor_sync(0xffffffffu, acc_b, 2);
}

// Blocks [0, route_blocks): four tokens' routers. The others: one warp per (span, token) of the hidden rows.
__global__ void __launch_bounds__(128)
moe_dec_prep_kernel(const float *__restrict__ logits, const float *__restrict__ router_bias, const float *__restrict__ sel_bias, int ntok,
                    int n_expert, int top_k, int norm, float scale, int32_t *__restrict__ sel, float *__restrict__ wt, int route_blocks,
                    const void *__restrict__ h, int h_dtype, __half *__restrict__ xh, float *__restrict__ xinv, int hidden) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nspan = hidden / 64;
    if ((int)blockIdx.x < route_blocks) {
        const int tok = blockIdx.x * 4 + warp;
        if (tok < ntok) moe_route_token(logits, router_bias, sel_bias, tok, lane, n_expert, top_k, norm, scale, sel, wt);
        return;
    }
    const int i = (blockIdx.x - route_blocks) * 4 + warp;
    if (i >= nspan * ntok) return;
    const int tok = i / nspan, sp = i - tok * nspan;
    const size_t at = (size_t)tok * hidden + (size_t)sp * 64 + 2 * lane;
    float2 v;
    if (h_dtype == JL_DT_F32) {
        v = *reinterpret_cast<const float2 *>(static_cast<const float *>(h) + at);
    } else {
        const uint32_t w = *reinterpret_cast<const uint32_t *>(static_cast<const uint16_t *>(h) + at);
        if (h_dtype == JL_DT_BF16) v = make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
        else v = __half22float2(*reinterpret_cast<const __half2 *>(&w));
    }
    __half2 hi, lo;
    const float inv = mx_split_span(v, hi, lo);
    __half *row = xh + (size_t)(2 * tok) * hidden + (size_t)sp * 64;
    reinterpret_cast<__half2 *>(row)[lane] = hi;
    reinterpret_cast<__half2 *>(row + hidden)[lane] = lo;
    if (lane == 0) xinv[(size_t)tok * nspan + sp] = inv;
}

struct moe_dec_params {
    int n_expert, top_k, hidden, ffn, act;
    const uint8_t *cg, *cu, *cd, *eg, *eu, *ed;        // code and scale planes of the three banks
    int eg_stride, ed_stride;
    const float *bg, *bu, *bd;                         // biases or NULL
    const int32_t *sel;
    const float *wt;                                   // NULL: given ids, out is written instead of added to
    const __half *xh; const float *xinv;               // hidden rows [2 tok][hidden], [tok][hidden / 64]
    __half *ah; float *ainv;                           // gated rows [2 pair][ffn], [pair][ffn / 64]
    float *out;
};

__global__ void __launch_bounds__(MXD_WARPS * 32, 2) moe_dec_gate_up_kernel(const moe_dec_params p) {
    __shared__ float red[2][2][64];                    // [k half][gate, up][row]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int pair = blockIdx.y, tok = pair / p.top_k;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int id = __ldg(p.sel + pair);
    if (id < 0 || id >= p.n_expert) return;
    const int m = warp & 1, rg = (warp >> 1) & 3, half = warp >> 3;
    const int nspan = p.hidden / 64;
    const size_t row = (size_t)id * p.ffn + blockIdx.x * 64 + rg * 16 + g;
    const size_t pitch = (size_t)p.hidden / 2;
    const uint8_t *c = (m ? p.cu : p.cg) + row * pitch, *e = (m ? p.eu : p.eg) + row * p.eg_stride;
    float a, b;
    mxd_dot(c, (uint32_t)(8 * pitch), e, 8u * p.eg_stride, p.xh + (size_t)(2 * tok + (g & 1)) * p.hidden, g, t,
            p.xinv + (size_t)tok * nspan, 2 * nspan, half, 2, a, b, [] {});
    if (t == 0) {
        red[half][m][rg * 16 + g] = a;
        red[half][m][rg * 16 + g + 8] = b;
    }
    __syncthreads();
    if (warp == 0) {
        float v[2];
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int r = 2 * lane + i;
            const size_t br = (size_t)id * p.ffn + blockIdx.x * 64 + r;
            const float gate = red[0][0][r] + red[1][0][r] + (p.bg ? __ldg(p.bg + br) : 0.f);
            const float up = red[0][1][r] + red[1][1][r] + (p.bu ? __ldg(p.bu + br) : 0.f);
            v[i] = moe_act(p.act, gate, up);
        }
        __half2 hi, lo;
        const float inv = mx_split_span(make_float2(v[0], v[1]), hi, lo);
        __half *dst = p.ah + (size_t)(2 * pair) * p.ffn + blockIdx.x * 64;
        reinterpret_cast<__half2 *>(dst)[lane] = hi;
        reinterpret_cast<__half2 *>(dst + p.ffn)[lane] = lo;
        if (lane == 0) p.ainv[(size_t)pair * (p.ffn / 64) + blockIdx.x] = inv;
    }
}

__global__ void __launch_bounds__(MXD_WARPS * 32, 2) moe_dec_down_kernel(const moe_dec_params p) {
    __shared__ int s_slot[32], s_id[32], s_n;
    __shared__ float red[32][16];                      // [expert of the token + n * slice][row]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int tok = blockIdx.y;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (warp == 0) {                                   // the token's valid slots in ascending expert id (ties: slot order)
        const int id = lane < p.top_k ? __ldcg(p.sel + (size_t)tok * p.top_k + lane) : -1;
        const bool ok = id >= 0 && id < p.n_expert;
        int rank = 0;
        for (int o = 0; o < 32; o++) {
            const int other = __shfl_sync(0xffffffffu, ok ? id : 0x7fffffff, o);
            rank += other < id || (other == id && o < lane);
        }
        if (ok) { s_slot[rank] = lane; s_id[rank] = id; }
        const unsigned mask = __ballot_sync(0xffffffffu, ok);
        if (lane == 0) s_n = __popc(mask);
    }
    __syncthreads();
    const int n = s_n;
    if (n == 0) {      // (never without the wait: the next launch counts on this grid ending after the one in front)
        asm volatile("griddepcontrol.wait;" ::: "memory");
        return;
    }
    const int slices = n >= MXD_WARPS ? 1 : MXD_WARPS / n, nspan = p.ffn / 64;
    const size_t pitch = (size_t)p.ffn / 2;
    bool waited = false;
    for (int task = warp; task < n * slices; task += MXD_WARPS) {
        const int j = task % n, slice = task / n, pair = tok * p.top_k + s_slot[j];
        const size_t row = (size_t)s_id[j] * p.hidden + blockIdx.x * 16 + g;
        const uint8_t *c = p.cd + row * pitch, *e = p.ed + row * p.ed_stride;
        float a, b;
        mxd_dot(c, (uint32_t)(8 * pitch), e, 8u * p.ed_stride, p.ah + (size_t)(2 * pair + (g & 1)) * p.ffn, g, t,
                p.ainv + (size_t)pair * nspan, 2 * nspan, slice, slices, a, b, [&] {
                    if (!waited) asm volatile("griddepcontrol.wait;" ::: "memory");
                    waited = true;
                });
        if (t == 0) {
            red[task][g] = a;
            red[task][g + 8] = b;
        }
    }
    if (!waited) asm volatile("griddepcontrol.wait;" ::: "memory");
    __syncthreads();
    if (tid < 16) {
        const int row = blockIdx.x * 16 + tid;
        float *o = p.out + (size_t)tok * p.hidden + row;
        float acc = p.wt ? *o : 0.f;
        for (int j = 0; j < n; j++) {
            float y = red[j][tid];
            for (int s = 1; s < slices; s++) y += red[j + n * s][tid];
            if (p.bd) y += __ldg(p.bd + (size_t)s_id[j] * p.hidden + row);
            acc = p.wt ? acc + __ldcg(p.wt + (size_t)tok * p.top_k + s_slot[j]) * y : y;
        }
        *o = acc;
    }
}
