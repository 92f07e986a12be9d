// Per-warp inner loops of the weight-streaming (1..8 row) projections, shared by the stand-alone skinny kernels
// (gemv.cu, parallel_block.cu, moe_rows.cu) and the persistent decode kernel (decode_mega.cu).
//
// `warp_dot_*`: a warp owns NPW weight rows over a K range: every lane streams 16-byte pieces (L1 no-allocate), multiplies them
// with the R activation rows in fp32 and the warp reduces with the xor tree of warp_sum, so every caller gets the same bits for the
// same (rows, K range).  `skinny_mma_*`: 16 weight rows on mma.sync, for one to eight rows and all but few outputs.
#pragma once

#include "common.cuh"
#include "moe_mma_core.cuh"

// ---------------------------------------------------------------------------------------------------
// Per-warp dot products.  acc[j][r] accumulates this lane's share of  sum_k w_j[k] * x_r[k].
template <int R, int NPW>
__device__ __forceinline__ void warp_dot_bf16(const bf16* const (&xr)[R], const bf16* const (&wp)[NPW], int kbeg, int kend,
                                              int lane, float (&acc)[NPW][R]) {
#pragma unroll (R * NPW <= 4 ? 4 : 2)
    for (int k = kbeg + lane * 8; k < kend; k += 256) {
        float wf[NPW][8];
#pragma unroll
        for (int j = 0; j < NPW; ++j) {
            const uint4 v = ld_stream16(wp[j] + k);
            wf[j][0] = bf16_lo(v.x); wf[j][1] = bf16_hi(v.x); wf[j][2] = bf16_lo(v.y); wf[j][3] = bf16_hi(v.y);
            wf[j][4] = bf16_lo(v.z); wf[j][5] = bf16_hi(v.z); wf[j][6] = bf16_lo(v.w); wf[j][7] = bf16_hi(v.w);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint4 v = ld_hot16(xr[r] + k);
            const float xf[8] = {bf16_lo(v.x), bf16_hi(v.x), bf16_lo(v.y), bf16_hi(v.y),
                                 bf16_lo(v.z), bf16_hi(v.z), bf16_lo(v.w), bf16_hi(v.w)};
#pragma unroll
            for (int j = 0; j < NPW; ++j)
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[j][r] = fmaf(wf[j][i], xf[i], acc[j][r]);
        }
    }
}

// FP8 (e4m3 + 128x128 fp32 block scales).  sp[j] points at the scale row of weight row j (K/128 entries).
template <int R, int NPW>
__device__ __forceinline__ void warp_dot_fp8(const bf16* const (&xr)[R], const uint8_t* const (&wp)[NPW],
                                             const float* const (&sp)[NPW], int K, int lane, float (&acc)[NPW][R]) {
#pragma unroll (R * NPW <= 2 ? 4 : 2)
    for (int k = lane * 16; k < K; k += 512) {
        float wf[NPW][16];
#pragma unroll
        for (int j = 0; j < NPW; ++j) {
            const uint4 v = ld_stream16(wp[j] + k);
            const float s = __ldg(sp[j] + (k >> 7));
            const uint32_t words[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float2 a = decode_e4m3x2(words[q], s);
                const float2 b = decode_e4m3x2(words[q] >> 16, s);
                wf[j][4 * q + 0] = a.x; wf[j][4 * q + 1] = a.y; wf[j][4 * q + 2] = b.x; wf[j][4 * q + 3] = b.y;
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint4 v0 = ld_hot16(xr[r] + k);
            const uint4 v1 = ld_hot16(xr[r] + k + 8);
            const float xf[16] = {bf16_lo(v0.x), bf16_hi(v0.x), bf16_lo(v0.y), bf16_hi(v0.y), bf16_lo(v0.z), bf16_hi(v0.z),
                                  bf16_lo(v0.w), bf16_hi(v0.w), bf16_lo(v1.x), bf16_hi(v1.x), bf16_lo(v1.y), bf16_hi(v1.y),
                                  bf16_lo(v1.z), bf16_hi(v1.z), bf16_lo(v1.w), bf16_hi(v1.w)};
#pragma unroll
            for (int j = 0; j < NPW; ++j)
#pragma unroll
                for (int i = 0; i < 16; ++i) acc[j][r] = fmaf(wf[j][i], xf[i], acc[j][r]);
        }
    }
}

template <int R, int NPW>
__device__ __forceinline__ void warp_reduce_all(float (&acc)[NPW][R]) {
#pragma unroll
    for (int j = 0; j < NPW; ++j)
#pragma unroll
        for (int r = 0; r < R; ++r) acc[j][r] = warp_sum(acc[j][r]);
}

// ---------------------------------------------------------------------------------------------------
// 16 weight rows as the M and one to eight activation rows as the N of mma.sync m16n8k16 (bf16 products, fp32 sums).  A row's bits depend neither on
// how many others there are nor on what they hold, where a row alone takes these kernels too.  With R rows the
// FMA loop above issues R + 2 instructions per weight and is bound by issue from four rows on; here a weight costs a sixteenth of an
// instruction whatever R is, and nothing is shuffled at the end.  Measured on a B200 (launches of their own), [6144 x 16384]: 2 rows 49.8 -> 32.2 us, 4 rows
// 58.0 -> 32.6, 8 rows 85.5 -> 32.9 (6.1 TB/s); [131072 x 4096]: 193 -> 154, 218 -> 158, 397 -> 163.
//
// The tensor core truncates what it adds to an accumulator, so every instruction starts from zero and its sixteen products' sum is added in
// rounded fp32: the four sums of a chunk in pairs, the chunk's to the warp's with Kahan's compensation, the warps' in pairs.  Error against
// 64 bits (2-norm, operands of either sign), [6144 x 16384] / [6144 x 6144] / [2048 x 2048]: 7.3e-8 / 7.1e-8 / 7.1e-8, with FMAs 12.6e-8 /
// 9.2e-8 / 7.5e-8, accumulated inside the tensor core 2.1e-6 / 7.3e-7 / 2.3e-7.  The additions hide behind the loads: [6144 x 16384] 31.6 ->
// 32.0 us, [4096 x 18432] 24.7 -> 25.0, [131072 x 4096] 154 -> 156.
//
// The k index inside an instruction is a permutation of the true k, the same for both operands: lane (g, t) holds 16 consecutive
// k values of weight rows g (w_lo) and g + 8 (w_hi) and of activation row g, at 16 t of a 64-wide chunk, so every load is a full
// 16-byte vector.  Chunks first, first + stride, .. enter the sum in ascending order, whatever DEPTH (chunks whose loads are in
// flight together) is.  `skinny_mma_span`: the SKM_WARPS warps of a CTA take the chunks of K round-robin; the bits depend on K only.
// w_lo, w_hi, xr: this lane's rows (NULL: zeros).  K a multiple of 8.  c: the C fragment, rows g and g + 8, columns 2t and 2t + 1.
#define SKM_WARPS 8
// d = a . b, the sums of sixteen products
__device__ __forceinline__ void mma_16816_alone(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
template <int DEPTH>
__device__ __forceinline__ void skinny_mma_chunks(const bf16* w_lo, const bf16* w_hi, const bf16* xr, int K, int first, int stride, int chunks, int t,
                                                  float (&c)[4]) {
    float lost[4] = {0.f, 0.f, 0.f, 0.f};
    for (int c0 = first; c0 < chunks; c0 += stride * DEPTH) {
        uint4 lo[DEPTH][2], hi[DEPTH][2], x[DEPTH][2];
#pragma unroll
        for (int u = 0; u < DEPTH; ++u)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int k = ((c0 + u * stride) << 6) + t * 16 + h * 8;
                const uint4 zero = make_uint4(0, 0, 0, 0);
                lo[u][h] = w_lo && k < K ? ld_stream16(w_lo + k) : zero;
                hi[u][h] = w_hi && k < K ? ld_stream16(w_hi + k) : zero;
                x[u][h] = xr && k < K ? ld_hot16(xr + k) : zero;
            }
#pragma unroll
        for (int u = 0; u < DEPTH; ++u) {
            float d[2][2][4];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                mma_16816_alone(d[h][0], lo[u][h].x, hi[u][h].x, lo[u][h].y, hi[u][h].y, x[u][h].x, x[u][h].y);
                mma_16816_alone(d[h][1], lo[u][h].z, hi[u][h].z, lo[u][h].w, hi[u][h].w, x[u][h].z, x[u][h].w);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float part = ((d[0][0][i] + d[0][1][i]) + (d[1][0][i] + d[1][1][i])) - lost[i], sum = c[i] + part;
                lost[i] = (sum - c[i]) - part;
                c[i] = sum;
            }
        }
    }
}
template <int DEPTH>
__device__ __forceinline__ void skinny_mma_span(const bf16* w_lo, const bf16* w_hi, const bf16* xr, int K, int warp, int t, float (&c)[4]) {
    skinny_mma_chunks<DEPTH>(w_lo, w_hi, xr, K, warp, SKM_WARPS, (K + 63) >> 6, t, c);
}

// Whether a projection of so many groups of 16 weight rows takes the kernels above: a CTA has one group.  Fewer than 64 CTAs leave the
// machine idle ([256 x 6144]: 16 CTAs 4.8 us, the FMA kernel's 128 CTAs of two rows 3.1; [2048 x 2048]: 3.8 against 4.4).  A row alone, in a step: from a CTA
// per SM on ([6144 x 16384] 36.0 -> 31.5 us, [2624 x 6144] 7.9 -> 6.8, [154880 x 6144] 273 -> 261, [4096 x 14336] 25.6 -> 19.8); with 128 the FMA
// kernel's smaller CTAs are done as early and let the next kernel in earlier ([2048 x 10240] 10.5 against 11.1).
__host__ __device__ static inline bool skinny_mma_takes(int rows, int groups) { return groups >= (rows > 1 ? 64 : 148); }

// Chunks in flight per warp: four with two CTAs per SM, or two with three.  The last wave decides: whichever fills its waves better ([4096 x
// 18432], 256 CTAs: 25.4 against 28.0 us; [6144 x 16384], 384 CTAs: 37.4 against 32.6).  Rows of fewer than two rounds of
// four chunks gain nothing from the deeper form beyond the first wave.
static inline int skinny_mma_depth(int groups, int K) {
    if (groups <= 2 * 148) return 4;
    const int full4 = (groups + 295) / 296 * 296, full2 = (groups + 443) / 444 * 444;
    return K >= 4096 && full4 < full2 ? 4 : 2;
}

// Fragments of a CTA's warps meet in shared memory, [column][row] with a stride of 20 floats (no bank conflict on the way in).
#define SKM_RED 20
__device__ __forceinline__ void skm_store_fragment(float* red, const float (&c)[4], int lane) {
    const int g = lane >> 2, t = lane & 3;
    red[(2 * t) * SKM_RED + g] = c[0]; red[(2 * t + 1) * SKM_RED + g] = c[1];
    red[(2 * t) * SKM_RED + g + 8] = c[2]; red[(2 * t + 1) * SKM_RED + g + 8] = c[3];
}
// Sum over the warps' K parts of (activation row r, weight row n), in pairs.
__device__ __forceinline__ float skm_sum(const float (*red)[8 * SKM_RED], int r, int n) {
    const int at = r * SKM_RED + n;
    return ((red[0][at] + red[1][at]) + (red[2][at] + red[3][at])) + ((red[4][at] + red[5][at]) + (red[6][at] + red[7][at]));
}
