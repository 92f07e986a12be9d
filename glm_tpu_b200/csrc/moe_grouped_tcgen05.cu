// Routed experts for many rows (prefill): grouped GEMM over expert-sorted routes with the FP8 weights decoded
// inside the kernel, on the 5th-generation tensor cores.
//
//   C[n, sorted route] = sum_k bf16(f32(e4m3 W[e][n][k]) * scale[e][n / 128][k / 128]) * A[sorted route, k]
//
// The WEIGHT rows are the M of the product and the routes its N: an expert has as many routes as the router sends it (2,048 rows over 256
// experts: 64 on average, 200 rows: 6), and N follows them in steps of 16, while M = 128 is always full.  A tile is 256 weight rows of one
// expert (gate/up: 128 gate rows and the 128 up rows of the same outputs) x up to 128 routes; one CTA per SM walks the tiles, all
// column blocks of a route tile after each other, so that neighbouring CTAs share the activations in L2.  Per 128-wide k step:
//
//   warp 0       TMA: the FP8 rows of both matrices (128-byte swizzle, four steps in flight), and the activations of the tile's routes
//                (32-row boxes, as many as there are routes)
//   warps 6-21   decode: a thread owns a weight row of every other step, 128 codes; block scale in fp32, rounded to bf16 (the
//                weight-decode contract), into TENSOR MEMORY, which the tensor core reads as its A operand: decoded weights that went
//                through shared memory (64 KB written and 64 KB read a step) were what bound this kernel.  Two stages per matrix
//   warp 1       issues tcgen05.mma (two matrices of M 128, N 16 .. 128)
//   warps 2-5    epilogue (more than 64 routes: a fifth of it) of the tile before, while the next one is decoded and multiplied: a thread owns a weight row (TMEM lane)
//                  gate/up mode  act = bf16( silu(bf16 gate) * bf16 up ), stored in sorted order
//                  down mode     dw[route] = bf16( bf16(acc) * bf16(route weight) ), scattered to the route's slot
//
// TMEM: 256 columns of accumulators (two tiles of up to 64 routes, or one of more), 256 of decoded weights.
//
// What bounds it: the FP8 bytes, which cross HBM once (5.3 - 5.8 TB/s up to 777 rows), and with many routes the decode, which is done again for every 128
// routes of an expert, and the activations from L2.  A tile of more than 64 routes has all the accumulators, so the next one waits for its epilogue: the decode
// warps, idle then, store four fifths of it.  Measured on a B200, [256 experts, 2 x 2048 x 6144] and back, 219 experts chosen: 777 rows 980 + 516 us
// (a kernel with the routes as the M and decoded weights in shared memory: 1,931 + 1,065), 2,048 rows 1,302 + 702 us (2,377 + 1,302); with the epilogue to
// four warps alone 2,048 rows 1,417 + 772, 128 routes for every expert 1,818 + 1,001 against 1,626 + 905.
//
// Short prefill chunks bring their routes as tiles of eight (`moe_tiles8_*`, behind glmb_moe_gateup_fp8 / glmb_moe_down_fp8): neighbouring tiles of an
// expert form an item of up to 64 routes, whose activations a warp of their own gathers.  All 256 experts, against a CTA per tile and 16 rows on mma.sync
// (moe_gemv_mma.cu), which decodes an expert again for every eight routes: 60 rows (218 experts) 1,115 + 680 -> 920 + 490 us, 200 rows 1,497 + 933
// -> 1,131 + 620, 256 rows 1,724 + 1,075 -> 1,160 + 623.  On the way there, 60 rows: the gather in warp 0, between the weights' copies, 1,321 + 682; sixteen
// decode warps on every step 1,128 + 582; a multiplication per code instead of one for two 976 + 523.
// Every mbarrier wait is bounded; on a timeout the kernel raises GLMB_STATUS_WAIT_TIMEOUT, skips its stores (tiles of eight: stores NaN, for callers that hand
// no status word) and still frees its TMEM.
//
// Replaces reference `glm_tpu/kernels/fp8_grouped_matmul/panel_kernel.py:31-153` + `layers/moe/routed_experts.py:27-127`
// (prefill: stable group-by-expert, M32 panels, three FP8 panel matmuls, bf16 SiLU, bf16 route weighting).
#include "common.cuh"
#include "moe_mma_core.cuh"
#include "tcgen05.cuh"

#define MG_ROUTES 128  // most routes of a tile
#define MG_BK 128
#define MG_BOX 16384   // bytes of 128 rows x 64 bf16 columns
#define MG_STAGES 3    // activations: two boxes each
#define MG_TILE8_ROUTES 64   // most routes of an item made of 8-route tiles
#define MG_TILE8_STAGES 4
#define MG_TILE8_BOX 8192    // 64 rows x 64 bf16 columns
#define MG_LIST 4096         // most 8-route tiles of a launch
#define MG_TILE8_THREADS (MG_THREADS + 32)
#define MG_RAW 4       // FP8 weights: 128 rows x 128 bytes of each matrix
#define MG_CONV_WARPS 16
#define MG_TEAMS (1 + MG_CONV_WARPS / 4)  // sets of four warps that store a tile of more than 64 routes
#define MG_THREADS (6 * 32 + 32 * MG_CONV_WARPS)
#define MG_SMEM_BYTES ((MG_STAGES * 2 + MG_RAW * 2) * MG_BOX + 1024)
#define MG_TILE8_SMEM_BYTES (MG_TILE8_STAGES * 2 * MG_TILE8_BOX + MG_RAW * 2 * MG_BOX + MG_LIST * 4 + 1024)
#define MG_A_COL 256   // TMEM column of the decoded weights: stage j of matrix m at 64 (2 m + j) from here

struct MoeGroupedArgs {
    const TcTile* tiles;      // [max_tiles] 128-route tiles of the expert-sorted route list (row0, the expert's row_end, local expert)
    const int* tile_expert;   // 8-route tiles: [max_tiles] global experts,
    const int* tile_routes;   //   [max_tiles, 8] route ids or -1,
    const bf16* x;            //   the activations: of route p the row p / divisor, rows x_stride apart
    int64_t x_stride;
    int divisor, expert_base, experts_local;
    const int* n_tiles;       // [1] on the device (8-route tiles: may be NULL, all of max_tiles)
    const float* scale0;      // block scales of the first weight [experts, ceil(N/128), ceil(K/128)]
    const float* scale1;      // ... of the second (gate/up mode: up; down mode: the same table)
    const int* perm;          // [sorted routes] -> route id (row * top_k + slot), -1 for none   (down mode)
    const float* route_weight;  // [routes] fp32                                                  (down mode)
    bf16* out;                // gate/up: act_sorted [sorted routes, N];  down: dw [routes, N]
    int N, K, mode;           // mode 0: gate/up (N = expert FFN width), 1: down (N = hidden size)
    int max_tiles;
    uint32_t* status;
};

// Which accumulator columns an item takes: a tile of up to 64 routes one of the two halves, in turn, a larger one both.  Every role that meets the
// accumulators walks the same items and keeps the same counts, which are the phases of the halves' barriers.
struct MgHalves {
    uint32_t uses[2] = {0, 0};
    bool wide = false;
    int half = 0;
    __device__ __forceinline__ void next(int routes) {
        wide = routes > 64;
        half = uses[0] <= uses[1] ? 0 : 1;
    }
    __device__ __forceinline__ bool takes(int h) const { return wide || h == half; }
    __device__ __forceinline__ uint32_t column(int matrix) const { return wide ? matrix * 128 : half * 128 + matrix * 64; }
    __device__ __forceinline__ void done() {
        if (takes(0)) ++uses[0];
        if (takes(1)) ++uses[1];
    }
};

__device__ __forceinline__ void mg_tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]),
        "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]) : "memory");
}

// 8-route tiles come in runs of the same expert: a piece is up to eight tiles of a run, and an item of the kernel below a piece and a column block.
// list[i] = first tile | (tiles - 1) << 12 | local expert << 16.  Tiles of other GPUs' experts are left out.  Every CTA makes the same list.
__device__ __forceinline__ int mg_list_pieces(const MoeGroupedArgs& a, int n, uint32_t* list, int* warp_counts) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int pieces = 0;
    for (int base = 0; base < n; base += MG_TILE8_THREADS) {
        const int t = base + threadIdx.x;
        bool first = false;
        int count = 0, e = 0;
        if (t < n) {
            e = a.tile_expert[t];
            if (e >= a.expert_base && e < a.expert_base + a.experts_local) {
                int before = 0;  // tiles of this expert ahead of t
                while (before < t && a.tile_expert[t - before - 1] == e) ++before;
                first = (before & (MG_TILE8_ROUTES / 8 - 1)) == 0;
                while (first && count < MG_TILE8_ROUTES / 8 && t + count < n && a.tile_expert[t + count] == e) ++count;
            }
        }
        const unsigned votes = __ballot_sync(0xffffffffu, first);
        if (lane == 0) warp_counts[warp] = __popc(votes);
        __syncthreads();
        int at = pieces;
        for (int w = 0; w < MG_TILE8_THREADS / 32; ++w) {
            if (w < warp) at += warp_counts[w];
            pieces += warp_counts[w];
        }
        if (first) list[at + __popc(votes & ((1u << lane) - 1))] = (uint32_t)t | (uint32_t)(count - 1) << 12 | (uint32_t)(e - a.expert_base) << 16;
        __syncthreads();
    }
    return pieces;
}

// Results of 16 routes from `r0` on for this warp's 32 weight rows: thread = weight row = TMEM lane; neighbouring lanes swap, so that each stores two columns
// of one route.  route16 / weight16: of column r0 + lane % 16 (-1: none).
template <bool TILES8>
__device__ __forceinline__ void mg_store16(const MoeGroupedArgs& a, uint32_t d0, uint32_t d1, int r0, int routes, int row0, int n0, int lane, int route16,
                                           float weight16) {
    if (a.mode == 0) {
        uint32_t g[16], u[16];
        tmem_ld16(d0 + r0, g);
        tmem_ld16(d1 + r0, u);
#pragma unroll
        for (int e = 0; e < 16; e += 2) {
            float v[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const float gv = bf16_round(__uint_as_float(g[e + q])), uv = bf16_round(__uint_as_float(u[e + q]));
                v[q] = gv * sigmoidf_precise(gv) * uv;
            }
            const float got = __shfl_xor_sync(0xffffffffu, (lane & 1) ? v[0] : v[1], 1);
            const int r = r0 + e + (lane & 1);
            const int to = TILES8 ? __shfl_sync(0xffffffffu, route16, e + (lane & 1)) : r < routes ? row0 + r : -1;
            if (to >= 0 && n0 < a.N)
                *reinterpret_cast<uint32_t*>(a.out + (int64_t)to * a.N + n0) = (lane & 1) ? pack_bf16(got, v[1]) : pack_bf16(v[0], got);
        }
    } else {
        uint32_t x[2][16];
        tmem_ld16(d0 + r0, x[0]);
        tmem_ld16(d1 + r0, x[1]);
#pragma unroll
        for (int e = 0; e < 16; e += 2) {
            const int to = __shfl_sync(0xffffffffu, route16, e + (lane & 1));
            const float w0 = __shfl_sync(0xffffffffu, weight16, e), w1 = __shfl_sync(0xffffffffu, weight16, e + 1);
            bf16* dst = a.out + (int64_t)to * a.N + n0;
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                const float v0 = bf16_round(__uint_as_float(x[m][e])) * w0, v1 = bf16_round(__uint_as_float(x[m][e + 1])) * w1;
                const float got = __shfl_xor_sync(0xffffffffu, (lane & 1) ? v0 : v1, 1);
                if (to >= 0 && n0 + m * 128 < a.N)
                    *reinterpret_cast<uint32_t*>(dst + m * 128) = (lane & 1) ? pack_bf16(got, v1) : pack_bf16(v0, got);
            }
        }
    }
}

// TILES8: the routes come as tiles of eight (row lists) instead of sorted rows, and their activations are gathered by warp 22 with cp.async.
template <bool TILES8>
__global__ void __launch_bounds__(TILES8 ? MG_TILE8_THREADS : MG_THREADS, 1)
moe_grouped_fp8w_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w0, const __grid_constant__ CUtensorMap map_w1,
                        MoeGroupedArgs a) {
    GLMB_PDL_PROLOGUE();
    constexpr int STAGES = TILES8 ? MG_TILE8_STAGES : MG_STAGES, XBOX = TILES8 ? MG_TILE8_BOX : MG_BOX;
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t x_full[STAGES], x_empty[STAGES], raw_full[MG_RAW], raw_empty[MG_RAW], w_full[4], w_empty[4], acc_full[2], acc_empty[2], wide_full, wide_done;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile uint32_t fail;
    __shared__ int warp_counts[MG_TILE8_THREADS / 32];
    unsigned char* x_s = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* raw_s = x_s + STAGES * 2 * XBOX;
    uint32_t* list = reinterpret_cast<uint32_t*>(raw_s + MG_RAW * 2 * MG_BOX);
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int cols = a.mode == 0 ? 128 : 256;  // output columns of a tile
    const int blocks = (a.N + cols - 1) / cols, steps = (a.K + MG_BK - 1) / MG_BK;
    const int n_tiles = a.n_tiles ? min(max(*a.n_tiles, 0), a.max_tiles) : a.max_tiles;
    const int items = (TILES8 ? mg_list_pieces(a, n_tiles, list, warp_counts) : n_tiles) * blocks;  // item = route tile * blocks + column block
    auto tile_of = [&](int it) {
        if constexpr (TILES8) {
            const uint32_t p = list[it / blocks];
            const int first = p & 0xfff;
            return TcTile{first * 8, (first + 1 + (int)(p >> 12 & 7)) * 8, (int)(p >> 16), 0};
        } else {
            return a.tiles[it / blocks];
        }
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(x_full + s, 1); mbar_init(x_empty + s, 1); }
        for (int s = 0; s < MG_RAW; ++s) { mbar_init(raw_full + s, 1); mbar_init(raw_empty + s, MG_CONV_WARPS / 2); }
        for (int j = 0; j < 4; ++j) { mbar_init(w_full + j, MG_CONV_WARPS / 4); mbar_init(w_empty + j, 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(acc_full + i, 1); mbar_init(acc_empty + i, 4); }
        mbar_init(&wide_full, 1);
        mbar_init(&wide_done, MG_CONV_WARPS);
        fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;

    if (warp == 0) {
        uint32_t g = 0;  // steps so far, over the items of this CTA
        bool ok = true;
        for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
            const TcTile t = tile_of(it);
            const int routes = min(t.row_end - t.row0, MG_ROUTES), boxes = (routes + 31) >> 5;
            const int w_row = t.expert * a.N + (it % blocks) * cols, w_row1 = a.mode == 0 ? w_row : w_row + 128;  // rows past N are never stored
            for (int kb = 0; kb < steps; ++kb, ++g) {
                const uint32_t s = g % STAGES, lap = g / STAGES, q = g % MG_RAW, raw_lap = g / MG_RAW;
                if (raw_lap > 0 && !mbar_wait_warp(raw_empty + q, (raw_lap - 1) & 1)) { fail = 1; ok = false; break; }
                if (elect_one()) {
                    mbar_expect_tx(raw_full + q, 2 * MG_BOX);
                    tma_load_2d(raw_s + q * 2 * MG_BOX, &map_w0, raw_full + q, kb * MG_BK, w_row);
                    tma_load_2d(raw_s + (q * 2 + 1) * MG_BOX, &map_w1, raw_full + q, kb * MG_BK, w_row1);
                }
                __syncwarp();
                if constexpr (!TILES8) {
                    if (lap > 0 && !mbar_wait_warp(x_empty + s, (lap - 1) & 1)) { fail = 1; ok = false; break; }
                    if (elect_one()) {
                        mbar_expect_tx(x_full + s, boxes * 2 * 4096);
                        for (int h = 0; h < 2; ++h)
                            for (int b = 0; b < boxes; ++b)
                                tma_load_2d(x_s + (s * 2 + h) * MG_BOX + b * 4096, &map_a, x_full + s, kb * MG_BK + h * 64, t.row0 + b * 32);
                    }
                    __syncwarp();
                }
            }
        }
    } else if (TILES8 && warp == MG_THREADS / 32) {
        // ---- gather: lane l copies 16-byte piece l % 8 of the rows l / 8 + 4 i; rows past the routes up to a multiple of 16 are zeros, as those of no route.
        // A step is handed on one step later, when its copies have arrived
        const int piece = lane & 7;
        uint32_t g = 0;
        bool ok = true;
        for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
            const TcTile t = tile_of(it);
            const int routes = t.row_end - t.row0, rows16 = (routes + 15) & ~15;
            int from[MG_TILE8_ROUTES / 4];
#pragma unroll
            for (int i = 0; i < MG_TILE8_ROUTES / 4; ++i) {
                const int r = i * 4 + (lane >> 3), p = r < routes ? a.tile_routes[t.row0 + r] : -1;
                from[i] = p >= 0 ? p / a.divisor : -1;
            }
            for (int kb = 0; kb < steps; ++kb, ++g) {
                const uint32_t s = g % STAGES, lap = g / STAGES;
                if (lap > 0 && !mbar_wait_warp(x_empty + s, (lap - 1) & 1)) { fail = 1; ok = false; break; }
                const uint32_t dst = smem_u32(x_s + s * 2 * XBOX);
#pragma unroll
                for (int i = 0; i < MG_TILE8_ROUTES / 4; ++i)
                    if (i * 4 < rows16) {
                        const int r = i * 4 + (lane >> 3);
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const int k = kb * MG_BK + h * 64 + piece * 8;
                            const bool live = from[i] >= 0 && k < a.K;
                            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                                         ::"r"(dst + h * XBOX + r * 128 + ((piece ^ (r & 7)) << 4)), "l"(a.x + (live ? from[i] * a.x_stride + k : 0)),
                                         "r"(live ? 16 : 0) : "memory");
                        }
                    }
                asm volatile("cp.async.commit_group;" ::: "memory");
                if (g >= 1) {
                    asm volatile("cp.async.wait_group 1;" ::: "memory");
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the copies -> visible to the tensor core
                    __syncwarp();
                    if (lane == 0) mbar_arrive(x_full + (g - 1) % STAGES);
                }
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (ok && g > 0 && lane == 0) mbar_arrive(x_full + (g - 1) % STAGES);
    } else if (warp == 1) {
        uint32_t g = 0, wides = 0;
        MgHalves at;
        for (int it = blockIdx.x; it < items; it += gridDim.x) {
            const TcTile t = tile_of(it);
            const int routes = min(max((t.row_end - t.row0 + 15) & ~15, 16), MG_ROUTES);
            const uint32_t idesc = umma_idesc_bf16(128, routes);
            at.next(routes);
            bool ok = true;
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (ok && at.takes(h) && at.uses[h] > 0) ok = mbar_wait_warp(acc_empty + h, (at.uses[h] - 1) & 1);
            if (ok && wides > 0) ok = mbar_wait_warp(&wide_done, (wides - 1) & 1);
            if (!ok) { fail = 1; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int kb = 0; kb < steps && ok; ++kb, ++g) {
                const uint32_t s = g % STAGES;
                ok = mbar_wait_warp(x_full + s, (g / STAGES) & 1);
                const uint32_t x_addr = smem_u32(x_s + s * 2 * XBOX);
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    const uint32_t j = m * 2 + (g & 1);
                    if (ok) ok = mbar_wait_warp(w_full + j, (g >> 1) & 1);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < MG_BK / 16; ++k)
                            umma_bf16_ts(tmem + at.column(m), tmem + MG_A_COL + j * 64 + k * 8, umma_desc_sw128(x_addr + (k >> 2) * XBOX + (k & 3) * 32), idesc,
                                         (kb > 0 || k > 0) ? 1u : 0u);
                        umma_commit(w_empty + j);
                        if (m == 1) umma_commit(x_empty + s);
                    }
                    __syncwarp();
                }
            }
            if (!ok) fail = 1;
            if (elect_one()) {  // complete, or abandoned after a timeout: either way release the epilogue
                if (at.takes(0)) umma_commit(acc_full);
                if (at.takes(1)) umma_commit(acc_full + 1);
                if (at.wide) umma_commit(&wide_full);
            }
            __syncwarp();
            if (!ok) break;
            wides += at.wide;
            at.done();
        }
    } else if (warp >= 6) {
        // ---- decode: thread = weight row = TMEM lane; four sets of four warps: (matrix, parity of the step).  While one set waits for the tensor core to
        // give its stage back and for its own stores, the other converts: sixteen warps on every step, a half row each, did all of that together
        // and spent a third of a step in waits
        const int set = (warp - 6) >> 2, m = set >> 1, j = set & 1, quarter = warp & 3, row = quarter * 32 + lane;
        const int n_srows = (a.N + 127) >> 7, n_scols = (a.K + 127) >> 7;
        const float* const scales = m ? a.scale1 : a.scale0;
        const uint32_t a_addr = tmem + ((uint32_t)(quarter * 32) << 16) + MG_A_COL + (m * 2 + j) * 64;
        const unsigned char* const line = raw_s + m * MG_BOX + row * 128;
        auto scales_of = [&](int it) {
            const int n0 = (it % blocks) * cols + (a.mode == 1 ? m * 128 : 0);
            return scales + ((int64_t)tile_of(it).expert * n_srows + min(n0 >> 7, n_srows - 1)) * n_scols;
        };
        uint32_t g = 0, wides = 0;
        bool ok = true, asked = false;
        float next = 0.f;  // the scale of this set's next step, asked for a step ahead
        for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
            const float* sc = scales_of(it);
            for (int kb = 0; kb < steps; ++kb, ++g) {
                if ((int)(g & 1) != j) continue;
                const uint32_t q = g % MG_RAW, lap = g >> 1;
                const float scale = asked ? next : __ldg(sc + kb);
                asked = kb + 2 < steps || (steps > 1 && it + (int)gridDim.x < items);
                if (asked) next = __ldg(kb + 2 < steps ? sc + kb + 2 : scales_of(it + gridDim.x) + kb + 2 - steps);
                if (!mbar_wait_warp(raw_full + q, (g / MG_RAW) & 1)) { fail = 1; ok = false; break; }
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    uint4 w[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) w[i] = *reinterpret_cast<const uint4*>(line + q * 2 * MG_BOX + (((half * 4 + i) ^ (row & 7)) << 4));
                    uint32_t v[32];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint32_t c[4] = {w[i].x, w[i].y, w[i].z, w[i].w};
#pragma unroll
                        for (int p = 0; p < 4; ++p) {
                            v[i * 8 + 2 * p] = dec2_packed(c[p], scale);
                            v[i * 8 + 2 * p + 1] = dec2_packed(c[p] >> 16, scale);
                        }
                    }
                    __syncwarp();
                    if (half == 1 && lane == 0) mbar_arrive(raw_empty + q);
                    if (half == 0) {
                        if (lap > 0 && !mbar_wait_warp(w_empty + m * 2 + j, (lap - 1) & 1)) { fail = 1; ok = false; break; }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    }
                    mg_tmem_st32(a_addr + half * 32, v);
                }
                if (!ok) break;
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(w_full + m * 2 + j);
            }
            if constexpr (!TILES8) {
                // A tile of more than 64 routes has all the accumulators, so the next one waits for its epilogue: these warps, which have nothing to decode
                // for meanwhile, take four of every five pieces of 16 routes
                const TcTile t = tile_of(it);
                const int routes = min(t.row_end - t.row0, MG_ROUTES), n0 = (it % blocks) * cols + quarter * 32 + (lane & ~1);
                if (routes <= 64 || !ok) continue;
                const bool done = mbar_wait_warp(&wide_full, wides++ & 1);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (!done || __any_sync(0xffffffffu, fail)) {
                    fail = 1;
                    if (lane == 0) raise_status(a.status, GLMB_STATUS_WAIT_TIMEOUT);
                    break;
                }
                const uint32_t d = tmem + ((uint32_t)(quarter * 32) << 16);
#pragma unroll 1
                for (int r0 = (set + 1) * 16; r0 < routes; r0 += MG_TEAMS * 16) {
                    const int r = r0 + (lane & 15), route = r < routes && a.mode == 1 ? a.perm[t.row0 + r] : -1;
                    mg_store16<TILES8>(a, d, d + 128, r0, routes, t.row0, n0, lane, route, route >= 0 ? bf16_round(a.route_weight[route]) : 0.f);
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&wide_done);
            }
        }
    } else {
        // ---- epilogue -----------
        const int quarter = warp & 3;
        const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
        MgHalves at;
        for (int it = blockIdx.x; it < items; it += gridDim.x) {
            const TcTile t = tile_of(it);
            const int routes = min(t.row_end - t.row0, MG_ROUTES), n0 = (it % blocks) * cols + quarter * 32 + (lane & ~1);
            at.next(min(max((routes + 15) & ~15, 16), MG_ROUTES));
            int route[4];  // of columns lane, lane + 32, ..: asked for while the products are still under way
            float weight[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = i * 32 + lane;
                route[i] = r >= routes ? -1 : TILES8 ? a.tile_routes[t.row0 + r] : a.mode == 1 ? a.perm[t.row0 + r] : -1;
                weight[i] = a.mode == 1 && route[i] >= 0 ? bf16_round(a.route_weight[route[i]]) : 0.f;
            }
            bool done = true;
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (done && at.takes(h)) done = mbar_wait_warp(acc_full + h, at.uses[h] & 1);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (!done || __any_sync(0xffffffffu, fail)) {
                fail = 1;
                if (lane == 0) raise_status(a.status, GLMB_STATUS_WAIT_TIMEOUT);
                if constexpr (TILES8)  // a caller may have no status word: what is missing becomes NaN
                    for (; it < items; it += gridDim.x) {
                        const TcTile rest = tile_of(it);
                        for (int r = rest.row0; r < rest.row_end; ++r)
                            for (int n = (it % blocks) * cols + quarter * 32 + lane; n < min((it % blocks + 1) * cols, a.N); n += 128)
                                if (a.tile_routes[r] >= 0) a.out[(int64_t)a.tile_routes[r] * a.N + n] = __ushort_as_bfloat16(0x7fff);
                    }
                break;
            }
            const uint32_t d0 = tmem + lanes + at.column(0), d1 = tmem + lanes + at.column(1);
#pragma unroll 1
            for (int r0 = 0; r0 < routes; r0 += at.wide ? MG_TEAMS * 16 : 16) {  // a tile of more than 64 routes: the decode warps take the others
                const int q = r0 >> 5, from = (r0 & 31) + (lane & 15);
                const int route16 = __shfl_sync(0xffffffffu, q < 2 ? (q ? route[1] : route[0]) : (q & 1 ? route[3] : route[2]), from);
                const float weight16 = __shfl_sync(0xffffffffu, q < 2 ? (q ? weight[1] : weight[0]) : (q & 1 ? weight[3] : weight[2]), from);
                mg_store16<TILES8>(a, d0, d1, r0, routes, t.row0, n0, lane, route16, weight16);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                if (at.takes(0)) mbar_arrive(acc_empty);
                if (at.takes(1)) mbar_arrive(acc_empty + 1);
            }
            at.done();
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// ---------------------------------------------------------------------------------------------------
// dst[i] = src[idx[i]] (rows of `width` bf16, width % 8 == 0); idx < 0 -> a row of zeros.  Expert-sorted copy of the
// activations, so that one TMA box covers 128 routes of one expert.
__global__ void __launch_bounds__(256)
gather_rows_kernel(const bf16* __restrict__ src, int64_t src_stride, const int* __restrict__ idx, int divisor, bf16* __restrict__ dst,
                   int width) {
    GLMB_PDL_PROLOGUE();
    const int i = blockIdx.x;
    const int from = idx[i];
    const uint4* s = reinterpret_cast<const uint4*>(src + (int64_t)(from >= 0 ? from / divisor : 0) * src_stride);
    uint4* d = reinterpret_cast<uint4*>(dst + (int64_t)i * width);
    for (int v = threadIdx.x; v < width / 8; v += blockDim.x) d[v] = from >= 0 ? s[v] : make_uint4(0, 0, 0, 0);
}

// ===================================================================================================
// a_sorted [sorted_rows, K] bf16 (expert-sorted routes), w0/w1 [experts, N, K] FP8 bytes with block scales s0/s1,
// tiles/n_tiles on the device (max_tiles entries).  mode 0: out = act_sorted [sorted_rows, N] (w0 gate, w1 up);
// mode 1: out = dw [routes, N] scattered through perm, scaled by route_weight (w1/s1 ignored, the kernel uses w0/s0).
GLMB_API int glmb_moe_grouped_fp8w(const void* a_sorted, int sorted_rows, const void* w0, const void* w1, const float* s0,
                                   const float* s1, int experts, int N, int K, const void* tiles, const int* n_tiles, int max_tiles,
                                   int mode, const int* perm, const float* route_weight, void* out, uint32_t* status, void* stream) {
    if (sorted_rows < 1 || experts < 1 || max_tiles < 1 || N < 8 || (N & 7) || K < 16 || (K & 15) || mode < 0 || mode > 1) return 1;
    if (mode == 1 && (!perm || !route_weight)) return 1;
    if ((reinterpret_cast<uintptr_t>(a_sorted) & 15) || (reinterpret_cast<uintptr_t>(w0) & 15) || (reinterpret_cast<uintptr_t>(out) & 15)) return 1;
    if (mode == 0 && (!w1 || !s1 || (reinterpret_cast<uintptr_t>(w1) & 15))) return 1;
    CUtensorMap map_a, map_w0, map_w1;
    if (make_map(&map_a, a_sorted, (uint64_t)sorted_rows, (uint64_t)K, (uint64_t)K, 32)) return 3;
    if (make_map_u8(&map_w0, w0, (uint64_t)experts * N, (uint64_t)K, (uint64_t)K, 128)) return 3;
    if (make_map_u8(&map_w1, mode == 0 ? w1 : w0, (uint64_t)experts * N, (uint64_t)K, (uint64_t)K, 128)) return 3;
    static DeviceOnce attr_set;
    const int attr_set_dev = attr_set.pending();
    if (attr_set_dev != DeviceOnce::SET) {
        cudaError_t e = cudaFuncSetAttribute(moe_grouped_fp8w_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, MG_SMEM_BYTES);
        if (e != cudaSuccess) return (int)e;
        attr_set.mark(attr_set_dev);
    }
    MoeGroupedArgs args = {};
    args.tiles = (const TcTile*)tiles;
    args.n_tiles = n_tiles;
    args.scale0 = s0;
    args.scale1 = mode == 0 ? s1 : s0;
    args.perm = perm;
    args.route_weight = route_weight;
    args.out = (bf16*)out;
    args.N = N; args.K = K; args.mode = mode; args.max_tiles = max_tiles;
    args.status = status;
    const int64_t most = (int64_t)(mode == 0 ? ceil_div(N, 128) : ceil_div(N, 256)) * max_tiles;
    GLMB_LAUNCH(moe_grouped_fp8w_kernel<false>, (int)(most < 148 ? most : 148), MG_THREADS, MG_SMEM_BYTES, (cudaStream_t)stream, map_a, map_w0, map_w1, args);
    return (int)cudaGetLastError();
}

// Tiles of eight routes (route_sort8), the weights as M: an expert's weights are read once for up to MG_TILE8_ROUTES routes, where a kernel with a tile per
// CTA reads and decodes them for every eight.  What it can take; with fewer than 512 columns the stretch of products is too short for its epilogue.
// mode 0: act [routes, N] of x [rows, K], route p of row p / divisor; mode 1: dw [routes, N] of x = act [routes, K], times route_weight.
bool moe_tiles8_takes(const void* x, int64_t x_stride, const void* w0, const void* w1, const void* out, const int* tile_routes, int tiles, int experts, int N, int K) {
    return tile_routes && tiles <= MG_LIST && experts <= 65536 && K >= 512 && !(K & 63) && N >= 256 && !(N & 15) && !(x_stride & 7) &&
           !((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w0) | reinterpret_cast<uintptr_t>(w1) | reinterpret_cast<uintptr_t>(out)) & 15);
}
// Whether it is expected to be the faster form.  Small experts, and few of them, end before its start is over ([8 x 1024 x 1024] and back, 9 rows of the top 2:
// 13.1 + 12.1 us against 6.0 + 4.0 on mma.sync), and a round of its 148 CTAs just begun costs as much as a full one ([256 x 256 x 6144], 12 rows of the top 8: 84
// against 67).  Here 10 us, and a round of items of 256 weight rows at 41 GB/s a CTA; there 3 us, and CTAs of 16 rows whose warps take chunks of 64 columns in
// turns of eight (the form for up to 512 columns: a warp to 16 rows).  `tiles` is an eighth of the routes and one per expert (the length of the list, not its
// count on the device); routes are taken to be dealt at random.  Of 231 measured launches (8 to 256 experts, 9 to 256 rows) the choice costs more than 9 % in three:
// 64 rows of [16 x 640 x 576] 13.6 us, not 11.2, and of the second half 200 rows of [8 x 1024 x 1024] 19.4, not 16.0, 100 of [16 x 4096 x 1024] 35.7, not 30.9.
static bool moe_tiles8_pays(int tiles, int experts, int N, int K, int mode) {
    const double routes = 8.0 * (tiles > experts ? tiles - experts : 0) + 4.0, chosen = experts * (1.0 - pow(1.0 - 1.0 / experts, routes));
    const double tiles8 = fmax(chosen, routes / 8 + chosen * 7 / 16), pieces = fmax(chosen, routes / MG_TILE8_ROUTES + chosen * 63 / 128);
    const double rounds = pieces * ceil_div(N, mode == 0 ? 128 : 256) / 148, columns = ceil_div(K, 512) * 512.0 * (mode == 0 ? 2 : 1);
    const double here = 10.0 + (rounds > 1.0 ? rounds + 0.5 : 1.0) * (256.0 * K / 41e3 + 1.25);
    const double there = 3.0 + tiles8 * N / 16 * (0.8e-3 + 3.8e-6 * columns) * (mode == 1 && K <= 512 ? 0.75 : 1.0);
    return here < there;
}
GLMB_API int glmb_moe_tiles8_pays(int tiles, int experts, int N, int K, int mode) { return experts > 0 && moe_tiles8_pays(tiles, experts, N, K, mode); }
int launch_moe_tiles8(const void* x, int64_t x_stride, int divisor, const int* tile_expert, const int* tile_routes, const int* n_tiles, int tiles,
                      const void* w0, const void* w1, const float* s0, const float* s1, int expert_base, int experts_local, int N, int K, int mode,
                      const float* route_weight, void* out, uint32_t* status, cudaStream_t stream) {
    CUtensorMap map_w0, map_w1;
    if (make_map_u8(&map_w0, w0, (uint64_t)experts_local * N, (uint64_t)K, (uint64_t)K, 128)) return 3;
    if (make_map_u8(&map_w1, mode == 0 ? w1 : w0, (uint64_t)experts_local * N, (uint64_t)K, (uint64_t)K, 128)) return 3;
    static DeviceOnce attr_set;
    const int dev = attr_set.pending();
    if (dev != DeviceOnce::SET) {
        cudaError_t e = cudaFuncSetAttribute(moe_grouped_fp8w_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, MG_TILE8_SMEM_BYTES);
        if (e != cudaSuccess) return (int)e;
        attr_set.mark(dev);
    }
    MoeGroupedArgs args = {};
    args.tile_expert = tile_expert; args.tile_routes = tile_routes; args.n_tiles = n_tiles; args.max_tiles = tiles;
    args.x = (const bf16*)x; args.x_stride = x_stride; args.divisor = divisor;
    args.expert_base = expert_base; args.experts_local = experts_local;
    args.scale0 = s0; args.scale1 = mode == 0 ? s1 : s0;
    args.route_weight = route_weight; args.out = (bf16*)out;
    args.N = N; args.K = K; args.mode = mode; args.status = status;
    const int64_t most = (int64_t)ceil_div(N, mode == 0 ? 128 : 256) * tiles;
    GLMB_LAUNCH(moe_grouped_fp8w_kernel<true>, (int)(most < 148 ? most : 148), MG_TILE8_THREADS, MG_TILE8_SMEM_BYTES, stream, map_w0, map_w0, map_w1, args);
    return (int)cudaGetLastError();
}

// dst [n, width] = src[idx[i] / divisor] (idx < 0: zeros).  width % 8 == 0, rows 16-byte aligned.
GLMB_API int glmb_gather_rows(const void* src, int64_t src_stride, const int* idx, int divisor, void* dst, int n, int width,
                              void* stream) {
    if (n < 1 || (width & 7) || divisor < 1 || (src_stride & 7)) return 1;
    GLMB_LAUNCH(gather_rows_kernel, n, 256, 0, (cudaStream_t)stream, (const bf16*)src, src_stride, idx, divisor, (bf16*)dst, width);
    return (int)cudaGetLastError();
}
