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
//   warps 6-21   decode, a team of eight warps per matrix: 64 codes per thread, straight from global memory (a piece is asked for again,
//                for two steps later, as soon as it has been decoded), block scale in fp32, rounded to bf16 (the weight-decode
//                contract), into two 64-column boxes in the 128-byte-swizzled K-major layout of the tensor core; a proxy fence
//                publishes them.  A team has two such stages, so that it decodes one while the tensor core reads the other
//   warp 0       TMA: the activations of the tile's routes (32-row boxes, as many as there are routes)
//   warp 1       issues tcgen05.mma (two matrices of M 128, N 16 .. 128) into one of two sets of TMEM accumulators
//   warps 2-5    epilogue of the tile before, while the next one is decoded and multiplied: a thread owns a weight row (TMEM lane)
//                  gate/up mode  act = bf16( silu(bf16 gate) * bf16 up ), stored in sorted order
//                  down mode     dw[route] = bf16( bf16(acc) * bf16(route weight) ), scattered to the route's slot
//
// What bounds it: shared-memory traffic (decoded weights in and out to the tensor core, activations) and the decoding, at 3.3 TB/s of weights
// whatever the number of routes; prefetching whole stretches of a row into the L2 changes nothing.  Measured on a B200, [256 experts, 2 x 2048 x
// 6144] and back, against routes as the M in tiles of 128 and weights through shared memory twice: 2,048 rows 2,377 + 1,302 -> 1,891 + 1,034 us,
// 777 rows 1,931 + 1,065 -> 1,680 + 856.
// Every mbarrier wait is bounded; on a timeout the kernel raises GLMB_STATUS_WAIT_TIMEOUT, skips its stores and
// still frees its TMEM.
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
#define MG_WSTAGES 4   // decoded weights: two of each matrix, two boxes each
#define MG_TEAM_WARPS 8
#define MG_THREADS (6 * 32 + 2 * 32 * MG_TEAM_WARPS)
#define MG_SMEM_BYTES ((MG_STAGES * 2 + MG_WSTAGES * 2) * MG_BOX + 1024)

struct MoeGroupedArgs {
    const TcTile* tiles;      // [max_tiles] 128-route tiles of the expert-sorted route list (row0, the expert's row_end, local expert)
    const int* n_tiles;       // [1] on the device
    const uint8_t* w0;        // [experts, N, K] FP8: gate, or down
    const uint8_t* w1;        // up (gate/up mode), or down again
    const float* scale0;      // block scales of w0 [experts, ceil(N/128), ceil(K/128)]
    const float* scale1;      // ... of w1
    const int* perm;          // [sorted routes] -> route id (row * top_k + slot), -1 for none   (down mode)
    const float* route_weight;  // [routes] fp32                                                  (down mode)
    bf16* out;                // gate/up: act_sorted [sorted routes, N];  down: dw [routes, N]
    int N, K, mode;           // mode 0: gate/up (N = expert FFN width), 1: down (N = hidden size)
    int max_tiles;
    uint32_t* status;
};

__global__ void __launch_bounds__(MG_THREADS, 1) moe_grouped_fp8w_kernel(const __grid_constant__ CUtensorMap map_a, MoeGroupedArgs a) {
    GLMB_PDL_PROLOGUE();
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t x_full[MG_STAGES], x_empty[MG_STAGES], w_full[MG_WSTAGES], w_empty[MG_WSTAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile uint32_t fail;
    unsigned char* x_s = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* w_s = x_s + MG_STAGES * 2 * MG_BOX;
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int cols = a.mode == 0 ? 128 : 256;  // output columns of a tile
    const int blocks = (a.N + cols - 1) / cols, steps = (a.K + MG_BK - 1) / MG_BK;
    const int items = min(max(*a.n_tiles, 0), a.max_tiles) * blocks;  // item = route tile * blocks + column block

    if (threadIdx.x == 0) {
        for (int s = 0; s < MG_STAGES; ++s) { mbar_init(x_full + s, 1); mbar_init(x_empty + s, 1); }
        for (int j = 0; j < MG_WSTAGES; ++j) { mbar_init(w_full + j, MG_TEAM_WARPS); mbar_init(w_empty + j, 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(acc_full + i, 1); mbar_init(acc_empty + i, 4); }
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
    const uint32_t tmem = tmem_slot;  // accumulator set i at 256 i: matrix 0, then matrix 1, a column per route

    if (warp == 0) {
        uint32_t g = 0;  // steps so far, over the items of this CTA
        bool ok = true;
        for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
            const TcTile t = a.tiles[it / blocks];
            const int boxes = (min(t.row_end - t.row0, MG_ROUTES) + 31) >> 5;
            for (int kb = 0; kb < steps; ++kb, ++g) {
                const uint32_t s = g % MG_STAGES, lap = g / MG_STAGES;
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
    } else if (warp == 1) {
        uint32_t g = 0, i = 0;
        for (int it = blockIdx.x; it < items; it += gridDim.x, ++i) {
            const TcTile t = a.tiles[it / blocks];
            const uint32_t acc = i & 1, use = i >> 1;
            const int routes = min(max((t.row_end - t.row0 + 15) & ~15, 16), MG_ROUTES);
            const uint32_t idesc = umma_idesc_bf16(128, routes);
            if (use > 0 && !mbar_wait_warp(acc_empty + acc, (use - 1) & 1)) { fail = 1; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            bool ok = true;
            for (int kb = 0; kb < steps; ++kb, ++g) {
                const uint32_t s = g % MG_STAGES;
                if (!mbar_wait_warp(x_full + s, (g / MG_STAGES) & 1)) { fail = 1; ok = false; break; }
                const uint32_t x_addr = smem_u32(x_s + s * 2 * MG_BOX);
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    const uint32_t j = m * 2 + (g & 1);
                    if (ok && !mbar_wait_warp(w_full + j, (g >> 1) & 1)) { fail = 1; ok = false; }
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t w_addr = smem_u32(w_s + j * 2 * MG_BOX);
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < MG_BK / 16; ++k) {
                            const uint32_t at = (k >> 2) * MG_BOX + (k & 3) * 32;
                            umma_bf16(tmem + acc * 256 + m * 128, umma_desc_sw128(w_addr + at), umma_desc_sw128(x_addr + at), idesc,
                                      (kb > 0 || k > 0) ? 1u : 0u);
                        }
                        umma_commit(w_empty + j);
                        if (m == 1) umma_commit(x_empty + s);
                    }
                    __syncwarp();
                }
                if (!ok) break;
            }
            if (elect_one()) umma_commit(acc_full + acc);  // complete, or abandoned after a timeout: either way release the epilogue
            __syncwarp();
            if (!ok) break;
        }
    } else if (warp >= 6) {
        // ---- decode: team = matrix; thread (row % 32, piece of 16 codes) of 128 rows ----------------------------------------------
        const int team = (warp - 6) / MG_TEAM_WARPS, dt = threadIdx.x - 192 - team * MG_TEAM_WARPS * 32, row = dt >> 3, c = dt & 7;
        const int n_srows = (a.N + 127) >> 7, n_scols = (a.K + 127) >> 7;
        const int mine = (int)blockIdx.x < items ? (items - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
        const int total = mine * steps, second = a.mode == 1 && team ? 128 : 0;  // where the team's columns begin in the tile
        const uint8_t* const table = team ? a.w1 : a.w0;
        const float* const scales = team ? a.scale1 : a.scale0;
        int l_it = blockIdx.x, l_kb = 0, l_step = 0, below = 0;  // the step whose codes are asked for next; rows from this thread's first one to N
        const uint8_t* base = nullptr;
        const float* sc = nullptr;
        auto aim = [&]() {
            if (l_step >= total) return;
            const int expert = a.tiles[l_it / blocks].expert, n0 = (l_it % blocks) * cols + second;
            below = a.N - n0 - row;
            base = table + ((int64_t)expert * a.N + n0 + row) * a.K + c * 16;
            sc = scales + ((int64_t)expert * n_srows + min(n0 >> 7, n_srows - 1)) * n_scols;
        };
        uint4 w[2][4];
        float s[2] = {0.f, 0.f};
        auto load = [&](uint4& to, int i) {
            const int k = l_kb * MG_BK;
            const bool in = l_step < total && k + c * 16 < a.K && i * 32 < below;
            to = in ? ld_stream16(base + (int64_t)(i * 32) * a.K + k) : make_uint4(0, 0, 0, 0);
        };
        auto onward = [&]() {
            ++l_step;
            if (++l_kb == steps) { l_kb = 0; l_it += gridDim.x; aim(); }
        };
        aim();
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            if (l_step < total) s[p] = __ldg(sc + l_kb);
#pragma unroll
            for (int i = 0; i < 4; ++i) load(w[p][i], i);
            onward();
        }
        // eight lanes hold a row's 128 columns: a quarter warp's first stores take the even chunks of the lower box and the odd ones
        // of the upper, so that they meet eight different groups of banks
        const int odd = c >> 2, chunk = (c & 3) * 2;
        unsigned char* line = w_s + team * 4 * MG_BOX + odd * MG_BOX + (row >> 3) * 1024 + (row & 7) * 128;
        unsigned char *at0 = line + (((chunk + odd) ^ (row & 7)) << 4), *at1 = line + (((chunk + 1 - odd) ^ (row & 7)) << 4);
        bool ok = true;
        for (int step = 0; step < total && ok; step += 2) {
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                if (step + p >= total) break;
                const uint32_t j = team * 2 + p, lap = step >> 1;
                if (lap > 0 && !mbar_wait_warp(w_empty + j, (lap - 1) & 1)) { fail = 1; ok = false; break; }
                const float scale = s[p];
                if (l_step < total) s[p] = __ldg(sc + l_kb);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint4 v = w[p][i];
                    const uint4 lo = make_uint4(dec2(v.x, scale), dec2(v.x >> 16, scale), dec2(v.y, scale), dec2(v.y >> 16, scale));
                    const uint4 hi = make_uint4(dec2(v.z, scale), dec2(v.z >> 16, scale), dec2(v.w, scale), dec2(v.w >> 16, scale));
                    load(w[p][i], i);
                    const int to = p * 2 * MG_BOX + i * 32 * 128;
                    *reinterpret_cast<uint4*>(at0 + to) = odd ? hi : lo;
                    *reinterpret_cast<uint4*>(at1 + to) = odd ? lo : hi;
                }
                onward();
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic-proxy stores -> visible to the tensor core
                __syncwarp();
                if (lane == 0) mbar_arrive(w_full + j);
            }
        }
    } else {
        // ---- epilogue: thread = weight row = TMEM lane; neighbouring lanes swap, so that each stores two columns of one route -----------
        const int quarter = warp & 3;
        const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
        uint32_t i = 0;
        for (int it = blockIdx.x; it < items; it += gridDim.x, ++i) {
            const TcTile t = a.tiles[it / blocks];
            const uint32_t acc = i & 1;
            const bool done = mbar_wait_warp(acc_full + acc, (i >> 1) & 1);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (!done || __any_sync(0xffffffffu, fail)) {
                fail = 1;
                if (lane == 0) raise_status(a.status, GLMB_STATUS_WAIT_TIMEOUT);
                break;
            }
            const int routes = min(t.row_end - t.row0, MG_ROUTES), n0 = (it % blocks) * cols + quarter * 32 + (lane & ~1);
            const uint32_t d = tmem + acc * 256 + lanes;
#pragma unroll 1
            for (int r0 = 0; r0 < routes; r0 += 16) {
                if (a.mode == 0) {
                    uint32_t g[16], u[16];
                    tmem_ld16(d + r0, g);
                    tmem_ld16(d + 128 + r0, u);
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
                        if (r < routes && n0 < a.N)
                            *reinterpret_cast<uint32_t*>(a.out + (int64_t)(t.row0 + r) * a.N + n0) = (lane & 1) ? pack_bf16(got, v[1]) : pack_bf16(v[0], got);
                    }
                } else {
                    int route = -1;  // of column r0 + lane
                    float weight = 0.f;
                    if (lane < 16 && r0 + lane < routes) route = a.perm[t.row0 + r0 + lane];
                    if (route >= 0) weight = bf16_round(a.route_weight[route]);
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        uint32_t x[16];
                        tmem_ld16(d + m * 128 + r0, x);
#pragma unroll
                        for (int e = 0; e < 16; e += 2) {
                            const float v0 = bf16_round(__uint_as_float(x[e])) * __shfl_sync(0xffffffffu, weight, e);
                            const float v1 = bf16_round(__uint_as_float(x[e + 1])) * __shfl_sync(0xffffffffu, weight, e + 1);
                            const float got = __shfl_xor_sync(0xffffffffu, (lane & 1) ? v0 : v1, 1);
                            const int to = __shfl_sync(0xffffffffu, route, e + (lane & 1));
                            if (to >= 0 && n0 + m * 128 < a.N)
                                *reinterpret_cast<uint32_t*>(a.out + (int64_t)to * a.N + n0 + m * 128) = (lane & 1) ? pack_bf16(got, v1) : pack_bf16(v0, got);
                        }
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty + acc);
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
    CUtensorMap map_a;
    if (make_map(&map_a, a_sorted, (uint64_t)sorted_rows, (uint64_t)K, (uint64_t)K, 32)) return 3;
    static DeviceOnce attr_set;
    const int attr_set_dev = attr_set.pending();
    if (attr_set_dev != DeviceOnce::SET) {
        cudaError_t e = cudaFuncSetAttribute(moe_grouped_fp8w_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MG_SMEM_BYTES);
        if (e != cudaSuccess) return (int)e;
        attr_set.mark(attr_set_dev);
    }
    MoeGroupedArgs args;
    args.tiles = (const TcTile*)tiles;
    args.n_tiles = n_tiles;
    args.w0 = (const uint8_t*)w0;
    args.w1 = (const uint8_t*)(mode == 0 ? w1 : w0);
    args.scale0 = s0;
    args.scale1 = mode == 0 ? s1 : s0;
    args.perm = perm;
    args.route_weight = route_weight;
    args.out = (bf16*)out;
    args.N = N; args.K = K; args.mode = mode; args.max_tiles = max_tiles;
    args.status = status;
    const int64_t most = (int64_t)(mode == 0 ? ceil_div(N, 128) : ceil_div(N, 256)) * max_tiles;
    GLMB_LAUNCH(moe_grouped_fp8w_kernel, (int)(most < 148 ? most : 148), MG_THREADS, MG_SMEM_BYTES, (cudaStream_t)stream, map_a, args);
    return (int)cudaGetLastError();
}

// dst [n, width] = src[idx[i] / divisor] (idx < 0: zeros).  width % 8 == 0, rows 16-byte aligned.
GLMB_API int glmb_gather_rows(const void* src, int64_t src_stride, const int* idx, int divisor, void* dst, int n, int width,
                              void* stream) {
    if (n < 1 || (width & 7) || divisor < 1 || (src_stride & 7)) return 1;
    GLMB_LAUNCH(gather_rows_kernel, n, 256, 0, (cudaStream_t)stream, (const bf16*)src, src_stride, idx, divisor, (bf16*)dst, width);
    return (int)cudaGetLastError();
}
