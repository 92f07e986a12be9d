// Dense bf16 GEMM of few rows (a short prompt, the tail of a long one), included by gemm_tcgen05.cu:  C[rows, N] = A[rows, K] . B[N, K]^T.
//
// The WEIGHT rows are the M of the product (128 at a time, always full) and the activation rows its N, in steps of 16 up to 128; more rows
// form several blocks.  A tile's K is dealt to the CTAs of a cluster, so that a projection with a few dozen tiles still has every SM streaming
// weights; the partial tiles meet in distributed shared memory and are added in the order of K, the same sums in every run.
//
//   warp 0      TMA producer (an elected lane issues)
//   warp 1      TMEM allocation, MMA issue
//   warps 2-5   partial tile TMEM -> shared memory (over the operand ring, whose last step has been multiplied)
//   all warps   the rows r = split, split + splits, .. of the tile: sums over the cluster, rounding, stores
//
// Bound by the latency of its start and of its two meetings in the cluster (13 us of a launch of its own, 2.6 of them the events') and, with several
// operands' worth of CTAs per SM, by the weights' bytes.  Measured on a B200, pairs of SMs (gemm_pair_tcgen05.cuh) -> here: [60 x 4096], K 18432: 69.6 -> 36.9 us,
// [60 x 6144], K 16384: 65.5 -> 43.0, [120 x 4096], K 12288: 49.2 -> 32.8, [120 x 2048], K 6144: 28.7 -> 22.5, [256 x 256], K 6144: 28.7 -> 18.4; [120 x
// 6144], K 4096: 24.6 either way; [200 x 12288], K 6144: 38.9 against 51.2.
//
// Every mbarrier wait is bounded; on a timeout the kernel raises GLMB_STATUS_WAIT_TIMEOUT, stores nothing of its share and still meets the
// cluster's barriers and frees its TMEM.
#pragma once

#include "tcgen05.cuh"

#define GF_THREADS 192
#define GF_A_BYTES (128 * 64 * 2)
#define GF_MAX_STAGES 8
#define GF_MAX_SPLITS 8
#define GF_ROWS 128              // most activation rows of a block
#define GF_RING (100 * 1024)     // two CTAs per SM

struct GemmFewArgs {
    void* c;
    int64_t ldc;
    const bf16* b;   // weights: only for the L2 prefetch ahead of the wait
    int64_t ldb;
    int rows, N, K, out_f32;
    int n_box;       // activation rows of a block, a multiple of 16
    int stages, splits, tiles_n, prefetch;
    uint32_t* status;
};

__device__ __forceinline__ void gf_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__global__ void __launch_bounds__(GF_THREADS)
gemm_few_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, GemmFewArgs p) {
    asm volatile("griddepcontrol.launch_dependents;");
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[GF_MAX_STAGES], empty_bar[GF_MAX_STAGES], acc_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile uint32_t fail;
    unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int split = blockIdx.x % p.splits, tile = blockIdx.x / p.splits;
    const int n0 = (tile % p.tiles_n) * 128, r0 = (tile / p.tiles_n) * p.n_box, rows = min(p.n_box, p.rows - r0);
    const int kblocks = (p.K + 63) / 64, per = (kblocks + p.splits - 1) / p.splits, k_first = split * per, steps = min(per, kblocks - k_first);  // >= 1
    const uint32_t stage_bytes = GF_A_BYTES + p.n_box * 128;
    const uint32_t columns = p.n_box <= 32 ? 32 : p.n_box <= 64 ? 64 : 128;

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) { mbar_init(full_bar + s, 1); mbar_init(empty_bar + s, 1); }
        mbar_init(&acc_bar, 1);
        fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (p.prefetch && warp >= 2) {  // this CTA's stretch of the weights, while the kernel before still runs
        const int row = n0 + (warp - 2) * 32 + lane;
        const uint32_t bytes = (uint32_t)min(steps * 128, (p.K - k_first * 64) * 2) & ~15u;
        if (row < p.N && bytes)
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p.b + (int64_t)row * p.ldb + k_first * 64), "r"(bytes) : "memory");
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");  // before the TMEM allocation: a kernel still running may need the columns to finish
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(columns) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;

    if (warp == 0) {
        for (int i = 0; i < steps; ++i) {
            const int s = i % p.stages, lap = i / p.stages;
            if (lap > 0 && !mbar_wait_warp(empty_bar + s, (lap - 1) & 1)) { fail = 1; break; }
            if (elect_one()) {
                unsigned char* dst = ring + s * stage_bytes;
                mbar_expect_tx(full_bar + s, stage_bytes);
                tma_load_2d(dst, &map_w, full_bar + s, (k_first + i) * 64, n0);
                tma_load_2d(dst + GF_A_BYTES, &map_x, full_bar + s, (k_first + i) * 64, r0);
            }
            __syncwarp();
        }
    } else if (warp == 1) {
        const uint32_t idesc = umma_idesc_bf16(128, p.n_box);
        for (int i = 0; i < steps; ++i) {
            const int s = i % p.stages;
            if (!mbar_wait_warp(full_bar + s, (i / p.stages) & 1)) { fail = 1; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_one()) {
                const uint32_t w_addr = smem_u32(ring + s * stage_bytes), x_addr = w_addr + GF_A_BYTES;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    umma_bf16(tmem, umma_desc_sw128(w_addr + k * 32), umma_desc_sw128(x_addr + k * 32), idesc, (i > 0 || k > 0) ? 1u : 0u);
                umma_commit(empty_bar + s);
            }
            __syncwarp();
        }
        if (elect_one()) umma_commit(&acc_bar);  // complete, or abandoned after a timeout: either way release the others
        __syncwarp();
    }
    // The accumulator is complete: every copy has arrived and been multiplied, so the ring may be written over.
    const bool ok = mbar_wait_warp(&acc_bar, 0);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (!ok) fail = 1;
    float* part = reinterpret_cast<float*>(ring);  // [rows][128 outputs]
    if (warp >= 2 && ok && !fail) {
        const int quarter = warp & 3, n = quarter * 32 + lane;
        const uint32_t at = tmem + ((uint32_t)(quarter * 32) << 16);
        for (int c = 0; c < rows; c += 16) {
            uint32_t v[16];
            tmem_ld16(at + c, v);
#pragma unroll
            for (int e = 0; e < 16; ++e)
                if (c + e < rows) part[(c + e) * 128 + n] = __uint_as_float(v[e]);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    gf_cluster_sync();
    const bool failed = fail != 0;  // of this CTA; what another one lacks, it reports itself
    if (failed && threadIdx.x == 0) raise_status(p.status, GLMB_STATUS_WAIT_TIMEOUT);
    if (!failed) {
        uint32_t from[GF_MAX_SPLITS];
#pragma unroll
        for (int q = 0; q < GF_MAX_SPLITS; ++q)
            asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(from[q]) : "r"(smem_u32(part)), "r"(q < p.splits ? q : 0));
        const int n = n0 + lane * 4, stride = p.splits * (GF_THREADS / 32);
        for (int first = split + warp * p.splits; first < rows; first += 4 * stride) {  // four rows together: a load from another SM takes long
            float4 sum[4];
#pragma unroll
            for (int q = 0; q < GF_MAX_SPLITS; ++q)
                if (q < p.splits) {
                    float4 v[4] = {};
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (first + i * stride < rows)
                            asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v[i].x), "=f"(v[i].y), "=f"(v[i].z), "=f"(v[i].w)
                                         : "r"(from[q] + (uint32_t)((first + i * stride) * 512 + lane * 16)) : "memory");
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (q == 0) sum[i] = v[i];
                        else { sum[i].x += v[i].x; sum[i].y += v[i].y; sum[i].z += v[i].z; sum[i].w += v[i].w; }
                    }
                }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = first + i * stride;
                if (r >= rows || n >= p.N) continue;  // N is a multiple of 8
                if (p.out_f32) *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.c) + (int64_t)(r0 + r) * p.ldc + n) = sum[i];
                else
                    *reinterpret_cast<uint2*>(reinterpret_cast<bf16*>(p.c) + (int64_t)(r0 + r) * p.ldc + n) =
                        make_uint2(pack_bf16(sum[i].x, sum[i].y), pack_bf16(sum[i].z, sum[i].w));
            }
        }
    }
    gf_cluster_sync();  // nobody leaves while another may still read its part
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(columns) : "memory");
}

struct GemmFewPlan { int n_box, blocks, splits, stages; double us; };

// How K is dealt, by the time expected of a launch of its own: 13 us, a 64-wide step of 0.29 us and 0.11 more with 128 rows (a CTA alone on its SM; beyond
// 148 CTAs they share the bandwidth), and 3 us to add 128 rows up over the cluster.  Measured against: [60 x 4096], K 18432, 1 to 8 splits: 92, 53, 41,
// 37, 37, 36 us, expected 112, 64, 48, 39, 36, 36; [120 x 2048], K 6144: 49, 31, 25, 23, 21, 23, expected 51, 35, 29, 25, 22, 21.
// splits: 0: chosen.
static GemmFewPlan gemm_few_plan(int rows, int N, int K, int splits = 0) {
    GemmFewPlan best = {0, 0, 0, 0, 1e30};
    const int blocks = ceil_div(rows, GF_ROWS), n_box = (ceil_div(rows, blocks) + 15) / 16 * 16, kblocks = ceil_div(K, 64);
    const int stage = GF_A_BYTES + n_box * 128;
    int stages = GF_RING / stage;
    if (stages > GF_MAX_STAGES) stages = GF_MAX_STAGES;
    const int tiles = ceil_div(N, 128) * blocks;
    const int choices[6] = {1, 2, 3, 4, 6, 8};
    for (int i = 0; i < 6; ++i) {
        const int s = choices[i], per = ceil_div(kblocks, s);
        if (s > kblocks || per * (s - 1) >= kblocks || (splits && s != splits)) continue;  // every CTA of a cluster has a step
        const double load = tiles * s / 148.0, step = 0.29 + 0.11 * n_box / 128;
        const double us = 13.0 + (load > 1 ? load : 1) * per * step + (s > 1 ? 3.0 * n_box / 128 : 0.0);
        if (us < best.us) best = {n_box, blocks, s, stages, us};
    }
    return best;
}

static int launch_gemm_few(const GemmFewPlan& plan, const void* a, int64_t lda, const void* b, int64_t ldb, void* c, int64_t ldc, int rows, int N, int K,
                           int out_f32, uint32_t* status, cudaStream_t stream) {
    CUtensorMap map_w, map_x;
    if (make_map(&map_w, b, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, 128)) return 3;
    if (make_map(&map_x, a, (uint64_t)rows, (uint64_t)K, (uint64_t)lda, (uint32_t)plan.n_box)) return 3;
    static DeviceOnce once;
    const int dev = once.pending();
    if (dev != DeviceOnce::SET) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_few_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GF_RING + 1024);
        if (e != cudaSuccess) return (int)e;
        once.mark(dev);
    }
    GemmFewArgs p;
    p.c = c; p.ldc = ldc; p.b = (const bf16*)b; p.ldb = ldb; p.rows = rows; p.N = N; p.K = K; p.out_f32 = out_f32;
    p.n_box = plan.n_box; p.stages = plan.stages; p.splits = plan.splits; p.tiles_n = ceil_div(N, 128); p.status = status;
    p.prefetch = (int64_t)N * K * 2 <= ((int64_t)48 << 20);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.tiles_n * plan.blocks * plan.splits);
    cfg.blockDim = dim3(GF_THREADS);
    cfg.dynamicSmemBytes = (size_t)plan.stages * (GF_A_BYTES + plan.n_box * 128) + 1024;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = g_glmb_pdl_enabled ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = plan.splits; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    (void)cudaLaunchKernelEx(&cfg, gemm_few_kernel, map_w, map_x, p);
    return (int)cudaGetLastError();
}
