// Dense bf16 GEMM of many rows on pairs of SMs (tcgen05 cta_group::2), included by gemm_tcgen05.cu.
//
//   plain   C[rows, N]  = A[rows, K] . B[N, K]^T                                        (bf16 or fp32)
//   gated   C[rows, N]  = bf16( f(bf16(A . G^T)) * bf16(A . U^T) ), G, U [N, K]         (bf16): a gated feed-forward's first half
//
// A cluster of two CTAs computes 256 rows x `bn` columns: each CTA stages its own 128 rows of A and HALF of the columns of B, and one
// tcgen05.mma issued by the first CTA reads both halves, so a CTA's shared memory takes in 32 KB per 64-wide k step where a CTA on its own
// (128 x 256) takes 48 KB for the same work.  The gated form has the first CTA stage gate rows and the second the up rows of the same
// outputs: both land in the same accumulator row, and the [rows, 2 N] intermediate never reaches memory.
//
//   warp 0      TMA producer of this CTA's operands; all bytes are counted on the first CTA's barrier
//   warp 1      TMEM allocation; in the first CTA it issues the MMAs of the pair
//   warps 2-5   epilogue of this CTA's 128 rows; the TMEM holds two accumulators, so it runs while the next tile is multiplied
//
// Tiles are walked by one pair per two SMs, in groups of eight row tiles by all column tiles (operand tiles shared in L2).
// The activation of the gated form is glu_activation, as in a launch of its own: the same bits (a quotient and a tanh without branches save nothing
// measurable: the epilogue runs beside the next tile's products).
// Bound by the tensor core (and the power it may draw).  Measured on a B200, single SMs -> pairs: [8192 x 8192], K 8192: 809 -> 717 us (1,534
// TFLOP/s); [4096 x 28672], K 4096: 718 -> 614; gated [4096 x 2 x 14336], K 4096, with its activation: 797 -> 609.
#pragma once

#include "tcgen05.cuh"
#include "vec8.cuh"

#define GP_STAGES 6
#define GP_A_BYTES (128 * 64 * 2)
#define GP_STAGE_BYTES (2 * GP_A_BYTES)  // B: up to 128 rows
#define GP_SMEM_BYTES (GP_STAGES * GP_STAGE_BYTES + 1024)
#define GP_THREADS 192

enum { GP_OUT_BF16 = 0, GP_OUT_F32 = 1, GP_OUT_GATED = 2 };

__device__ __forceinline__ uint32_t gp_in_first_cta(uint32_t addr) {  // the same shared-memory address in the cluster's first CTA
    uint32_t at;
    asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(at) : "r"(addr));
    return at;
}
__device__ __forceinline__ void gp_tma_load(void* smem_dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(map), "r"(bar), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void gp_mma(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void gp_commit(uint64_t* bar) {  // arrives at this barrier of both CTAs
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void gp_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

struct GemmPairArgs {
    void* c;
    int64_t ldc;
    int rows, N, K;
    int bn;    // columns of the accumulator (gated: bn / 2 outputs)
    int out;   // GP_OUT_*
    int glu;   // gated: GLU_*
    uint32_t* status;
};

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GP_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b0, const __grid_constant__ CUtensorMap map_b1,
                 GemmPairArgs p) {
    GLMB_PDL_PROLOGUE();
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full[GP_STAGES], empty[GP_STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile uint32_t fail;
    unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    uint32_t rank;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const bool gated = p.out == GP_OUT_GATED;
    const int cols = gated ? p.bn >> 1 : p.bn;  // output columns of a tile
    const int m_tiles = (p.rows + 255) >> 8, n_blocks = (p.N + cols - 1) / cols, total = m_tiles * n_blocks, kblocks = (p.K + 63) >> 6;

    if (threadIdx.x == 0) {
        for (int s = 0; s < GP_STAGES; ++s) { mbar_init(full + s, 1); mbar_init(empty + s, 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(acc_full + a, 1); mbar_init(acc_empty + a, 8); }
        fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    gp_cluster_sync();  // the barriers of both CTAs are ready
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;

    auto place = [&](int t, int& m, int& n) {
        const int group = 8 * n_blocks, first = (t / group) * 8, gm = min(m_tiles - first, 8);
        m = first + (t % group) % gm;
        n = (t % group) / gm;
    };
    if (warp == 0) {
        const uint32_t bytes = 2 * (GP_A_BYTES + (uint32_t)(p.bn >> 1) * 128);
        const CUtensorMap* map_b = gated && rank ? &map_b1 : &map_b0;
        uint32_t g = 0;  // k steps issued so far, across tiles
        bool ok = true;
        for (int t = pair; t < total && ok; t += pairs) {
            int m, n;
            place(t, m, n);
            const int a_row = m * 256 + (int)rank * 128, b_row = n * cols + (gated ? 0 : (int)rank * (p.bn >> 1));
            for (int kb = 0; kb < kblocks; ++kb, ++g) {
                const uint32_t s = g % GP_STAGES, lap = g / GP_STAGES;
                if (lap > 0 && !mbar_wait_warp(empty + s, (lap - 1) & 1)) { fail = 1; ok = false; break; }
                unsigned char* dst = ring + s * GP_STAGE_BYTES;
                const uint32_t bar = gp_in_first_cta(smem_u32(full + s));
                if (elect_one()) {
                    if (rank == 0) mbar_expect_tx(full + s, bytes);
                    gp_tma_load(dst, &map_a, bar, kb * 64, a_row);
                    gp_tma_load(dst + GP_A_BYTES, map_b, bar, kb * 64, b_row);
                }
                __syncwarp();
            }
        }
    } else if (warp == 1) {
        const uint32_t idesc = umma_idesc_bf16(256, p.bn);
        uint32_t g = 0, i = 0;
        for (int t = pair; t < total && rank == 0; t += pairs, ++i) {
            const uint32_t acc = i & 1, use = i >> 1;
            if (use > 0 && !mbar_wait_warp(acc_empty + acc, (use - 1) & 1)) { fail = 1; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            bool ok = true;
            for (int kb = 0; kb < kblocks; ++kb, ++g) {
                const uint32_t s = g % GP_STAGES;
                if (!mbar_wait_warp(full + s, (g / GP_STAGES) & 1)) { fail = 1; ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t a_addr = smem_u32(ring + s * GP_STAGE_BYTES), b_addr = a_addr + GP_A_BYTES;
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        gp_mma(tmem + acc * 256, umma_desc_sw128(a_addr + k * 32), umma_desc_sw128(b_addr + k * 32), idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    gp_commit(empty + s);
                }
                __syncwarp();
            }
            if (elect_one()) gp_commit(acc_full + acc);  // complete, or abandoned after a timeout: either way release the epilogues
            __syncwarp();
            if (!ok) break;
        }
    } else {
        const int quarter = warp & 3;
        uint32_t i = 0;
        for (int t = pair; t < total; t += pairs, ++i) {
            const uint32_t acc = i & 1;
            const bool done = mbar_wait_warp(acc_full + acc, (i >> 1) & 1);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (!done || __any_sync(0xffffffffu, fail)) {
                fail = 1;
                if (lane == 0) raise_status(p.status, GLMB_STATUS_WAIT_TIMEOUT);
                break;
            }
            int m, n;
            place(t, m, n);
            const int row = m * 256 + (int)rank * 128 + quarter * 32 + lane, n0 = n * cols;
            const uint32_t d = tmem + acc * 256 + ((uint32_t)(quarter * 32) << 16);
            if (gated) {
                bf16* dst = reinterpret_cast<bf16*>(p.c) + (int64_t)row * p.ldc + n0;
#pragma unroll 1
                for (int cb = 0; cb < cols; cb += 16) {
                    uint32_t g[16], u[16], o[8];
                    tmem_ld16(d + cb, g);
                    tmem_ld16(d + cols + cb, u);
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        float v[2];
#pragma unroll
                        for (int q = 0; q < 2; ++q)
                            v[q] = glu_activation(p.glu, bf16_round(__uint_as_float(g[2 * e + q]))) * bf16_round(__uint_as_float(u[2 * e + q]));
                        o[e] = pack_bf16(v[0], v[1]);
                    }
                    if (row < p.rows)
#pragma unroll
                        for (int q = 0; q < 2; ++q)
                            if (n0 + cb + 8 * q < p.N) *reinterpret_cast<uint4*>(dst + cb + 8 * q) = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
                }
            } else {
#pragma unroll 1
                for (int cb = 0; cb < cols; cb += 32) {
                    uint32_t v[32];
                    tmem_ld32(d + cb, v);
                    if (row < p.rows && p.out == GP_OUT_F32) {
                        float* dst = reinterpret_cast<float*>(p.c) + (int64_t)row * p.ldc + n0 + cb;
#pragma unroll
                        for (int e = 0; e < 32; e += 4)
                            if (n0 + cb + e < p.N)
                                *reinterpret_cast<float4*>(dst + e) = make_float4(__uint_as_float(v[e]), __uint_as_float(v[e + 1]), __uint_as_float(v[e + 2]),
                                                                                  __uint_as_float(v[e + 3]));
                    } else if (row < p.rows) {
                        bf16* dst = reinterpret_cast<bf16*>(p.c) + (int64_t)row * p.ldc + n0 + cb;
#pragma unroll
                        for (int e = 0; e < 32; e += 8)
                            if (n0 + cb + e < p.N)
                                *reinterpret_cast<uint4*>(dst + e) =
                                    make_uint4(pack_bf16(__uint_as_float(v[e]), __uint_as_float(v[e + 1])), pack_bf16(__uint_as_float(v[e + 2]), __uint_as_float(v[e + 3])),
                                               pack_bf16(__uint_as_float(v[e + 4]), __uint_as_float(v[e + 5])), pack_bf16(__uint_as_float(v[e + 6]), __uint_as_float(v[e + 7])));
                    }
                }
            }
            // this warp's quarter of the accumulator has been read: hand it back to the CTA that issues the MMAs
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(gp_in_first_cta(smem_u32(acc_empty + acc))) : "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    gp_cluster_sync();  // neither CTA leaves while the other may still signal it or read its operands
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// b1: the up table of the gated form (NULL otherwise).
static int launch_gemm_pair(const void* a, int64_t lda, const void* b0, const void* b1, int64_t ldb, void* c, int64_t ldc, int rows, int N, int K, int bn,
                            int out, int glu, uint32_t* status, cudaStream_t stream) {
    CUtensorMap map_a, map_b0, map_b1;
    if (make_map(&map_a, a, (uint64_t)rows, (uint64_t)K, (uint64_t)lda)) return 3;
    if (make_map(&map_b0, b0, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, (uint32_t)bn / 2)) return 3;
    if (make_map(&map_b1, b1 ? b1 : b0, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, (uint32_t)bn / 2)) return 3;
    static DeviceOnce once;
    const int dev = once.pending();
    if (dev != DeviceOnce::SET) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GP_SMEM_BYTES);
        if (e != cudaSuccess) return (int)e;
        once.mark(dev);
    }
    GemmPairArgs p;
    p.c = c; p.ldc = ldc; p.rows = rows; p.N = N; p.K = K; p.bn = bn; p.out = out; p.glu = glu; p.status = status;
    const int total = ceil_div(rows, 256) * ceil_div(N, out == GP_OUT_GATED ? bn / 2 : bn);
    GLMB_LAUNCH(gemm_pair_kernel, 2 * (total < 74 ? total : 74), GP_THREADS, GP_SMEM_BYTES, stream, map_a, map_b0, map_b1, p);
    return (int)cudaGetLastError();
}
