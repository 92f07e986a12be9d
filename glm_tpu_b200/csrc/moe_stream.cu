// Routed FP8 experts of a decode step (a route per tile, moe_gateup_fp8 / moe_down_fp8): the weights of the chosen experts streamed once.
//
// Routes to the same expert (up to eight) form a group and share its weights as the columns of mma.sync m16n8k16.  An item is a group and 32 weight rows
// (gate/up: 16 gate rows and their 16 up rows); two CTAs per SM walk the items, and every warp keeps MS_DEPTH of its 64-wide chunks in flight with
// cp.async, over the ends of items: a CTA per item and tile spent its life in the latency of one chunk after another, and read an expert
// again for every route.  A lane copies the very 16 bytes that it multiplies, so nothing is exchanged before the fragments meet.
//
// Bound by the bytes (slope 5.6 TB/s) behind a fixed 10 - 15 us.  All chosen experts different, 2 x 2048 x 6144 and back on a B200, moe_gemv_mma.cu ->
// here: 16 routes 99 + 55 -> 94 + 55 us, 32 routes 178 + 102 -> 170 + 97, 64 routes 345 + 195 -> 312 + 181; 8 routes 56 + 33 either way.  Depths of two to
// four and two to four CTAs per SM differ by 3 %.  In a step of four GLM layers, four chats at 5,000: 1,729 -> 1,650 us.
//
// Fragments, the order of the sums (chunks c = warp, warp + 8, .. in a warp's accumulator, the warps in order) and so the bits are those of
// moe_gemv_mma.cu, which takes what this file does not, and of the persistent decode kernel.
#include "common.cuh"
#include "moe_mma_core.cuh"

#define MS_WARPS 8
#define MS_THREADS (MS_WARPS * 32)
#define MS_DEPTH 3
#define MS_CTAS (2 * 148)
#define MS_SLOT 3072   // two weight panels of 16 rows x 64 bytes, 8 activation rows x 64 bf16
#define MS_ROUTES 256
#define MS_COLS 8
#define MS_SMEM (MS_WARPS * MS_DEPTH * (MS_SLOT + 16))

struct MoeStreamArgs {
    const bf16* x;           // mode 0: rows, route p reads row p / top_k; mode 1: activations, a row per route
    int64_t xs;
    int top_k, routes;
    const int* experts;      // [routes] global expert of a route
    const uint8_t *w0, *w1;  // mode 0: gate, up [local, N, K]; mode 1: down [local, N, K] twice
    const float *s0, *s1;
    const float* route_weight;  // mode 1
    int expert_base, experts_local, N, K, mode;
    bf16* out;               // [routes, N]
};

__device__ __forceinline__ void ms_copy16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ uint4 ms_lds16(uint32_t at) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at));
    return v;
}

__global__ void __launch_bounds__(MS_THREADS, 2) moe_stream_kernel(const MoeStreamArgs a) {
    GLMB_PDL_PROLOGUE();
    extern __shared__ __align__(16) unsigned char ms_ring[];
    __shared__ int id_s[MS_ROUTES], leaders_s[MS_WARPS];
    __shared__ short member_s[MS_ROUTES][MS_COLS];  // per group: its routes, -1 past the last
    __shared__ int expert_s[MS_ROUTES];             // per group: local expert
    __shared__ float red[MS_WARPS][2][16][MS_COLS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;

    // ---- groups, in the order of their first routes
    int e = -1;
    if (tid < a.routes) {
        e = a.experts[tid] - a.expert_base;
        if (e < 0 || e >= a.experts_local) e = -1;  // another GPU's
        id_s[tid] = e;
    }
#pragma unroll
    for (int r = 0; r < MS_COLS; ++r) member_s[tid][r] = -1;
    __syncthreads();
    int nth = 0, leader = tid;
    if (e >= 0)
        for (int j = 0; j < tid; ++j)
            if (id_s[j] == e) {
                if ((nth & (MS_COLS - 1)) == 0) leader = j;
                ++nth;
            }
    if ((nth & (MS_COLS - 1)) == 0) leader = tid;
    const unsigned firsts = __ballot_sync(0xffffffffu, e >= 0 && leader == tid);
    if (lane == 0) leaders_s[warp] = __popc(firsts);
    __syncthreads();
    int groups = 0, before = 0;
#pragma unroll
    for (int w = 0; w < MS_WARPS; ++w) {
        if (w < warp) before += leaders_s[w];
        groups += leaders_s[w];
    }
    __syncthreads();
    const int own_group = before + __popc(firsts & ((1u << lane) - 1));
    if (e >= 0 && leader == tid) { id_s[tid] = own_group; expert_s[own_group] = e; }  // from here on: the group of a leader
    __syncthreads();
    if (e >= 0) member_s[id_s[leader]][nth & (MS_COLS - 1)] = (short)tid;
    __syncthreads();

    const int rows = a.mode == 0 ? 16 : 32, blocks = (a.N + rows - 1) / rows, items = groups * blocks;
    const int chunks = a.K >> 6, kb = (a.K + 127) >> 7, n_srows = (a.N + 127) >> 7;
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(ms_ring) + warp * MS_DEPTH * MS_SLOT;
    float* scale_ring = reinterpret_cast<float*>(ms_ring + MS_WARPS * MS_DEPTH * MS_SLOT) + warp * MS_DEPTH * 4;
    const bool idle = warp >= chunks;  // fewer chunks than warps

    // ---- the chunk that is asked for next: addresses of the item it belongs to
    int ask_item = blockIdx.x, ask_chunk = warp;
    const uint8_t *p0 = nullptr, *p1 = nullptr;
    const float* ps = nullptr;
    const bf16* px = nullptr;
    bool second = false;
    auto open_item = [&]() {
        if (ask_item >= items || idle) return;
        const int group = ask_item / blocks, n0 = (ask_item - group * blocks) * rows, expert = expert_s[group];
        second = a.mode == 0 || n0 + 16 < a.N;
        p0 = a.w0 + ((int64_t)expert * a.N + n0 + g) * a.K + t * 16;
        p1 = a.mode == 0 ? a.w1 + ((int64_t)expert * a.N + n0 + g) * a.K + t * 16 : p0 + (int64_t)16 * a.K;
        // lanes 0 and 1 copy the panels' scales
        ps = (lane == 0 ? a.s0 : a.s1) + ((int64_t)expert * n_srows + ((a.mode == 1 && lane == 1 && second ? n0 + 16 : n0) >> 7)) * kb;
        const int route = member_s[group][g];
        px = route < 0 ? nullptr : a.x + (int64_t)(a.mode == 0 ? route / a.top_k : route) * a.xs + t * 16;
    };
    open_item();
    auto ask = [&](int slot) {
        if (ask_item < items && !idle) {
            const uint32_t at = ring + slot * MS_SLOT + lane * 16;
            const int k = ask_chunk << 6;
            const int64_t down8 = (int64_t)8 * a.K;
            ms_copy16(at, p0 + k);
            ms_copy16(at + 512, p0 + down8 + k);
            if (second) {
                ms_copy16(at + 1024, p1 + k);
                ms_copy16(at + 1536, p1 + down8 + k);
            }
            if (px) {
                ms_copy16(at + 2048, px + k);
                ms_copy16(at + 2560, px + k + 8);
            }
            if (lane < 2)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;"
                             ::"r"((uint32_t)__cvta_generic_to_shared(scale_ring + slot * 4 + lane)), "l"(ps + (ask_chunk >> 1)) : "memory");
            ask_chunk += MS_WARPS;
            if (ask_chunk >= chunks) { ask_chunk = warp; ask_item += gridDim.x; open_item(); }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int d = 0; d < MS_DEPTH; ++d) ask(d);

    int slot = 0;
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
        const int group = item / blocks, n0 = (item - group * blocks) * rows;
        const bool both = a.mode == 0 || n0 + 16 < a.N, column = member_s[group][g] >= 0;
        float acc[2][4] = {};
        for (int c = warp; c < chunks; c += MS_WARPS) {
            asm volatile("cp.async.wait_group %0;" ::"n"(MS_DEPTH - 1) : "memory");
            __syncwarp();  // the scales are other lanes' copies
            const uint32_t at = ring + slot * MS_SLOT + lane * 16;
            uint4 x0 = make_uint4(0, 0, 0, 0), x1 = x0;
            if (column) { x0 = ms_lds16(at + 2048); x1 = ms_lds16(at + 2560); }
            const float sc0 = scale_ring[slot * 4], sc1 = scale_ring[slot * 4 + 1];
            chunk_mma<true>(acc[0], ms_lds16(at), ms_lds16(at + 512), sc0, x0, x1);
            if (both) chunk_mma<true>(acc[1], ms_lds16(at + 1024), ms_lds16(at + 1536), sc1, x0, x1);
            __syncwarp();
            ask(slot);
            slot = slot + 1 == MS_DEPTH ? 0 : slot + 1;
        }
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            red[warp][m][g][2 * t] = acc[m][0]; red[warp][m][g][2 * t + 1] = acc[m][1];
            red[warp][m][g + 8][2 * t] = acc[m][2]; red[warp][m][g + 8][2 * t + 1] = acc[m][3];
        }
        __syncthreads();
        if (a.mode == 0) {
            const int n = tid & 15, col = tid >> 4;
            const int route = tid < 16 * MS_COLS ? member_s[group][col] : -1;
            if (route >= 0 && n0 + n < a.N) {
                float gs = 0.f, us = 0.f;
#pragma unroll
                for (int w = 0; w < MS_WARPS; ++w) { gs += red[w][0][n][col]; us += red[w][1][n][col]; }
                const float gv = bf16_round(gs), uv = bf16_round(us);
                a.out[(int64_t)route * a.N + n0 + n] = __float2bfloat16_rn(gv * sigmoidf_precise(gv) * uv);
            }
        } else {
            const int n = tid & 31, col = tid >> 5, route = member_s[group][col];
            if (route >= 0 && n0 + n < a.N) {
                float s = 0.f;
#pragma unroll
                for (int w = 0; w < MS_WARPS; ++w) s += red[w][n >> 4][n & 15][col];
                a.out[(int64_t)route * a.N + n0 + n] = __float2bfloat16_rn(bf16_round(s) * bf16_round(a.route_weight[route]));
            }
        }
        __syncthreads();
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// A route per tile, shapes and alignments as the kernels of moe_gemv_mma.cu take them (K a multiple of 64, N of 16), 16-byte aligned weights.  With fewer
// than six items per CTA their tail costs what the rest gains: eight routes in a step 53 + 30 us there, 57 + 31 here.
bool moe_stream_takes(const void* x, const void* w0, const void* w1, int tiles, int N, int K, int64_t xs, int mode) {
    return tiles <= MS_ROUTES && (int64_t)tiles * ceil_div(N, mode == 0 ? 16 : 32) >= 6 * MS_CTAS && !(K & 63) && !(N & 15) && !(xs & 7) &&
           !((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w0) | reinterpret_cast<uintptr_t>(w1)) & 15);
}
int launch_moe_stream(const void* x, int64_t xs, int top_k, const int* experts, int routes, const void* w0, const void* w1, const float* s0, const float* s1,
                      int expert_base, int experts_local, int N, int K, int mode, const float* route_weight, void* out, cudaStream_t stream) {
    static DeviceOnce once;
    const int dev = once.pending();
    if (dev != DeviceOnce::SET) {
        const cudaError_t e = cudaFuncSetAttribute(moe_stream_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MS_SMEM);
        if (e != cudaSuccess) return (int)e;
        once.mark(dev);
    }
    MoeStreamArgs a;
    a.x = (const bf16*)x; a.xs = xs; a.top_k = top_k; a.routes = routes; a.experts = experts;
    a.w0 = (const uint8_t*)w0; a.w1 = (const uint8_t*)(mode == 0 ? w1 : w0); a.s0 = s0; a.s1 = mode == 0 ? s1 : s0;
    a.route_weight = route_weight; a.expert_base = expert_base; a.experts_local = experts_local;
    a.N = N; a.K = K; a.mode = mode; a.out = (bf16*)out;
    const int64_t most = (int64_t)routes * ceil_div(N, mode == 0 ? 16 : 32);
    GLMB_LAUNCH(moe_stream_kernel, (int)(most < MS_CTAS ? most : MS_CTAS), MS_THREADS, MS_SMEM, stream, a);
    return (int)cudaGetLastError();
}
