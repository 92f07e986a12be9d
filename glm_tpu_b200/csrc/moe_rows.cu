// Routed experts with unquantized (bf16 or fp32) tables, where a token's weight scales the expert's input:
//
//   out_r = sum over the row's routes (e, w) of  W_down^e (f(W_gate^e (w h_r)) * (W_up^e (w h_r))) .
//
// The projections are linear, so w multiplies their fp32 sums and nothing is rounded twice.
//
//   expert_glu    decode and the 32-bit path: act[route] from the rows themselves
//   expert_down   the same for the second half: the routes of a row are added in slot order in fp32
//                 (bf16, up to eight rows: an expert's weights are read once for all rows that chose it, 16 weight rows against the
//                 eight activation rows of mma.sync; otherwise a warp per output channel and route)
//   route_combine prefill: expert-sorted outputs of the grouped GEMM back to rows, added in slot order
//   gather_routes prefill: rows into expert order (zeros where there is no route)
#include "common.cuh"
#include "gemv_core.cuh"
#include "vec8.cuh"

#define MR_WARPS 8
#define MR_THREADS (MR_WARPS * 32)

template <typename T> struct ExpertDot;
template <> struct ExpertDot<bf16> {
    template <int N>
    static __device__ __forceinline__ void run(const bf16* x, const bf16* const (&w)[N], int K, int lane, float (&acc)[N]) {
        const bf16* const xr[1] = {x};
        float sum[N][1] = {};
        warp_dot_bf16<1, N>(xr, w, 0, K, lane, sum);
#pragma unroll
        for (int j = 0; j < N; ++j) acc[j] += warp_sum(sum[j][0]);
    }
};
template <> struct ExpertDot<float> {
    template <int N>
    static __device__ __forceinline__ void run(const float* x, const float* const (&w)[N], int K, int lane, float (&acc)[N]) {
        float sum[N] = {};
        for (int k = lane; k < K; k += 32)
#pragma unroll
            for (int j = 0; j < N; ++j) sum[j] = fmaf(x[k], w[j][k], sum[j]);
#pragma unroll
        for (int j = 0; j < N; ++j) acc[j] += warp_sum(sum[j]);
    }
};

// grid (pieces of MR_WARPS expert channels, routes).  gate_up [E, 2 F, K]: gate rows, then up rows.
template <typename T>
__global__ void __launch_bounds__(MR_THREADS)
expert_glu_kernel(const T* __restrict__ x, int64_t xs, int top, const int* __restrict__ ids, const float* __restrict__ weights, const T* __restrict__ gate_up,
                  int E, int F, int K, int kind, T* __restrict__ act, uint32_t* status) {
    GLMB_PDL_PROLOGUE();
    const int p = blockIdx.y, n = blockIdx.x * MR_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    int e = ids[p];
    if (e < 0 || e >= E) {
        if (threadIdx.x == 0) raise_status(status, GLMB_STATUS_BAD_INDEX);
        e = min(max(e, 0), E - 1);
    }
    if (n >= F) return;
    const T* const w[2] = {gate_up + ((int64_t)e * 2 * F + n) * K, gate_up + ((int64_t)e * 2 * F + F + n) * K};
    float acc[2] = {0.f, 0.f};
    ExpertDot<T>::template run<2>(x + (int64_t)(p / top) * xs, w, K, lane, acc);
    if (lane == 0) from_f32(glu_activation(kind, acc[0] * weights[p]) * (acc[1] * weights[p]), act[(int64_t)p * F + n]);
}

// grid (pieces of MR_WARPS output columns, rows).  down [E, N, F].
template <typename T>
__global__ void __launch_bounds__(MR_THREADS)
expert_down_kernel(const T* __restrict__ act, int top, const int* __restrict__ ids, const T* __restrict__ down, int E, int N, int F, float* __restrict__ out,
                   int64_t os) {
    GLMB_PDL_PROLOGUE();
    const int r = blockIdx.y, n = blockIdx.x * MR_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (n >= N) return;
    float total = 0.f;
    for (int s = 0; s < top; ++s) {
        const int64_t p = (int64_t)r * top + s;
        const int e = min(max(ids[p], 0), E - 1);
        const T* const w[1] = {down + ((int64_t)e * N + n) * F};
        float acc[1] = {0.f};
        ExpertDot<T>::template run<1>(act + p * F, w, F, lane, acc);
        total += acc[0];
    }
    if (lane == 0) out[(int64_t)r * os + n] = total;
}

// ---------------------------------------------------------------------------------------------------
// Up to eight rows: routes to the same expert form a group (a row that names an expert twice: its second naming belongs to another group), and
// the group's first route stands for it.  Eight chats of four experts out of 64 have 26 groups in 32 routes; the bytes of the groups are what
// bounds both kernels.
#define MR_ROWS 8
#define MR_ROUTES 256

// This thread's route (threadIdx.x < routes <= MR_ROUTES == MR_THREADS): its group's first route.  ids_s: the clamped ids of all routes.
__device__ __forceinline__ int route_leader(const int* ids_s, int top) {
    const int i = threadIdx.x, e = ids_s[i], row0 = i / top * top;
    int nth = 0;  // namings of the expert before this one in the row
    for (int j = row0; j < i; ++j) nth += ids_s[j] == e;
    for (int r0 = 0; r0 < row0; r0 += top) {
        int seen = 0;
        for (int j = r0; j < r0 + top; ++j)
            if (ids_s[j] == e && seen++ == nth) return j;
    }
    return i;
}
__device__ __forceinline__ void load_route_ids(const int* ids, int routes, int E, int* ids_s) {
    if ((int)threadIdx.x < routes) ids_s[threadIdx.x] = min(max(ids[threadIdx.x], 0), E - 1);
    __syncthreads();
}

// grid (pieces of 8 expert channels, routes): the CTA of a group's first route computes the group, 8 gate rows and their 8 up rows, K split
// over its warps.
// Two chunks in flight a warp and three CTAs per SM: most of a CTA's time that is not loads is its start (ids, groups) and its sum, which the others cover.  With
// four chunks and two CTAs (as for the second half, whose CTAs go through all groups: 52 us, with two chunks 56) 122 -> 110 us for eight rows of the top 4 of
// 64 experts, [2 x 1536 x 4096]; 67 -> 63, 38.2 -> 36.1, 21.3 -> 19.9 for four, two and one.  The weights asked for in L2 by the CTA's first thread: 120.
__global__ void __launch_bounds__(MR_THREADS, 3)
expert_glu_mma_kernel(const bf16* __restrict__ x, int64_t xs, int rows, int top, const int* __restrict__ ids, const float* __restrict__ weights,
                      const bf16* __restrict__ gate_up, int E, int F, int K, int kind, bf16* __restrict__ act, uint32_t* status) {
    GLMB_PDL_PROLOGUE();
    __shared__ int ids_s[MR_ROUTES], member_s[MR_ROWS];
    __shared__ float red[SKM_WARPS][8 * SKM_RED];
    const int p = blockIdx.y, routes = rows * top;
    if (threadIdx.x < MR_ROWS) member_s[threadIdx.x] = -1;
    load_route_ids(ids, routes, E, ids_s);
    const int e = ids_s[p];
    const int own = (int)threadIdx.x < routes && ids_s[threadIdx.x] == e ? route_leader(ids_s, top) : -1;
    if (own == p) member_s[threadIdx.x / top] = threadIdx.x;
    if ((int)threadIdx.x == p && ids[p] != e) raise_status(status, GLMB_STATUS_BAD_INDEX);
    if (__syncthreads_or((int)threadIdx.x == p && own != p)) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, n = blockIdx.x * 8;
    const bf16* w = gate_up + ((int64_t)e * 2 * F + n + g) * K;
    float c[4] = {0.f, 0.f, 0.f, 0.f};
    skinny_mma_span<2>(w, w + (int64_t)F * K, member_s[g] >= 0 ? x + (int64_t)g * xs : nullptr, K, warp, lane & 3, c);
    skm_store_fragment(red[warp], c, lane);
    __syncthreads();
    const int r = threadIdx.x >> 3, j = threadIdx.x & 7;
    if (threadIdx.x >= 64 || member_s[r] < 0) return;
    const float weight = weights[member_s[r]];
    act[(int64_t)member_s[r] * F + n + j] = __float2bfloat16_rn(glu_activation(kind, skm_sum(red, r, j) * weight) * (skm_sum(red, r, j + 8) * weight));
}

// grid (pieces of 16 output columns).  A warp takes (group, half of K) pairs; the products of every route meet in shared memory and a row's are
// added in slot order.
__global__ void __launch_bounds__(MR_THREADS, 2)
expert_down_mma_kernel(const bf16* __restrict__ act, int rows, int top, const int* __restrict__ ids, const bf16* __restrict__ down, int E, int N, int F,
                       float* __restrict__ out, int64_t os) {
    GLMB_PDL_PROLOGUE();
    extern __shared__ float y_s[];  // [routes][2 halves][16 columns]
    __shared__ int ids_s[MR_ROUTES], group_s[MR_ROUTES], count_s[MR_WARPS];
    __shared__ short member_s[MR_ROUTES][MR_ROWS];
    const int routes = rows * top, i = threadIdx.x, warp = i >> 5, lane = i & 31, g = lane >> 2, t = lane & 3;
    load_route_ids(ids, routes, E, ids_s);
    const int leader = i < routes ? route_leader(ids_s, top) : -1;
    const unsigned first = __ballot_sync(0xffffffffu, i < routes && leader == i);
    if (lane == 0) count_s[warp] = __popc(first);
#pragma unroll
    for (int r = 0; r < MR_ROWS; ++r) member_s[i][r] = -1;
    __syncthreads();
    int groups = 0, before = 0;
#pragma unroll
    for (int w = 0; w < MR_WARPS; ++w) {
        if (w < warp) before += count_s[w];
        groups += count_s[w];
    }
    if (leader == i) group_s[i] = before + __popc(first & ((1u << lane) - 1));
    __syncthreads();
    if (i < routes) member_s[group_s[leader]][i / top] = (short)i;
    __syncthreads();
    const int n = blockIdx.x * 16 + g, chunks = (F + 63) >> 6;
    for (int u = warp; u < 2 * groups; u += MR_WARPS) {
        const short* member = member_s[u >> 1];
        const int half = u & 1, mine = member[g];
        int e = 0;
#pragma unroll
        for (int r = 0; r < MR_ROWS; ++r)
            if (member[r] >= 0) e = ids_s[member[r]];
        const bf16* w_lo = n < N ? down + ((int64_t)e * N + n) * F : nullptr;
        const bf16* w_hi = n + 8 < N ? down + ((int64_t)e * N + n + 8) * F : nullptr;
        const bf16* xr = mine >= 0 ? act + (int64_t)mine * F : nullptr;
        float c[4] = {0.f, 0.f, 0.f, 0.f};
        skinny_mma_chunks<4>(w_lo, w_hi, xr, F, half, 2, chunks, t, c);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int route = member[2 * t + q];
            if (route >= 0) {
                y_s[(route * 2 + half) * 16 + g] = c[q];
                y_s[(route * 2 + half) * 16 + g + 8] = c[2 + q];
            }
        }
    }
    __syncthreads();
    const int r = i >> 4, col = i & 15;
    if (r < rows && (int)blockIdx.x * 16 + col < N) {
        float total = 0.f;
        for (int s = 0; s < top; ++s) total += y_s[(r * top + s) * 32 + col] + y_s[(r * top + s) * 32 + 16 + col];
        out[(int64_t)r * os + blockIdx.x * 16 + col] = total;
    }
}

// out[r] = sum over slots of y[place[r * top + slot]], place: route -> expert-sorted row.
__global__ void __launch_bounds__(256)
route_combine_kernel(const float* __restrict__ y, const int* __restrict__ place, int top, int routes, float* __restrict__ out, int width) {
    GLMB_PDL_PROLOGUE();
    const int r = blockIdx.x;
    for (int c = threadIdx.x * 4; c < width; c += 1024) {
        float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int s = 0; s < top; ++s) {
            const int at = place[r * top + s];
            if (at < 0 || at >= routes) continue;
            const float4 v = *reinterpret_cast<const float4*>(y + (int64_t)at * width + c);
            t.x += v.x; t.y += v.y; t.z += v.z; t.w += v.w;
        }
        *reinterpret_cast<float4*>(out + (int64_t)r * width + c) = t;
    }
}

__global__ void __launch_bounds__(256)
gather_routes_kernel(const uint4* __restrict__ src, int64_t src_stride8, const int* __restrict__ perm, int top, int* __restrict__ place, uint4* __restrict__ dst,
                     int width8) {
    GLMB_PDL_PROLOGUE();
    const int i = blockIdx.x, p = perm[i];
    if (threadIdx.x == 0 && p >= 0) place[p] = i;
    for (int v = threadIdx.x; v < width8; v += 256) dst[(int64_t)i * width8 + v] = p >= 0 ? src[(int64_t)(p / top) * src_stride8 + v] : make_uint4(0, 0, 0, 0);
}

// ===================================================================================================
// x [rows, xs], ids / weights [rows, top], gate_up [E, 2 F, K], act [rows * top, F]; K and F multiples of 8.
GLMB_API int glmb_expert_glu(const void* x, int64_t xs, int rows, int top, const int* ids, const float* weights, const void* gate_up, int E, int F, int K,
                             int kind, void* act, int is_f32, uint32_t* status, void* stream) {
    if (rows < 1 || top < 1 || (int64_t)rows * top > 65535 || E < 1 || F < 1 || (K & 7) || K < 8 || (xs & 7) || (kind != GLU_SILU && kind != GLU_GELU_TANH)) return 1;
    const dim3 grid(ceil_div(F, MR_WARPS), rows * top);
    if (!is_f32 && rows <= MR_ROWS && rows * top <= MR_ROUTES && !(F & 7))
        GLMB_LAUNCH_L1(expert_glu_mma_kernel, grid, MR_THREADS, 0, (cudaStream_t)stream, (const bf16*)x, xs, rows, top, ids, weights, (const bf16*)gate_up, E, F, K,
                    kind, (bf16*)act, status);
    else if (is_f32)
        GLMB_LAUNCH(expert_glu_kernel<float>, grid, MR_THREADS, 0, (cudaStream_t)stream, (const float*)x, xs, top, ids, weights, (const float*)gate_up, E, F, K, kind,
                    (float*)act, status);
    else
        GLMB_LAUNCH(expert_glu_kernel<bf16>, grid, MR_THREADS, 0, (cudaStream_t)stream, (const bf16*)x, xs, top, ids, weights, (const bf16*)gate_up, E, F, K, kind,
                    (bf16*)act, status);
    return (int)cudaGetLastError();
}

// out [rows, os] fp32, N columns; act [rows * top, F], down [E, N, F].
GLMB_API int glmb_expert_down(const void* act, int rows, int top, const int* ids, const void* down, int E, int N, int F, float* out, int64_t os, int is_f32,
                              void* stream) {
    if (rows < 1 || rows > 65535 || top < 1 || E < 1 || N < 1 || (F & 7) || F < 8) return 1;
    const dim3 grid(ceil_div(N, MR_WARPS), rows);
    if (!is_f32 && rows <= MR_ROWS && rows * top <= MR_ROUTES)
        GLMB_LAUNCH_L1(expert_down_mma_kernel, ceil_div(N, 16), MR_THREADS, rows * top * 32 * sizeof(float), (cudaStream_t)stream, (const bf16*)act, rows, top, ids,
                    (const bf16*)down, E, N, F, out, os);
    else if (is_f32)
        GLMB_LAUNCH(expert_down_kernel<float>, grid, MR_THREADS, 0, (cudaStream_t)stream, (const float*)act, top, ids, (const float*)down, E, N, F, out, os);
    else
        GLMB_LAUNCH(expert_down_kernel<bf16>, grid, MR_THREADS, 0, (cudaStream_t)stream, (const bf16*)act, top, ids, (const bf16*)down, E, N, F, out, os);
    return (int)cudaGetLastError();
}

// y [routes, width] fp32 in expert order -> out [rows, width]; width a multiple of 4, both contiguous.
GLMB_API int glmb_route_combine(const float* y, const int* place, int rows, int top, float* out, int width, void* stream) {
    if (rows < 1 || top < 1 || width < 4 || (width & 3)) return 1;
    GLMB_LAUNCH(route_combine_kernel, rows, 256, 0, (cudaStream_t)stream, y, place, top, rows * top, out, width);
    return (int)cudaGetLastError();
}

// dst [routes, width] = rows of src in the order of perm (route ids, -1: zeros); place becomes the inverse of perm.
GLMB_API int glmb_gather_routes(const void* src, int64_t src_stride, const int* perm, int routes, int top, int* place, void* dst, int width, void* stream) {
    if (routes < 1 || top < 1 || (width & 7) || width < 8 || (src_stride & 7)) return 1;
    GLMB_LAUNCH(gather_routes_kernel, routes, 256, 0, (cudaStream_t)stream, (const uint4*)src, src_stride / 8, perm, top, place, (uint4*)dst, width / 8);
    return (int)cudaGetLastError();
}
